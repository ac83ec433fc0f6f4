"""The tensor-core coarse pass where its visits have edges: probes or none, one tile, odd lists, the
three operand forms, candidate buffers of both widths. The answer equals the oracle's bit for bit and
every rescored candidate stays inside its row's error bound."""

import numpy as np
import pytest

from conftest import clustered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,margin", [
    (2, 4, 1, None), (128, 21, 5, None), (129, 22, 10, None), (300, 32, 16, None), (513, 33, 20, 12),  # one to three tiles
    (900, 42, 30, None), (1111, 64, 10, 0), (2000, 15, 31, 33),                                        # cap 60, k alone, 64
    (32_641, 9, 10, None), (32_769, 32, 10, None), (33_000, 40, 30, None), (40_001, 24, 32, None),     # probes (128 tiles)
])
@pytest.mark.parametrize("prune", [True, False])
def test_tc_pass_at_its_edges(ext, oracle, n, d, k, margin, prune):
    x = clustered(n, d, 2 * n + d) - 1.5
    x[n // 3] = x[0]
    want = oracle.knn_bruteforce(x, k) if n < 5000 else oracle.knn_exact(x, k)[0]
    (idx, cos, norms), st = ext._knn_exact(x, k, margin=margin, matmul="bf16", prune=prune)
    for a, b in zip((idx.view(np.uint32), cos, norms), want):
        np.testing.assert_array_equal(a, b)
    assert st["max_err_ratio"] < 1.0 and st["coarse_kind"] == "bf16"


@pytest.mark.parametrize("n,d,k,matmul", [(700, 256, 15, "fp32"), (900, 259, 10, "bf16"), (600, 513, 30, "fp8"),
                                          (500, 1000, 60, "fp32")])
def test_deep_rescoring_drops_by_f32_cosines(ext, oracle, n, d, k, matmul):
    """Deep rows: the candidates an f32 cosine rules out are not rescored. Rows whose norms are far out
    of f32's comfortable range get no such estimate, zero and repeated rows stay exact."""
    x = clustered(n, d, n + d)
    x[: n // 4] *= np.float32(1e-18)
    x[n // 4: n // 2] *= np.float32(1e16)
    x[n - 40:] = x[n - 1]
    x[[1, n // 2]] = 0.0
    want = oracle.knn_bruteforce(x, k)
    (idx, cos, norms), st = ext._knn_exact(x, k, matmul=matmul)
    for a, b in zip((idx.view(np.uint32), cos, norms), want):
        np.testing.assert_array_equal(a, b)
