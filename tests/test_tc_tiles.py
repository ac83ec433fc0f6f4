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
