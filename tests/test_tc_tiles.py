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


@pytest.mark.parametrize("n,d,matmul", [(17, 20, "bf16"), (20, 21, "bf16"), (33, 36, "bf16"), (34, 40, "bf16"), (40, 64, "bf16"),
                                        (50, 100, "bf16"), (60, 600, "bf16"), (65, 600, "fp8"), (64, 70, "fp8")])
def test_lists_with_room_for_every_row(ext, n, d, matmul):
    """k + m ≥ n − 1: every other row is a candidate. Orthonormal rows have cosines of ~1e-8 with random
    signs, so their exact order is far inside the coarse error: a row that a starting threshold left out
    (the zero padding's score) shows."""
    q = np.linalg.qr(np.random.default_rng(n).standard_normal((d, d)))[0]
    x = np.ascontiguousarray(q[:n], dtype=np.float32)
    for k in (1, n // 3, n // 2, n - 2):
        want = ext._knn_bruteforce(x, k)
        got, st = ext._knn_exact(x, k, matmul=matmul, margin=n)
        assert st["coarse_kind"] != "fp32" and st["margin"] + k >= n - 1
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,d", [(17, 20), (34, 40), (40, 64)])
def test_labels_of_lists_with_room_for_every_row(ext, n, d):
    """The same in training: labels from lists of n − 1 candidates equal those from n − 2 (certified)."""
    q = np.linalg.qr(np.random.default_rng(n).standard_normal((d, d)))[0]
    x, k = np.ascontiguousarray(q[:n], dtype=np.float32), n // 2
    trained = []
    for margin in (n, n - 2 - k):
        st = ext._mlp_train(x, k, sample=n, epochs=1, batch=32, margin=margin)
        trained.append((st["loss"], st["mae"], st["coverage"]))
    assert trained[0] == trained[1]


@pytest.mark.parametrize("matmul,d,k,margin,kept", [
    ("bf16", 50, 40, None, 64), ("bf16", 64, 63, None, 64), ("bf16", 41, 33, 95, 64), ("fp8", 64, 50, 10, 64),
    ("fp32", 64, 40, None, 64), ("fp32", 48, 60, 100, 64), ("fp32", 40, 40, None, 80), ("fp32", 65, 40, None, 80),
    ("fp32", 64, 64, None, 128), ("fp32", 64, 30, None, 60)])
def test_candidates_kept_where_the_passes_hold_64(ext, oracle, matmul, d, k, margin, kept):
    """k + m above 64 at 40 < d ≤ 64: 64 candidates while k is below, which the tensor-core pass holds."""
    x = clustered(700, d, d + k)
    (idx, cos, norms), st = ext._knn_exact(x, k, margin=margin, matmul=matmul)
    assert st["margin"] == kept - k
    assert (st["coarse_kind"] == "fp32") == (matmul == "fp32")
    for a, b in zip((idx.view(np.uint32), cos, norms), oracle.knn_bruteforce(x, k)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,d", [(24_400, 2048), (24_415, 2048), (97_657, 512)])
def test_split_fp8_with_either_buffer(ext, n, d):
    """Both sides of the size from which the split-FP8 kind takes three stages and 80-entry buffers
    (n·d = 50,000,000): the answer equals the FP32 pass's."""
    x = clustered(n, d, n + d, n_centers=40, noise=1.5)
    got, st = ext._knn_exact(x, 10, matmul="bf16")
    assert st["coarse_kind"] == "fp8" and st["max_err_ratio"] < 1.0
    for a, b in zip(got, ext._knn_exact(x, 10)[0]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("matmul,n,d", [("fp32", 1500, 24), ("bf16", 1500, 24), ("fp8", 900, 600)])
def test_error_ratio_is_the_f64_quotient(ext, matmul, n, d):
    """max_err_ratio is the largest f64 quotient itself, not an f32 above it: 29 and more of its low bits are
    zero only by a chance of 2⁻²⁹. (FP32: the bound is one number, so the quotient of the maxima.)"""
    x = clustered(n, d, n + d)
    for seed in range(3):
        _, st = ext._knn_exact(x + np.float32(0.01 * seed), 10, matmul=matmul)
        r = st["max_err_ratio"]
        assert 0.0 < r < 1.0 and float(np.float32(r)) != r
        if matmul == "fp32":
            assert r == st["max_coarse_err"] / ((d + 4.0) * 2.0**-23)


@pytest.mark.parametrize("n,d", [(25_000, 43), (25_000, 64), (40_001, 50)])
def test_split_fp8_forced_where_bf16_has_lists(ext, n, d):
    """The split-FP8 kind has no lists: forced at 43 ≤ d ≤ 64 it runs its tiles in row order at any size."""
    x = clustered(n, d, n + d)
    got, st = ext._knn_exact(x, 10, matmul="fp8")
    assert st["coarse_kind"] == "fp8" and st["blocks_stopped"] == 0
    for a, b in zip(got, ext._knn_exact(x, 10)[0]):
        np.testing.assert_array_equal(a, b)
