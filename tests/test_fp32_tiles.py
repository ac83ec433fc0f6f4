"""The FP32 coarse pass at the sizes where its tiles, stages, segments and buffers have edges: the
answer equals the oracle's brute force bit for bit."""

import numpy as np
import pytest

from conftest import clustered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,margin", [
    (2, 1, 1, None), (127, 8, 5, None), (128, 9, 10, None), (129, 3, 16, None),  # one tile, its remainders
    (257, 64, 16, None), (1000, 64, 32, None), (385, 63, 20, 13),                # resident, 2 stages; cap 32 | 33
    (300, 5, 64, None), (700, 40, 50, 14), (900, 8, 64, 64),                     # cap 64 and 128: streamed
    (640, 65, 10, None), (513, 72, 30, None), (513, 130, 60, 60), (129, 2000, 15, None),
    (12_011, 17, 10, None),                                                      # several segments a block
])
@pytest.mark.parametrize("select", ["cosine", "tanimoto"])
def test_fp32_pass_at_its_edges(ext, oracle, n, d, k, margin, select):
    x = clustered(n, d, n + d)
    if select == "tanimoto":
        x = np.ascontiguousarray(x * np.random.default_rng(n).uniform(0.5, 2.0, size=(n, 1)).astype(np.float32))
    want = oracle.knn_bruteforce(x, k, select=select)
    for prune in (True, False):
        (idx, cos, norms), st = ext._knn_exact(x, k, margin=margin, select=select, prune=prune)
        np.testing.assert_array_equal(idx.view(np.uint32), want[0])
        np.testing.assert_array_equal(cos, want[1])
        np.testing.assert_array_equal(norms, want[2])
        assert st["max_err_ratio"] < 1.0


@pytest.mark.parametrize("d", [6, 70])
def test_fp32_pass_with_repeated_and_zero_rows(ext, oracle, d):
    """Columns equal to a query, rows of zeros and whole tiles of equal scores: buffers overflow with ties."""
    rng = np.random.default_rng(d)
    x = np.floor(rng.uniform(0, 2, size=(1500, d))).astype(np.float32)
    x[200:600] = x[200]
    x[[0, 1499]] = 0.0
    for select in ("cosine", "tanimoto"):
        want = oracle.knn_bruteforce(x, 12, select=select)
        got, _ = ext._knn_exact(x, 12, select=select)
        for a, b in zip((got[0].view(np.uint32), got[1], got[2]), want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,d,k,margin", [(16_384, 2, 10, None), (40_000, 33, 30, None), (33_100, 64, 10, 3),
                                          (36_000, 17, 70, None)])
def test_fp32_pass_by_lists(ext, oracle, n, d, k, margin):
    """Enough rows for the column lists and the early stop (ragged last blocks, repeated rows): the
    answer equals the oracle's and the pass over all tiles in order."""
    x = clustered(n, d, n + d)
    x[n // 2:n // 2 + 300] = x[5]
    x[7] = 0.0
    want, _ = oracle.knn_exact(x, k)
    for prune in (True, False):
        (idx, cos, norms), st = ext._knn_exact(x, k, margin=margin, prune=prune)
        for a, b in zip((idx.view(np.uint32), cos, norms), want):
            np.testing.assert_array_equal(a, b)
        assert prune or st["blocks_stopped"] == 0


@pytest.mark.parametrize("n,d,k,spread,signed", [(130, 3, 5, 4.0, False), (5001, 30, 10, 9.0, False), (16_383, 7, 12, 3.0, True),
                                                 (16_385, 5, 10, 6.0, False), (30_001, 40, 30, 2.0, False),
                                                 (25_000, 64, 70, 5.0, True)])
def test_tanimoto_by_lists(ext, oracle, n, d, k, spread, signed):
    """Tanimoto selection by the norm order's lists (few rows) and by cosine bounds with norm ranges
    (16,384 rows and more): zero rows, repeated rows, thresholds below zero."""
    rng = np.random.default_rng(n)
    x = clustered(n, d, n + d) - (2.0 if signed else 0.0)
    x = x * np.exp(rng.uniform(0, np.log(spread), size=(n, 1)))
    x[n // 2:n // 2 + 40] = x[4]
    x[:2] = 0.0
    x = np.ascontiguousarray(x, dtype=np.float32)
    want, _ = oracle.knn_exact(x, k, select="tanimoto")
    for prune in (True, False):
        got, st = ext._knn_exact(x, k, select="tanimoto", prune=prune)
        for a, b in zip((got[0].view(np.uint32), got[1], got[2]), want):
            np.testing.assert_array_equal(a, b)
        assert prune or st["blocks_skipped"] == 0


@pytest.mark.parametrize("n,d,k,margin", [(19_456, 30, 10, None), (19_457, 30, 10, None),  # all tiles | lists
                                          (19_456, 64, 30, None), (19_457, 64, 30, None),  # one CTA an SM | two, streamed
                                          (20_001, 41, 60, None), (21_000, 56, 63, None), (16_001, 48, 64, None)])
@pytest.mark.parametrize("select", ["cosine", "tanimoto"])
def test_fp32_pass_on_either_shape(ext, oracle, n, d, k, margin, select):
    """Both sides of the size from which the lists are taken and a query operand that leaves room for one CTA
    to an SM is streamed instead; the candidates kept (60, 64, 126, 128) decide the buffers."""
    x = clustered(n, d, n + d)
    if select == "tanimoto":
        x = np.ascontiguousarray(x * np.random.default_rng(n).uniform(0.5, 2.0, size=(n, 1)).astype(np.float32))
    want, _ = oracle.knn_exact(x, k, select=select)
    got, st = ext._knn_exact(x, k, margin=margin, select=select)
    for a, b in zip((got[0].view(np.uint32), got[1], got[2]), want):
        np.testing.assert_array_equal(a, b)
    assert st["max_err_ratio"] < 1.0
    if select == "cosine":
        assert (st["blocks_stopped"] > 0) == (n > 19_456)
