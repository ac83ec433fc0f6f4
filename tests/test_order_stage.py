"""The order stage (k-means cells, stable sort by cell, block geometry) at its edges, through the test
hook that returns the working order and the blocks' bounds."""

import numpy as np
import pytest

from conftest import clustered

pytestmark = pytest.mark.gpu


def _cells(x):
    """The library's k-means restated in numpy (f32 dots; near ties may fall on either side)."""
    n = len(x)
    xn = x / np.linalg.norm(x.astype(np.float64), axis=1, keepdims=True)
    m = min(n, 65536)
    s = xn[(np.arange(m, dtype=np.int64) * n) // m]
    c = s[(np.arange(256, dtype=np.int64) * m) // 256].copy()
    for _ in range(8):
        a = (s @ c.T).argmax(1)
        for j in range(256):
            if (a == j).any():
                v = s[a == j].sum(0)
                c[j] = v / np.linalg.norm(v)
    return (xn @ c.T).argmax(1)


@pytest.mark.parametrize("n,d", [(2, 1), (129, 5), (1023, 8), (1025, 33), (4099, 64), (5000, 16)])
def test_order_is_the_stable_sort_by_cell(ext, n, d):
    x = clustered(n, d, 3 * n + d) - 1.0
    perm, _, cradius, _, _ = ext._block_bounds(x)
    np.testing.assert_array_equal(np.sort(perm), np.arange(n, dtype=np.uint32))
    assert np.isfinite(cradius).all()
    # inside a cell rows keep their order, so the order descends in index only where a new cell starts
    assert (np.diff(perm.astype(np.int64)) < 0).sum() <= 255
    if n >= 1023:
        cell = _cells(x)[perm]
        runs = 1 + (np.diff(cell) != 0).sum()  # (a few near ties and drifted centroids split runs)
        assert runs <= 256 + n // 20, runs


@pytest.mark.parametrize("matmul,n,k", [("fp32", 16385, 5), ("fp32", 131_201, 3), ("bf16", 24_577, 5), ("bf16", 131_073, 3)])
def test_every_query_block_runs_in_the_list_length_order(ext, matmul, n, k):
    """Query blocks start by descending list weight, in 1,024 classes: with lists of very different
    lengths, and with more than 1,024 blocks, every row is still computed exactly once."""
    d = 12
    x = clustered(n, d, n)
    x[: n // 3] += 6.0  # a third of the rows in one narrow cone: long lists beside short ones
    (idx, cos, norms), st = ext._knn_exact(x, k, matmul=matmul)
    assert st["blocks_skipped"] + st.get("blocks_stopped", 0) > 0
    (want, wcos, wnorms), _ = ext._knn_exact(x, k, matmul="fp32", prune=False)
    np.testing.assert_array_equal(idx, want)
    np.testing.assert_array_equal(cos, wcos)
    np.testing.assert_array_equal(norms, wnorms)
