"""Which calls take the column lists, and the passes that go without: all tiles in order, and for Tanimoto
selection the walk outward in the norm order."""

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, clustered


def _list_bytes(n, d, select="cosine", free=1 << 40, prune=1, backend=0, k=10):
    from costal_gb300 import _lib as L

    o = L.KnnOpts(margin=0xFFFFFFFF, select=L.SELECT[select], backend=backend, sort_by_norm=1, prune=prune, learned_prune=0)
    out, (err, size) = C.c_uint64(1), L.errbuf()
    L.check(L.lib().costal_fp32_list_bytes(n, d, k, C.byref(o), free, C.byref(out), err, size), err)
    return out.value


def test_lists_are_bounded(ext):
    """The lists' memory grows with n², so they end where their sort does (16,384 column blocks) and where
    they do not fit; the pass goes on without them."""
    assert _list_bytes(19_456, 32) == 0 and _list_bytes(16_383, 32, "tanimoto") == 0
    for select in ("cosine", "tanimoto"):
        for n, d in ((19_457, 1), (161_443, 32), (1_048_577, 40), (4_194_304, 64)):
            need = _list_bytes(n, d, select)
            blocks = -(-n // (128 if n <= 1_048_576 else 256))
            assert need > 12 * -(-n // 128) * blocks
            assert _list_bytes(n, d, select, free=need + need // 4) == need
            assert _list_bytes(n, d, select, free=need) == 0
            assert _list_bytes(n, d, select, prune=0) == 0
        for n in (4_194_305, 10_000_000, 30_000_000, 2**31 - 1):
            assert _list_bytes(n, 10, select) == 0
        assert _list_bytes(161_443, 65, select) == 0
    assert _list_bytes(161_443, 32, backend=1) == 0
    # few query blocks: shallow rows, or more than 20 candidates at d ≤ 40
    assert [_list_bytes(16_384, d, k=k) > 0 for d, k in ((16, 5), (17, 10), (40, 11), (41, 30))] == [True, False, True, False]
    assert _list_bytes(16_383, 10, k=30) == 0
    with pytest.raises(ValueError):
        _list_bytes(0, 5)


def _norms(kind, n, rng):
    if kind == "equal":
        return np.ones(n)
    if kind == "two":
        return np.where(rng.random(n) < 0.5, 1.0, 40.0)
    if kind == "outlier":
        s = rng.uniform(1.0, 1.1, n)
        s[n // 3] = 1e6
        return s
    return np.exp(rng.uniform(0.0, 6.0, n))


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,k", [(2, 1, 1), (129, 3, 5), (1_300, 17, 30), (6_145, 40, 10), (12_300, 64, 60), (16_000, 5, 70)])
@pytest.mark.parametrize("norms", ["equal", "two", "outlier", "spread"])
def test_walk_in_the_norm_order(ext, oracle, n, d, k, norms):
    """One tile, ragged tiles, one and several segments; norms that overlap everywhere, in two groups far apart
    (a block that spans both), with an outlier (one bucket holds the rest), spread; rows of zeros."""
    rng = np.random.default_rng(n + d)
    x = clustered(n, d, n + d) - (2.0 if d > 4 else 0.0)
    x = x / np.maximum(np.linalg.norm(x, axis=1, keepdims=True), 1e-6) * _norms(norms, n, rng)[:, None]
    if n > 1000:
        x[rng.integers(0, n, 150)] = 0.0
        x[n // 2:n // 2 + 30] = x[4]
    x = np.ascontiguousarray(x, dtype=np.float32)
    got, st = ext._knn_exact(x, k, select="tanimoto")
    want, _ = oracle.knn_exact(x, k, select="tanimoto")
    for a, b in zip((got[0].view(np.uint32), got[1], got[2]), want):
        np.testing.assert_array_equal(a, b)
    assert st["blocks_skipped"] <= st["blocks_total"] and st["max_err_ratio"] < 1.0
    if norms == "spread" and n >= 1_300 and d > 4:
        assert st["blocks_skipped"] > 0


_ABOVE = """
import sys
import numpy as np, torch
from costal_gb300 import _costal as ext
n, d, k, select = 4_194_433, 8, 3, sys.argv[1]
rng = np.random.default_rng(5)
x = rng.standard_normal((n, d), dtype=np.float32)
x /= np.linalg.norm(x, axis=1, keepdims=True)
if select == "tanimoto":
    x *= np.exp(rng.uniform(0.0, 7.0, (n, 1))).astype(np.float32)
ext._knn_exact(x[:1000], k)
free = torch.cuda.mem_get_info()[0]
(idx, cos, norms), st = ext._knn_exact(x, k, select=select)
assert free - torch.cuda.mem_get_info()[0] < 3 << 30, free - torch.cuda.mem_get_info()[0]
assert st["col_block"] == 128 and st["blocks_stopped"] == 0
assert (st["blocks_skipped"] > st["blocks_total"] // 2) == (select == "tanimoto"), st
x64 = torch.from_numpy(x).cuda().double()
nn = x64.norm(dim=1)
for i in rng.integers(0, n, 40):
    dot = x64 @ x64[i]
    t = dot / (nn * nn[i]) if select == "cosine" else dot / (nn**2 + nn[i]**2 - dot)
    t[i] = -9
    best = torch.topk(t, k)
    assert sorted(best.indices.tolist()) == sorted(idx[i].tolist()), i
"""


@pytest.mark.gpu
@pytest.mark.parametrize("select", ["cosine", "tanimoto"])
def test_above_the_longest_sorted_lists(ext, select):
    """4,194,433 rows, one query block past the longest lists: O(n) memory (lists would take 6.4 GB), and
    Tanimoto selection still leaves out what the norms rule out."""
    env = dict(os.environ, PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", _ABOVE, select], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("matmul,select,n,d", [
    ("fp32", "cosine", 20_001, 12), ("fp32", "cosine", 20_001, 40), ("fp32", "cosine", 9_000, 70),  # lists, all tiles
    ("fp32", "tanimoto", 300, 5), ("fp32", "tanimoto", 20_001, 12),                                 # walk, lists
    ("bf16", "cosine", 5_000, 12), ("bf16", "cosine", 25_000, 40), ("bf16", "cosine", 3_000, 520)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_rows_on_every_route(ext, matmul, select, n, d, bad):
    """The error names the first bad row wherever the rows have been by then, and the next call is right."""
    x = clustered(n, d, n + d)
    want, _ = ext._knn_exact(x, 5, matmul=matmul, select=select)
    y = x.copy()
    y[n - 7, d - 1] = bad
    y[n - 3] = np.nan
    with pytest.raises(ValueError, match=f"row {n - 7} contains NaN or inf"):
        ext._knn_exact(y, 5, matmul=matmul, select=select)
    got, _ = ext._knn_exact(x, 5, matmul=matmul, select=select)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
def test_non_finite_rows_in_training(ext):
    x = clustered(20_001, 12, 9)
    ext._mlp_train(x, 5, sample=2000, epochs=1)
    before = ext._mlp_get()
    x[17_000, 3] = np.inf
    with pytest.raises(ValueError, match="row 17000 contains NaN or inf"):
        ext._mlp_train(x, 5, sample=2000, epochs=1)
    np.testing.assert_array_equal(ext._mlp_get()[0], before[0])


@pytest.mark.gpu
@pytest.mark.parametrize("select,spread", [("cosine", 1.0), ("tanimoto", 1.2), ("tanimoto", 400.0)])
def test_lists_of_256_row_blocks(ext, select, spread):
    """Above 1,048,576 rows a list entry is two column tiles (their own geometry and norm ranges beside the
    query blocks'), with a last entry of one: the answer equals the pass over all tiles, in the cells' order and (norms
    spread 400-fold) in the norm order."""
    n, d, k = 1_048_577 + 128 * 3 + 40, 8, 3
    rng = np.random.default_rng(3)
    centres = rng.standard_normal((60, d))
    x = centres[rng.integers(0, 60, n)] + 0.15 * rng.standard_normal((n, d), dtype=np.float32)
    x = np.ascontiguousarray(x * np.exp(rng.uniform(0, np.log(spread), (n, 1))), dtype=np.float32)
    got, st = ext._knn_exact(x, k, select=select)
    want, st0 = ext._knn_exact(x, k, select=select, prune=False)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    left_out = "blocks_stopped" if select == "cosine" else "blocks_skipped"
    assert st["col_block"] == 256 and st[left_out] > st["blocks_total"] // 4
    assert st0["col_block"] == 128 and st0[left_out] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["cells", "norms"])
def test_the_two_orders_of_tanimoto_selection(ext, order):
    """Enough rows for lists. Forty tight clusters with norms within 5 %: only the cells' order leaves blocks out.
    One cluster with norms spread 55-fold: only the norm order does."""
    n, d, k = 30_000, 12, 10
    rng = np.random.default_rng(8)
    x = clustered(n, d, 8, n_centers=40 if order == "cells" else 1, noise=0.1 if order == "cells" else 0.5).astype(np.float64)
    x *= (rng.uniform(1.0, 1.05, n) if order == "cells" else np.exp(rng.uniform(0.0, 4.0, n)))[:, None] / np.linalg.norm(
        x, axis=1, keepdims=True)
    x = np.ascontiguousarray(x, dtype=np.float32)
    got, st = ext._knn_exact(x, k, select="tanimoto")
    want, _ = ext._knn_exact(x, k, select="tanimoto", prune=False)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert st["blocks_skipped"] > 0.3 * st["blocks_total"]
