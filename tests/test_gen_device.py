"""Device graph builder against the host builder: the same arrays, bit for
bit (both follow the counter-based R-MAT / ER draws of gen_common.h)."""
import numpy as np
import pytest

import apspie_b200 as ap


@pytest.mark.gpu
@pytest.mark.parametrize("scale,ef,sym,scr", [(8, 4, True, True), (12, 16, True, True),
                                              (12, 16, False, True), (14, 8, True, False),
                                              (16, 16, True, True)])
def test_rmat_device_matches_host(ctx, scale, ef, sym, scr):
    h = ap.gen_rmat(scale, ef, seed=3, symmetric=sym, scramble=scr)
    d = ap.gen_rmat_device(ctx, scale, ef, seed=3, symmetric=sym, scramble=scr)
    assert d.m == h.m and d.nnz == h.nnz
    np.testing.assert_array_equal(d.ptr.cpu().numpy(), h.ptr)
    np.testing.assert_array_equal(d.ind.cpu().numpy(), h.ind)


@pytest.mark.gpu
@pytest.mark.parametrize("n,deg", [(2, 1), (1000, 8), (1 << 16, 16)])
def test_er_device_matches_host(ctx, n, deg):
    h = ap.gen_er(n, deg, seed=5)
    d = ap.gen_er_device(ctx, n, deg, seed=5)
    assert d.nnz == h.nnz
    np.testing.assert_array_equal(d.ptr.cpu().numpy(), h.ptr)
    np.testing.assert_array_equal(d.ind.cpu().numpy(), h.ind)


@pytest.mark.gpu
def test_rmat22_device_properties(ctx):
    """At the benchmark size: rows sorted and strictly increasing, no
    self-loops, symmetric (checked by the transpose having the same nnz and
    a checksum of (row, col) pairs equal in both orientations)."""
    import torch
    d = ap.gen_rmat_device(ctx, 22, 16, seed=1)
    ptr, ind = d.ptr.long(), d.ind.long()
    rows = torch.repeat_interleave(torch.arange(d.m, device=ptr.device), ptr[1:] - ptr[:-1])
    assert int(ptr[-1]) == d.nnz
    assert not bool((rows == ind).any())
    key = rows * d.m + ind
    assert bool((key[1:] > key[:-1]).all())
    tkey = ind * d.m + rows
    assert int((key * 2654435761 % (1 << 61)).sum()) == int((tkey * 2654435761 % (1 << 61)).sum())


@pytest.mark.gpu
def test_weights_device_match_host(ctx):
    h = ap.gen_rmat(12, 16, seed=3)
    wu = ap.weights_u32(h, seed=9)
    wf = ap.weights_f32(h, seed=9)
    d = ap.weights_device(ctx, h.to_device(), seed=9)
    np.testing.assert_array_equal(d.w_u32.cpu().numpy().view(np.uint32), wu)
    np.testing.assert_array_equal(d.w_f32.cpu().numpy(), wf)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(1000, 1000), (700, 1500), (3000, 40)])
def test_csr_transpose_matches_host(ctx, m, n):
    """apspie_csr_transpose = the CSC: offsets, row ids ascending within a
    column, values carried along (scipy's csr -> csc as the reference)."""
    import scipy.sparse as sp
    import torch
    rng = np.random.default_rng(m + n)
    a = sp.random(m, n, density=0.01, format="csr", random_state=rng, dtype=np.float32)
    a.sort_indices()
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    tp, ti, tv = ap.csr_transpose(ctx, m, n, t(a.indptr.astype(np.int32)),
                                  t(a.indices.astype(np.int32)), t(a.data))
    c = a.tocsc()
    c.sort_indices()
    np.testing.assert_array_equal(tp.cpu().numpy(), c.indptr)
    np.testing.assert_array_equal(ti.cpu().numpy(), c.indices)
    np.testing.assert_array_equal(tv.cpu().numpy(), c.data)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,nnz", [(1, 1, 1), (5, 3, 31), (4000, 70, 2047), (3, 5000, 2048),
                                     (300000, 257, 2049), (700, 300, 40961)])
def test_csr_transpose_rows_across_tiles(ctx, m, n, nnz):
    """Rows that span tiles of 2,048 entries (one row holds half of them), long
    runs of empty rows, entry counts at and around a tile, 1 to 2 sort passes;
    columns may repeat in a row (their order is then the input's)."""
    import torch
    rng = np.random.default_rng(nnz)
    rows = np.sort(np.concatenate([np.full(nnz // 2, m // 2),
                                   rng.integers(0, m, size=nnz - nnz // 2)]))
    ind = rng.integers(0, n, size=nnz).astype(np.int32)
    val = rng.random(nnz, dtype=np.float32)
    ptr = np.searchsorted(rows, np.arange(m + 1)).astype(np.int32)
    t = lambda x: torch.from_numpy(x).cuda()
    tp, ti, tv = ap.csr_transpose(ctx, m, n, t(ptr), t(ind), t(val))
    order = np.argsort(ind, kind="stable")
    assert np.array_equal(tp.cpu().numpy(), np.searchsorted(ind[order], np.arange(n + 1)))
    assert np.array_equal(ti.cpu().numpy(), rows[order])
    assert np.array_equal(tv.cpu().numpy(), val[order])
    _, _, ones = ap.csr_transpose(ctx, m, n, t(ptr), t(ind))
    assert bool((ones == 1.0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("leaves,extra", [(1, 0), (2047, 0), (2049, 64), (9000, 20000)])
def test_tc_prepare_hub_rows_across_tiles(ctx, leaves, extra):
    """L of a star with random edges among its leaves: the hub's row spans
    tiles, and isolated vertices leave empty rows."""
    import torch
    rng = np.random.default_rng(leaves)
    m = leaves + 50
    hub = m // 3
    others = np.setdiff1d(rng.permutation(m)[:leaves + 1], [hub])
    e = np.concatenate([np.stack([np.full(len(others), hub), others]),
                        rng.choice(others, size=(2, extra))], axis=1)
    e = e[:, e[0] != e[1]]
    keys = np.unique(np.concatenate([e[0] * m + e[1], e[1] * m + e[0]]))
    rows, cols = keys // m, keys % m
    ptr = np.searchsorted(rows, np.arange(m + 1)).astype(np.int32)
    g = ap.DeviceGraph(m, len(cols), torch.from_numpy(ptr).cuda(),
                       torch.from_numpy(cols.astype(np.int32)).cuda(), symmetric=True)
    perm, lp, li = ap.tc_prepare(ctx, g)
    want = np.empty(m, np.int64)
    want[np.lexsort((np.arange(m), np.diff(ptr)))] = np.arange(m)
    assert np.array_equal(perm.cpu().numpy(), want)
    r, c = want[rows], want[cols]
    low = np.sort((r * m + c)[c < r])
    assert np.array_equal(lp.cpu().numpy(), np.searchsorted(low // m, np.arange(m + 1)))
    assert np.array_equal(li.cpu().numpy(), low % m)


@pytest.mark.gpu
@pytest.mark.parametrize("nnz", [1, 2, 33, 511, 512, 4095, 4096, 4097, 8191, 8192, 8193])
@pytest.mark.parametrize("n", [3, 256, 257, 100000])
def test_csr_transpose_small_sorts(ctx, nnz, n):
    """Entry and column counts around the one-block sort and scan, one to
    three digit passes, with columns that repeat."""
    import torch
    rng = np.random.default_rng(nnz + n)
    m = 50
    rows = np.sort(rng.integers(0, m, size=nnz))
    ind = rng.integers(0, n, size=nnz).astype(np.int32)
    ptr = np.searchsorted(rows, np.arange(m + 1)).astype(np.int32)
    val = rng.random(nnz, dtype=np.float32)
    t = lambda x: torch.from_numpy(x).cuda()
    tp, ti, tv = ap.csr_transpose(ctx, m, n, t(ptr), t(ind), t(val))
    order = np.argsort(ind, kind="stable")
    assert np.array_equal(tp.cpu().numpy(), np.searchsorted(ind[order], np.arange(n + 1)))
    assert np.array_equal(ti.cpu().numpy(), rows[order])
    assert np.array_equal(tv.cpu().numpy(), val[order])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8190, 8191, 8192, 12287, 12288, 1 << 22, (1 << 22) + 5])
def test_offset_scan_sizes(ctx, n):
    """The offset scan around its one-launch, few-tile and many-tile forms:
    the offsets of a transpose with n columns."""
    import torch
    rng = np.random.default_rng(n)
    ind = rng.integers(0, n, size=5000).astype(np.int32)
    ind[:3] = (0, n - 1, n // 2)
    t = lambda x: torch.from_numpy(x).cuda()
    tp, ti, _ = ap.csr_transpose(ctx, 1, n, t(np.array([0, 5000], np.int32)), t(ind))
    want = np.zeros(n + 1, np.int64)
    np.add.at(want, ind + 1, 1)
    assert np.array_equal(tp.cpu().numpy(), np.cumsum(want))
    assert int(ti.abs().max()) == 0
