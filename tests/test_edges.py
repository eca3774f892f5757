"""The passes over a CSR's entries in tiles (edges.cuh): row offsets that
index a part of larger arrays, and counts that the offsets correct."""
import ctypes as C

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _csr(m, n, nnz, seed):
    rng = np.random.default_rng(seed)
    deg = np.bincount(rng.integers(0, m, nnz), minlength=m)
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    ind = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in deg]).astype(np.int32)
    return ptr, ind, rng.uniform(-1, 1, nnz).astype(np.float32)


@pytest.mark.parametrize("rows", [(1, 400), (37, 38), (200, 395), (399, 400)])
def test_spgemm_of_a_slice_of_rows(ctx, rows):
    """A's offsets taken from the middle of a larger matrix, its entries'
    arrays left whole: C is the product of those rows."""
    import apspie_b200 as ap
    m, n = 400, 300
    ptr, ind, val = _csr(m, n, 20000, 1)
    bptr, bind, bval = _csr(n, n, 3000, 2)
    r0, r1 = rows
    d_ptr, d_ind, d_val = _t(ptr), _t(ind), _t(val)
    B = (n, n, _t(bptr), _t(bind), _t(bval))
    got = ap.spgemm(ctx, (r1 - r0, n, d_ptr[r0:r1 + 1], d_ind, d_val), B)
    lo, hi = ptr[r0], ptr[r1]
    own = (r1 - r0, n, _t(ptr[r0:r1 + 1] - lo), _t(ind[lo:hi]), _t(val[lo:hi]))
    ref = ap.spgemm(ctx, own, B)
    rp, ri, _ = oracle.spgemm(r1 - r0, n, ptr[r0:r1 + 1] - lo, ind[lo:hi], val[lo:hi], bptr, bind,
                              bval)
    np.testing.assert_array_equal(got[0].cpu().numpy(), rp)
    np.testing.assert_array_equal(got[1].cpu().numpy(), ri)
    # the same rows through the same kernels: sums of two or more products may
    # differ in the last bit of their rounding only
    np.testing.assert_allclose(got[2].cpu().numpy(), ref[2].cpu().numpy(), rtol=2.0**-22,
                               atol=2.0**-40)


@pytest.mark.parametrize("nnz", [0, 1, 2048, 19999])
def test_spgemm_reads_the_offsets_not_the_count(ctx, nnz):
    """apspie_csr's nnz below what its offsets hold leaves no entry out."""
    import torch
    from apspie_b200._native import Csr, check, lib
    m = n = 400
    ptr, ind, _ = _csr(m, n, 20000, 3)
    bptr, bind, _ = _csr(n, n, 3000, 4)
    t = [_t(a) for a in (ptr, ind, bptr, bind)]
    p = [C.c_void_p(x.data_ptr()) for x in t]
    A, B = Csr(m, n, nnz, p[0], p[1], None), Csr(n, n, len(bind), p[2], p[3], None)
    out, total = torch.empty(m + 1, dtype=torch.int32, device="cuda"), C.c_int64(0)
    check(lib.apspie_spgemm_symbolic(ctx.handle, C.byref(A), C.byref(B),
                                     C.c_void_p(out.data_ptr()), C.byref(total)), ctx.handle)
    rp, _, _ = oracle.spgemm(m, n, ptr, ind, None, bptr, bind, None)
    np.testing.assert_array_equal(out.cpu().numpy(), rp)
    assert total.value == rp[-1]


def test_triangles_of_graphs_packed_in_one_array(ctx):
    """Graphs whose rows lie one after the other in one index array, each with
    its part of the offsets, and an L placed behind other entries."""
    import torch
    import apspie_b200 as ap
    hs = [ap.gen_rmat(11, 16, seed=1), ap.gen_er(3000, 20, seed=2), ap.gen_rmat(9, 8, seed=3)]
    base = np.concatenate([[0], np.cumsum([h.nnz for h in hs])])
    ind = _t(np.concatenate([h.ind for h in hs]))
    for h, b in zip(hs, base):
        g = ap.HostGraph(h.m, h.ptr, h.ind, symmetric=True).to_device()
        perm, lp, li = ap.tc_prepare(ctx, g)
        _, olp, oli = oracle.tc_build_lower(h.m, h.ptr, h.ind)
        want = oracle.tc_lower(h.m, olp, oli)
        assert ap.triangle_count(ctx, h.m, lp, li) == want
        g.ptr, g.ind = _t(h.ptr + np.int32(b)), ind
        perm2, lp2, li2 = ap.tc_prepare(ctx, g)
        assert torch.equal(perm, perm2) and torch.equal(lp, lp2) and torch.equal(li, li2)
        behind = torch.cat([torch.zeros(5000, dtype=torch.int32, device="cuda"), li])
        assert ap.triangle_count(ctx, h.m, lp + 5000, behind) == want


@pytest.mark.parametrize("m", [8192, 8193, 8194, 8195, 20001, 300000])
@pytest.mark.parametrize("nnz", [2, 2047, 2048, 2049, 6000])
def test_tiles_over_runs_of_empty_rows(ctx, m, nnz):
    """Tiles that span about as many rows as are marked, and more: the first
    and the last row hold an entry, the others lie in a few clusters."""
    import apspie_b200 as ap
    rng = np.random.default_rng(m + nnz)
    where = np.concatenate([[0, m - 1], rng.integers(0, m, 5), np.arange(4000, 4100)])
    row = np.sort(np.concatenate([[0, m - 1], rng.choice(where, nnz - 2)]))
    ptr = np.searchsorted(row, np.arange(m + 1)).astype(np.int32)
    ind = rng.integers(0, 700, nnz).astype(np.int32)
    val = rng.uniform(-1, 1, nnz).astype(np.float32)
    tp, ti, tv = ap.csr_transpose(ctx, m, 700, _t(ptr), _t(ind), _t(val))
    order = np.argsort(ind, kind="stable")
    np.testing.assert_array_equal(tp.cpu().numpy(), np.searchsorted(ind[order], np.arange(701)))
    np.testing.assert_array_equal(ti.cpu().numpy(), row[order])
    np.testing.assert_array_equal(tv.cpu().numpy(), val[order])


def _fastest_ms(call):
    import torch
    best = float("inf")
    for _ in range(6):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        call()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("op", ["transpose", "spgemm", "spmspv"])
def test_empty_rows_are_not_one_blocks_work(ctx, op):
    """Millions of rows (or frontier columns) with 2,000 entries in one tile:
    0.1 to 0.3 ms.  A block that walks every one of them takes 5 to 19 ms."""
    import torch
    import apspie_b200 as ap
    from apspie_b200.graph import DeviceGraph
    m, nnz = (4000000 if op == "spmspv" else 10000000), 2000
    rng = np.random.default_rng(1)
    row = np.sort(rng.integers(0, m, nnz))
    ptr = _t(np.searchsorted(row, np.arange(m + 1)).astype(np.int32))
    ind = rng.integers(0, 1000, nnz).astype(np.int32)
    d_ind = _t(ind)
    if op == "transpose":
        call = lambda: ap.csr_transpose(ctx, m, 1000, ptr, d_ind)
        np.testing.assert_array_equal(call()[1].cpu().numpy(), row[np.argsort(ind, kind="stable")])
    elif op == "spgemm":
        one = (1000, 5, _t(np.arange(1001, dtype=np.int32)),
               _t((np.arange(1000) % 5).astype(np.int32)), None)
        call = lambda: ap.spgemm_symbolic(ctx, (m, 1000, ptr, d_ind, None), one)
        assert call()[1] == len(np.unique(row * 5 + ind % 5))
    else:
        g = DeviceGraph(m, nnz, ptr, d_ind)
        every = torch.arange(m, dtype=torch.int32, device="cuda")
        call = lambda: ap.spmspv(ctx, 1, g, every)
        assert call()[0].tolist() == np.unique(ind).tolist()
    assert _fastest_ms(call) < 2.0


def _symmetric(m, pairs):
    """CSR of the undirected multigraph of the given pairs."""
    r = np.concatenate([pairs[:, 0], pairs[:, 1]])
    c = np.concatenate([pairs[:, 1], pairs[:, 0]])
    order = np.lexsort((c, r))
    return np.searchsorted(r[order], np.arange(m + 1)).astype(np.int32), c[order].astype(np.int32)


@pytest.mark.parametrize("kind", ["tiny", "warp", "units", "parts"])
@pytest.mark.parametrize("repeats", [0, 1, 500])
def test_triangles_of_a_multigraph(ctx, kind, repeats):
    """Repeated edges count once in the mask and each time in the product,
    whatever the column lengths: columns of a quarter warp, a warp, a block and
    a block in parts."""
    import scipy.sparse as sp
    import apspie_b200 as ap
    from apspie_b200.graph import DeviceGraph
    rng = np.random.default_rng(repeats)
    m, clique = {"tiny": (400, 8), "warp": (400, 60), "units": (500, 300),
                 "parts": (1500, 1300)}[kind]
    a, b = np.triu_indices(clique, 1)
    pairs = np.concatenate([np.stack([a, b], 1), rng.integers(0, m, (3 * m, 2))])
    pairs = np.unique(np.sort(pairs, axis=1), axis=0)
    pairs = pairs[pairs[:, 0] != pairs[:, 1]]
    # some edges two or three times, those of the clique among them
    pairs = np.concatenate([pairs, pairs[rng.integers(0, len(pairs), repeats)], pairs[:repeats]])
    ptr, ind = _symmetric(m, pairs)
    g = DeviceGraph(m, len(ind), _t(ptr), _t(ind), symmetric=True)
    _, lp, li = ap.tc_prepare(ctx, g)
    hl, hi = lp.cpu().numpy(), li.cpu().numpy()
    M = sp.csr_matrix((np.ones(len(hi)), hi, hl), shape=(m, m))   # repeats are summed in products
    M.sum_duplicates()
    want = int(round((M @ M).multiply(M > 0).sum()))
    for _ in range(2):
        assert ap.triangle_count(ctx, m, lp, li) == want


@pytest.mark.parametrize("more", [0, 1, 1 << 33])
def test_triangle_count_takes_a_buffers_size_for_the_entries(ctx, more):
    """nnz(L) given as more than int32 offsets can name: the offsets tell."""
    import apspie_b200 as ap
    from apspie_b200._native import lib
    h = ap.gen_rmat(10, 16, seed=1)
    _, lp, li = ap.tc_prepare(ctx, h.to_device())
    n = C.c_int64(-1)
    rc = lib.apspie_tc(ctx.handle, h.m, C.c_int64(2**31 - 1 + more), C.c_void_p(lp.data_ptr()),
                       C.c_void_p(li.data_ptr()), C.byref(n))
    assert rc == 0 and n.value == ap.triangle_count(ctx, h.m, lp, li)
