"""Generic SpMSpV parity (both mXv forms, every semiring, both the radix-sort
and the bitmap path) against the oracle's restatement of src/mXv.cuh."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SEMIRINGS = [0, 1, 2, 3]   # PLUS_TIMES, MIN_PLUS, MAX_TIMES, OR_AND
PLUS_REL_TOL = 1e-5        # float sums vs the FP64 oracle, relative to sum |terms|


def _graph(scale=12, seed=3, positive=False):
    import apspie_b200 as ap
    h = ap.gen_rmat(scale, 16, seed=seed, symmetric=False)
    rng = np.random.default_rng(seed)
    vals = rng.uniform(0.01, 1.0, h.nnz) if positive else rng.uniform(-1, 1, h.nnz)
    return h, vals.astype(np.float32)


def _compare(sr, got_i, got_v, ref_i, ref_v, h, vals, xind, xval):
    np.testing.assert_array_equal(got_i, ref_i)
    if sr == 0:
        # bound on the rounding of a float sum: relative to the sum of |terms|
        absref = oracle.spmspv(0, h.m, h.ptr, h.ind, np.abs(vals), xind, np.abs(xval))[1]
        assert np.all(np.abs(got_v - ref_v) <= PLUS_REL_TOL * absref + 1e-30)
    else:
        np.testing.assert_array_equal(got_v.astype(np.float32), ref_v.astype(np.float32))


@pytest.mark.parametrize("sr", SEMIRINGS)
@pytest.mark.parametrize("path", ["sort", "bitmap"])
@pytest.mark.parametrize("density", [0.001, 0.05])
def test_spmspv_vs_oracle(ctx, sr, path, density):
    import torch
    import apspie_b200 as ap
    h, vals = _graph(positive=(sr == 1))
    g = h.to_device(with_transpose=False)
    rng = np.random.default_rng(int(density * 1000) + sr)
    xind = np.flatnonzero(rng.random(h.m) < density).astype(np.int32)
    xval = rng.uniform(0.1, 2.0, xind.size).astype(np.float32)
    ap.spmspv_set_params(ctx, 0.0 if path == "sort" else 1e12)
    try:
        yi, yv, e = ap.spmspv(ctx, sr, g, torch.from_numpy(xind).cuda(),
                              torch.from_numpy(xval).cuda(), torch.from_numpy(vals).cuda())
    finally:
        ap.spmspv_set_params(ctx)
    ri, rv = oracle.spmspv(sr, h.m, h.ptr, h.ind, vals, xind, xval)
    assert e == int(h.degrees()[xind].sum())
    _compare(sr, yi.cpu().numpy(), yv.cpu().numpy().astype(np.float64), ri, rv, h, vals, xind,
             xval)


def test_spmspv_hub_columns_and_empty(ctx):
    import torch
    import apspie_b200 as ap
    h, vals = _graph(scale=14, seed=5)
    g = h.to_device(with_transpose=False)
    deg = h.degrees()
    hubs = np.sort(np.argsort(deg)[-20:]).astype(np.int32)  # columns far above the chunk size
    assert deg[hubs].max() > 256
    xval = np.ones(hubs.size, np.float32)
    for path in (0.0, 1e12):
        ap.spmspv_set_params(ctx, path)
        yi, yv, _ = ap.spmspv(ctx, 0, g, torch.from_numpy(hubs).cuda(),
                              torch.from_numpy(xval).cuda(), torch.from_numpy(vals).cuda())
        ri, rv = oracle.spmspv(0, h.m, h.ptr, h.ind, vals, hubs, xval)
        _compare(0, yi.cpu().numpy(), yv.cpu().numpy().astype(np.float64), ri, rv, h, vals, hubs,
                 xval)
    ap.spmspv_set_params(ctx)
    yi, yv, e = ap.spmspv(ctx, 0, g, torch.zeros(0, dtype=torch.int32, device="cuda"))
    assert yi.numel() == 0 and e == 0


@pytest.mark.parametrize("sr", [0, 1])
def test_mxv_dense_reference_semantics(ctx, sr):
    """Dense in / dense out: frontier by bitify (> 0.5) or finite (< 1e38),
    untouched rows 0 (or 1.70141e38), return value = expanded size."""
    import torch
    import apspie_b200 as ap
    h, vals = _graph(positive=True)
    g = h.to_device(with_transpose=False)
    rng = np.random.default_rng(7)
    if sr == 0:
        x = np.where(rng.random(h.m) < 0.01, 1.0, 0.0).astype(np.float32)
        front = np.flatnonzero(x > 0.5)
    else:
        x = np.where(rng.random(h.m) < 0.01, rng.uniform(0, 5, h.m),
                     np.float32(1.70141e38)).astype(np.float32)
        front = np.flatnonzero((x > -1) & (x < 1e38))
    y, total = ap.mxv_dense(ctx, sr, g, torch.from_numpy(x).cuda(), torch.from_numpy(vals).cuda())
    y = y.cpu().numpy()
    ri, rv = oracle.spmspv(sr, h.m, h.ptr, h.ind, vals, front, x[front])
    assert total == int(h.degrees()[front].sum())
    empty = np.float32(0.0) if sr == 0 else np.float32(1.70141e38)
    expect = np.full(h.m, empty, np.float32)
    expect[ri] = rv.astype(np.float32)
    untouched = np.ones(h.m, bool)
    untouched[ri] = False
    np.testing.assert_array_equal(y[untouched], expect[untouched])
    np.testing.assert_allclose(y[ri], expect[ri], rtol=1e-5)


def test_spmspv_bfs_step_matches_bfs(ctx):
    """One OR_AND SpMSpV from a source = the source's out-neighbours."""
    import torch
    import apspie_b200 as ap
    h, _ = _graph()
    g = h.to_device(with_transpose=False)
    s = int(np.argmax(h.degrees()))
    yi, _, _ = ap.spmspv(ctx, 3, g, torch.tensor([s], dtype=torch.int32, device="cuda"))
    np.testing.assert_array_equal(yi.cpu().numpy(), np.unique(h.ind[h.ptr[s]:h.ptr[s + 1]]))


@pytest.mark.gpu
@pytest.mark.parametrize("semiring", [0, 1, 2, 3])
def test_dense_spmv_all_rows(ctx, semiring):
    """apspie_spmv against an FP64 / exact restatement: power-law rows with
    a few hubs above the block threshold (4096) and empty rows."""
    import torch
    import apspie_b200 as ap
    rng = np.random.default_rng(semiring)
    m = 6000
    lens = rng.integers(0, 20, m)
    lens[::997] = 0
    lens[[5, 1234, 4321]] = [5000, 9000, 4097]
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ind = rng.integers(0, m, int(ptr[-1])).astype(np.int32)
    val = rng.uniform(-1, 1, int(ptr[-1])).astype(np.float32)
    x = rng.uniform(-1, 1, m).astype(np.float32)
    x[::5] = 0
    t = lambda a: torch.from_numpy(a).cuda()
    y = ap.spmv(ctx, m, t(ptr), t(ind), t(val), t(x), semiring).cpu().numpy()
    for r in range(m):
        a, xs = val[ptr[r]:ptr[r + 1]], x[ind[ptr[r]:ptr[r + 1]]]
        if semiring == 0:
            ref = float(np.sum(a.astype(np.float64) * xs.astype(np.float64)))
            tol = 1e-6 * max(1.0, float(np.sum(np.abs(a.astype(np.float64) * xs))))
            assert abs(y[r] - ref) <= tol, (r, y[r], ref)
        elif semiring == 1:
            ref = np.float32(np.min(a + xs)) if len(a) else np.finfo(np.float32).max
            assert y[r] == ref, (r, y[r], ref)
        elif semiring == 2:
            ref = np.float32(np.max(a * xs)) if len(a) else -np.finfo(np.float32).max
            assert y[r] == ref, (r, y[r], ref)
        else:
            ref = 1.0 if np.any((a != 0) & (xs != 0)) else 0.0
            assert y[r] == ref, (r, y[r], ref)


@pytest.mark.parametrize("sr", [0, 1, 2, 3])
@pytest.mark.parametrize("path", ["sort", "bitmap"])
@pytest.mark.parametrize("total", [1, 2047, 2048, 2049, 40961])
def test_spmspv_tile_edges(ctx, sr, path, total):
    """Expanded sizes at and around a tile of 2,048 entries, half of them in
    one column that spans tiles, between runs of empty columns; a repeated
    frontier vertex counts twice."""
    import torch
    import apspie_b200 as ap
    rng = np.random.default_rng(total)
    m = 3001
    xind = np.sort(rng.choice(m, size=200, replace=False)).astype(np.int32)
    deg = np.zeros(m, np.int64)
    np.add.at(deg, rng.choice(xind[100:140], size=total - total // 2), 1)
    deg[xind[60]] += total // 2
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    ind = rng.integers(0, m, size=total).astype(np.int32)
    vals = rng.uniform(0.5, 2, size=total).astype(np.float32)
    if total > 1:
        xind = np.append(xind, xind[110]).astype(np.int32)
    xval = rng.uniform(0.5, 2, size=len(xind)).astype(np.float32)
    h = ap.HostGraph(m, ptr, ind)
    g = h.to_device(with_transpose=False)
    ap.spmspv_set_params(ctx, 0.0 if path == "sort" else 1e12)
    try:
        yi, yv, e = ap.spmspv(ctx, sr, g, torch.from_numpy(xind).cuda(),
                              torch.from_numpy(xval).cuda(), torch.from_numpy(vals).cuda())
    finally:
        ap.spmspv_set_params(ctx)
    ri, rv = oracle.spmspv(sr, m, ptr, ind, vals, xind, xval)
    assert e == int(deg[xind].sum())
    np.testing.assert_array_equal(yi.cpu().numpy(), ri)
    np.testing.assert_allclose(yv.cpu().numpy(), rv, rtol=1e-6)


def test_spmspv_bitmap_extreme_terms(ctx):
    """Negative, zero, infinite and not-a-number terms in the minimum and the
    maximum: a row that only infinities of the identity's sign or NaN terms
    touch is in y with the identity."""
    import torch
    import apspie_b200 as ap
    inf, nan = np.inf, np.nan
    # column 0 -> rows 0..6, column 1 -> the same rows
    terms0 = np.array([-1.5, 0.0, inf, -inf, nan, 3.0, nan], np.float32)
    terms1 = np.array([2.5, -2.0, inf, 7.0, nan, nan, -4.0], np.float32)
    ptr = np.array([0, 7, 14] + [14] * 6, np.int32)
    ind = np.tile(np.arange(7), 2).astype(np.int32)
    val = torch.from_numpy(np.concatenate([terms0, terms1])).cuda()
    g = ap.HostGraph(8, ptr, ind).to_device(with_transpose=False)
    xi = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    zero, one = torch.zeros(2, device="cuda"), torch.ones(2, device="cuda")
    yi, yv, _ = ap.spmspv(ctx, 1, g, xi, zero, val)
    assert yi.tolist() == list(range(7))
    assert yv.tolist() == [-1.5, -2.0, inf, -inf, inf, 3.0, -4.0]
    yi, yv, _ = ap.spmspv(ctx, 2, g, xi, one, val)
    assert yi.tolist() == list(range(7))
    assert yv.tolist() == [2.5, 0.0, inf, 7.0, -inf, 3.0, -4.0]


@pytest.mark.parametrize("sr", [1, 2])
@pytest.mark.parametrize("m", [55, 56, 57])
def test_spmspv_nan_rows_below_the_threshold(ctx, sr, m):
    """14 products at the default factor of 4: up to 55 rows a row of NaN
    terms keeps the identity, from 56 on it is NaN, as the sort path has it."""
    import torch
    import apspie_b200 as ap
    inf, nan = np.inf, np.nan
    terms = np.array([-1.5, 0.0, inf, -inf, nan, 3.0, nan,
                      2.5, -2.0, inf, 7.0, nan, nan, -4.0], np.float32)
    ptr = np.array([0, 7] + [14] * (m - 1), np.int32)
    ind = np.tile(np.arange(7), 2).astype(np.int32)
    g = ap.HostGraph(m, ptr, ind).to_device(with_transpose=False)
    xi = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    xv = torch.full((2,), 0.0 if sr == 1 else 1.0, device="cuda")
    val = torch.from_numpy(terms).cuda()
    yi, yv, _ = ap.spmspv(ctx, sr, g, xi, xv, val)
    ap.spmspv_set_params(ctx, 0.0)
    try:
        si, sv, _ = ap.spmspv(ctx, sr, g, xi, xv, val)
    finally:
        ap.spmspv_set_params(ctx)
    assert yi.tolist() == si.tolist() == list(range(7))
    expect = sv.cpu().numpy()
    assert np.isnan(expect[4])
    if m < 56:
        expect[4] = inf if sr == 1 else -inf
    np.testing.assert_array_equal(yv.cpu().numpy(), expect)


@pytest.mark.parametrize("m", [31, 32, 33, 2049])
def test_spmspv_zero_sums(ctx, m):
    """PLUS_TIMES rows whose terms are zeros of either sign or cancel are in y
    with +0.0, at the ends of the accumulator too."""
    import torch
    import apspie_b200 as ap
    rows = np.array([0, 1, m - 2, m - 1], np.int32)
    ptr = np.array([0, 4, 8] + [8] * (m - 2), np.int32)
    ind = np.tile(rows, 2).astype(np.int32)
    val = np.array([-0.0, 1.5, 0.0, -0.0, -0.0, -1.5, -0.0, 2.0], np.float32)
    g = ap.HostGraph(m, ptr, ind).to_device(with_transpose=False)
    xi = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    yi, yv, _ = ap.spmspv(ctx, 0, g, xi, torch.ones(2, device="cuda"),
                          torch.from_numpy(val).cuda())
    assert yi.tolist() == rows.tolist()
    assert yv.tolist() == [0.0, 0.0, 0.0, 2.0]
    assert not np.signbit(yv.cpu().numpy()).any()


@pytest.mark.parametrize("guess", ["sparse", "dense"])
def test_spmspv_sparse_sums_run_in_the_frontiers_order(ctx, guess):
    """PLUS_TIMES with products * factor <= m: every row's terms are added in
    the order of the frontier's columns, in double, whatever the mean column
    length makes of the frontier; one row less and the sum is only close."""
    import torch
    import apspie_b200 as ap
    m, cols, rows = 1 << 16, 512, 32       # 16,384 products: 4 * 16,384 = m
    rng = np.random.default_rng(5)
    xind = np.sort(rng.choice(m, cols, replace=False)).astype(np.int32)
    deg = np.zeros(m, np.int64)
    if guess == "dense":
        deg[:] = 30
    deg[xind] = rows
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    ind = rng.integers(0, m, int(ptr[-1])).astype(np.int32)
    val = rng.uniform(1, 2, ind.size).astype(np.float32)
    target = np.arange(rows, dtype=np.int32) * 1000
    # small terms among huge ones that cancel: which of the small ones are left
    # depends on the order of the additions
    huge = np.concatenate([np.full(cols // 4, 2.0**60), np.full(cols // 4, -2.0**60),
                           np.zeros(cols // 2)])
    order = np.stack([rng.permutation(huge) for _ in range(rows)], axis=1)
    for k, c in enumerate(xind):
        ind[ptr[c]:ptr[c + 1]] = target
        row = val[ptr[c]:ptr[c + 1]]
        row[order[k] != 0] = order[k][order[k] != 0]
    ref = np.zeros(rows)
    for c in xind:
        ref += val[ptr[c]:ptr[c + 1]].astype(np.float64)
    t = lambda a: torch.from_numpy(a).cuda()
    g = ap.HostGraph(m, ptr, ind).to_device(with_transpose=False)
    for _ in range(3):
        yi, yv, e = ap.spmspv(ctx, 0, g, t(xind), None, t(val))
        assert e == cols * rows and yi.tolist() == target.tolist()
        np.testing.assert_array_equal(yv.cpu().numpy(), ref.astype(np.float32))
    x = np.zeros(m, np.float32)
    x[xind] = 1.0
    y, e = ap.mxv_dense(ctx, 0, g, t(x), t(val))
    assert e == cols * rows
    np.testing.assert_array_equal(y.cpu().numpy()[target], ref.astype(np.float32))
    # one more product: the bitmap path
    ptr[xind[-1] + 1:] += 1
    ind = np.insert(ind, ptr[xind[-1]] + rows, 0).astype(np.int32)
    val = np.insert(val, ptr[xind[-1]] + rows, 0.0).astype(np.float32)
    g = ap.HostGraph(m, ptr, ind).to_device(with_transpose=False)
    yi, yv, e = ap.spmspv(ctx, 0, g, t(xind), None, t(val))
    assert e == cols * rows + 1 and yi.tolist() == target.tolist()
    mag = np.zeros(rows)
    for c in xind:
        mag += np.abs(val[ptr[c]:ptr[c] + rows].astype(np.float64))
    # 512 double additions and one rounding to float
    assert np.all(np.abs(yv.cpu().numpy() - ref) <= 512 * 2.0**-52 * mag + 2.0**-23 * np.abs(ref))


@pytest.mark.parametrize("sr", SEMIRINGS)
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("m", [1 << 22, (1 << 22) + 1])
def test_spmspv_both_sides_of_the_row_limit(ctx, sr, dense, m):
    """The rows up to which the bitmap path starts by itself, with products
    on either side of m / factor, against the oracle."""
    import torch
    import apspie_b200 as ap
    rng = np.random.default_rng(m + dense)
    cols = 3000
    xind = np.sort(rng.choice(m, cols, replace=False)).astype(np.int32)
    deg = np.zeros(m, np.int64)
    deg[xind] = rng.integers(0, 900 if dense else 20, cols)
    total = int(deg.sum())
    assert (total * 4 > m) == dense
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    ind = (rng.integers(0, m, total) // 3 * 3).astype(np.int32)
    ind[::7] = m - 1
    val = rng.uniform(0.5, 2, total).astype(np.float32)
    xval = rng.uniform(0.5, 2, cols).astype(np.float32)
    g = ap.HostGraph(m, ptr, ind).to_device(with_transpose=False)
    yi, yv, e = ap.spmspv(ctx, sr, g, torch.from_numpy(xind).cuda(), torch.from_numpy(xval).cuda(),
                          torch.from_numpy(val).cuda())
    ri, rv = oracle.spmspv(sr, m, ptr, ind, val, xind, xval)
    assert e == total
    np.testing.assert_array_equal(yi.cpu().numpy(), ri)
    np.testing.assert_allclose(yv.cpu().numpy(), rv, rtol=1e-6)
