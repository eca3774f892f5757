"""BFS parity: apspie_bfs (sm_100a, through the C ABI) against the reference's
CPU BFS (golden vectors) and the oracle, bit-exact, including the fixed
iteration count of the reference driver and both traversal directions."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _dev(ptr, ind):
    import apspie_b200 as ap
    return ap.HostGraph(len(ptr) - 1, np.asarray(ptr, np.int32), np.asarray(ind, np.int32)).to_device()


@pytest.mark.parametrize("kind", ["dir", "und"])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_bfs_fixtures_every_source(ctx, golden, fixture_names, kind, mode):
    import apspie_b200 as ap
    ap.bfs_set_params(ctx, mode=mode)
    try:
        for name in fixture_names:
            ptr, ind = golden[f"mtx/{name}/{kind}_ptr"], golden[f"mtx/{name}/{kind}_ind"]
            g = _dev(ptr, ind)
            ref = golden[f"mtx/{name}/{kind}_bfs"]
            for s in range(g.m):
                d = ap.bfs(ctx, g, s).cpu().numpy()
                np.testing.assert_array_equal(d, ref[s], err_msg=f"{name}/{kind} src {s}")
                st = ap.bfs_stats(ctx)
                assert st["levels"] == int(ref[s].max()) + 1
                assert st["vertices_reached"] == int((ref[s] >= 0).sum())
    finally:
        ap.bfs_set_params(ctx)


@pytest.mark.parametrize("scale,symmetric", [(14, True), (16, True), (14, False)])
def test_bfs_rmat_vs_oracle(ctx, scale, symmetric):
    import apspie_b200 as ap
    h = ap.gen_rmat(scale, 16, seed=scale, symmetric=symmetric)
    g = h.to_device()
    deg = h.degrees()
    for s in ap.seeded_sources(h, 6, seed=1) + [int(np.argmax(deg))]:
        d = ap.bfs(ctx, g, s).cpu().numpy()
        ref, depth = oracle.bfs(h.m, h.ptr, h.ind, s)
        np.testing.assert_array_equal(d, ref)
        st = ap.bfs_stats(ctx)
        assert st["levels"] == depth
        assert st["edges_traversed"] == int(deg[ref >= 0].sum())


def test_bfs_directions_agree(ctx):
    import apspie_b200 as ap
    h = ap.gen_rmat(15, 16, seed=9)
    g = h.to_device()
    s = ap.seeded_sources(h, 1, seed=2)[0]
    ref, _ = oracle.bfs(h.m, h.ptr, h.ind, s)
    pulls = []
    try:
        for mode in (0, 1, 2):
            ap.bfs_set_params(ctx, mode=mode)
            np.testing.assert_array_equal(ap.bfs(ctx, g, s).cpu().numpy(), ref)
            pulls.append(ap.bfs_stats(ctx)["pull_levels"])
    finally:
        ap.bfs_set_params(ctx)
    assert pulls[1] == 0 and pulls[2] > 0 and pulls[0] > 0


def test_bfs_fixed_iteration_count(ctx):
    """max_levels = the reference driver's `depth` argument (src/bfs.cuh:87)."""
    import apspie_b200 as ap
    h = ap.gen_rmat(13, 16, seed=4)
    g = h.to_device()
    s = ap.seeded_sources(h, 1, seed=3)[0]
    full, depth = oracle.bfs(h.m, h.ptr, h.ind, s)
    for k in (1, 2, 3, depth, depth + 5):
        d = ap.bfs(ctx, g, s, max_levels=k).cpu().numpy()
        expect = np.where(full < k, full, -1) if k < depth else full
        np.testing.assert_array_equal(d, expect, err_msg=f"max_levels={k}")


def test_bfs_edge_cases(ctx):
    import apspie_b200 as ap
    # isolated source, single vertex, edgeless graph
    g = _dev([0, 0, 1, 2], [2, 1])
    np.testing.assert_array_equal(ap.bfs(ctx, g, 0).cpu().numpy(), [0, -1, -1])
    np.testing.assert_array_equal(ap.bfs(ctx, g, 1).cpu().numpy(), [-1, 0, 1])
    g1 = _dev([0, 0], [])
    np.testing.assert_array_equal(ap.bfs(ctx, g1, 0).cpu().numpy(), [0])
    # a hub above the chunking threshold and a long path (many levels)
    n = 5000
    rows = np.concatenate([np.zeros(n - 1, np.int64), np.arange(1, n)])
    cols = np.concatenate([np.arange(1, n), np.zeros(n - 1, np.int64)])
    star = ap.from_edges(n, rows, cols)
    ref, _ = oracle.bfs(n, star.ptr, star.ind, 7)
    np.testing.assert_array_equal(ap.bfs(ctx, star.to_device(), 7).cpu().numpy(), ref)
    grid = ap.gen_grid(256, 256)
    ref, depth = oracle.bfs(grid.m, grid.ptr, grid.ind, 0)
    np.testing.assert_array_equal(ap.bfs(ctx, grid.to_device(), 0).cpu().numpy(), ref)
    assert ap.bfs_stats(ctx)["levels"] == depth == 511
    with pytest.raises(ap.ApspieError):
        ap.bfs(ctx, grid.to_device(), grid.m)


def test_bfs_rmat22_full_size(ctx):
    """The benchmark graph: bit-exact against the oracle at full size."""
    import apspie_b200 as ap
    h = ap.gen_rmat(22, 16, seed=1)
    g = h.to_device()
    s = ap.seeded_sources(h, 1, seed=0)[0]
    d = ap.bfs(ctx, g, s).cpu().numpy()
    ref, depth = oracle.bfs(h.m, h.ptr, h.ind, s)
    np.testing.assert_array_equal(d, ref)
    st = ap.bfs_stats(ctx)
    assert st["levels"] == depth and st["pull_levels"] > 0
    assert st["edges_traversed"] == int(h.degrees()[ref >= 0].sum())


def test_bfs_repeated_runs_with_direction_switches(ctx):
    """Repeated traversals that switch push -> pull -> push are all exact.
    (A frontier rebuilt for a push level once shared its counters with the
    level's direction decision; slower blocks then chose a different
    direction in a few percent of the runs.)"""
    import apspie_b200 as ap
    h = ap.gen_rmat(16, 16, seed=16)
    g = h.to_device()
    for s in (2300, 30945):
        ref, _ = oracle.bfs(h.m, h.ptr, h.ind, s)
        dirs = None
        for _ in range(40):
            np.testing.assert_array_equal(ap.bfs(ctx, g, s).cpu().numpy(), ref)
            tr = ap.bfs_trace(ctx)
            dirs = [t["dir"] for t in tr]
            for t in tr:
                if t["dir"] == "push":
                    assert t["expanded"] == t["frontier_edges"]
                    if t["queued"]:
                        assert t["queued"] == t["frontier"]
        assert "pull" in dirs and dirs[-1] == "push"


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("mode", [0, 2])
def test_bfs_prepared_in_adjacency(ctx, symmetric, mode):
    """apspie_bfs_prepare: each in-row is the set of in-neighbours ordered by
    out-degree (highest first, ties by id), and BFS over it gives the same
    depths as the oracle."""
    import apspie_b200 as ap
    h = ap.gen_rmat(14, 16, seed=21, symmetric=symmetric)
    g = ap.bfs_prepare(ctx, h.to_device(with_transpose=False))
    tptr, tind = g.tptr.cpu().numpy(), g.tind.cpu().numpy()
    tr = h.transpose()
    deg = np.diff(h.ptr)
    np.testing.assert_array_equal(tptr, tr.ptr)
    for v in range(0, h.m, 97):
        row = tind[tptr[v]:tptr[v + 1]]
        exp = sorted(tr.ind[tr.ptr[v]:tr.ptr[v + 1]], key=lambda u: (-deg[u], u))
        np.testing.assert_array_equal(row, exp, err_msg=f"row {v}")
    ap.bfs_set_params(ctx, mode=mode)
    try:
        for s in ap.seeded_sources(h, 6, seed=2):
            ref, _ = oracle.bfs(h.m, h.ptr, h.ind, s)
            np.testing.assert_array_equal(ap.bfs(ctx, g, s).cpu().numpy(), ref)
    finally:
        ap.bfs_set_params(ctx, mode=0)


def _tree(*fanouts):
    """Undirected tree given the number of children of every vertex, level by
    level (a number for all vertices of a level, or one per vertex)."""
    parent, level, n = [], np.array([0]), 1
    for f in fanouts:
        kids = np.broadcast_to(np.asarray(f), level.shape)
        parent.append(np.repeat(level, kids))
        level = np.arange(n, n + int(kids.sum()))
        n += len(level)
    p, c = np.concatenate(parent), np.arange(1, n)
    return np.concatenate([p, c]), np.concatenate([c, p]), n


def _layers(*sizes):
    """Undirected graph of layers; every vertex has an edge to a random vertex
    of the layer before, so depth = layer from vertex 0."""
    rng = np.random.default_rng(0)
    first = np.concatenate([[0], np.cumsum(sizes)])
    u = np.arange(1, first[-1])
    layer = np.searchsorted(first, u, side="right") - 1
    v = first[layer - 1] + (rng.random(len(u)) * np.asarray(sizes)[layer - 1]).astype(np.int64)
    return np.concatenate([u, v]), np.concatenate([v, u]), int(first[-1])


@pytest.mark.parametrize("edges", [
    _layers(*[1] * 700),
    _layers(1, 15, 16, 17, 511, 512, 513, 8191, 8192, 8193, 3),  # shares and warps
    _layers(1, 1000, 5000, 24000, 24600, 30000, 200, 1, 1),      # thin, wide, thin
    _layers(1, 40, 4000, 1, 5000, 7),                            # hubs below and above the limit
    # one block finds 150 * 31 vertices, more than its queue holds
    _tree(16, 150, np.repeat([31, 7], [150, 2250]), 1, 1),
], ids=["path", "shares", "wide", "hubs", "spill"])
@pytest.mark.parametrize("mode", [0, 1])
def test_bfs_thin_levels(ctx, edges, mode):
    """Graphs of few edges per vertex, whose thin levels one cluster runs:
    frontiers around a block's share, levels that are too wide or too
    hub-heavy, a block's queue that overflows, and a level limit before and
    after the hand-over."""
    import apspie_b200 as ap
    r, c, m = edges
    h = ap.from_edges(m, r, c)
    h.symmetric = True
    g = h.to_device()
    ap.bfs_set_params(ctx, mode=mode)
    try:
        for src in (0, m - 1, m // 2):
            ref, depth = oracle.bfs(h.m, h.ptr, h.ind, src)
            np.testing.assert_array_equal(ap.bfs(ctx, g, src).cpu().numpy(), ref)
            st = ap.bfs_stats(ctx)
            assert st["levels"] == depth
            assert st["vertices_reached"] == int((ref >= 0).sum())
            assert st["edges_traversed"] == int(h.degrees()[ref >= 0].sum())
            for lim in (1, 2, 4, depth - 1, depth, depth + 1):
                if lim < 1:
                    continue
                d = ap.bfs(ctx, g, src, max_levels=lim).cpu().numpy()
                np.testing.assert_array_equal(d, np.where(ref < lim, ref, -1))
    finally:
        ap.bfs_set_params(ctx)


_RESET_CHILD = """
import ctypes as C, glob, sys
import numpy as np
import nvidia.cuda_runtime
import apspie_b200 as ap
from apspie_b200._native import lib
rt = C.CDLL(glob.glob(list(nvidia.cuda_runtime.__path__)[0] + "/lib/libcudart.so*")[0])
h = ap.gen_grid(200, 300)
for turn in range(2):
    ctx, dev = C.c_void_p(), []
    assert lib.apspie_ctx_create(0, None, C.byref(ctx)) == 0
    for a in (h.ptr, h.ind, np.zeros(h.m, np.int32)):
        p = C.c_void_p()
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
        assert rt.cudaMemcpy(p, C.c_void_p(a.ctypes.data), C.c_size_t(a.nbytes), 1) == 0
        dev.append(p)
    rc = lib.apspie_bfs(ctx, 0, C.c_int64(h.nnz), h.m, dev[0], dev[1], dev[0], dev[1], dev[2], 0)
    assert rc == 0, (turn, rc, lib.apspie_last_error(ctx))
    assert lib.apspie_ctx_sync(ctx) == 0
    out = np.empty(h.m, np.int32)
    assert rt.cudaMemcpy(C.c_void_p(out.ctypes.data), dev[2], C.c_size_t(out.nbytes), 2) == 0
    r, c = np.divmod(np.arange(h.m), 300)
    np.testing.assert_array_equal(out, r + c)
    lib.apspie_ctx_destroy(ctx)
    assert rt.cudaDeviceReset() == 0
print("both turns")
"""


def test_sparse_bfs_after_the_device_was_reset():
    """A process that resets its device (its own CUDA context) and goes on
    with a new context, in a process of its own."""
    import subprocess
    import sys
    from pathlib import Path
    res = subprocess.run([sys.executable, "-c", _RESET_CHILD], capture_output=True, text=True,
                         timeout=300, cwd=Path(__file__).resolve().parents[1])
    assert res.returncode == 0 and "both turns" in res.stdout, res.stdout + res.stderr[-2000:]
