"""MIS parity: apspie_mis against the oracle's greedy MIS (same mt19937
priorities) bit-exact, plus the reference's own validity rule
(test/mis/main.cu:217-221: neighbour flag + membership == 1 everywhere)
computed on the GPU with apspie_neighbor_flags."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _run(ctx, h, prio, delta=1.0):
    import torch
    import apspie_b200 as ap
    g = h.to_device()
    p = torch.from_numpy(prio.view(np.int32)).cuda()
    out = ap.mis(ctx, g, p, delta=delta)
    flags = ap.neighbor_flags(ctx, g, out)
    return out.cpu().numpy(), flags.cpu().numpy(), ap.mis_rounds(ctx)


def _check(ctx, h, prio, delta=1.0):
    got, flags, rounds = _run(ctx, h, prio, delta)
    ref = oracle.mis(h.m, h.ptr, h.ind, prio)
    np.testing.assert_array_equal(got, ref)
    # the reference's check (uncompareResults): flag(v) + mis(v) == 1
    np.testing.assert_array_equal(flags + got, np.ones(h.m, np.int32))
    assert oracle.mis_check(h.m, h.ptr, h.ind, got) == 0
    return rounds


def test_mis_fixtures(ctx, golden, fixture_names):
    import apspie_b200 as ap
    for name in fixture_names:
        ptr, ind = golden[f"mtx/{name}/und_ptr"], golden[f"mtx/{name}/und_ind"]
        h = ap.HostGraph(len(ptr) - 1, ptr, ind, symmetric=True)
        for seed in (1, 5489):
            got, flags, _ = _run(ctx, h, ap.mt19937(seed, h.m))
            np.testing.assert_array_equal(got, oracle.mis(h.m, ptr, ind, ap.mt19937(seed, h.m)))
            # fixtures with self-loops: a looped vertex counts as its own neighbour in the
            # flag check only if it is in the set, so check independence + maximality directly
            assert oracle.mis_check(h.m, ptr, ind, got) == 0 or name == "test_spgemm"


def test_mis_matches_reference_kernel_goldens(ctx, golden):
    """apspie_mis against the membership that the reference's own round
    kernels and loop (src/spmspvMis.cuh:10-78, 232-318) produced with the
    same mt19937(5489) priorities, stored in the goldens, at both of their
    step sizes."""
    import apspie_b200 as ap
    names = sorted({k.split("/")[1] for k in golden if k.startswith("mis/")})
    for name in names:
        ptr, ind = golden[f"mis/{name}/ptr"], golden[f"mis/{name}/ind"]
        h = ap.HostGraph(len(ptr) - 1, ptr, ind, symmetric=True)
        for delta in (0.1, 1.0):
            got, _, _ = _run(ctx, h, ap.mt19937(5489, h.m), delta)
            np.testing.assert_array_equal(got, golden[f"mis/{name}/d{delta}"].astype(np.int32),
                                          err_msg=f"{name} delta {delta}")


@pytest.mark.parametrize("delta", [1.0, 0.5, 0.1])
def test_mis_er_and_grid_any_delta(ctx, delta):
    import apspie_b200 as ap
    h = ap.gen_er(1 << 15, 8, seed=3)
    _check(ctx, h, ap.mt19937(11, h.m), delta)
    grid = ap.gen_grid(128, 128)
    _check(ctx, grid, ap.mt19937(12, grid.m), delta)


def test_mis_ties_broken_by_id(ctx):
    import apspie_b200 as ap
    h = ap.gen_er(4096, 8, seed=4)
    prio = (np.arange(h.m) % 7).astype(np.uint32)
    _check(ctx, h, prio)
    _check(ctx, h, np.zeros(h.m, np.uint32))


def test_mis_rmat_with_hubs(ctx):
    import apspie_b200 as ap
    h = ap.gen_rmat(14, 16, seed=7)
    _check(ctx, h, ap.mt19937(3, h.m))


def test_neighbor_flags_vs_oracle(ctx):
    import torch
    import apspie_b200 as ap
    h = ap.gen_rmat(12, 16, seed=1, symmetric=False)
    g = h.to_device()
    rng = np.random.default_rng(0)
    fl = (rng.random(h.m) < 0.05).astype(np.int32)
    out = ap.neighbor_flags(ctx, g, torch.from_numpy(fl).cuda()).cpu().numpy()
    np.testing.assert_array_equal(out, oracle.neighbor_flags(h.m, h.ptr, h.ind, fl))


@pytest.mark.parametrize("which", ["er", "grid"])
def test_mis_full_size_configs(ctx, which):
    """ER n=2^20 mean degree 8 and the 1024x1024 grid, mt19937 priorities."""
    import apspie_b200 as ap
    h = ap.gen_er(1 << 20, 8, seed=1) if which == "er" else ap.gen_grid(1024, 1024)
    rounds = _check(ctx, h, ap.mt19937(5489, h.m))
    assert rounds < 100


@pytest.mark.parametrize("delta", [1.0, 0.1])
@pytest.mark.parametrize("leaves", [1, 3, 4, 7, 8, 9, 31, 32, 33, 127, 128, 129, 136, 137, 5000])
def test_mis_scan_lengths(ctx, leaves, delta):
    """Stars whose hub's scan ends in a lane's batches of four, at their end,
    or in the warp's batches of 128, with the hub's key the largest, the
    smallest and in between; leaves are paired up, one has a self-loop."""
    import apspie_b200 as ap
    hub = leaves // 2
    others = np.setdiff1d(np.arange(leaves + 1), [hub])
    r = np.concatenate([np.full(leaves, hub), others])
    c = np.concatenate([others, np.full(leaves, hub)])
    pair = others[: 2 * (leaves // 2)].reshape(-1, 2)
    r = np.concatenate([r, pair[:, 0], pair[:, 1], others[-1:]])
    c = np.concatenate([c, pair[:, 1], pair[:, 0], others[-1:]])
    order = np.lexsort((c, r))
    h = ap.from_edges(leaves + 1, r[order], c[order])
    prio = ap.mt19937(leaves, h.m)
    for hp in (0, 0xFFFFFFFF, 1 << 31, 0xFFFFFFFF - (1 << 24)):
        p = prio.copy()
        p[hub] = hp
        got, _, _ = _run(ctx, h, p, delta)
        np.testing.assert_array_equal(got, oracle.mis(h.m, h.ptr, h.ind, p))
    got, _, _ = _run(ctx, h, np.zeros(h.m, np.uint32), delta)
    np.testing.assert_array_equal(got, oracle.mis(h.m, h.ptr, h.ind, np.zeros(h.m, np.uint32)))


def test_mis_first_call_allocates_once():
    """A context's first call grows its workspace in one piece: it takes a
    warm call and about one allocation of that size (three or four pieces:
    three or four times as long)."""
    import ctypes as C
    import glob
    import time
    import nvidia.cuda_runtime
    import torch
    import apspie_b200 as ap
    rt = C.CDLL(glob.glob(list(nvidia.cuda_runtime.__path__)[0] + "/lib/libcudart.so*")[0])
    h = ap.gen_er(1 << 20, 8, seed=1)
    g = h.to_device()
    prio = torch.from_numpy(ap.mt19937(1, h.m).view(np.int32)).cuda()

    def clock(call):
        torch.cuda.synchronize()
        t = time.perf_counter()
        call()
        torch.cuda.synchronize()
        return time.perf_counter() - t

    first, warm, alloc = [], [], []
    for _ in range(8):
        with ap.Context(0) as own:
            first.append(clock(lambda: ap.mis(own, g, prio)))
            warm.append(clock(lambda: ap.mis(own, g, prio)))
            size = own.workspace_bytes
        p = C.c_void_p()
        alloc.append(clock(lambda: rt.cudaMalloc(C.byref(p), C.c_size_t(size))))
        rt.cudaFree(p)
    assert min(first) < min(warm) + 2.5 * min(alloc), (first, warm, alloc)
