"""The stand-alone neighbour query against brute force in the same 32-bit
arithmetic: crowds that leave the grid, crowd single cells, tie, or are too
sparse for the first search disc, at list sizes around the kernels' capacities
(8, 16, 32) and warp-sized remainders.  Ids and counts are whole numbers:
equal, no tolerance."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _query(L, pos, act, k, r, box, cell, shift=0):
    import torch

    n = len(pos)
    b = tuple(map(ctypes.c_float, (*box, cell)))
    p = torch.from_numpy(pos).cuda()
    a = torch.from_numpy(act).cuda()
    scratch = torch.empty(L.ecmg_knn_scratch_bytes(n, *b), dtype=torch.uint8, device="cuda")
    ids = torch.full((n * k + shift,), -7, dtype=torch.int32, device="cuda")[shift:]
    cnt = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    assert L.ecmg_knn(p.data_ptr(), a.data_ptr(), n, k, r, *b, ids.data_ptr(), cnt.data_ptr(), scratch.data_ptr(),
                      scratch.numel(), None) == 0
    torch.cuda.synchronize()
    return ids.cpu().numpy().reshape(n, k), cnt.cpu().numpy()


def _brute(pos, act, k, r):
    idx = np.nonzero(act)[0]
    ids = np.full((len(pos), k), -1, np.int32)
    cnt = np.zeros(len(pos), np.int32)
    r2 = np.float32(r) * np.float32(r)
    with np.errstate(invalid="ignore", over="ignore"):
        for i in idx:
            dx, dy = pos[idx, 0] - pos[i, 0], pos[idx, 1] - pos[i, 1]
            d2 = dx * dx + dy * dy
            near = np.nonzero((d2 > np.float32(1e-4)) & (d2 < r2))[0]
            near = near[np.argsort(d2[near], kind="stable")][:k]  # slots ascend among equal distances
            ids[i, : near.size] = idx[near]
            cnt[i] = near.size
    return ids, cnt


def _crowd(name, rng):
    f = np.float32
    if name == "uniform":
        return rng.uniform(0, 13, (1025, 2)).astype(f), 5.0, (0, 0, 13, 13), 0.6
    if name == "lattice":  # equal distances: ties inside and across the k-th
        g = np.stack(np.meshgrid(np.arange(33) * 0.5, np.arange(31) * 0.5), -1).reshape(-1, 2)
        return g.astype(f), 3.0, (0, 0, 17, 16), 0.6
    if name == "one cell":  # hundreds of agents in one cell
        return rng.normal(50, 0.2, (900, 2)).astype(f), 2.0, (0, 0, 100, 100), 4.0
    if name == "outside":  # most of the crowd beyond the grid, on every side
        return rng.uniform(-60, 160, (1000, 2)).astype(f), 9.0, (40, 40, 60, 60), 2.0
    if name == "far away":  # everybody in one border cell
        return (rng.uniform(0, 30, (500, 2)) + [1e4, -1e4]).astype(f), 7.0, (0, 0, 50, 50), 1.0
    if name == "sparse":  # fewer than k within the radius for many
        return rng.uniform(0, 400, (700, 2)).astype(f), 40.0, (0, 0, 400, 400), 3.0
    if name == "coincident":
        return np.repeat(rng.uniform(0, 9, (90, 2)), 9, 0).astype(f), 5.0, (0, 0, 9, 9), 1.0
    if name == "two densities":  # discs that start too small and too large
        p = rng.uniform(0, 60, (1200, 2))
        p[:600] *= 0.05
        return p.astype(f), 30.0, (0, 0, 60, 60), 0.9
    if name == "not finite":
        p = rng.uniform(0, 20, (800, 2)).astype(f)
        p[::7] = np.nan
        p[::11, 0] = np.inf
        p[::13, 1] = -np.inf
        return p, 5.0, (0, 0, 20, 20), 1.0
    if name == "offset":  # coordinates whose ulp is 3 cm
        return (rng.uniform(0, 30, (900, 2)) + 5e5).astype(f), 5.0, (5e5, 5e5, 5e5 + 30, 5e5 + 30), 0.7
    p = np.stack([rng.uniform(0, 3e5, 900), rng.uniform(0, 2, 900)], 1)  # "strip"
    return p.astype(f), 3000.0, (0, 0, 3e5, 2), 0.5


@pytest.mark.parametrize("name", ["uniform", "lattice", "one cell", "outside", "far away", "sparse", "coincident",
                                  "two densities", "not finite", "offset", "strip"])
@pytest.mark.parametrize("k", [1, 5, 8, 9, 16, 17, 32])
def test_knn_equals_brute_force(lib, name, k):
    rng = np.random.default_rng(7)
    pos, r, box, cell = _crowd(name, rng)
    act = (rng.random(len(pos)) < 0.95).astype(np.uint8)
    ids, cnt = _query(lib, pos, act, k, r, box, cell)
    want_ids, want_cnt = _brute(pos, act, k, r)
    live = act == 1
    assert np.array_equal(cnt, want_cnt)
    assert np.array_equal(ids[live], want_ids[live])


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 129])
def test_knn_few_agents_and_unaligned_output(lib, n):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 5, (n, 2)).astype(np.float32)
    act = np.ones(n, np.uint8)
    for k in (8, 16):
        for shift in (0, 1):
            ids, cnt = _query(lib, pos, act, k, 5.0, (0, 0, 5, 5), 0.5, shift)
            want_ids, want_cnt = _brute(pos, act, k, 5.0)
            assert np.array_equal(ids, want_ids) and np.array_equal(cnt, want_cnt)


def test_tick_with_agents_outside_the_scene(lib):
    """agents beyond the grid on all sides (pushed out by a dense crowd): the
    tick's lists equal the stand-alone query's on the same positions"""
    from ecmgenerator_gb300 import agents as ag
    from ecmgenerator_gb300.simulator import Simulator

    cfg = ag.scaled("c1", agents=600)
    scene = ag.build_scene(cfg, seed=5)
    rng = np.random.default_rng(3)
    pos = rng.uniform(-45, 145, (600, 2)).astype(np.float32)
    goal = rng.uniform(10, 90, (600, 2)).astype(np.float32)
    sim = Simulator(scene, 600, 1.0 / 60.0, max_neighbors=10, tau_agent=2.0, tau_obst=2.0)
    sim.set_record(True)
    sim.add_agents(pos, np.full(600, 0.3, np.float32), np.full(600, 1.3, np.float32),
                   [np.stack([p, g]) for p, g in zip(pos, goal)])
    sim.update()
    rec = sim.get_record()
    want, cnt = _brute(pos, np.ones(600, np.uint8), 10, 5.0)
    live = rec["nbr_count"] >= 0
    assert live.sum() > 500
    assert np.array_equal(rec["nbr_count"][live], cnt[live])
    assert np.array_equal(rec["nbr_ids"][live], want[live])
    sim.close()
