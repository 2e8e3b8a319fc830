"""Neighbour searches whose grid does not fit their crowd: the lists (against
brute force in the same 32-bit arithmetic; ids and counts are whole numbers, no
tolerance) and the time beside that of a crowd that fits, with room to spare
for another clock or another box."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _query(L, pos, k, r, box, cell, repeats=1):
    """ids, counts and the least time (us)"""
    import torch

    n = len(pos)
    b = tuple(map(ctypes.c_float, (*box, cell)))
    p = torch.from_numpy(np.ascontiguousarray(pos, np.float32)).cuda()
    a = torch.ones(n, dtype=torch.uint8, device="cuda")
    scratch = torch.empty(L.ecmg_knn_scratch_bytes(n, *b), dtype=torch.uint8, device="cuda")
    ids = torch.full((n, k), -7, dtype=torch.int32, device="cuda")
    cnt = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    best = float("inf")
    for _ in range(repeats):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        assert L.ecmg_knn(p.data_ptr(), a.data_ptr(), n, k, r, *b, ids.data_ptr(), cnt.data_ptr(), scratch.data_ptr(),
                          scratch.numel(), torch.cuda.current_stream().cuda_stream) == 0
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, 1e3 * e[0].elapsed_time(e[1]))
    return ids.cpu().numpy(), cnt.cpu().numpy(), best


def _check(pos, k, r, ids, cnt, rows):
    """the lists of the agents `rows`"""
    pos = np.ascontiguousarray(pos, np.float32)
    r2 = np.float32(r) * np.float32(r)
    for i in rows:
        d = pos - pos[i]
        d2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]
        near = np.nonzero((d2 > np.float32(1e-4)) & (d2 < r2))[0]
        near = near[np.argsort(d2[near], kind="stable")][:k]  # slots ascend among equal distances
        assert cnt[i] == near.size and np.array_equal(ids[i, : near.size], near), i
        assert (ids[i, near.size:] == -1).all()


def test_few_agents_in_many_cells(lib):
    rng = np.random.default_rng(1)
    box = (0, 0, 5000, 5000)
    few, many = rng.uniform(0, 5000, (300, 2)), rng.uniform(0, 5000, (20000, 2))
    ids, cnt, _ = _query(lib, few, 8, 500.0, box, 1.0)
    _check(few, 8, 500.0, ids, cnt, range(300))
    assert _query(lib, few, 8, 5.0, box, 1.0, 5)[2] < 3.0 * _query(lib, many, 8, 5.0, box, 1.0, 5)[2]


def test_tick_of_few_agents_in_many_cells(lib, c1_small):
    """2 M cells (binning by several blocks) and the usual ones: the same bits"""
    from ecmgenerator_gb300.simulator import Simulator

    scene, st, paths = c1_small
    n, out = st.num_agents, []
    for cell in (0.0, 0.08):
        sim = Simulator(scene, n, 1.0 / 60.0, max_neighbors=10, tau_agent=2.0, tau_obst=2.0, grid_cell=cell)
        sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
        sim.update(ticks=5)
        out.append((sim.get_position_data(), sim.get_velocity_data()))
        sim.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("k", [5, 8, 14, 16, 27, 32])
def test_lattice(lib, k):
    """a crowd on a lattice: distances tie across the k-th place"""
    rng = np.random.default_rng(2)
    pos = 0.4 * np.stack(np.meshgrid(np.arange(317), np.arange(316)), -1).reshape(-1, 2)
    pos = pos[rng.permutation(len(pos))]
    box, cell = (0, 0, 127, 127), max(0.3, 0.5 * (k / 6.25) ** 0.5)
    ids, cnt, t = _query(lib, pos, k, 5.0, box, cell, 5)
    _check(pos, k, 5.0, ids, cnt, rng.integers(0, len(pos), 300))
    assert t < 3.0 * _query(lib, rng.uniform(0, 126.6, pos.shape), k, 5.0, box, cell, 5)[2]


def _crowded(name, rng, m):
    """crowds far denser than their cells, about m agents: positions, radius,
    box, cell"""
    box, cell = (0, 0, 100, 100), 4.0
    if name == "cluster":
        return rng.normal(50, 0.5, (m, 2)), 5.0, box, cell
    if name == "cluster and strays":
        return np.concatenate([rng.normal(50, 0.1, (m, 2)), rng.uniform(0, 100, (1500, 2))]), 30.0, box, cell
    if name == "lattice in a cell":  # ties across every k-th place
        side = int(m**0.5)
        g = np.stack(np.meshgrid(np.arange(side), np.arange(side)), -1).reshape(-1, 2)
        return 48.5 + 0.04 * g[rng.permutation(len(g))], 5.0, box, cell
    if name == "coincident":  # more agents at one distance than a list, a column or a warp holds
        return np.repeat(rng.uniform(48.1, 51.9, (m // 100, 2)), 100, 0), 5.0, box, cell
    if name == "few in reach":  # fewer than k within the radius
        return rng.uniform(48, 52, (m, 2)), 0.05, box, cell
    if name == "outside":  # one corner cell holds everybody
        return rng.uniform(0, 60, (m, 2)) + 500, 5.0, box, 1.0
    p = rng.uniform(48, 52, (m, 2))  # "not finite"
    p[::7] = np.nan
    p[::11, 0] = np.inf
    return p, 5.0, box, cell


@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("m", [900, 4000])  # on both sides of the sizes at which another variant is taken
@pytest.mark.parametrize("name", ["cluster", "cluster and strays", "lattice in a cell", "coincident", "few in reach",
                                  "outside", "not finite"])
def test_crowded_cells(lib, name, m, k):
    rng = np.random.default_rng(4)
    pos, r, box, cell = _crowded(name, rng, m)
    ids, cnt, _ = _query(lib, pos, k, r, box, cell)
    with np.errstate(invalid="ignore", over="ignore"):
        _check(pos, k, r, ids, cnt, rng.integers(0, len(pos), 300))


def test_crowded_cell_in_time(lib):
    """every agent has to look at all 4,000: beside a crowd in cells that fit"""
    rng = np.random.default_rng(4)
    pos, r, box, cell = _crowded("cluster", rng, 4000)
    fit = _query(lib, rng.uniform(0, 26, pos.shape), 16, 5.0, (0, 0, 26, 26), 0.8, 5)[2]
    assert _query(lib, pos, 16, r, box, cell, 5)[2] < 60.0 * fit


@pytest.mark.parametrize("n,slots,cell", [(300, 300, 40.0), (300, 8193, 40.0), (4000, 4000, 60.0), (4000, 8193, 60.0)])
def test_tick_with_crowded_cells(lib, c1_small, n, slots, cell):
    """cells with hundreds or thousands of agents in the 3 x 3 around one, and
    the usual ones: the same lists and the same bits"""
    from ecmgenerator_gb300.simulator import Simulator

    scene, st, paths = c1_small
    rng = np.random.default_rng(6)
    pos, goal = (st.pos[:n], None) if n <= 300 else (rng.uniform(5, 95, (n, 2)).astype(np.float32),
                                                     rng.uniform(5, 95, (n, 2)).astype(np.float32))
    ways = paths[:n] if n <= 300 else [np.stack([p, g]) for p, g in zip(pos, goal)]
    for k in (7, 16, 25):
        out = []
        for c in (0.0, cell):
            sim = Simulator(scene, slots, 1.0 / 60.0, max_neighbors=k, tau_agent=2.0, tau_obst=2.0, grid_cell=c,
                            neighbor_dist=15.0)
            sim.set_record(True)
            sim.add_agents(pos, np.full(n, 0.25, np.float32), np.full(n, 1.3, np.float32), ways)
            sim.update(ticks=3)
            rec = sim.get_record()
            out.append((sim.get_position_data(), sim.get_velocity_data(), rec["nbr_ids"][:n], rec["nbr_count"][:n]))
            sim.close()
        for a, b in zip(*out):
            assert np.array_equal(a, b, equal_nan=True)
