"""Crowds on both sides of the sizes at which the tick takes another kernel
(one-block binning to 8,192 slots, several lanes per agent in the attraction
kernel to 16,000 agents and in the per-agent kernel to 8,000, kd-tree segments
built by one block to 4,096 agents), against the C oracle: whole states, equal
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORCA = dict(tau_agent=2.0, tau_obst=2.0, neighbor_dist=5.0)


@pytest.fixture(scope="module")
def crowd():
    from ecmgenerator_gb300 import agents as ag
    from ecmgenerator_gb300.simulator import Planner

    cfg = ag.scaled("c1", agents=16001, overlap=True)
    scene = ag.build_scene(cfg, seed=5)
    st = ag.spawn_agents(cfg, scene, seed=5)
    paths = Planner(scene).find_paths(st.pos, st.goal, st.clear)
    return scene, st, [p if p is not None else np.stack([st.pos[i], st.goal[i]]) for i, p in enumerate(paths)]


@pytest.mark.parametrize("mode", ["exact", "kdtree"])
@pytest.mark.parametrize("n,slots", [(4096, 4096), (4097, 8191), (8000, 8192), (8001, 8193), (16000, 16000),
                                     (16001, 16001)])
def test_tick_bitexact_at_size_rules(port, crowd, mode, n, slots):
    from ecmgenerator_gb300.agents import AgentState
    from ecmgenerator_gb300.simulator import Simulator, set_neighbor_mode

    scene, full, paths = crowd
    st = AgentState.empty(slots)
    for f in ("pos", "clear", "pref_speed", "active", "goal"):
        getattr(st, f)[:n] = getattr(full, f)[:n]
    st.num_agents, st.last_idx = n, n - 1
    st.set_paths(paths[:n])
    sim = Simulator(scene, slots, 1.0 / 60.0, max_neighbors=8, **ORCA)
    set_neighbor_mode(sim, mode)
    sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
    O, E = port.obstacles(scene), port.ecm(scene.ecm)
    P = port.params(k=8, libm=0, knn_mode=int(mode == "kdtree"), **ORCA)
    kd = port.kdtree(8) if mode == "kdtree" else None
    for t in range(3):
        stats = sim.update()
        res = port.tick(O, E, st, P, kd=kd)
        assert stats.destroyed == len(res["destroyed"]) and stats.replans == len(res["replan"])
        for got, want in ((sim.get_active_flags(), st.active), (sim.get_position_data(), st.pos),
                          (sim.get_velocity_data(), st.vel), (sim.get_attraction_point_data(), st.attr)):
            assert np.array_equal(got, want, equal_nan=True), t
        if np.isnan(st.pos[st.active == 1]).any():  # stale kd-tree entries: no further tick is defined
            break
        for s in res["replan"]:
            st.replace_path(int(s), sim.get_path(int(s)))
    if kd:
        port.lib.og_kdtree_destroy(kd)
    sim.close()
