"""The kd-tree neighbour mode where its other tests do not go: crowds hardly
larger than the list (the carried cache moves between slots from tick to tick)
and the per-agent kernel with one thread per agent, whose entries outside the
tick's grid no automatic layout reaches.  Against the oracle's kd-tree tick,
bit for bit, until stale entries make a position NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORCA = dict(tau_agent=2.0, tau_obst=2.0, neighbor_dist=5.0)


def _run(port, scene, st, paths, ticks, k, layout=None):
    from ecmgenerator_gb300.simulator import Simulator, set_lp_mode, set_neighbor_mode

    st = st.copy()
    n = st.num_agents
    sim = Simulator(scene, st.n_slots, 1.0 / 60.0, max_neighbors=k, **ORCA)
    set_neighbor_mode(sim, "kdtree")
    if layout:
        set_lp_mode(sim, layout, 1)
    sim.set_record(True)
    sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
    O, E = port.obstacles(scene), port.ecm(scene.ecm)
    P = port.params(k=k, libm=0, knn_mode=1, **ORCA)
    kd = port.kdtree(k)
    done = outside = 0
    for t in range(ticks):
        started = st.active.copy()
        sim.update()
        res = port.tick(O, E, st, P, kd=kd)
        live = st.active == 1
        rec = sim.get_record()
        assert np.array_equal(rec["nbr_count"][live], res["nbr_count"][live]), t
        assert np.array_equal(rec["nbr_ids"][live], res["nbr_ids"][live]), t
        for got, want in ((rec["v_orca"][live], res["v_orca"][live]), (sim.get_active_flags(), st.active),
                          (sim.get_position_data(), st.pos), (sim.get_velocity_data(), st.vel)):
            assert np.array_equal(got, want, equal_nan=True), t
        for a in np.nonzero(live)[0]:
            outside += int(np.sum(started[res["nbr_ids"][a][: res["nbr_count"][a]]] == 0))
        done = t + 1
        if np.isnan(st.pos[live]).any():
            break
        for s in res["replan"]:
            st.replace_path(int(s), sim.get_path(int(s)))
    port.lib.og_kdtree_destroy(kd)
    sim.close()
    return done, outside


def _crowd(n, slots, leave_first):
    from ecmgenerator_gb300 import agents as ag
    from ecmgenerator_gb300.simulator import Planner

    cfg = ag.scaled("c1", agents=n)
    scene = ag.build_scene(cfg, seed=3)
    st = ag.spawn_agents(cfg, scene, seed=3, n_slots=slots)
    if leave_first:
        st.goal[0] = st.pos[0]  # removed in the first tick
    paths = Planner(scene).find_paths(st.pos[:n], st.goal[:n], st.clear[:n])
    paths = [p if p is not None else np.stack([st.pos[i], st.goal[i]]) for i, p in enumerate(paths)]
    st.set_paths(paths)
    return scene, st, paths


@pytest.mark.parametrize("n,k", [(34, 32), (33, 31), (18, 16), (9, 7)])
def test_crowds_hardly_larger_than_the_list(port, n, k):
    done, _ = _run(port, *_crowd(n, n + 3, False), 60, k)
    assert done == 60


@pytest.mark.parametrize("layout", [None, "thread"])
@pytest.mark.parametrize("n,k", [(6, 8), (6, 16), (12, 32)])
def test_entries_outside_the_grid(port, n, k, layout):
    """fewer agents than list places: what the cache starts with (slot 0, an
    agent that leaves) is carried through every list"""
    done, outside = _run(port, *_crowd(n, n + 3, True), 40, k, layout)
    assert done == 40 and outside > 0


def test_tuner_reports_the_layout_it_timed(lib, c1_small):
    """in the kd-tree mode the tuner times the automatic layout, one trial per
    cell size (nothing else is read there), and what it reports can be set"""
    from ecmgenerator_gb300._lib import EcmgError
    from ecmgenerator_gb300.simulator import Simulator, autotune, set_lp_mode, set_neighbor_mode

    scene, st, paths = c1_small
    n = st.num_agents
    out = []
    for tuned in (False, True):
        sim = Simulator(scene, n, 1.0 / 60.0, max_neighbors=10, **ORCA)
        set_neighbor_mode(sim, "kdtree")
        sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
        if tuned:
            set_lp_mode(sim, "thread", 1)
            r = autotune(sim, ticks_per_trial=1)
            assert r["lp_mode"] == "auto" and r["trials"] == 7
            set_lp_mode(sim, r["lp_mode"])
            with pytest.raises(EcmgError):
                set_lp_mode(sim, "warp")
        sim.update(ticks=5)
        out.append((sim.get_position_data(), sim.get_velocity_data()))
        sim.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_back_to_the_automatic_layout(lib, c1_small):
    from ecmgenerator_gb300.simulator import Simulator, set_lp_mode

    scene, st, paths = c1_small
    n = st.num_agents
    out = []
    for switch in (False, True):
        sim = Simulator(scene, n, 1.0 / 60.0, max_neighbors=10, **ORCA)
        sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
        for mode in ("thread", "auto", "warp", "auto") if switch else ("auto",) * 4:
            set_lp_mode(sim, mode)
            sim.update(ticks=3)
        out.append((sim.get_position_data(), sim.get_velocity_data()))
        sim.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
