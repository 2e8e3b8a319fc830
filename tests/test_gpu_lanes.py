"""The per-agent kernel with 1, 4, 8, 16 and 32 lanes per agent: the layouts
take the same steps on the same numbers, so whole states are equal bit for
bit (lists of up to 8, 16 and 32 neighbours, agents that do not fill a warp's
groups, and the layout chosen by the agent count)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ticks(scene, st, paths, n, k, layout, ticks, tau=2.0):
    from ecmgenerator_gb300.simulator import Simulator, set_lp_mode

    sim = Simulator(scene, n, 1.0 / 60.0, max_neighbors=k, tau_agent=tau, tau_obst=2.0)
    if layout is not None:
        set_lp_mode(sim, *layout)
    sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
    s = sim.update(ticks=ticks)
    out = sim.get_position_data(), sim.get_velocity_data(), sim.get_active_flags(), s.lp3d
    sim.close()
    return out


@pytest.mark.parametrize("k,n", [(5, 33), (8, 300), (10, 299), (16, 1), (16, 900), (20, 257), (32, 600)])
def test_layouts_agree(lib, k, n):
    from ecmgenerator_gb300 import agents as ag
    from ecmgenerator_gb300.simulator import Planner

    # a crowd dense enough for the 3D linear program at the larger counts
    cfg = ag.scaled("c1", agents=n, w=30.0, h=30.0, boxes=6, side=(1.0, 4.0), overlap=True)
    scene = ag.build_scene(cfg, seed=9)
    st = ag.spawn_agents(cfg, scene, seed=9)
    paths = Planner(scene).find_paths(st.pos, st.goal, st.clear)
    paths = [p if p is not None else np.stack([st.pos[i], st.goal[i]]) for i, p in enumerate(paths)]
    want = _ticks(scene, st, paths, n, k, ("thread", 1), 6)
    if n >= 600:
        assert want[3] > n  # the 3D program ran
    for layout in (None, ("warp", 1), ("warp", 2), ("warp", 4), ("warp", 8), ("fused", 1)):
        got = _ticks(scene, st, paths, n, k, layout, 6)
        for a, b in zip(want, got):
            assert np.array_equal(a, b, equal_nan=True) if isinstance(a, np.ndarray) else a == b
