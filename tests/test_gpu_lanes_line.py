"""The per-agent kernel's automatic layout on both sides of 160,000 agents (four
lanes per agent, then one thread): the bits of the other layout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def crowd():
    from ecmgenerator_gb300 import agents as ag

    cfg = ag.scaled("c3", agents=160001)
    scene = ag.build_scene(cfg, seed=2)
    st = ag.spawn_agents(dict(cfg, overlap=True), scene, seed=2)
    return scene, st, [np.stack([p, g]) for p, g in zip(st.pos, st.goal)]


@pytest.mark.parametrize("n,other", [(160000, ("thread", 1)), (160001, ("warp", 8))])
def test_layouts_agree_at_the_line(lib, crowd, n, other):
    from ecmgenerator_gb300.simulator import Simulator, set_lp_mode

    scene, st, paths = crowd
    out = []
    for layout in (None, other):
        sim = Simulator(scene, n, 1.0 / 60.0, max_neighbors=16, tau_agent=2.0, tau_obst=2.0)
        if layout:
            set_lp_mode(sim, *layout)
        sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
        s = sim.update(ticks=3)
        out.append((sim.get_position_data(), sim.get_velocity_data(), sim.get_active_flags(), s.lp3d))
        sim.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
