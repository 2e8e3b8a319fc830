"""ecmg_kernels_per_tick: with the graph the binning is chosen for all slots,
without it for those in use (one launch to 8,192, else three)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,graph,binning", [(8192, True, 1), (8193, True, 3), (8193, False, 1)])
def test_launches_of_a_tick(lib, c1_small, slots, graph, binning):
    from ecmgenerator_gb300.simulator import Simulator

    scene, st, paths = c1_small
    n = st.num_agents
    sim = Simulator(scene, slots, 1.0 / 60.0, max_neighbors=10, tau_agent=2.0, tau_obst=2.0, use_graph=graph)
    sim.add_agents(st.pos[:n], st.clear[:n], st.pref_speed[:n], paths[:n])
    sim.update()
    assert lib.ecmg_kernels_per_tick(sim.h) == binning + 3
    sim.close()
