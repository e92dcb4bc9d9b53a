"""GPU: the cluster build of the register-resident solver (plans of at most
16 CTAs of 512 rows) at the edges of its range.  It adds the same partials in
the same order as the other two synchronisation schemes, so its iterates must
equal those of the polled mode bit for bit: grids of one partial slice, of
exactly one CTA's rows and one more, of 8 and 9 CTAs (the portable cluster
size and one above) and of 16; 17 CTAs take the grid barrier again.  A CTA
that holds several instances stops each at its own count."""
import numpy as np
import pytest

from chysx import capi, scenes
from chysx.runner import GpuCloth

pytestmark = pytest.mark.gpu


def _run(sc, mode, warm="zero", offs=None, steps=2):
    g = GpuCloth(sc, max_iter=20000, rel_tol=1e-6, warm_start="zero", instances=offs)
    g.sim.set_sync_mode(mode)
    g.sim.set_solver(20000, 1e-6, warm)
    its = g.run(steps)
    return g, its


@pytest.mark.parametrize("warm", ["zero", "previous_scaled"])
@pytest.mark.parametrize("side,ctas", [(4, 1), (22, 1), (23, 2), (64, 8), (65, 9), (90, 16), (91, 17)])
def test_cluster_iterates_equal_polled_mode(side, ctas, warm):
    sc = scenes.config_large(side=side, steps=2)
    (a, ia), (b, ib) = (_run(sc, mode, warm) for mode in (0, 1))
    assert a.sim.solver_info() == ("resident", ctas, 512)
    assert a.stats()[2] == capi.SOLVE_CONVERGED
    assert np.array_equal(ia, ib)
    assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.velocities(), b.velocities())


def test_instances_in_one_cta_stop_alone():
    sc, offs = scenes.concat(scenes.batch_instances(count=3, seed=21, lo=6, hi=11, steps=2, max_iter=20000))
    (a, _), (b, _) = (_run(sc, mode, offs=offs) for mode in (0, 1))
    assert a.sim.solver_info() == ("resident", 1, 512)
    ia, ib = a.sim.instance_stats(), b.sim.instance_stats()
    assert len(set(ia[0].tolist())) > 1 and (ia[2] == capi.SOLVE_CONVERGED).all()
    assert all(np.array_equal(x, y) for x, y in zip(ia, ib))
    assert np.array_equal(a.positions(), b.positions())


def test_iteration_limits_without_a_rebuild():
    # the graph's cluster node takes new solver parameters in place
    g = GpuCloth(scenes.config_small(), max_iter=50, rel_tol=0.0, warm_start="zero")
    for n in (50, 7, 0):
        g.sim.set_solver(n, 0.0, "zero")
        g.step()
        assert g.stats()[0] == n and g.stats()[2] == capi.SOLVE_CONVERGED
