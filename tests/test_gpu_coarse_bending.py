"""GPU: the coarse level of systems with bending, whose off-diagonal blocks are
general 3x3 (nine planes instead of six)."""
import numpy as np
import pytest

from chysx import capi, scenes
from chysx.runner import GpuCloth

pytestmark = pytest.mark.gpu


def _gpu(sc, coarse, offs=None):
    g = GpuCloth(sc, max_iter=20000, rel_tol=1e-6, warm_start="zero", instances=offs)
    g.sim.set_row_order(1)
    if coarse:
        g.sim.set_preconditioner("chebyshev_coarse", 7, 30.0)
    return g


def _compare(sc, offs=None):
    """Three steps, each from the two-level run's state: same solutions, fewer iterations (measured 0.71 of the plain
    solves' for 128 x 128, 0.57 for the batch; a level whose inversion fails leaves them equal)."""
    g, p = _gpu(sc, True, offs), _gpu(sc, False, offs)
    its = np.zeros(2)
    for _ in range(3):
        p.pos.copy_(g.pos)
        p.vel.copy_(g.vel)
        g.step()
        p.step()
        assert g.sim.preconditioner()[3] == 3 and p.sim.preconditioner()[3] == 0
        assert g.sim.solver_info()[0] == "streamed"
        assert g.stats()[2] == p.stats()[2] == capi.SOLVE_CONVERGED
        # both stop at 1e-6 of the load: the bound of the other solver tests
        assert np.abs(g.positions() - p.positions()).max() < 1e-5
        its += g.stats()[0], p.stats()[0]
    assert its[0] < 0.8 * its[1]
    return g


def test_coarse_matrix_with_bending():
    # 16,384 rows on 5,120-row blocks.  Between two blocks the translations' entry is the plain sum of A_ij over the
    # pairs across their border (a few hundred, in FP32: 2^-24 of the largest each)
    side = 128
    sc = scenes.config_large(side=side)
    sc["k_bend"] = 5.0e-3
    g = _compare(sc)
    info, ac, _ = g.sim.debug_coarse()
    assert (info["on"], info["fields"], info["blocks"]) == (1, 4, 4)
    block = np.searchsorted(g.sim.debug_coarse_rows(), g.sim.row_of_particles(side * side), side="right") - 1
    _, rp, col, vals, _, _ = g.dump()
    assert np.abs(vals - np.transpose(vals, (0, 2, 1))).max() > 0
    b, c = block[np.repeat(np.arange(side * side), np.diff(rp))], block[col]
    want = np.zeros((4, 4, 3, 3))
    np.add.at(want, (b, c), vals.astype(np.float64))
    got = ac.reshape(4, 4, 3, 4, 4, 3)[:, 0, :, :, 0, :].transpose(0, 2, 1, 3)
    off = ~np.eye(4, dtype=bool)
    assert np.abs(want[off]).max() > 1e4
    np.testing.assert_allclose(got[off], want[off], atol=1e-5 * np.abs(want[off]).max())


def test_coarse_level_of_a_batch_with_bending():
    sc, offs = scenes.concat(scenes.batch_instances(count=6, seed=21, lo=40, hi=64, steps=1, max_iter=20000))
    sc["k_bend"] = 5.0e-3
    _compare(sc, offs)
