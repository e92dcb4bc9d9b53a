"""GPU: the tiled solver kernel (matrix streamed, solver vectors on the SM) at
the edges of its range, against the streamed kernel on the same systems.

Both run the same PCG in FP32 with FP64 dots and differ in summation order
only.  Over 10 iterations from a zero guess each of the ~10 FP32 operations
per vector entry and iteration adds at most 2^-24 of |dx| < 0.02 m: 10 * 10 *
6e-8 * 0.02 = 1.2e-7 m, and the positions round to 1.2e-7 m (values up to 2):
bound 5e-7 m.  Converged solves are compared at 1e-5 m, the bound of the other
solver tests."""
import numpy as np
import pytest

from chysx import capi, scenes
from chysx.runner import GpuCloth

pytestmark = pytest.mark.gpu


def _run(sc, path, warm="zero", its=10, tol=0.0, offs=None, order=0, coarse=False, steps=1):
    g = GpuCloth(sc, max_iter=its, rel_tol=tol, warm_start="zero", instances=offs)
    g.sim.set_tuning(path)
    g.sim.set_row_order(order)
    if coarse:
        g.sim.set_preconditioner("chebyshev_coarse", 7, 30.0)
    g.sim.set_solver(its, tol, warm)
    for _ in range(steps):
        g.step()
    return g


def _second_step(sc, warm, **kw):
    """Two simulators (default kernel, streamed) after a second step that both
    take from the first one's state, each from its own previous dx."""
    a, b = (_run(sc, p, warm, **kw) for p in (0, 2))
    b.pos.copy_(a.pos)
    b.vel.copy_(a.vel)
    for g in (a, b):
        g.step()
    return a, b


def _rect(w, h, seed=0):
    """A jittered w x h grid in the default material, one edge pinned."""
    pos, tris = scenes.grid_mesh(w, h)
    rng = np.random.default_rng(seed)
    pos = pos + rng.uniform(-0.01, 0.01, pos.shape) / max(w, h)
    pos[:, 1] += 0.002 * np.sin(7.0 * pos[:, 0]) + 0.002 * np.cos(9.0 * pos[:, 2])
    return scenes._finish(f"rect{w}x{h}", pos, tris, 1.0e3, 1.0e4, np.arange(w), 1, 10, 0.0, det_eps=1.0e-12)


# one slice above the register-resident kernel's 75,776 rows (276 x 276 = 76,176, whole slices and not: 277 x 275 =
# 76,175 ends in a slice of 15 rows; the matrix fits shared memory, 512 threads), and 224 slices on every SM (1,060,864 rows) and one grid row more
@pytest.mark.parametrize("w,h,block", [(276, 276, 512), (277, 275, 512), (1036, 1024, 1024), (1037, 1024, 256)])
def test_size_limits(w, h, block):
    sc = _rect(w, h)
    a, b = _run(sc, 0), _run(sc, 2)
    assert a.sim.solver_info()[::2] == ("tiled" if block > 256 else "streamed", block)
    assert b.sim.solver_info()[::2] == ("streamed", 256)
    assert a.stats()[0] == b.stats()[0] == 10
    assert np.abs(a.positions() - b.positions()).max() < 5e-7


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("warm", ["previous", "previous_scaled"])
@pytest.mark.parametrize("w,h,block", [(300, 280, 512), (401, 380, 1024)])
def test_warm_starts(w, h, block, warm, order):
    sc = _rect(w, h)
    a, b = _second_step(sc, warm, order=order, its=20000, tol=1e-6)
    assert a.sim.solver_info()[::2] == ("tiled", block)
    assert a.stats()[2] == capi.SOLVE_CONVERGED and a.stats()[1] <= 1e-6
    assert np.abs(a.positions() - b.positions()).max() < 1e-5


@pytest.mark.parametrize("w,h", [(320, 320), (321, 317)])
def test_particles_without_elements(w, h):
    # inertia and pins alone, more rows than the register-resident kernel takes: a matrix without entries
    sc = dict(_rect(w, h), k_spring=None, k_stretch=None)
    a, b = _run(sc, 0, its=20, tol=1e-6, steps=2), _run(sc, 2, its=20, tol=1e-6, steps=2)
    assert a.sim.num_off_diag_blocks() == 0 and a.sim.solver_info()[::2] == ("tiled", 512)
    assert a.stats()[2] == capi.SOLVE_CONVERGED
    assert np.abs(a.positions() - b.positions()).max() < 5e-7
    # two steps of free fall from rest: 3 g dt^2 down
    free = np.arange(w, w * h)
    assert np.abs(a.positions()[free, 1] - sc["pos"][free, 1] + 3 * 9.81 / 3600.0).max() < 1e-6


# Long solves with several slices per warp: the stage then holds another slice's blocks at every use (three and four
# slices a warp at 801 x 643, seven at 1024 x 1024).  A block of another slice, or a halo value that is not its owner's,
# costs conjugacy and shows in the count; over thousands of iterations the two kernels' roundings move it by less than
# 0.3%.  A solution at 1e-6 of the load lies within 1e-5 m (as above) once the cloth moves: the first step, from rest,
# is left out of the comparison of positions.
@pytest.mark.parametrize("sc", [_rect(801, 643), scenes.config_huge()], ids=["801x643", "1024x1024"])
def test_long_plain_solves(sc):
    a, b = (_run(sc, p, its=60000, tol=1e-6) for p in (0, 2))
    for k in range(3):
        if k > 0:
            b.pos.copy_(a.pos)
            b.vel.copy_(a.vel)
            for g in (a, b):
                g.step()
        ia, ib = a.stats(), b.stats()
        assert ia[2] == ib[2] == capi.SOLVE_CONVERGED and max(ia[1], ib[1]) <= 1e-6
        assert abs(ia[0] - ib[0]) <= 0.01 * ib[0]
        if k > 0:
            assert np.abs(a.positions() - b.positions()).max() < 1e-5


def test_wide_rows_on_one_cta():
    # a 60-triangle fan: too wide for the register-resident kernel, two slices
    ang = np.linspace(0.0, 2.0 * np.pi, 60, endpoint=False)
    pos = np.concatenate([[[0.0, 1.0, 0.0]], np.stack([0.5 * np.cos(ang), np.ones(60), 0.5 * np.sin(ang)], 1)])
    tris = np.array([[0, 1 + k, 1 + (k + 1) % 60] for k in range(60)], np.int32)
    sc = scenes._finish("fan", pos, tris, 1.0e3, 1.0e4, [1, 31], 1, 10, 0.0)
    a, b = _run(sc, 0), _run(sc, 2)
    assert a.sim.solver_info()[::2] == ("tiled", 512)
    assert np.abs(a.positions() - b.positions()).max() < 5e-7


def test_scattered_particles_keep_the_streamed_kernel():
    # neighbours all over the row range: the halo fits shared memory at 400 x 400 and not at 700 x 700
    for side, block in ((400, 1024), (700, 256)):
        sc = _rect(side, side)
        perm = np.random.default_rng(1).permutation(sc["pos"].shape[0])
        inv = np.argsort(perm)
        pos, tris = sc["pos"][perm], inv[sc["tris"]].astype(np.int32)
        sh = scenes._finish("shuffled", pos.astype(np.float64), tris, 1.0e3, 1.0e4, inv[:side], 1, 10, 0.0,
                            det_eps=1.0e-12)
        a, b = _run(sh, 0), _run(sh, 2)
        assert a.sim.solver_info()[::2] == ("tiled" if block > 256 else "streamed", block)
        assert np.abs(a.positions() - b.positions()).max() < 5e-7


@pytest.mark.parametrize("coarse", [False, True])
@pytest.mark.parametrize("lo,hi,count", [(100, 128, 9), (6, 40, 300)])
def test_batches_stop_alone(lo, hi, count, coarse):
    # few large instances, and many small ones (a dozen per CTA)
    sc, offs = scenes.concat(scenes.batch_instances(count=count, seed=3, lo=lo, hi=hi, steps=1, max_iter=20000))
    a, b = (_run(sc, p, its=20000, tol=1e-6, offs=offs, order=1, coarse=coarse, steps=2) for p in (0, 2))
    assert a.sim.solver_info()[::2] == ("tiled", 1024) and a.sim.preconditioner()[3] == (3 if coarse else 0)
    ia, ib = a.sim.instance_stats(), b.sim.instance_stats()
    assert (ia[2] == capi.SOLVE_CONVERGED).all() and (ia[1] <= 1e-6).all()
    assert len(set(ia[0].tolist())) > 1
    if not coarse:  # the same preconditioner: the same counts overall (single instances move with rounding)
        assert abs(ia[0].sum() - ib[0].sum()) <= 0.02 * ib[0].sum()
    assert np.abs(a.positions() - b.positions()).max() < 1e-5


def test_two_level_converges_to_the_streamed_solution():
    sc = scenes.config_large(side=300, steps=2, max_iter=20000)
    a, b = (_run(sc, p, its=20000, tol=1e-6, order=1, coarse=True) for p in (0, 2))
    assert a.sim.solver_info()[::2] == ("tiled", 1024) and a.sim.preconditioner()[3] == 3
    assert a.stats()[2] == capi.SOLVE_CONVERGED and a.stats()[1] <= 1e-6
    assert a.stats()[0] < 1.5 * b.stats()[0]
    assert np.abs(a.positions() - b.positions()).max() < 1e-5


# general 3x3 blocks (bending) and the matrix in shared memory: one cluster (3 and 16 CTAs), every SM, and above
# what fits the SMs (301 x 290) streamed; the last slices are ragged
@pytest.mark.parametrize("w,h", [(9, 9), (61, 47), (91, 90), (301, 290)])
def test_bending_systems(w, h):
    sc = _rect(w, h)
    sc["k_bend"], sc["k_shear"] = 5.0e-3, 5.0e3
    a, b = _run(sc, 0), _run(sc, 2)
    assert a.sim.solver_info()[0] == "tiled" and b.sim.solver_info()[0] == "streamed"
    assert a.sim.solver_info()[2] == (1024 if w > 200 else 512)
    assert (a.sim.solver_info()[1] <= 16) == (w * h < 4000)
    assert np.abs(a.positions() - b.positions()).max() < 5e-7


@pytest.mark.parametrize("warm", ["previous", "previous_scaled"])
@pytest.mark.parametrize("w,h", [(30, 31), (91, 90)])
def test_bending_warm_starts_and_stops(w, h, warm):
    sc = _rect(w, h)
    sc["k_bend"] = 5.0e-3
    a, b = _second_step(sc, warm)
    assert np.abs(a.positions() - b.positions()).max() < 2e-6  # guesses, dt * velocities and the step's own 5e-7 m each
    for n in (3, 0):  # other limits on the same graph
        a.sim.set_solver(n, 0.0, warm)
        a.step()
        assert a.stats()[0] == n and a.stats()[2] == capi.SOLVE_CONVERGED
    a.sim.set_solver(20000, 1e-6, "zero")
    a.step()
    assert a.stats()[2] == capi.SOLVE_CONVERGED and a.stats()[1] <= 1e-6
