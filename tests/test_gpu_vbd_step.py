"""GPU: the one-kernel VBD step at the edges of its plan, against the FP64
oracle with the same colouring.  Sizes with 16, 8 and 4 lanes per vertex, the
largest colours it takes and the first ones that a launch per colour takes;
a colour smaller than a warp's tile, empty energies, particles without
elements and a single colour.  One step's FP32 rounding: the 10 x 10 fixture
tests hold it to 2e-6 m, positions being of order one."""
import numpy as np
import pytest

import oracle.oracle as O
from chysx import capi, scenes, vbd_scenes
from test_gpu_vbd import GpuVbd

pytestmark = pytest.mark.gpu


def _hinges(w, h):
    """Interior edges (o0, o1, v2, v3) of chysx.scenes.grid_mesh: diagonals, then the edges along x and z."""
    def at(i, j):
        return (j * w + i).ravel()

    i, j = np.meshgrid(np.arange(w - 1), np.arange(h - 1), indexing="xy")
    e = [np.stack([at(i, j + 1), at(i + 1, j), at(i, j), at(i + 1, j + 1)], 1)]
    i, j = np.meshgrid(np.arange(w - 1), np.arange(1, h - 1), indexing="xy")
    e.append(np.stack([at(i + 1, j + 1), at(i, j - 1), at(i, j), at(i + 1, j)], 1))
    i, j = np.meshgrid(np.arange(1, w - 1), np.arange(h - 1), indexing="xy")
    e.append(np.stack([at(i - 1, j), at(i + 1, j + 1), at(i, j), at(i, j + 1)], 1))
    return np.concatenate(e).astype(np.int32)


def _problem(w, h, loose=0):
    pos, tris = scenes.grid_mesh(w, h)
    rng = np.random.default_rng(w * h)
    pos = pos + rng.uniform(-0.01, 0.01, pos.shape) / max(w, h)
    poses, area = vbd_scenes.rest_frames(pos, tris)
    edges = _hinges(w, h)
    inv_mass = vbd_scenes.lumped_inv_mass(pos, tris, 0.1)
    inv_mass[[w * (h - 1), w * h - 1]] = 0.0
    cur = pos * np.array([1.01, 1.0, 1.02]) + np.array([0.0, 0.01, 0.0]) * np.sin(8.0 * pos[:, :1])
    vel = 0.2 * np.stack([np.sin(5 * pos[:, 2]), np.cos(4 * pos[:, 0]), 0 * pos[:, 0]], 1)
    if loose:  # particles without elements
        cur = np.concatenate([cur, rng.uniform(-1, 1, (loose, 3))])
        vel = np.concatenate([vel, rng.uniform(-1, 1, (loose, 3))])
        inv_mass = np.concatenate([inv_mass, np.full(loose, 50.0)])
    ii = np.arange(w * h)
    colors = np.concatenate([(ii % w) % 2 + 2 * ((ii // w) % 2), np.zeros(loose, np.int64)])
    return dict(pos=cur.astype(np.float32), vel=vel.astype(np.float32), inv_mass=inv_mass.astype(np.float32),
                tri_indices=tris.astype(np.int32), tri_poses=poses.astype(np.float32),
                tri_areas=area.astype(np.float32),
                tri_materials=np.tile(np.array([2e3, 2e3, 1e-3], np.float32), (len(tris), 1)), edge_indices=edges,
                edge_rest_angle=np.zeros(len(edges), np.float32),
                edge_rest_length=np.linalg.norm(pos[edges[:, 3]] - pos[edges[:, 2]], axis=1).astype(np.float32),
                edge_bending_props=np.tile(np.array([5e-3, 1e-3], np.float32), (len(edges), 1)),
                gravity=np.array([0.0, -9.81, 0.0], np.float32), dt=1.0 / 60.0, colors=colors.astype(np.int32))


def _compare(vb, iterations):
    g = GpuVbd(vb, colors=vb["colors"])
    for _ in range(2):  # the second from the first one's state: no state is left over in the solver
        p0, v0 = g.state()
        g.step(iterations)
        p, v = O.vbd_step(vb, p0, v0, iterations, vb["dt"])
        gp, gv = g.state()
        assert np.abs(gp - p).max() < 2e-6
        assert np.abs(gv - v).max() < 2e-6 * 60 * 2


# colours of at most 4,736, 9,472 and 18,944 vertices take 16, 8 and 4 lanes (512 x 148 threads); above, a launch each
@pytest.mark.parametrize("w,h", [(3, 3), (33, 20), (137, 138), (139, 138), (195, 194), (197, 194), (275, 275),
                                 (277, 276)])
def test_lane_counts(w, h):
    _compare(_problem(w, h), 3)


@pytest.mark.parametrize("drop", ["tri", "edge", "both"])
def test_energies_left_out(drop):
    vb = _problem(12, 9, loose=5)
    for k in [q for q in vb if (drop != "edge" and q.startswith("tri_")) or (drop != "tri" and q.startswith("edge_"))]:
        vb[k] = vb[k][:0]
    _compare(vb, 4)


def test_single_color_of_loose_particles():
    # one colour: every sweep updates the vertices that the next one reads
    vb = _problem(3, 3, loose=400)
    for k in [q for q in vb if q.startswith("tri_") or q.startswith("edge_")]:
        vb[k] = vb[k][:0]
    vb["colors"][:] = 0
    _compare(vb, 6)


@pytest.mark.parametrize("api", ["capi", "pybind"])
def test_failed_barrier_is_reported_and_leaves_the_state(api):
    vb = _problem(33, 20)
    g = GpuVbd(vb, colors=vb["colors"], api=api)
    g.step(3)
    assert g.s.last_status() == capi.SOLVE_CONVERGED
    p0, v0 = g.state()
    if api == "pybind":  # the error flag of a barrier is set through the C ABI only
        return
    g.s.debug_fail_barrier(True)
    g.step(3)
    assert all(np.array_equal(a, b) for a, b in zip(g.state(), (p0, v0)))
    g.s.debug_fail_barrier(False)
    with pytest.raises(RuntimeError, match="barrier"):  # the next step, which does not run
        g.step(3)
    g.s.debug_fail_barrier(True)
    g.step(3)
    assert g.s.last_status() == capi.SOLVE_KERNEL_ERROR and g.s.last_status() == capi.SOLVE_CONVERGED
    assert all(np.array_equal(a, b) for a, b in zip(g.state(), (p0, v0)))
    # and from there as if nothing had been
    g.s.debug_fail_barrier(False)
    g.step(3)
    h = GpuVbd(dict(vb, pos=p0.astype(np.float32), vel=v0.astype(np.float32)), colors=vb["colors"])
    h.step(3)
    assert all(np.array_equal(a, b) for a, b in zip(g.state(), h.state()))
    # a launch per colour has no barrier to fail
    vb = _problem(277, 276)
    g = GpuVbd(vb, colors=vb["colors"])
    g.s.debug_fail_barrier(True)
    g.step(1)
    assert g.s.last_status() == capi.SOLVE_CONVERGED and not np.array_equal(g.state()[0], vb["pos"])
