"""GPU: the contact operator in the register-resident solver (one cluster up
to 16 CTAs, the grid barrier above) against the streamed kernel on the same
contacts.  Converged solves (rel-res 1e-8) agree to the 1e-5 m of the other
solver tests; over 10 fixed iterations from a zero guess each FP32 operation
adds at most 2^-24 of |dx| < 0.02 m, about ten per entry and iteration, and
the positions round to 1.2e-7 m: 5e-7 m."""
import numpy as np
import pytest

from chysx import capi, scenes
from chysx.runner import GpuCloth

pytestmark = pytest.mark.gpu


class Contacts:
    """Random four-particle contacts, some on one particle twice as often, with slips."""

    def __init__(self, n, m, seed, same=None):
        import torch

        rng = np.random.default_rng(seed)
        pairs = np.stack([rng.choice(n, 4, replace=False) for _ in range(m)]).astype(np.int32)
        k = m // 4 if same is None else same
        pairs[:k, 0] = pairs[0, 0]  # a row with many slots
        pairs[:k, 1:] = np.sort((pairs[0, 0] + 1 + rng.permuted(np.tile(np.arange(n - 1), (k, 1)), axis=1)[:, :3]) % n)
        w = np.zeros((m, 8), np.float32)
        w[:, 0] = 1.0
        w[:, 1:4] = -rng.dirichlet((1, 1, 1), m)
        nrm = rng.standard_normal((m, 3))
        w[:, 4:7] = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
        w[:, 7] = 1.0e-3
        u = np.zeros((m, 4), np.float32)
        u[:, :3] = 1.0e-4 * rng.standard_normal((m, 3))
        u[:, 3] = np.linalg.norm(u[:, :3], axis=1)
        self.m = m
        self.dev = [torch.from_numpy(a).cuda() for a in (pairs, w, u)]
        self.count = torch.tensor([m], dtype=torch.int32, device="cuda")

    def attach(self, sim, mode=0):
        p, w, u = self.dev
        sim.set_contact_op(p.data_ptr(), w.data_ptr(), self.count.data_ptr(), self.m, 50.0, slips=u.data_ptr(),
                           friction_mu=0.2, residual_mode=mode)


def _run(sc, c, path, its, tol, warm="zero", steps=1, mode=0):
    g = GpuCloth(sc, max_iter=its, rel_tol=tol, warm_start="zero")
    g.sim.set_tuning(path)
    c.attach(g.sim, mode)
    g.sim.set_solver(its, tol, warm)
    for _ in range(steps):
        g.step()
    return g


# one CTA, eight, sixteen (clusters), and the grid barrier
@pytest.mark.parametrize("side,grid", [(20, 1), (64, 8), (90, 16), (100, 20)])
def test_matches_streamed(side, grid):
    sc = scenes.config_large(side=side)
    c = Contacts(side * side, 40, side)
    a, b = (_run(sc, c, p, 10, 0.0) for p in (0, 2))
    assert a.sim.solver_info() == ("resident", grid, 512) and b.sim.solver_info()[0] == "streamed"
    assert np.abs(a.positions() - b.positions()).max() < 5e-7
    a, b = (_run(sc, c, p, 20000, 1e-8) for p in (0, 2))
    assert a.stats()[2] == b.stats()[2] == capi.SOLVE_CONVERGED
    assert np.abs(a.positions() - b.positions()).max() < 1e-5


@pytest.mark.parametrize("side", [20, 100])
@pytest.mark.parametrize("mode", [0, 1])
def test_warm_residual(side, mode):
    # the second step starts from the first one's dx with either residual: positions, dt * velocities and guess may
    # each differ by 5e-7 m after the first step, the second adds its own
    sc = scenes.config_large(side=side)
    c = Contacts(side * side, 30, 5)
    a, b = (_run(sc, c, p, 10, 0.0, "previous", 2, mode) for p in (0, 2))
    assert np.abs(a.positions() - b.positions()).max() < 2e-6


# more entries than a CTA keeps in shared memory (2048): the rest is read from the list; one CTA, eight, the grid barrier
@pytest.mark.parametrize("side,m", [(20, 700), (64, 6000), (100, 14000)])
def test_long_lists(side, m):
    sc = scenes.config_large(side=side)
    c = Contacts(side * side, m, side, 12)
    a, b = (_run(sc, c, p, 10, 0.0) for p in (0, 2))
    assert np.abs(a.positions() - b.positions()).max() < 5e-7
    a, b = (_run(sc, c, p, 20000, 1e-8) for p in (0, 2))
    assert a.stats()[2] == b.stats()[2] == capi.SOLVE_CONVERGED
    assert np.abs(a.positions() - b.positions()).max() < 1e-5


def test_autotune_tells_the_kernels_apart():
    # 100 x 100: the resident and the streamed kernel both run 20 CTAs of 512 threads
    sc = scenes.config_large(side=100)
    g = _run(sc, Contacts(10000, 40, 3), 0, 50, 0.0)
    table = g.sim.autotune(sc["dt"], 1)
    kinds = {(t["kernel"], t["threads"], t["grid"]) for t in table if t["sync"] == 0}
    assert ("resident", 512, 20) in kinds and ("streamed", 512, 20) in kinds
