"""The benchmark's comparison arms on a fake simulator: every step's solve
status counts, the warm-up ones' too."""
import bench
import pytest
import torch


class _Event:
    def __init__(self, enable_timing):
        pass

    def record(self):
        pass

    def elapsed_time(self, other):
        return 4.0


class _Sim:
    def __init__(self, fails_at):
        self.k, self.fails_at, self.sim = 0, fails_at, self

    def step(self):
        self.k += 1

    def stats(self):
        return 100 + self.k, 1e-7, int(self.k == self.fails_at)

    def last_timing(self):
        return 1.0, 2.0, 1.0

    def solver_info(self):
        return "tiled", 148, 1024

    def preconditioner(self):
        return "block_jacobi", 0, 0.0, 0


@pytest.mark.parametrize("fails_at", [0, 2, 5])
def test_unconverged_step_is_reported(monkeypatch, fails_at):
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    arm = bench.timed_arm(_Sim(fails_at), 2, 3, torch.zeros(4))
    if fails_at:
        assert f"step {fails_at} (3 warm-up)" in arm["failed"] and "steps_per_s" not in arm
    else:
        assert arm["steps_per_s"] == pytest.approx(250.0) and arm["pcg_iters_per_step"] == 104.5 and arm["steps"] == 2
