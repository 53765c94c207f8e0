"""What the 'auto' imaging cache and the batched gradient keep, from the
memory there is, on the host: the allocator and the driver are fakes."""
import numpy as np
import pytest
import torch

from geobrain_b200.wave import batched, engine, kernel3d


class _Memory:
    """unused bytes in blocks of at most `largest`, `free` more at the driver."""

    def __init__(self, monkeypatch, unused, free=0, largest=None):
        self.unused, self.largest, self.held, self.asked = unused, largest, 0, 0
        monkeypatch.setattr(engine, "unused_pool", lambda device: unused)
        monkeypatch.setattr(engine, "workspace", self.take)
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: self.ask(free))

    def ask(self, free):
        self.asked += 1
        return free, free

    def take(self, nbytes, device):
        if self.largest is not None and nbytes > self.largest:
            raise torch.OutOfMemoryError("no block of that size")
        return torch.empty(0, dtype=torch.uint8)


def _plan(n_rcv=400):
    geo = engine.Geometry(40, 600, 8, 200, 1e-3, 10.0, 2, False)
    return engine.Plan(geo, np.array([3, 9]), np.array([1, 1]), np.arange(n_rcv), np.ones(n_rcv, np.int64))


def _choose(plan):
    return engine.choose_cached_steps(plan, "auto", False, "cuda:0", "fp32", 10, "fp32")


def _needs(plan):
    nt = plan.geo.nt
    fixed = plan.imaging_bytes(nt) + max(plan.workspace_bytes(0, 0), plan.gradient_workspace_bytes(False, 1))
    return fixed, plan.n_shots * nt * plan.n_rcv * 4


@pytest.mark.parametrize("fields", [0, 1, 3, 5])
def test_unused_blocks_must_hold_every_trace_field(monkeypatch, fields):
    """A gradient holds three recorded trace fields and up to three of its
    loss's; with room for fewer, and nothing free beside it, the driver's
    answer and its margin decide, and they leave no room for the cache."""
    plan = _plan()
    fixed, trace = _needs(plan)
    mem = _Memory(monkeypatch, fixed + fields * trace + trace // 2)
    assert _choose(plan) < plan.geo.nt and mem.asked == 1


def test_unused_blocks_that_hold_a_gradient_settle_it(monkeypatch):
    plan = _plan()
    fixed, trace = _needs(plan)
    mem = _Memory(monkeypatch, (fixed + 6 * trace) * 257 // 256 + 1)
    assert _choose(plan) == plan.geo.nt and mem.asked == 0


def test_unused_bytes_in_small_blocks_do_not(monkeypatch):
    """The sum suffices, but no block takes the imaging fields."""
    plan = _plan()
    fixed, trace = _needs(plan)
    mem = _Memory(monkeypatch, 2 * (fixed + 6 * trace), largest=plan.imaging_bytes(plan.geo.nt) - 1)
    assert _choose(plan) < plan.geo.nt and mem.asked == 1


def test_batched_and_3d_gradients_count_their_traces(monkeypatch):
    plans = [_plan(), _plan(200)]
    blocks, traces = batched.batch_hold_blocks(plans, False, "fp24")
    assert traces == sum(6 * _needs(p)[1] for p in plans)
    assert sum(blocks) >= sum(p.imaging_bytes(p.geo.nt, False, "fp24") for p in plans)

    class Lib:
        gb3_backward_workspace_bytes = staticmethod(lambda *a: 1000)
        gb3_workspace_bytes = staticmethod(lambda *a: 3000)

    class Run:
        from geobrain_b200._lib import Desc3
        L, device, desc = Lib, "cuda:0", Desc3(8, 8, 8, 2, 50, 2, 30, 0, 1e-3, 10.0, 10.0, 10.0)

    need = 100000 + 3000 + 8 * 4 * 2 * 50 * 30
    mem = _Memory(monkeypatch, need)
    assert not kernel3d._imaging_fits(Run, 100000) and mem.asked == 1
    mem = _Memory(monkeypatch, need * 257 // 256 + 1)
    assert kernel3d._imaging_fits(Run, 100000) and mem.asked == 0
