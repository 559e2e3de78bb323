"""Solvers that Python collects while another one records a graph (CPU only, the library stubbed)."""
import contextlib
import gc

import numpy as np
import pytest


class FakeLib:
    """A capture between begin and end; waits in it are counted, graphs freed once."""

    def __init__(self):
        self.open, self.waits, self.made, self.freed, self.inside = 0, 0, 0, [], lambda: None

    def begin(self, *a):
        self.open += 1

    def end(self, exec_):
        self.open -= 1
        self.made += 1
        exec_._obj.value = 1000 + self.made

    def wait(self, *a):
        self.waits += self.open

    def lpb_capture_end(self, st, exec_):
        self.end(exec_)

    def lpb_while_end(self, st, outer, exec_):
        self.end(exec_)

    lpb_capture_begin = lpb_while_begin = begin

    def lpb_mma_loop_body(self, *a):
        self.inside()

    def lpb_graph_free(self, exec_):
        assert not self.open and exec_.value not in self.freed
        self.freed.append(exec_.value)

    def lpb_mma_part_len(self, m):
        return 4

    def lpb_mma_state_len(self):
        return 64

    def __getattr__(self, name):
        return lambda *a: 0


@pytest.fixture
def fake(monkeypatch):
    import loadpath_b200.mg as mg
    import loadpath_b200.mma as mma

    f = FakeLib()
    for mod in (mg, mma):
        monkeypatch.setattr(mod, "lib", lambda: f)
        monkeypatch.setattr(mod, "stream_handle", lambda: 0)
    for name in ("device", "stream", "Stream"):
        monkeypatch.setattr(mg.torch.cuda, name, lambda *a: contextlib.nullcontext())
    monkeypatch.setattr(mg.torch.cuda, "current_stream", lambda *a: type("S", (), {"synchronize": f.wait})())
    monkeypatch.setattr(mg.torch.cuda, "synchronize", f.wait)

    def solver():
        ge = object.__new__(mg.GridElasticity)
        ge._gcache, ge._gen, ge._cap_stream, ge.device = {}, 0, None, "cpu"
        return ge

    def update(m):
        m.update(np.full(m.n, 0.5), 1.0, -np.ones(m.n), np.zeros(m.m), np.ones((m.m, m.n)))

    f.solver, f.mma, f.update = solver, lambda: mma.MMA(5, 1, device="cpu"), update
    gc.collect()
    gc.disable()
    yield f
    gc.enable()


@pytest.mark.parametrize("old", ["solver", "mma"])
@pytest.mark.parametrize("new", ["solver", "mma"])
def test_a_solver_collected_during_a_capture_is_freed_behind_it(fake, old, new):
    gone, here = getattr(fake, old)(), getattr(fake, new)()
    if old == "solver":
        gone._graph("a", lambda: None)
    else:
        fake.update(gone)
    gone.cycle = gone
    del gone
    seen = []

    def inside():
        gc.collect()
        seen.append((fake.open, list(fake.freed)))

    fake.inside = inside
    if new == "solver":
        here._graph("b", inside)
    else:
        fake.update(here)
    assert seen == [(1, [])]
    assert fake.waits == 0 and fake.freed == [1001]
    del here, inside
    fake.inside = None
    gc.collect()
    assert fake.freed == [1001, 1002]
