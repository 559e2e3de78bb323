"""What an MMA object keeps between updates, with the library stubbed (CPU only)."""
import copy
import ctypes
import pickle

import numpy as np
import pytest


class FakeLib:
    """Records the buffers each graph names; a graph is freed once."""

    def __init__(self):
        self.graphs, self.freed, self.launched, self.hosts = {}, [], [], []

    def lpb_mma_part_len(self, m):
        return 4

    def lpb_mma_state_len(self):
        return 64

    def lpb_while_begin(self, st, handle, outer):
        pass

    def lpb_mma_loop_body(self, handle, n, m, *bufs_and_stream):
        self._bufs = bufs_and_stream[:-1]

    def lpb_while_end(self, st, outer, exec_):
        exec_._obj.value = 1000 + len(self.graphs)
        self.graphs[exec_._obj.value] = self._bufs

    def lpb_graph_launch(self, exec_, st):
        assert exec_.value not in self.freed
        self.launched.append(self.graphs[exec_.value])

    def lpb_graph_free(self, exec_):
        assert exec_.value not in self.freed
        self.freed.append(exec_.value)

    def lpb_mma_loop_begin(self, m, state, out, a, c, d, f, a0, epsimin, st):
        self.hosts.append([np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_double)), (m,)).copy()
                           for p in (a, c, d, f)])

    def __getattr__(self, name):
        return lambda *a: 0


@pytest.fixture
def fake(monkeypatch):
    import contextlib

    import loadpath_b200.mma as mod

    lib = FakeLib()
    monkeypatch.setattr(mod, "lib", lambda: lib)
    monkeypatch.setattr(mod, "stream_handle", lambda: 0)
    for name in ("device", "stream", "Stream"):
        monkeypatch.setattr(mod.torch.cuda, name, lambda *a: contextlib.nullcontext())
    monkeypatch.setattr(mod.torch.cuda, "synchronize", lambda *a: None)
    lib.mma = lambda n=5, m=1: mod.MMA(n, m, device="cpu")
    lib.update = lambda mma: mma.update(np.full(mma.n, 0.5), 1.0, -np.ones(mma.n), np.zeros(mma.m),
                                        np.ones((mma.m, mma.n)))
    return lib


def test_replaced_state_is_what_the_loop_reads(fake):
    """low and upp restored between updates (a resumed run): the loop names the new tensors."""
    mma = fake.mma()
    fake.update(mma)
    fake.update(mma)
    assert len(fake.graphs) == 1
    old = mma.low                      # kept alive, so its address is not given out again
    mma.low, mma.upp = mma.low.clone(), mma.upp.clone()
    fake.update(mma)
    assert fake.launched[-1][:2] == (mma.low.data_ptr(), mma.upp.data_ptr())
    assert old.data_ptr() not in fake.launched[-1]
    assert len(fake.graphs) == 2 and len(fake.freed) == 1


@pytest.mark.parametrize("make", [copy.copy, copy.deepcopy, lambda m: pickle.loads(pickle.dumps(m))])
def test_copies_have_a_loop_of_their_own(fake, make):
    """A copy after an update works, and each graph is freed once."""
    mma = fake.mma()
    fake.update(mma)
    other = make(mma)
    fake.update(other)
    assert fake.launched[-1][0] == other.low.data_ptr()
    n = len(fake.graphs)
    del mma, other
    assert sorted(fake.freed) == sorted(fake.graphs) and n == 2


def test_penalty_weights_one_for_all(fake):
    """d as one number for all constraints; a and c of another length are refused, not read past their end."""
    mma = fake.mma(m=3)
    mma.d = 2.0
    fake.update(mma)
    a, c, d, f = fake.hosts[-1]
    assert a.tolist() == [0.0] * 3 and c.tolist() == [1000.0] * 3 and d.tolist() == [2.0] * 3
    for name in ("a", "c"):
        short = fake.mma(m=3)
        setattr(short, name, np.ones(2))
        with pytest.raises(ValueError):
            fake.update(short)
