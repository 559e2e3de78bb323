"""Solvers that Python collects while another one records a graph (GPU)."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS = (20, 12, 8)


def _elasticity():
    from loadpath_b200.mg import BoxMesh, GridElasticity

    fixed = np.zeros((3,) + tuple(d + 1 for d in DIMS), bool)
    fixed[:, 0] = True
    return GridElasticity(BoxMesh(DIMS), 0.3, np.moveaxis(fixed.reshape(3, -1), 0, 1).reshape(-1), element="im")


def _solve(ge):
    f = np.zeros((3,) + tuple(d + 1 for d in DIMS))
    f[2, -1] = -1.0
    ge.set_moduli(np.ones(int(np.prod(DIMS))))
    return ge.solve_device(ge.g0.nodes_to_dev(f, torch.float64)).clone()


def _mma(n=300):
    from loadpath_b200.mma import MMA

    m = MMA(n, 1)
    x = torch.full((n,), 0.5, dtype=torch.float64, device="cuda")
    m.update(x, 1.0, -x, np.zeros(1), torch.ones((1, n), dtype=torch.float64, device="cuda"))
    return m


@pytest.mark.parametrize("kind", ["solver", "mma"])
def test_capture_outlives_a_collected_solver(kind, monkeypatch):
    """Every capture of a solve collects a solver, or an MMA, held by a cycle: same solution."""
    import loadpath_b200.mg as mg

    want = _solve(_elasticity())
    gone = []

    def cycle():
        if kind == "solver":
            other = _elasticity()
            _solve(other)
        else:
            other = _mma()
        other.cycle = other
        gone.append(1)

    plain = mg.GridElasticity._graph
    inner = [False]

    def graph(self, key, fn, loop=False):
        if inner[0] or key in self._gcache:
            return plain(self, key, fn, loop)
        inner[0] = True          # the solver made here captures as it always does
        cycle()
        inner[0] = False

        def collected(*a):
            gc.collect()
            return fn(*a)

        return plain(self, key, collected, loop)

    ge = _elasticity()
    gc.collect()
    gc.disable()
    try:
        monkeypatch.setattr(mg.GridElasticity, "_graph", graph)
        got = _solve(ge)
    finally:
        gc.enable()
    assert gone and torch.equal(got, want)
