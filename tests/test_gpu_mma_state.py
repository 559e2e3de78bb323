"""MMA state restored and copied between updates, on the device (GPU)."""
import copy

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(257, 1), (5000, 3)])
def test_resumed_and_copied_runs_continue_as_the_run_itself(n, m):
    """low and upp replaced by saved ones after two updates, or the object copied there: the third update
    has the bits of a run that went on."""
    from loadpath_b200.mma import MMA

    rng = np.random.default_rng(n)
    x = torch.tensor(0.2 + 0.6 * rng.random(n), device="cuda")
    steps = [(torch.tensor(-rng.random(n), device="cuda"), 0.1 * rng.standard_normal(m),
              torch.tensor(rng.random((m, n)) / n, device="cuda")) for _ in range(3)]
    mma = MMA(n, m, move=0.3)
    for df0, f, df in steps[:2]:
        x = mma.update(x, 1.0, df0, f, df)
    saved = mma.low.clone(), mma.upp.clone()
    other = copy.deepcopy(mma)
    df0, f, df = steps[2]
    want = mma.update(x, 1.0, df0, f, df)
    got = other.update(x, 1.0, df0, f, df)
    assert torch.equal(got, want) and np.array_equal(other.lam, mma.lam)
    other = copy.deepcopy(mma)              # after the third update: back to the saved asymptotes
    other._xold1, other._xold2, other.iter = mma._xold2.clone(), mma._xold2.clone(), 2
    first = other.low
    other.low, other.upp = saved
    first.fill_(float("nan"))               # what the loop must not read any more
    assert torch.isfinite(other.update(x, 1.0, df0, f, df)).all()
