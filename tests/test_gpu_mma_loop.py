"""The MMA subproblem's device-side loop at its ends (GPU): one variable, a block and one variable around
its end, every instantiated number of constraints, several objects and streams, infeasible constraints
(y > 0), against the oracle. Sums in another order and shared reciprocals change an iterate by
rounding; the subproblem is solved to 1e-7 and its Newton steps contract, so designs agree to the
1e-9 of the span that the host-driven loops were held to."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (2, 2), (255, 3), (257, 4), (1000, 5), (4097, 8), (75_777, 2)])
@pytest.mark.parametrize("shift", [-0.2, 3.0])
def test_loop_matches_oracle(n, m, shift):
    from loadpath_b200.mma import MMA
    from oracle import ref_numpy as R

    rng = np.random.default_rng(n + m)
    dev, ref = MMA(n, m, move=0.3), R.MMA(n, m, move=0.3)
    x = 0.2 + 0.6 * rng.random(n)
    for it in range(3):
        df0 = -np.abs(rng.standard_normal(n)) * (1 + rng.random(n))
        f = rng.standard_normal(m) * 0.1 + shift   # (3: no design in reach is feasible)
        df = (0.2 + rng.random((m, n))) / n
        want = ref.update(x, 1.0, df0, f, df)
        got = dev.update(x, 1.0, df0, f, df)
        np.testing.assert_allclose(got, want, rtol=1e-9, atol=1e-9)
        np.testing.assert_allclose(dev.lam, ref.lam, rtol=1e-6, atol=1e-6)
        x = want


def test_two_objects_on_two_streams():
    """Two problems solved in turn on two streams give the bits each gives alone."""
    from loadpath_b200.mma import MMA

    rng = np.random.default_rng(0)
    n = 30_000
    args = [(torch.tensor(0.2 + 0.6 * rng.random(n), device="cuda"), 1.0,
             torch.tensor(-np.abs(rng.standard_normal(n)), device="cuda"), np.array([0.1]),
             torch.tensor(rng.random((1, n)) / n, device="cuda")) for _ in range(2)]
    alone = [MMA(n, 1).update(*a) for a in args]
    torch.cuda.synchronize()
    both = [MMA(n, 1), MMA(n, 1)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    got = []
    for mma, st, a in zip(both, streams, args):
        with torch.cuda.stream(st):
            got.append(mma.update(*a))
    torch.cuda.synchronize()
    for g, w in zip(got, alone):
        assert torch.equal(g, w)
