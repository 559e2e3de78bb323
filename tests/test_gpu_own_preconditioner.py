"""A preconditioner of the caller's own (precondition_device overridden) in the float64 CG (GPU)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_loop", [True, False])
def test_every_iteration_asks_it(device_loop):
    """With the operator's diagonal in the V-cycle's place a solve gives the same answer, in the many iterations
    that a diagonal takes (over three times the V-cycle's on this design)."""
    from loadpath_b200.mg import BoxMesh, GridElasticity
    from oracle import ref_numpy as R

    dims = (24, 12, 10)
    fixed = np.zeros((3,) + tuple(d + 1 for d in dims), bool)
    fixed[:, 0] = True
    f = np.zeros(fixed.shape)
    f[2, -1, :, 0] = -1.0
    order = lambda a: np.ascontiguousarray(np.moveaxis(a.reshape(3, -1), 0, 1)).reshape(-1)  # noqa: E731

    class Diagonal(GridElasticity):
        def precondition_device(self, r64, z_out):
            return torch.mul(r64, self.levels[0].dinv, out=z_out)

    got = []
    for cls in (GridElasticity, Diagonal):
        ge = cls(BoxMesh(dims), 0.3, order(fixed), rtol=1e-10, dtype=np.float64, element="im", coarse_cells=100,
                 maxiter=5000)
        ge.device_loop = device_loop
        ge.set_moduli(R.simp_moduli(R.log_uniform_density(dims, 3)).reshape(-1))
        got.append((ge.solve_many([order(f)])[0], ge.last_iters))
    (want, iters), (u, its) = got
    assert its > 3 * iters
    np.testing.assert_allclose(u, want, rtol=1e-6, atol=1e-8 * np.abs(want).max())
