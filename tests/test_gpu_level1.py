"""The level-1 march (lpb_apply_level1_*) at the ends of its tiles, chunks and unit splits (GPU): against
the general kernel on the same level, patch cells on faces and inside, and its Chebyshev modes against
apply + vector kernel.

Tolerances: an output sums 8 cells x 24 products of O(1) relative size whose partial sums are bounded by
the row's absolute sum s; in any order the error is below 400 eps s, and s is below 30 times the largest
output here: 1.2e4 eps of the largest, 1e-3 in float32 and 3e-12 in float64 as worst cases; the
rounding errors add up as a random walk, sqrt(200) eps s: 5e-5 and 1e-13."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _hierarchy(dims, dtype, inside):
    from loadpath_b200.mg import BoxMesh, GridElasticity
    from oracle import ref_numpy as R

    rng = np.random.default_rng(sum(dims))
    fixed = np.zeros((3,) + tuple(d + 1 for d in dims), bool)
    fixed[:, 0] = True
    if inside:   # held dofs scattered over the grid: patch cells in every warp, several per row
        fixed |= rng.random(fixed.shape) < 0.01
    mesh = BoxMesh(dims)
    fx = np.moveaxis(fixed.reshape(3, -1), 0, 1).reshape(-1)
    ge = GridElasticity(mesh, 0.3, fx, coarse_cells=dims[0] * dims[1] * dims[2] // 9 + 1, dtype=dtype, element="im")
    ge.set_moduli(R.simp_moduli(R.log_uniform_density(dims, 3)).reshape(-1))
    assert ge.levels[1].kind == "weights"
    return ge, rng


def _field(lv, rng):
    g = lv.grid
    t = g.nodes_to_dev(rng.standard_normal(g.node_shape), lv.dtype)
    bits = torch.stack([((lv.mask >> c) & 1) for c in range(3)]).to(lv.dtype)
    return t * bits


# fine cells; the coarse grid's nodes end one before, at and after a tile of 15 x 7 columns, a chunk of 4
@pytest.mark.parametrize("dims", [(28, 12, 6), (30, 14, 8), (32, 16, 10), (58, 26, 14), (10, 6, 60)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("inside", [False, True])
def test_march_matches_general_kernel(dims, dtype, inside):
    ge, rng = _hierarchy(dims, dtype, inside)
    lv = ge.levels[1]
    u = _field(lv, rng)
    want = lv.apply(lv.grid.node_field(lv.dtype), u, fine_kernel=False)
    out = torch.full_like(u, 7.0)
    lv.apply(out, u)
    ge.check_device()
    tol = 5e-5 if dtype == np.float32 else 1e-13
    assert float((out - want).abs().max()) <= tol * float(want.abs().max())
    pad = out.permute(0, 3, 2, 1, 4).reshape(3, lv.grid.NX, lv.grid.NY, lv.grid.pz)[..., lv.grid.NZ:]
    assert torch.count_nonzero(pad) == 0
    from loadpath_b200._lib import lib

    knob = 3 if dtype == np.float32 else 4
    try:   # one block per SM: other segment ends, the same operator
        lib().lpb_tune_set(knob, lv.grid.nx, lv.grid.ny, lv.grid.nz, 1)
        out1 = lv.apply(torch.full_like(u, 7.0), u)
        assert float((out1 - want).abs().max()) <= tol * float(want.abs().max())
    finally:
        lib().lpb_tune_set(knob, lv.grid.nx, lv.grid.ny, lv.grid.nz, 0)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_chebyshev_modes_match_two_launches(dtype):
    """The fused updates against apply + vector kernel, to the bit (the same expressions)."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import stream_handle

    ge, rng = _hierarchy((44, 20, 18), dtype, True)
    lv = ge.levels[1]
    sfx = "f32" if dtype == np.float32 else "f64"
    L, st, n = lib(), stream_handle(), lv.grid.n_node_field
    b, x0, d0 = (_field(lv, rng) for _ in range(3))
    coef, dinv = lv.coef.data_ptr(), lv.dinv.data_ptr()
    t = torch.zeros_like(b)
    # mode 1
    lv.apply(t, d0)
    want, got = torch.zeros_like(b), torch.zeros_like(b)
    getattr(L, f"lpb_cheb2_zero_{sfx}")(want.data_ptr(), b.data_ptr(), t.data_ptr(), d0.data_ptr(), dinv, coef, n, st)
    lv.level1(1, None, d0, x=got, d=d0, b=b, coef=coef)
    assert torch.equal(got, want)
    # mode 2
    lv.apply(t, x0)
    rw, dw, rg, dg = (torch.zeros_like(b) for _ in range(4))
    getattr(L, f"lpb_residual_scaled_{sfx}")(b.data_ptr(), t.data_ptr(), dinv, coef, rw.data_ptr(), dw.data_ptr(), n, st)
    lv.level1(2, None, x0, x=x0, r=rg, d=dg, b=b, coef=coef)
    assert torch.equal(rg, rw) and torch.equal(dg, dw)
    # mode 3
    lv.apply(t, dw)
    xw, xg = x0.clone(), x0.clone()
    getattr(L, f"lpb_cheb2_{sfx}")(xw.data_ptr(), dw.data_ptr(), rw.data_ptr(), t.data_ptr(), dinv, coef, n, st)
    lv.level1(3, None, dg, x=xg, r=rg, d=dg, coef=coef)
    assert torch.equal(xg, xw)
