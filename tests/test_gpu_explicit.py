"""The explicit levels' apply (cells shared by the warps of a block) at cell counts around its blocks
of 32 cells, against the assembled operator in float64 (GPU).

Tolerances: a node's value sums 8 cells x 24 products; in any order the error is below
(24 + 8 + 8) eps s with s the row's absolute sum (two factors rounded to the type add 2 eps s), and s is
below 30 times the largest output for these random operands: 1300 eps of the largest, 1.6e-4 in
float32 and 3e-13 in float64. The corner-parity form adds two transforms of 8 sums and 8 corner
values, whose terms grow by up to 8: 8 x as much, with the 1e-5 (its float32 storage's relative
tolerance) of a listed cell's entries on top."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CORNERS = [(k & 1, (k >> 1) & 1, k >> 2) for k in range(8)]


def _assembled(k, u, dims):
    """sum over cells of K u in float64: k (nx, ny, nz, 24, 24), u (3, nx+1, ny+1, nz+1)"""
    out = np.zeros_like(u)
    nx, ny, nz = dims
    uc = np.stack([u[:, a:a + nx, b:b + ny, c:c + nz] for a, b, c in CORNERS])   # (8, 3, ...)
    f = np.einsum("xyzrs,sxyz->rxyz", k, uc.reshape(24, nx, ny, nz)).reshape(8, 3, nx, ny, nz)
    for q, (a, b, c) in enumerate(CORNERS):
        out[:, a:a + nx, b:b + ny, c:c + nz] += f[q]
    return out


def _cells_dev(grid, k, dtype):
    """(nx, ny, nz, r, c) to the device's cell order with zero padding: (cells, 576)"""
    nx, ny, nz = k.shape[:3]
    pad = np.zeros((nx, ny, grid.cpz, 576))
    pad[:, :, :nz] = k.reshape(nx, ny, nz, 576)
    pad = pad.reshape(nx, ny, -1, 4, 576).transpose(2, 1, 0, 3, 4)
    return torch.tensor(np.ascontiguousarray(pad.reshape(-1, 576)), device="cuda", dtype=dtype)


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 5), (8, 1, 4), (3, 3, 4), (11, 3, 4), (5, 4, 7), (8, 4, 12)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_explicit_apply(dims, dtype):
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid

    rng = np.random.default_rng(sum(dims))
    g = DevGrid(dims)
    k = rng.standard_normal(dims + (24, 24))
    k = k + np.swapaxes(k, -1, -2)
    u = rng.standard_normal(g.node_shape)
    kd = _cells_dev(g, k, dtype)
    ncp = kd.shape[0]
    ud = g.nodes_to_dev(u, dtype)
    mask = torch.full_like(ud[0], 7, dtype=torch.uint8)
    kp = torch.empty(300, ncp, device="cuda", dtype=dtype)
    ft = torch.full((24, ncp), float("nan"), device="cuda", dtype=dtype)
    out = torch.full_like(ud, 7.0)
    sfx = "f32" if dtype == torch.float32 else "f64"
    st = torch.cuda.current_stream().cuda_stream
    assert getattr(lib(), f"lpb_pack_sym_{sfx}")(kp.data_ptr(), kd.data_ptr(), ncp, st) == 0
    rc = getattr(lib(), f"lpb_apply_explicit_sym_{sfx}")(out.data_ptr(), ud.data_ptr(), kp.data_ptr(), ft.data_ptr(),
                                                         mask.data_ptr(), *g.args, st)
    assert rc == 0
    want = _assembled(k, u, dims)
    err = np.abs(g.nodes_to_host(out) - want).max()
    assert err <= (1.6e-4 if dtype == torch.float32 else 3e-13) * np.abs(want).max()
    if dtype != torch.float32:
        return
    # the corner-parity form: every other cell's matrix holds the pattern, the rest are listed
    from loadpath_b200 import fem

    ke, on, n = np.ascontiguousarray(fem.hex8_ke(0.3, "im")), np.zeros((8, 24, 24)), np.zeros((64, 576))
    lib().lpb_level1_products(ke.ctypes.data, on.ctypes.data, n.ctypes.data)
    w = rng.random(dims + (8,)) + 0.5
    kk = np.einsum("xyzm,mrs->xyzrs", w, on)   # a level-1 matrix of each cell
    sel = np.indices(dims).sum(0) % 2 == 1
    kk[sel] = k[sel]
    kd = _cells_dev(g, kk, dtype)
    km = torch.empty(150, ncp, device="cuda")
    kpc = torch.empty(ncp, 300, device="cuda")
    glist = torch.empty(ncp, device="cuda", dtype=torch.int32)
    gcount = torch.zeros(1, device="cuda", dtype=torch.int32)
    assert lib().lpb_pack_modal_f32(km.data_ptr(), glist.data_ptr(), gcount.data_ptr(), kpc.data_ptr(), kd.data_ptr(),
                                    ncp, 1e-5, st) == 0
    assert int(gcount) == int(sel.sum())
    ft.fill_(float("nan"))
    rc = lib().lpb_apply_explicit_modal_f32(out.fill_(7.0).data_ptr(), ud.data_ptr(), km.data_ptr(), kpc.data_ptr(),
                                            glist.data_ptr(), gcount.data_ptr(), ft.data_ptr(), mask.data_ptr(), *g.args, st)
    assert rc == 0
    want = _assembled(kk, u, dims)
    err = np.abs(g.nodes_to_host(out) - want).max()
    assert err <= 1.3e-3 * np.abs(want).max()


@pytest.mark.parametrize("dims", [(1, 1, 1), (11, 3, 4), (8, 4, 12)])
def test_float64_updates_match_two_launches(dims):
    """The Chebyshev updates in the float64 gather, to the bit as the apply and the vector kernel."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid

    L, st = lib(), torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(sum(dims))
    g = DevGrid(dims)
    k = rng.standard_normal(dims + (24, 24))
    kd = _cells_dev(g, k + np.swapaxes(k, -1, -2), torch.float64)
    ncp = kd.shape[0]
    kp = torch.empty(300, ncp, device="cuda", dtype=torch.float64)
    ft = torch.empty(24, ncp, device="cuda", dtype=torch.float64)
    L.lpb_pack_sym_f64(kp.data_ptr(), kd.data_ptr(), ncp, st)
    b, d0, x0, r0, dinv = (g.nodes_to_dev(rng.standard_normal(g.node_shape), torch.float64) for _ in range(5))
    mask = torch.randint(0, 8, b.shape[1:], device="cuda", dtype=torch.uint8)
    coef = torch.rand(16, device="cuda", dtype=torch.float64)
    n = b.numel()

    def fused(mode, x, r, d, u):
        assert L.lpb_apply_explicit_sym_cheb_f64(mode, x.data_ptr(), r.data_ptr(), d.data_ptr(), u.data_ptr(),
                                                 b.data_ptr(), dinv.data_ptr(), coef.data_ptr(), kp.data_ptr(),
                                                 ft.data_ptr(), mask.data_ptr(), *g.args, st) == 0

    def apply(u):
        t = torch.zeros_like(u)
        L.lpb_apply_explicit_sym_f64(t.data_ptr(), u.data_ptr(), kp.data_ptr(), ft.data_ptr(), mask.data_ptr(), *g.args, st)
        return t

    def same(a, w):   # (the padding aside: the fused form leaves it)
        assert np.array_equal(g.nodes_to_host(a), g.nodes_to_host(w))

    xa, xb = x0.clone(), x0.clone()
    fused(1, xa, r0.clone(), d0, d0)
    L.lpb_cheb2_zero_f64(xb.data_ptr(), b.data_ptr(), apply(d0).data_ptr(), d0.data_ptr(), dinv.data_ptr(),
                         coef.data_ptr(), n, st)
    same(xa, xb)
    ra, da, rb, db = r0.clone(), d0.clone(), r0.clone(), d0.clone()
    fused(2, x0, ra, da, x0)
    L.lpb_residual_scaled_f64(b.data_ptr(), apply(x0).data_ptr(), dinv.data_ptr(), coef.data_ptr(), rb.data_ptr(),
                              db.data_ptr(), n, st)
    same(ra, rb)
    same(da, db)
    xa, xb = x0.clone(), x0.clone()
    fused(3, xa, r0, d0, d0)
    L.lpb_cheb2_f64(xb.data_ptr(), d0.data_ptr(), r0.data_ptr(), apply(d0).data_ptr(), dinv.data_ptr(),
                    coef.data_ptr(), n, st)
    same(xa, xb)
