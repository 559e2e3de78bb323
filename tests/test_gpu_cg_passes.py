"""The PCG's and the power iteration's passes with folded reductions, several columns at once, against
the same formulas in float64 (GPU): one quad, a block and one quad around its end, more than one
round of every block.

Tolerances: a sum adds at most 4 x 3 values a thread, 8 warp and block steps, 3 x 592 / 256 partials a
thread and 10 more steps: below 60 eps of the sum of magnitudes, 1.4e-14. Elementwise results take
three roundings of their terms and carry the scalars' errors: 3e-14 (float64), 3e-7 (float32 fields) of
the largest term. The power step adds the float32 roundings of dinv av / |v|: 4e-7."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
SUM = 1.4e-14


def _parts(t, n, cols):
    from loadpath_b200._lib import lib

    return t[: cols * lib().lpb_cg_parts(n)].view(cols, -1)


@pytest.mark.parametrize("n", [4, 1020, 1024, 1028, 4 * 256 * 592, 4 * 256 * 592 * 2 + 4])
@pytest.mark.parametrize("cols", [1, 3, 9])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_cg_passes(n, cols, dtype):
    from loadpath_b200._lib import lib

    L, st = lib(), torch.cuda.current_stream().cuda_stream
    sfx = "f32" if dtype == torch.float32 else "f64"
    tol = 3e-7 if dtype == torch.float32 else 3e-14
    gen = torch.Generator("cuda").manual_seed(n + cols)
    f64 = dict(dtype=torch.float64, device="cuda", generator=gen)
    r, ap, p, x = (torch.randn(cols, n, **f64) for _ in range(4))
    z = torch.randn(cols, n, **f64).to(dtype)
    dinv = torch.rand(n, **f64).to(dtype)
    coef = torch.rand(16, **f64) + 0.5
    sc = torch.rand(cols, 8, **f64) + 0.5
    pap_part = torch.rand(cols, 5, **f64)
    part = torch.zeros(cols * L.lpb_reduce_blocks(), dtype=torch.float64, device="cuda")
    r32 = torch.zeros(cols, n, device="cuda")
    d = torch.zeros(cols, n, device="cuda", dtype=dtype)
    rz0 = sc[:, 2].clone()
    alpha = rz0 / pap_part.sum(1)
    want_r = r - alpha[:, None] * ap
    top = float(want_r.abs().max())
    rc = getattr(L, f"lpb_cg_r_{sfx}")(r.data_ptr(), ap.data_ptr(), r32.data_ptr(), d.data_ptr(), dinv.data_ptr(),
                                       coef.data_ptr(), n, sc.data_ptr(), pap_part.data_ptr(), 5, part.data_ptr(), cols, st)
    assert rc == 0
    assert float((r - want_r).abs().max()) <= 3e-14 * top
    assert torch.equal(r32, r.float())
    assert float((d - coef[1] * dinv * r).abs().max()) <= tol * top * float(coef[1])
    assert torch.equal(sc[:, 1], rz0)
    assert float((sc[:, 3] - pap_part.sum(1)).abs().max()) <= SUM * 5
    rr = (r * r).sum(1)
    assert float(((_parts(part, n, cols).sum(1) - rr) / rr).abs().max()) <= 2 * SUM
    assert L.lpb_cg_rr(sc.data_ptr(), part.data_ptr(), n, cols, st) == 0
    assert float(((sc[:, 4] - rr) / rr).abs().max()) <= 2 * SUM
    assert getattr(L, f"lpb_cg_rz_{sfx}")(r.data_ptr(), z.data_ptr(), n, part.data_ptr(), cols, st) == 0
    rz = (r * z.double()).sum(1)
    mag = (r * z.double()).abs().sum(1)
    assert float(((_parts(part, n, cols).sum(1) - rz) / mag).abs().max()) <= 2 * SUM
    part.copy_(torch.rand(part.shape, **f64))   # (r.z itself may cancel: any partials serve the update)
    rz = _parts(part, n, cols).sum(1)
    want_x = x + (sc[:, 1] / sc[:, 3])[:, None] * p
    want_p = z.double() + (rz / sc[:, 1])[:, None] * p
    rc = getattr(L, f"lpb_cg_p_{sfx}")(p.data_ptr(), x.data_ptr(), z.data_ptr(), n, sc.data_ptr(), part.data_ptr(), cols, st)
    assert rc == 0
    assert float((x - want_x).abs().max()) <= 3e-14 * float(want_x.abs().max())
    assert float((p - want_p).abs().max()) <= 3e-14 * float(want_p.abs().max())
    assert float(((sc[:, 2] - rz) / rz).abs().max()) <= 2 * SUM


@pytest.mark.parametrize("dims", [(1, 1, 1), (7, 5, 9), (40, 30, 50), (150, 70, 60)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("zero", [False, True])
def test_power_passes(dims, dtype, zero):
    """Two steps with A = 2 I; a zero start stays zero and leaves the interval's fixed upper end."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid

    L, st = lib(), torch.cuda.current_stream().cuda_stream
    sfx = "f32" if dtype == torch.float32 else "f64"
    tol = 4e-7 if dtype == torch.float32 else 8e-16
    g = DevGrid(dims)
    rng = np.random.default_rng(sum(dims))
    v0 = g.nodes_to_dev(0.0 * rng.standard_normal(g.node_shape) if zero else rng.standard_normal(g.node_shape), dtype)
    mask = torch.randint(0, 8, v0.shape[1:], device="cuda", dtype=torch.uint8)
    bits = torch.stack([(mask >> c) & 1 for c in range(3)]).to(torch.float64)
    dinv = torch.rand(v0.shape, device="cuda", dtype=torch.float64).to(dtype) + 0.5
    n = g.n_node_field
    part = torch.zeros(4 * L.lpb_reduce_blocks(), dtype=torch.float64, device="cuda")
    vv = torch.zeros(16, dtype=torch.float64, device="cuda")
    coef = torch.zeros(16, dtype=torch.float64, device="cuda")
    v, av = torch.empty_like(v0), torch.empty_like(v0)
    assert getattr(L, f"lpb_pw_start_{sfx}")(v.data_ptr(), v0.data_ptr(), mask.data_ptr(), *g.args, part.data_ptr(), st) == 0
    assert torch.equal(v.double(), v0.double() * bits)
    for k in range(2):
        torch.mul(v, 2, out=av)
        vd = v.double()
        s = (vd * vd).sum()
        want = bits * dinv.double() * av.double() / (torch.sqrt(s) if s > 0 else 1.0)
        lam = (vd * want).sum() / torch.sqrt(s)
        rc = getattr(L, f"lpb_pw_step_{sfx}")(av.data_ptr(), v.data_ptr(), dinv.data_ptr(), mask.data_ptr(), *g.args, k,
                                              part.data_ptr(), vv.data_ptr(), st)
        assert rc == 0
        assert float((av.double() - want).abs().max()) <= tol * float(want.abs().max())
        assert abs(float(vv[k] - s)) <= 2 * SUM * float(s)
        v, av = av, v
    assert L.lpb_pw_coef(coef.data_ptr(), vv.data_ptr(), part.data_ptr(), n, 2, 2, 1.3, st) == 0
    if zero:
        assert float(coef[0]) == 2.0
    else:
        assert abs(float(coef[0]) - 1.3 * float(lam)) <= (tol + 2 * SUM) * 1.3 * float(lam)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dims,cdims", [((14, 6, 6), (7, 3, 3)), ((62, 9, 17), (31, 5, 9)),
                                        ((62, 40, 60), (31, 20, 30))])   # (the last: one column and three fall on either side of a rule)
def test_transfers_with_columns(dtype, dims, cdims):
    """Three columns at once and the first direction, to the bit as one column's passes."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid

    L, st = lib(), torch.cuda.current_stream().cuda_stream
    sfx = "f32" if dtype == torch.float32 else "f64"
    gf, gc = DevGrid(dims), DevGrid(cdims)
    gen = torch.Generator("cuda").manual_seed(5)

    def rnd(g, k=3):
        return torch.randn((k,) + tuple(g.node_field(dtype).shape), device="cuda", dtype=torch.float64, generator=gen).to(dtype)

    b, ax, xc, x = rnd(gf), rnd(gf), rnd(gc), rnd(gf)
    dinv = rnd(gc, 1)[0]
    m = torch.randint(0, 8, b.shape[2:], device="cuda", dtype=torch.uint8, generator=gen)
    cm = torch.randint(0, 8, xc.shape[2:], device="cuda", dtype=torch.uint8, generator=gen)
    coef = torch.rand(16, device="cuda", dtype=torch.float64, generator=gen)
    rc, d = torch.empty_like(xc), torch.empty_like(xc)
    args = (*gf.args, *gc.args)
    assert getattr(L, f"lpb_restrict_start_{sfx}")(rc.data_ptr(), d.data_ptr(), dinv.data_ptr(), coef.data_ptr(),
                                                   b.data_ptr(), ax.data_ptr(), m.data_ptr(), cm.data_ptr(), *args, 3, st) == 0
    one, d1 = torch.empty_like(dinv), torch.empty_like(dinv)
    xs = x.clone()
    assert getattr(L, f"lpb_prolong_add_cols_{sfx}")(xs.data_ptr(), xc.data_ptr(), cm.data_ptr(), m.data_ptr(), *args, 3, st) == 0
    for j in range(3):
        getattr(L, f"lpb_restrict_residual_{sfx}")(one.data_ptr(), b[j].data_ptr(), ax[j].data_ptr(), m.data_ptr(),
                                                   cm.data_ptr(), *args, st)
        getattr(L, f"lpb_cheb_d_start_{sfx}")(one.data_ptr(), dinv.data_ptr(), coef.data_ptr(), d1.data_ptr(), one.numel(), st)
        assert torch.equal(rc[j], one) and torch.equal(d[j], d1)
        xj = x[j].clone()
        getattr(L, f"lpb_prolong_add_{sfx}")(xj.data_ptr(), xc[j].data_ptr(), cm.data_ptr(), m.data_ptr(), *args, st)
        assert torch.equal(xs[j], xj)
