"""The C entries that the package itself no longer calls, against what took their place or the formula (GPU):
the PCG's and the power iteration's passes with reductions of their own, the device loop's test
alone, the level-1 apply in two launches, its float64 columns, and the MMA passes that a host loop drives."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _lib():
    from loadpath_b200._lib import lib

    return lib(), torch.cuda.current_stream().cuda_stream


def _near(got, want, tol):
    assert float((got.double() - want.double()).abs().max()) <= tol * float(want.double().abs().max())


@pytest.mark.parametrize("n", [4, 1021, 700_001])
def test_cg_passes_with_their_own_reductions(n):
    """Elementwise results within three roundings (float32 copies: its own one), dots within 60 roundings of
    the sum of magnitudes."""
    L, st = _lib()
    gen = torch.Generator("cuda").manual_seed(n)
    x, r, p, ap, z = (torch.randn(n, device="cuda", dtype=F64, generator=gen) for _ in range(5))
    part, out = torch.zeros(4 * L.lpb_reduce_blocks(), device="cuda", dtype=F64), torch.zeros(1, device="cuda", dtype=F64)
    num, den, new = (torch.tensor([v], device="cuda", dtype=F64) for v in (0.7, 1.3, 0.4))
    alpha, beta, z32 = 0.7 / 1.3, 0.4 / 0.7, z.float()
    ptr = lambda *t: [None if v is None else v.data_ptr() for v in t]  # noqa: E731
    L.lpb_dot_f64_f32(*ptr(x, z32), n, *ptr(part, out), st)
    assert abs(float(out) - float((x * z32.double()).sum())) <= 1.4e-14 * float((x * z32.double()).abs().sum())
    xs, rs, r32 = x.clone(), r.clone(), torch.zeros(n, device="cuda")
    L.lpb_cg_step(*ptr(xs, rs, p, ap, r32), n, *ptr(num, den, part, out), st)
    _near(xs, x + alpha * p, 1e-15)
    _near(rs, r - alpha * ap, 1e-15)
    _near(r32, rs, 6e-8)
    assert abs(float(out) - float((rs * rs).sum())) <= 1.4e-14 * float(out)
    ra, rb32 = r.clone(), torch.zeros(n, device="cuda")
    L.lpb_cg_step_r(*ptr(ra, ap, rb32), n, *ptr(num, den, part, out), st)
    assert torch.equal(ra, rs) and torch.equal(rb32, r32)
    for sfx, zz in (("f32", z32), ("f64", z)):
        q = p.clone()
        getattr(L, f"lpb_xpby_{sfx}")(*ptr(q, zz), n, *ptr(new, num), st)
        _near(q, zz.double() + beta * p, 1e-15)
        q, xx = p.clone(), x.clone()
        getattr(L, f"lpb_xpby_x_{sfx}")(*ptr(q, xx, zz), n, *ptr(num, den, new), st)
        _near(q, zz.double() + beta * p, 1e-15)
        _near(xx, x + alpha * p, 1e-15)
        v = zz.clone()
        s = (zz.double() ** 2).sum().reshape(1)
        getattr(L, f"lpb_scale_rsqrt_{sfx}")(v.data_ptr(), n, s.data_ptr(), st)
        _near(v, zz.double() / s.sqrt(), 2e-7 if sfx == "f32" else 1e-15)


def test_power_iteration_passes():
    from loadpath_b200.grid import DevGrid

    L, st = _lib()
    g = DevGrid((9, 5, 6))
    gen = torch.Generator("cuda").manual_seed(1)
    mask = torch.randint(0, 8, g.mask_shape, device="cuda", dtype=torch.uint8, generator=gen)
    bits = torch.stack([(mask >> c) & 1 for c in range(3)])
    for dtype, sfx in ((torch.float32, "f32"), (F64, "f64")):
        a, d = (torch.randn(bits.shape, device="cuda", dtype=dtype, generator=gen) for _ in range(2))
        out = a.clone()
        getattr(L, f"lpb_dinv_mask_{sfx}")(out.data_ptr(), d.data_ptr(), mask.data_ptr(), *g.args, st)
        assert torch.equal(out, torch.where(bits.bool(), d * a, torch.zeros_like(a)))
    vv, vav = torch.ones(12, device="cuda", dtype=F64), torch.linspace(1.0, 1.9, 12, device="cuda", dtype=F64)
    coef = torch.zeros(16, device="cuda", dtype=F64)
    L.lpb_cheb_coef(coef.data_ptr(), vv.data_ptr(), vav.data_ptr(), 12, 2, 1.3, st)
    hi = 1.3 * 1.9
    theta, delta = 0.5 * (hi + hi / 30), 0.5 * (hi - hi / 30)
    sigma, rho, want = theta / delta, delta / theta, [hi, 1 / theta]
    for _ in range(2):
        new = 1.0 / (2.0 * sigma - rho)
        want += [new * rho, 2.0 * new / delta]
        rho = new
    np.testing.assert_allclose(coef[:6].cpu().numpy(), want, rtol=1e-14)


def _while(L, body):
    """body(handle, stream) as a device loop's, run once."""
    side = torch.cuda.Stream()
    handle, outer, exec_ = ctypes.c_longlong(), ctypes.c_void_p(), ctypes.c_void_p()
    L.lpb_while_begin(side.cuda_stream, ctypes.byref(handle), ctypes.byref(outer))
    body(handle.value, side.cuda_stream)
    L.lpb_while_end(side.cuda_stream, outer, ctypes.byref(exec_))
    L.lpb_graph_launch(exec_, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    L.lpb_graph_free(exec_)


@pytest.mark.parametrize("bb,pap,rr,want", [(1.0, 1.0, 1e-20, (1, 1)), (0.0, 1.0, 1.0, (1, 2)), (1.0, -1.0, 1.0, (1, 3)),
                                            (1.0, 1.0, 1.0, (7, 0))])
def test_stopping_test_alone(bb, pap, rr, want):
    """Statuses 1 to 3 stop the loop at once; a running solve stops at maxiter (7). The column form: every
    column its own, the loop as long as one runs; and the snapshot of a column that converged in the last
    iteration."""
    from loadpath_b200.grid import DevGrid

    L, st = _lib()
    sc = torch.zeros(8, device="cuda", dtype=F64)
    sc[0], sc[3], sc[4] = bb, pap, rr
    state = torch.zeros(2, device="cuda", dtype=torch.int64)
    _while(L, lambda h, s: L.lpb_cg_continue(h, sc.data_ptr(), state.data_ptr(), 1e-6, 7, s))
    assert tuple(state.tolist()) == want
    cols = torch.stack([sc, sc.clone()])
    cols[1, 0], cols[1, 3], cols[1, 4] = 1.0, 1.0, 1e-20
    states = torch.zeros(3, 2, device="cuda", dtype=torch.int64)
    _while(L, lambda h, s: L.lpb_cg_continue_cols(h, cols.data_ptr(), states.data_ptr(), 2, 1e-6, 7, s))
    got = states.tolist()
    assert got[1] == [1, 1] and got[2][0] == want[0] and got[0] == ([0, 0] if want[1] == 0 else list(want))
    g = DevGrid((4, 3, 5))
    mask = torch.randint(0, 8, g.mask_shape, device="cuda", dtype=torch.uint8)
    x = g.node_field(F64).normal_()
    snap = torch.full_like(x, 7.0)
    L.lpb_snapshot_converged(snap.data_ptr(), x.data_ptr(), mask.data_ptr(), states.data_ptr(), 1, 2, *g.args, st)
    kept = torch.where(torch.stack([(mask >> c) & 1 for c in range(3)]).bool(), x, torch.zeros_like(x))
    assert torch.equal(snap, kept if want[0] == 1 else torch.full_like(x, 7.0))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_level1_entries(dtype):
    """The apply in two launches against the package's (5e-5 and 1e-13 of the largest entry), and the columns
    entry to the bit as one column at a time."""
    from loadpath_b200.mg import BoxMesh, GridElasticity
    from oracle import ref_numpy as R

    dims = (30, 22, 26)
    fixed = np.zeros((3,) + tuple(d + 1 for d in dims), bool)
    fixed[:, 0] = True
    ge = GridElasticity(BoxMesh(dims), 0.3, np.moveaxis(fixed.reshape(3, -1), 0, 1).reshape(-1), dtype=dtype, element="im",
                        coarse_cells=2000)
    ge.set_moduli(R.simp_moduli(R.log_uniform_density(dims, 3)).reshape(-1))
    lv = ge.levels[1]
    assert lv.kind == "weights" and lv.npatch > 0
    L, st = _lib()
    g, sfx, k = lv.grid, lv._sfx(), 3
    bits = torch.stack([((lv.mask >> c) & 1) for c in range(3)]).to(lv.dtype)
    u, b, x0, r0 = (torch.randn((k,) + bits.shape, device="cuda", dtype=lv.dtype) * bits for _ in range(4))
    want, got = lv.apply(torch.zeros_like(u[0]), u[0]), torch.full_like(u[0], 7.0)
    getattr(L, f"lpb_apply_weights_tma_{sfx}")(got.data_ptr(), u.data_ptr(), lv.wc.data_ptr(), lv.patch_id.data_ptr(),
                                               lv.patch_k.data_ptr(), lv.mask.data_ptr(), lv.g1.ctypes.data,
                                               lv.pbox.ctypes.data, lv.err.data_ptr(), *g.args, st)
    _near(got, want, 5e-5 if dtype == np.float32 else 1e-13)
    coef = lv.coef.data_ptr()
    for mode in range(4):
        x, r, d = (u.clone() if mode == 2 else x0.clone()), r0.clone(), (u.clone() if mode != 2 else r0.clone())
        xs, rs, ds = x.clone(), r.clone(), d.clone()
        src = x if mode == 2 else d
        out, outs = torch.zeros_like(u), torch.zeros_like(u)
        getattr(L, f"lpb_apply_level1_cols_{sfx}")(
            mode, out.data_ptr(), x.data_ptr(), r.data_ptr(), d.data_ptr(), src.data_ptr(), b.data_ptr(), lv.dinv.data_ptr(),
            coef, lv.wc.data_ptr(), lv.patch_id.data_ptr(), lv.patch_m.data_ptr(), lv.patch_k.data_ptr(), lv.mask.data_ptr(),
            lv.g1.ctypes.data, lv.pbox.ctypes.data, lv.err.data_ptr(), *g.args, k, st)
        for j in range(k):
            lv.level1(mode, outs[j], (xs if mode == 2 else ds)[j], x=xs[j], r=rs[j], d=ds[j], b=b[j], coef=coef)
        assert torch.equal(x, xs) and torch.equal(r, rs) and torch.equal(d, ds)
        assert mode or torch.equal(out, outs)
    ge.check_device()


@pytest.mark.parametrize("n,m", [(1, 1), (3000, 1), (5001, 3)])
def test_mma_passes_driven_by_the_host(n, m):
    """loadpath's subproblem loops on the host around lpb_mma_newton_a, _newton_b and _trial, against the
    device's loop on the same terms: solved to 1e-7, so designs agree to 1e-9 of the span."""
    from loadpath_b200.mma import MMA

    L, st = _lib()
    rng = np.random.default_rng(n + m)
    mma = MMA(n, m, move=0.3)
    f = 0.1 * rng.standard_normal(m)
    mma.update(0.2 + 0.6 * rng.random(n), 1.0, -rng.random(n) - 0.1, f, (0.2 + rng.random((m, n))) / n)
    M, ntri = mma.M, mma.M * (mma.M + 1) // 2
    arrays = [t.data_ptr() for t in (mma.low, mma.upp, mma._alfa, mma._beta)]
    pq = [t.data_ptr() for t in (mma._P, mma._Q)]
    z_ = lambda: torch.zeros(n, dtype=F64, device="cuda")  # noqa: E731
    cur, nxt = [[z_() for _ in range(3)] for _ in range(2)]
    dx, dxsi, deta, delx, diagx = (z_() for _ in range(5))
    part, out = torch.zeros(int(L.lpb_mma_part_len(m)), dtype=F64, device="cuda"), torch.zeros(64, dtype=F64, device="cuda")
    L.lpb_mma_sub_init(n, arrays[2], arrays[3], *(t.data_ptr() for t in cur), st)
    # b = sum_j P_ij / (upp_j - x_j) + Q_ij / (x_j - low_j) - f at the design the terms were formed at
    b = (mma._P / (mma.upp - mma._x) + mma._Q / (mma._x - mma.low)).sum(1).cpu().numpy() - f

    def residual(src, dst, step, steg, lam, y, z, mu, zet, s, epsi):
        lam = np.ascontiguousarray(lam, float)
        L.lpb_mma_trial(n, m, *arrays, mma._p0.data_ptr(), mma._q0.data_ptr(), *pq, *(t.data_ptr() for t in src),
                        *((dx.data_ptr(), dxsi.data_ptr(), deta.data_ptr()) if step else (None, None, None)), float(steg),
                        lam.ctypes.data, float(epsi), *(t.data_ptr() for t in dst), part.data_ptr(), out.data_ptr(), st)
        o = out[:2 + M].cpu().numpy()
        small = np.concatenate([mma.c + mma.d * y - mu - lam, [mma.a0 - zet - mma.a @ lam],
                                o[2:2 + m] - mma.a * z - y + s - b, mu * y - epsi, [zet * z - epsi], lam * s - epsi])
        return np.sqrt(o[0] + small @ small), max(o[1], np.abs(small).max())

    y, z, lam, mu, zet, s, epsi = np.ones(m), 1.0, np.ones(m), np.maximum(1.0, 0.5 * mma.c), 1.0, np.ones(m), 1.0
    while epsi > 1e-7:
        norm, rmax = residual(cur, cur, False, 0.0, lam, y, z, mu, zet, s, epsi)
        it = 0
        while rmax > 0.9 * epsi and it < 200:
            it += 1
            keep = np.ascontiguousarray(lam, float)
            L.lpb_mma_newton_a(n, m, *arrays, mma._p0.data_ptr(), mma._q0.data_ptr(), *pq, *(t.data_ptr() for t in cur),
                               keep.ctypes.data, float(epsi), delx.data_ptr(), diagx.data_ptr(), part.data_ptr(),
                               out.data_ptr(), st)
            o = out[:2 * M + ntri].cpu().numpy()
            tri = np.zeros((M, M))
            tri[np.triu_indices(M)] = o[2 * M:]
            dely, diagy = mma.c + mma.d * y - lam - epsi / y, mma.d + mu / y
            rhs = o[:m] - mma.a * z - y - b + epsi / lam + dely / diagy - o[M:M + m]
            aa = np.zeros((m + 1, m + 1))
            aa[:m, :m] = np.diag(s / lam + 1.0 / diagy) + (tri + np.triu(tri, 1).T)[:m, :m]
            aa[:m, m] = aa[m, :m] = mma.a
            aa[m, m] = -zet / z
            sol = np.linalg.solve(aa, np.append(rhs, mma.a0 - mma.a @ lam - epsi / z))
            dlam, dz = np.ascontiguousarray(sol[:m]), sol[m]
            L.lpb_mma_newton_b(n, m, *arrays, *pq, *(t.data_ptr() for t in cur), delx.data_ptr(), diagx.data_ptr(),
                               dlam.ctypes.data, float(epsi), dx.data_ptr(), dxsi.data_ptr(), deta.data_ptr(),
                               part.data_ptr(), out.data_ptr(), st)
            mx = out[:4].cpu().numpy()
            dy = (dlam - dely) / diagy
            dmu, dzet = -mu + epsi / y - mu * dy / y, -zet + epsi / z - zet * dz / z
            ds = -s + epsi / lam - s * dlam / lam
            small = np.concatenate([dy, [dz], dlam, dmu, [dzet], ds]) / np.concatenate([y, [z], lam, mu, [zet], s])
            steg = 1.0 / max(mx[2], mx[3], np.max(-1.01 * small), mx[0], mx[1], 1.0)
            old = (y, z, lam, mu, zet, s)
            for _ in range(50):
                y, z, lam, mu, zet, s = (v + steg * d for v, d in zip(old, (dy, dz, dlam, dmu, dzet, ds)))
                newnorm, rmax = residual(cur, nxt, True, steg, lam, y, z, mu, zet, s, epsi)
                if newnorm < 2.0 * norm:
                    break
                steg /= 2.0
            cur, nxt, norm = nxt, cur, newnorm
        epsi *= 0.1
    want = torch.minimum(torch.maximum(cur[0], mma._alfa), mma._beta)
    assert float((mma._xnew - want).abs().max()) <= 1e-9
    np.testing.assert_allclose(mma.lam, lam, rtol=1e-6, atol=1e-6)
