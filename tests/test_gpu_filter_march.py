"""The marched cone filter (lp_filter.cu) at the sizes where its tiles, chunks and segments end, and
the fused volume trial against the separate passes (GPU).

A cell's sum has at most 343 positive terms, so a float64 sum in any order is within 343 eps =
7.7e-14 of the exact one; the volume trial's sums over the cells are within cells * eps of each other."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("radius", [1.0, 2.0, 3.0, 3.9, 4.5])
@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 15, 3), (32, 16, 4), (33, 17, 5), (65, 2, 41), (2, 35, 8)])
def test_filter_at_tile_edges(dims, radius):
    from loadpath_b200.grid import DevGrid
    from loadpath_b200.simp import DeviceFilter
    from oracle import ref_numpy as R

    rng = np.random.default_rng(sum(dims))
    g = DevGrid(dims)
    flt = DeviceFilter(g, radius)
    taps = R.filter_taps(radius)
    v = rng.random(dims) + 0.1
    hs = R.filter_row_sums(dims, taps)
    src = torch.full_like(flt.hs, float("nan"))          # values outside the grid are never read
    full = src.permute(2, 1, 0, 3).reshape(g.nx, g.ny, g.cpz).clone()
    full[..., :g.nz] = torch.from_numpy(v).cuda()
    src.copy_(full.reshape(g.nx, g.ny, g.cpz // 4, 4).permute(2, 1, 0, 3))
    out = g.cell_field(torch.float64)
    flt.apply(out, src, hs_in=flt.hs)
    np.testing.assert_allclose(g.cells_to_host(out), R.grid_filter(v / hs, taps), rtol=400 * EPS)
    # the same taps in reverse: not sorted, so gathered cell by cell
    flt.toff = flt.toff.reshape(-1, 3).flip(0).reshape(-1).contiguous()
    flt.tw = flt.tw.flip(0).contiguous()
    flt.apply(out, src, hs_out=flt.hs)
    np.testing.assert_allclose(g.cells_to_host(out), R.grid_filter(v, taps) / hs, rtol=400 * EPS)


def test_filter_takes_an_unaligned_field():
    """A field that starts 8 bytes off a 16-byte boundary."""
    from loadpath_b200.grid import DevGrid
    from loadpath_b200.simp import DeviceFilter

    g = DevGrid((20, 18, 7))
    flt = DeviceFilter(g, 2.5)
    a = g.set_cells(g.cell_field(torch.float64), torch.rand(g.cells, dtype=torch.float64))
    off = torch.zeros(a.numel() + 1, dtype=torch.float64, device="cuda")[1:]
    off.copy_(a.reshape(-1))
    assert off.data_ptr() % 16 == 8
    want = flt.apply(g.cell_field(torch.float64), a)
    got = flt.apply(g.cell_field(torch.float64), off.reshape(a.shape))   # gathered cell by cell
    np.testing.assert_allclose(g.cells_to_host(got), g.cells_to_host(want), rtol=800 * EPS)


@pytest.mark.parametrize("radius", [1.5, 2.5, 3.5])
@pytest.mark.parametrize("dims", [(33, 17, 5), (64, 16, 12)])
def test_fused_trial_equals_separate_passes(dims, radius):
    """lpb_oc_trial against step, filter and projection one after another: the design, its filtered and
    its projected form to the bit, the volume to the sums' rounding."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid, stream_handle
    from loadpath_b200.simp import DeviceFilter, ProjectedDesign

    rng = np.random.default_rng(5)
    g = DevGrid(dims)
    flags = rng.choice([0, 0, 0, 1, 2], size=dims).astype(np.uint8)
    w = rng.random(dims)
    pd = ProjectedDesign(DeviceFilter(g, radius, pad=True), w=g.cells_to_dev(w, torch.float64),
                         flags=g.set_cells(g.cell_field(torch.uint8), torch.from_numpy(flags)))
    x, dc, dv = (g.cells_to_dev(a, torch.float64) for a in (rng.random(dims), -rng.random(dims), rng.random(dims) + 0.1))
    st = stream_handle()
    lm, beta, eta = 0.7, 4.0, 0.5
    L = lib()
    L.lpb_oc_stepped(pd.xn.data_ptr(), x.data_ptr(), dc.data_ptr(), dv.data_ptr(), lm, 0.2, pd.flags.data_ptr(),
                     *g.args, st)
    vol = pd.physical(pd.xn, beta, eta)
    ts, xn, xt, xp = (g.cell_field(torch.float64) for _ in range(4))
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    L.lpb_oc_step_base(ts.data_ptr(), x.data_ptr(), dc.data_ptr(), dv.data_ptr(), *g.args, st)
    for bufs in ((xn, xt, xp), (None, None, None)):
        L.lpb_oc_trial(*(b.data_ptr() if b is not None else None for b in bufs), ts.data_ptr(), x.data_ptr(), lm, 0.2,
                       pd.flags.data_ptr(), pd.flt.toff.data_ptr(), pd.flt.tw.data_ptr(), pd.flt.ntaps,
                       pd.flt.reach, pd.flt.hs.data_ptr(), beta, eta, pd.w.data_ptr(), pd._part.data_ptr(), out.data_ptr(), *g.args,
                       st)
        assert abs(out.item() - vol) <= w.size * EPS * vol
    for got, want in ((xn, pd.xn), (xt, pd.xt), (xp, pd.xp)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("beta", [1e-7, 0.499, 0.5, 64.0])
def test_trial_volume_at_any_slope(beta):
    """A volume trial alone, at slopes on both sides of where it leaves tanh, against the projection in
    extended precision: a cell's share is within 16 roundings (the filter's sum and division, the
    argument's, tanh's two, den's) of its own size or, on a steep slope, beta / 2 roundings of xt."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid, stream_handle
    from loadpath_b200.simp import DeviceFilter, ProjectedDesign

    dims, eta = (33, 17, 5), 0.5
    rng = np.random.default_rng(6)
    g = DevGrid(dims)
    w = rng.random(dims)
    pd = ProjectedDesign(DeviceFilter(g, 2.0, pad=True), w=g.cells_to_dev(w, torch.float64))
    x, ts = rng.random(dims), 0.5 * rng.random(dims)
    xd, td = (g.cells_to_dev(a, torch.float64) for a in (x, ts))
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    lib().lpb_oc_trial(None, None, None, td.data_ptr(), xd.data_ptr(), 1.0, 0.2, None, pd.flt.toff.data_ptr(),
                       pd.flt.tw.data_ptr(), pd.flt.ntaps, pd.flt.reach, pd.flt.hs.data_ptr(), beta, eta,
                       pd.w.data_ptr(), pd._part.data_ptr(), out.data_ptr(), *g.args, stream_handle())
    xn = g.set_cells(g.cell_field(torch.float64), torch.from_numpy(np.clip(ts, np.maximum(0, x - 0.2), np.minimum(1, x + 0.2))))
    xt = g.cells_to_host(pd.flt.apply(g.cell_field(torch.float64), xn, hs_out=pd.flt.hs)).astype(np.longdouble)
    b, e = np.longdouble(beta), np.longdouble(eta)
    xp = (np.tanh(b * e) + np.tanh(b * (xt - e))) / (np.tanh(b * e) + np.tanh(b * (1 - e)))
    want = (xp * w).sum()
    assert abs(out.item() - want) <= (16 + beta / 2) * EPS * w.sum()
