"""Tap lists and fields that the filter's march does not take: cones past reach 3, lists out of order, any
weights, repeats, fields 8 bytes off a 16-byte boundary; against numpy, tap by tap (GPU)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(v, taps, w, hs_in, hs_out):
    u = v / hs_in if hs_in is not None else v
    nx, ny, nz = v.shape
    r = int(np.abs(taps).max())
    p = np.pad(u, r)
    out = np.zeros_like(v)
    size = np.zeros_like(v)
    for (dx, dy, dz), wt in zip(taps, w):
        t = wt * p[r + dx:r + dx + nx, r + dy:r + dy + ny, r + dz:r + dz + nz]
        out += t
        size += np.abs(t)
    return (out / hs_out, size / hs_out) if hs_out is not None else (out, size)


@pytest.mark.parametrize("kind", ["cone", "shuffled", "weights", "repeats", "off"])
@pytest.mark.parametrize("radius", [1.5, 3.0, 3.5, 4.5, 6.2])
@pytest.mark.parametrize("dims", [(1, 1, 1), (33, 9, 5), (70, 20, 21)])
def test_any_list(dims, radius, kind):
    """Both entries: the sum of n taps is within n + 3 roundings of the sizes of its terms."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid, stream_handle
    from loadpath_b200.simp import filter_taps

    rng = np.random.default_rng(int(10 * radius) + len(kind))
    taps, w = (np.array(a) for a in zip(*filter_taps(radius)))
    if kind == "shuffled":
        p = rng.permutation(len(w))
        taps, w = taps[p], w[p]
    elif kind == "weights":
        w = rng.standard_normal(len(w))
    elif kind == "repeats":
        taps, w = np.concatenate([taps, taps[:3]]), np.concatenate([w, w[:3]])
    reach = int(np.abs(taps).max())
    g = DevGrid(dims)
    v, h = rng.standard_normal(dims), 1.0 + rng.random(dims)
    vd, hd = (g.cells_to_dev(a, torch.float64) for a in (v, h))
    if kind == "off":
        held = torch.zeros(vd.numel() + 1, dtype=torch.float64, device="cuda")
        held[1:] = vd.reshape(-1)
        vd = held[1:].view(vd.shape)
        assert vd.data_ptr() % 16 == 8
    toff = torch.tensor(taps.reshape(-1), dtype=torch.int32, device="cuda")
    tw = torch.tensor(w, dtype=torch.float64, device="cuda")
    L, st = lib(), stream_handle()
    for hs_in, hs_out in ((None, hd), (hd, None)):
        want, size = _want(v, taps, w, None if hs_in is None else h, None if hs_out is None else h)
        tol = (len(w) + 3) * np.finfo(float).eps * size
        ptrs = [None if t is None else t.data_ptr() for t in (hs_in, hs_out)]
        for entry in (lambda o: L.lpb_filter(o.data_ptr(), vd.data_ptr(), toff.data_ptr(), tw.data_ptr(), len(w), *ptrs,
                                             None, 3.0, 1e-9, *g.args, st),
                      lambda o: L.lpb_filter_reach(o.data_ptr(), vd.data_ptr(), toff.data_ptr(), tw.data_ptr(), len(w),
                                                   reach, *ptrs, None, 3.0, 1e-9, *g.args, st)):
            out = g.cell_field(torch.float64)
            out.fill_(7.0)
            entry(out)
            assert (np.abs(g.cells_to_host(out) - want) <= tol).all()


@pytest.mark.parametrize("radius", [4.5, 2.0])
def test_design_update_past_the_fused_pass(radius):
    """The design update with a cone past the fused trial's reach, or a design 8 bytes off, gives the
    multiplier of the update that is not fused."""
    from loadpath_b200.grid import DevGrid
    from loadpath_b200.simp import DeviceFilter, ProjectedDesign

    dims = (24, 12, 8)
    rng = np.random.default_rng(3)
    g = DevGrid(dims)
    x, dc, dv = (g.cells_to_dev(a, torch.float64) for a in (rng.random(dims), -rng.random(dims), 0.1 + rng.random(dims)))
    flt = DeviceFilter(g, radius, pad=True)
    target = 0.4 * np.prod(dims)
    got = ProjectedDesign(flt).oc_step(x, dc, dv, 0.2, 2.0, 0.5, target)
    held = torch.zeros(x.numel() + 1, dtype=torch.float64, device="cuda")
    held[1:] = x.reshape(-1)
    off = held[1:].view(x.shape)
    assert off.data_ptr() % 16 == 8
    again = ProjectedDesign(flt).oc_step(off, dc, dv, 0.2, 2.0, 0.5, target)
    assert got[2] and again[2] and abs(got[1] - again[1]) <= 1e-12 * got[1]
    np.testing.assert_allclose(g.cells_to_host(got[0]), g.cells_to_host(again[0]), rtol=1e-12, atol=1e-13)
