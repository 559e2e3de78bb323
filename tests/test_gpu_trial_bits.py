"""A volume trial's values against the accepted design's: the same bits (GPU)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [1e-7, 0.49, 0.5, 1.0, 2.0, 8.0, 64.0])
@pytest.mark.parametrize("radius", [1.5, 3.0, 3.5])
def test_a_trial_measures_the_design_it_would_write(beta, radius):
    """The volume alone (xn, xt, xp NULL) and with the design written are summed in the same order, so
    they are equal to the bit when, and only as long as, every cell's step and projection are; ts covers
    the clipped ends, infinities and NaN (dv = 0)."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid, stream_handle
    from loadpath_b200.simp import DeviceFilter, ProjectedDesign

    dims = (61, 35, 22)
    rng = np.random.default_rng(7)
    g = DevGrid(dims)
    w = np.exp(rng.uniform(-3, 3, dims))
    pd = ProjectedDesign(DeviceFilter(g, radius), w=g.cells_to_dev(w, torch.float64))
    x = rng.random(dims)
    ts = x * np.exp(rng.standard_normal(dims))
    ts[rng.random(dims) < 0.01] = np.inf
    ts[rng.random(dims) < 0.01] = np.nan
    ts[rng.random(dims) < 0.01] = 1e-310
    xd, td = (g.cells_to_dev(a, torch.float64) for a in (x, ts))
    bufs = [g.cell_field(torch.float64) for _ in range(3)]
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    for lm in (0.7, 3.0, 1e-12, 1e12):
        vols = []
        for b in (bufs, (None, None, None)):
            lib().lpb_oc_trial(*(t.data_ptr() if t is not None else None for t in b), td.data_ptr(), xd.data_ptr(), lm,
                               0.2, None, pd.flt.toff.data_ptr(), pd.flt.tw.data_ptr(), pd.flt.ntaps, pd.flt.reach,
                               pd.flt.hs.data_ptr(), beta, 0.5, pd.w.data_ptr(), pd._part.data_ptr(), out.data_ptr(),
                               *g.args, stream_handle())
            vols.append(out.item())
        assert vols[0] == vols[1] and np.isfinite(vols[0])
