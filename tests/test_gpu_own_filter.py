"""The design update with a filter or a physical density of the caller's own: what the caller overrode is what
each trial of the volume multiplier is measured with (GPU)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem():
    from loadpath_b200.grid import DevGrid

    dims = (20, 11, 9)
    rng = np.random.default_rng(2)
    g = DevGrid(dims)
    return g, [g.cells_to_dev(a, torch.float64) for a in (rng.random(dims), -rng.random(dims), 0.1 + rng.random(dims))]


@pytest.mark.parametrize("how", ["class", "instance", "other"])
def test_filter_of_the_callers_own(how):
    """A filter that doubles its result: the volume of the design that oc_step returns, measured through it, is
    the target."""
    from loadpath_b200.simp import DeviceFilter, ProjectedDesign

    class Doubled(DeviceFilter):
        def apply(self, out, v, *a, **kw):
            return super().apply(out, v, *a, **kw).mul_(2.0)

    class Other:     # grid, hs and apply are all that the update asks for
        def __init__(self, flt):
            self.grid, self.hs, self._flt = flt.grid, flt.hs, flt

        def apply(self, out, v, **kw):
            return self._flt.apply(out, v, **kw).mul_(2.0)

    g, (x, dc, dv) = _problem()
    flt = Doubled(g, 2.0) if how == "class" else DeviceFilter(g, 2.0)
    if how == "class":
        flt.hs = DeviceFilter(g, 2.0).hs
    elif how == "instance":
        plain = flt.apply
        flt.apply = lambda out, v, **kw: plain(out, v, **kw).mul_(2.0)
    else:
        flt = Other(flt)
    pd = ProjectedDesign(flt)
    target = 0.6 * x.numel()
    xn, lm, held = pd.oc_step(x, dc, dv, 0.2, 2.0, 0.5, target)
    assert held
    vol = pd.physical(xn.clone(), 2.0, 0.5)
    assert abs(vol - target) <= 1e-10 * target


def test_physical_density_of_the_callers_own():
    from loadpath_b200.simp import DeviceFilter, ProjectedDesign

    class Half(ProjectedDesign):
        def physical(self, *a, **kw):
            return 0.5 * super().physical(*a, **kw)

    g, (x, dc, dv) = _problem()
    pd = Half(DeviceFilter(g, 2.0))
    target = 0.2 * x.numel()
    xn, lm, held = pd.oc_step(x, dc, dv, 0.2, 2.0, 0.5, target)
    assert held and abs(pd.physical(xn.clone(), 2.0, 0.5) - target) <= 1e-10 * target
