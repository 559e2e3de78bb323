"""Level-1 patch cells behind the march in boxes of every shape: thin ones on a face (a warp per node or
per quad of nodes), and whole-grid ones with few patch cells in them (blocks that list the nodes to take), on
grids on both sides of the box size that decides (GPU).

Tolerances as for the smaller boxes: A u differs by the order of its sums, 5e-5 and 1e-13 of the largest entry;
the updates scale that by s dinv or c2 dinv."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fixed(dims, support):
    fixed = np.zeros((3,) + tuple(d + 1 for d in dims), bool)
    if support == "points":
        rng = np.random.default_rng(1)
        for _ in range(30):
            fixed[rng.integers(0, 3), rng.integers(0, dims[0] + 1), rng.integers(0, dims[1] + 1), rng.integers(0, dims[2] + 1)] = True
        fixed[:, 0, 0, 0] = fixed[:, -1, -1, -1] = True
    elif support == "slab":
        fixed[:, :, :, :3] = True
    else:   # faces, each low one of an axis and then its high one
        for k, a in enumerate(support):
            fixed[(slice(None),) + tuple((0, -1)[k] if a == b else slice(None) for b in "xyz")] = True
    return np.moveaxis(fixed.reshape(3, -1), 0, 1).reshape(-1)


@pytest.mark.parametrize("dims", [(128, 128, 64), (136, 40, 50), (257, 129, 63)])
@pytest.mark.parametrize("support", ["x", "y", "z", "xx", "zz", "points", "slab"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_boxes_match_the_general_kernel(dims, support, dtype):
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import stream_handle
    from loadpath_b200.mg import BoxMesh, GridElasticity

    rng = np.random.default_rng(sum(dims))
    ge = GridElasticity(BoxMesh(dims), 0.3, _fixed(dims, support), dtype=dtype, element="im")
    ge.set_moduli(np.exp(rng.uniform(-5, 0, int(np.prod(dims)))))
    lv = ge.levels[1]
    assert lv.kind == "weights" and lv.npatch > 0
    g, L, st, sfx = lv.grid, lib(), stream_handle(), lv._sfx()
    gen = torch.Generator(device="cuda").manual_seed(1)
    bits = torch.stack([((lv.mask >> c) & 1) for c in range(3)]).to(lv.dtype)
    u, b, x0, r0 = (torch.randn(bits.shape, generator=gen, device="cuda", dtype=lv.dtype) * bits for _ in range(4))
    tol = 5e-5 if dtype == np.float32 else 1e-13
    want = lv.apply(torch.zeros_like(u), u, fine_kernel=False)
    top = float(want.abs().max())
    assert float((lv.apply(torch.full_like(u, 7.0), u) - want).abs().max()) <= tol * top
    s, c2, dmax, coef = float(lv.coef[1]), float(lv.coef[3]), float(lv.dinv.abs().max()), lv.coef.data_ptr()
    n, near = u.numel(), lambda p, q, scale: float((p - q).abs().max()) <= 2 * tol * top * scale
    call = lambda name, *a: getattr(L, f"{name}_{sfx}")(*(t.data_ptr() for t in a), coef, n, st)  # noqa: E731
    # mode 1: x = d + (c1 d + c2 dinv (b - A d)); 2: r = b - A x, d = s dinv r; 3: x = (x + d) + (c1 d + c2 dinv (r - A d))
    x, w = torch.zeros_like(u), torch.zeros_like(u)
    lv.level1(1, torch.full_like(u, 7.0), u, x=x, d=u, b=b, coef=coef)
    call("lpb_cheb2_zero", w, b, want, u, lv.dinv)
    assert near(x, w, c2 * dmax)
    r, d, rw, dw = (torch.zeros_like(u) for _ in range(4))
    lv.level1(2, torch.full_like(u, 7.0), u, x=u, r=r, d=d, b=b, coef=coef)
    getattr(L, f"lpb_residual_scaled_{sfx}")(b.data_ptr(), want.data_ptr(), lv.dinv.data_ptr(), coef, rw.data_ptr(),
                                             dw.data_ptr(), n, st)
    assert near(r, rw, 1.0) and near(d, dw, s * dmax)
    x, w = x0.clone(), x0.clone()
    lv.level1(3, torch.full_like(u, 7.0), u, x=x, r=r0, d=u, coef=coef)
    call("lpb_cheb2", w, u, r0, want, lv.dinv)
    assert near(x, w, c2 * dmax)
    ge.check_device()
