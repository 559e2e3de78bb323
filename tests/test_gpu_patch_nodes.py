"""Level-1 patch cells in a launch behind the march (with scratch given) against the same cells in the
march (without): supports on each face, whose boxes start and end inside chunks of four planes, and
scattered ones (GPU).

Tolerances: A u differs by the order of its sums, 5e-5 and 1e-13 of the largest entry (as derived for
the march against the general kernel); the updates scale that by s dinv or c2 dinv."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(32, 16, 12), (30, 22, 26)])
@pytest.mark.parametrize("support", ["x", "y", "z", "zmid", "inside"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_apart_matches_in_march(dims, support, dtype):
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import ptr, stream_handle
    from loadpath_b200.mg import BoxMesh, GridElasticity
    from oracle import ref_numpy as R

    rng = np.random.default_rng(sum(dims))
    fixed = np.zeros((3,) + tuple(d + 1 for d in dims), bool)
    if support == "inside":
        fixed[:, 0] = True
        fixed |= rng.random(fixed.shape) < 0.01
    elif support == "zmid":
        fixed[:, 3:9, 2:7, 5] = True
    else:
        fixed[(slice(None),) + tuple(0 if a == support else slice(None) for a in "xyz")] = True
    fx = np.moveaxis(fixed.reshape(3, -1), 0, 1).reshape(-1)
    ge = GridElasticity(BoxMesh(dims), 0.3, fx, coarse_cells=dims[0] * dims[1] * dims[2] // 9 + 1, dtype=dtype,
                        element="im")
    ge.set_moduli(R.simp_moduli(R.log_uniform_density(dims, 3)).reshape(-1))
    lv = ge.levels[1]
    assert lv.kind == "weights" and lv.npatch > 0
    g, L, st = lv.grid, lib(), stream_handle()
    bits = torch.stack([((lv.mask >> c) & 1) for c in range(3)]).to(lv.dtype)
    u, b, x0, r0 = (g.nodes_to_dev(rng.standard_normal(g.node_shape), lv.dtype) * bits for _ in range(4))
    fn = L.lpb_apply_level1_f32 if dtype == np.float32 else L.lpb_apply_level1_f64

    def run(mode, out):
        x, r, d = (u.clone() if mode == 2 else x0.clone()), r0.clone(), (u.clone() if mode != 2 else r0.clone())
        src = x if mode == 2 else d
        assert fn(mode, ptr(out), x.data_ptr(), r.data_ptr(), d.data_ptr(), src.data_ptr(), b.data_ptr(),
                  lv.dinv.data_ptr(), lv.coef.data_ptr(), lv.wc.data_ptr(), lv.patch_id.data_ptr(),
                  lv.patch_m.data_ptr(), lv.patch_k.data_ptr(), lv.mask.data_ptr(), lv.g1.ctypes.data,
                  lv.pbox.ctypes.data, lv.err.data_ptr(), *g.args, st) == 0
        return x, r, d

    tol = 5e-5 if dtype == np.float32 else 1e-13
    au = torch.zeros_like(u)
    lv.apply(au, u)
    want = lv.apply(torch.zeros_like(u), u, fine_kernel=False)
    top = float(want.abs().max())
    assert float((au - want).abs().max()) <= tol * top
    s, c2 = float(lv.coef[1]), float(lv.coef[3])
    dmax = float(lv.dinv.abs().max())
    for mode in (1, 2, 3):
        scratch = torch.full_like(u, 7.0)
        apart, march = run(mode, scratch), run(mode, None)
        ge.check_device()
        for name, p, q in zip("xrd", apart, march):
            scale = {1: {"x": c2 * dmax}, 2: {"r": 1.0, "d": s * dmax}, 3: {"x": c2 * dmax}}[mode].get(name, 0.0)
            assert float((p - q).abs().max()) <= 2 * tol * top * scale, (mode, name)
