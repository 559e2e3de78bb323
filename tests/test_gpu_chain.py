"""The coarsest level's chain of planes (lp_chain.cu) against numpy on the dense operator the same level
assembles (GPU): planes of odd and even dofs, two to eight segments, segments of unequal length,
one to nine right-hand sides, both field precisions; and the pivot test that hands a level to the band.

Tolerance: these operators' condition numbers are below 1e6 (two ends of the density range in
[1e-3, 1] smoothed and cubed), so a float64 inverse's error is below 1e6 * n * eps ~ 1e-7 in the
worst case and, the rounding errors adding up as a random walk, about 1e6 sqrt(n) eps ~ 1e-8;
float32 fields round the answer at 6e-8."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _level(dims, cc, dtype):
    from loadpath_b200.mg import BoxMesh, GridElasticity
    from oracle import ref_numpy as R

    x = R.log_uniform_density(dims, 7)
    fixed, _ = R.cantilever_bc(dims)
    mesh = BoxMesh(dims)
    fx = np.empty(mesh.n_dof, bool)
    for i in range(3):
        fx[i::3] = fixed[i].reshape(-1)
    ge = GridElasticity(mesh, 0.3, fx, rtol=1e-10, maxiter=3000, coarse_cells=cc, dtype=dtype, element="im")
    ge.set_moduli(R.simp_moduli(x).reshape(-1))
    return ge


def _dense(ge):
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import ptr, stream_handle

    lv = ge.levels[-1]
    gr = lv.grid
    n = 3 * gr.NX * gr.NY * gr.NZ
    a = torch.empty((n, n), dtype=torch.float64, device="cuda")
    f = getattr(lib(), "lpb_coarse_dense_f32" if lv.dtype == torch.float32 else "lpb_coarse_dense_f64")
    if lv.kind == "weights":
        f(a.data_ptr(), 1, lv.w.data_ptr(), lv.mcat.data_ptr(), ptr(lv.patch_id), ptr(lv.patch_k), None,
          lv.mask.data_ptr(), *gr.args, stream_handle())
    else:
        f(a.data_ptr(), 2, None, None, None, None, lv.k.data_ptr(), lv.mask.data_ptr(), *gr.args, stream_handle())
    return a.cpu().numpy()


# fine cells, coarse_cells; the coarsest level's cells: (4, 2, 2), (8, 4, 4), (6, 16, 8), (10, 12, 8), (30, 6, 4)
@pytest.mark.parametrize("dims,cc", [((16, 8, 8), 40), ((16, 8, 8), 200), ((12, 32, 16), 1000), ((20, 24, 14), 1500),
                                     ((60, 12, 8), 1000)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_chain_solve_matches_dense(dims, cc, dtype):
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import stream_handle

    ge = _level(dims, cc, dtype)
    gr = ge.levels[-1].grid
    L = lib()
    plan = np.zeros(5, np.int64)
    words = L.lpb_chain_dims(gr.nx, gr.ny, gr.nz, plan.ctypes.data)
    assert words > 0 and ge._coarse["chain"] is not None and plan[0] >= 2
    dense = _dense(ge)
    sfx, tdt = ("f32", torch.float32) if dtype == np.float32 else ("f64", torch.float64)
    rng = np.random.default_rng(4)
    ws = ge._coarse["chain"]
    for k in (1, 2, 3, 4, 9):
        b = rng.standard_normal((k,) + gr.node_shape).astype(dtype)
        bd = torch.stack([gr.nodes_to_dev(v, tdt) for v in b])
        xd = torch.zeros_like(bd)
        if k == 1:
            getattr(L, f"lpb_chain_solve_{sfx}")(xd.data_ptr(), bd.data_ptr(), ws.data_ptr(), *gr.args, stream_handle())
        else:
            getattr(L, f"lpb_chain_solve_cols_{sfx}")(xd.data_ptr(), bd.data_ptr(), xd[0].numel(), k, ws.data_ptr(),
                                                      *gr.args, stream_handle())
        want = np.linalg.solve(dense, b.astype(np.float64).reshape(k, -1).T).T
        got = np.stack([gr.nodes_to_host(v) for v in xd]).astype(np.float64).reshape(k, -1)
        err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() < (2e-7 if dtype == np.float32 else 1e-8), (k, err)
    # the dense inverse on request, from the same band
    ainv = ge._coarse["ainv"]
    assert ainv.shape[0] >= dense.shape[0] and ge._coarse["ainv"] is ainv


def test_lost_pivots_go_to_the_band():
    """A bar in 1e-9 void, whose coarsest operator is indefinite by rounding: the chain reports it, the
    hierarchy holds the band's inverse instead, and keeps to the band when it is rebuilt."""
    from loadpath_b200.mg import BoxMesh, GridElasticity

    dims = (24, 8, 8)
    fixed = np.zeros((3,) + tuple(d + 1 for d in dims), bool)
    fixed[:, 0] = True
    xp = np.full(dims, 1e-6)
    xp[:, 2:6, 2:6] = 1.0
    xp[10:14, 0, 0] = 1.0
    e = (1e-9 + xp ** 3).reshape(-1)
    mesh = BoxMesh(dims)
    fx = np.moveaxis(fixed.reshape(3, -1), 0, 1).reshape(-1)
    ge = GridElasticity(mesh, 0.3, fx, rtol=1e-10, maxiter=3000, coarse_cells=200, element="im")
    for _ in range(3):
        ge.set_moduli(e)
        assert not ge.strict and ge._coarse["chain"] is None and ge._plan["band"]
        assert [int(v) for v in ge._work["band_info"].cpu()] == [0, 0]


def test_planned_rebuild_leaves_the_chain_when_a_design_breaks_it():
    """A design the chain takes, then (same structure, so a planned rebuild) one it does not, then the
    first again: every build holds its own operator's inverse, to the bits of a build from scratch
    where both hold the band's."""
    from loadpath_b200.mg import BoxMesh, GridElasticity

    dims = (24, 8, 8)
    fixed = np.zeros((3,) + tuple(d + 1 for d in dims), bool)
    fixed[:, 0] = True
    bad = np.full(dims, 1e-6)
    bad[:, 2:6, 2:6] = 1.0
    bad[10:14, 0, 0] = 1.0
    good = np.full(dims, 0.5)
    mesh = BoxMesh(dims)
    fx = np.moveaxis(fixed.reshape(3, -1), 0, 1).reshape(-1)
    f = np.zeros(fixed.shape)
    f[2, -1, 4, 4] = -1.0
    fm = np.moveaxis(f.reshape(3, -1), 0, 1).reshape(-1)
    ge = GridElasticity(mesh, 0.3, fx, rtol=1e-10, maxiter=3000, coarse_cells=200, element="im")
    ref = GridElasticity(mesh, 0.3, fx, rtol=1e-10, maxiter=3000, coarse_cells=200, element="im")
    chains = []
    for x in (good, bad, good):
        e = (1e-9 + x ** 3).reshape(-1)
        ge.set_moduli(e)
        chains.append(ge._coarse["chain"] is not None)
        ref._plan = None
        ref.set_moduli(e)
        if x is bad:
            assert torch.equal(ge._coarse["ainv"], ref._coarse["ainv"])
        else:
            c = [float(fm @ s.solve_many([fm])[0]) for s in (ge, ref)]
            assert abs(c[0] - c[1]) <= 1e-9 * abs(c[1])
    assert chains == [True, False, False]     # the plan keeps to the band from there on
