"""Several right-hand sides in one launch (GPU): every level's apply and Chebyshev modes on a block of
columns, to the bit as the same entry on each column; and the block solve with and without it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solver(dims, coarse=60):
    from loadpath_b200.mg import BoxMesh, GridElasticity
    from oracle import ref_numpy as R

    mesh = BoxMesh(dims)
    fixed = np.zeros(mesh.n_dof, bool)
    fixed[3 * np.flatnonzero(mesh.node_ijk[:, 0] == 0)[:, None] + np.arange(3)] = True
    ge = GridElasticity(mesh, 0.3, fixed, coarse_cells=coarse, dtype=np.float32, element="im")
    ge.set_moduli(R.simp_moduli(R.log_uniform_density(dims, 3)).reshape(-1))
    return ge


@pytest.mark.parametrize("dims", [(32, 16, 16), (29, 14, 11)])
@pytest.mark.parametrize("k", [2, 5])
def test_level_columns_match_single(dims, k):
    ge = _solver(dims)
    kinds = []
    for i, lv in enumerate(ge._op(j) for j in range(len(ge.levels) - 1)):
        assert ge._batched(i, k)
        kinds.append(lv.kind)
        g = lv.grid
        gen = torch.Generator("cuda").manual_seed(i)
        bits = torch.stack([((lv.mask >> c) & 1) for c in range(3)]).float()
        u, b, x, r = (torch.randn((k,) + tuple(bits.shape), device="cuda", generator=gen) * bits for _ in range(4))
        for mode in range(4):
            def run(cols):
                o = [t.clone() for t in (u, b, x, r)]
                out = torch.zeros_like(u)
                uu, bb, xx, rr = o
                for s in ([slice(0, k)] if cols else [slice(j, j + 1) for j in range(k)]):
                    if mode == 0:
                        ge._apply_cols(i, 0, out[s], uu[s])
                    elif mode == 1:
                        ge._apply_cols(i, 1, None, uu[s], x=xx[s], d=uu[s], b=bb[s])
                    elif mode == 2:
                        ge._apply_cols(i, 2, None, xx[s], x=xx[s], r=rr[s], d=uu[s], b=bb[s])
                    else:
                        ge._apply_cols(i, 3, None, uu[s], x=xx[s], r=rr[s], d=uu[s])
                return [out, uu, xx, rr]

            for got, want in zip(run(True), run(False)):
                assert torch.equal(got, want)
        single = torch.zeros_like(u[1])
        lv.apply(single, u[1])
        out = torch.zeros_like(u)
        ge._apply_cols(i, 0, out, u)
        assert torch.equal(out[1], single)
    ge.check_device()
    assert kinds[:2] == ["scaled", "weights"]


def test_block_solve_with_and_without_columns(monkeypatch):
    dims = (32, 16, 16)
    ge = _solver(dims)
    rng = np.random.default_rng(1)
    g = ge.g0
    loads = [g.nodes_to_dev(rng.standard_normal(g.node_shape) * (rng.random(g.node_shape) < 0.01), torch.float64)
             for _ in range(3)]
    xs = ge.solve_block_device(loads)
    its = ge.last_iters
    other = _solver(dims)
    batched = other._batched
    for rule in (lambda i, k: False, lambda i, k: i != 1 and batched(i, k), lambda i, k: i == 1 and batched(i, k)):
        monkeypatch.setattr(other, "_batched", rule)
        other._free_graphs()
        ys = other.solve_block_device(loads)
        assert other.last_iters == its
        for x, y in zip(xs, ys):
            assert torch.equal(x, y)
        other = _solver(dims)
        batched = other._batched
