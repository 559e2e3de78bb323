"""An explicit apply reads what the launch just before it on the stream wrote, its matrices too (GPU)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(5, 3, 4), (48, 32, 32)])
@pytest.mark.parametrize("noalloc", [False, True])
def test_matrices_written_by_the_launch_ahead(dims, noalloc):
    """kp filled by lpb_cast_f64_f32 right before the apply: the bits of an apply of the finished kp."""
    from loadpath_b200._lib import lib
    from loadpath_b200.grid import DevGrid

    L, st = lib(), torch.cuda.current_stream().cuda_stream
    g = DevGrid(dims)
    u = g.nodes_to_dev(np.random.default_rng(1).standard_normal(g.node_shape), torch.float32)
    mask = torch.full(g.mask_shape, 7, device="cuda", dtype=torch.uint8)
    ncp = g.cell_field(torch.float32).numel()
    kp64 = torch.randn(300, ncp, device="cuda", dtype=torch.float64)
    kp, ft = torch.empty(300, ncp, device="cuda"), torch.empty(24, ncp, device="cuda")

    def apply(out):
        if noalloc:
            L.lpb_apply_explicit_sym_noalloc_f32(out.data_ptr(), u.data_ptr(), kp.data_ptr(), mask.data_ptr(), *g.args, st)
        else:
            L.lpb_apply_explicit_sym_f32(out.data_ptr(), u.data_ptr(), kp.data_ptr(), ft.data_ptr(), mask.data_ptr(),
                                         *g.args, st)
        return out

    kp.copy_(kp64)
    torch.cuda.synchronize()
    want = apply(torch.zeros_like(u))
    torch.cuda.synchronize()
    outs = []
    for _ in range(10):
        kp.fill_(1e6)
        outs.append(torch.zeros_like(u))
        L.lpb_cast_f64_f32(kp.data_ptr(), kp64.data_ptr(), kp.numel(), st)
        apply(outs[-1])
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
