"""The plane backward at every side it takes (32 and 28: four warps per image; 12 and 6: two and three images per warp, idle lanes), against
the CPU oracle at the kernels' own pooled positions: ragged batches, one image, parts of the batch, channels whose taps all name
one plane, an upstream gradient in the flat layers' layout (the same bits as for the ordinary one)."""

import pytest
import torch

import oracle
from tests.util import assert_close

pytestmark = pytest.mark.gpu
GEOM = (1, 1, 1, 1, 3, 3)


@pytest.mark.parametrize("n,ci,c,side", [(1, 16, 5, 32), (9, 20, 3, 32), (5, 4, 2, 32), (40, 16, 4, 28), (1, 17, 2, 28), (1, 16, 7, 12), (35, 16, 3, 12),
                                         (130, 40, 2, 12), (1, 12, 3, 6), (38, 48, 10, 6), (300, 20, 4, 6),
                                         (3, 4, 6, 16), (17, 4, 3, 8), (9, 4, 5, 4)])
def test_plane_backward_sides(n, ci, c, side):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib, ops
    from convlogic_b200._lib import W_SOFTMAX

    torch.manual_seed(n + side)
    sel = cb.ConvLogicLayer(ci, c, padding=1, complete=True).selection.clone()
    sel[0] = (sel[0] & 0xFFFF) | (2 << 16)  # all taps of the first output channel on one plane
    x, logits, gy = torch.rand(n, ci, side, side), torch.randn(c, 7, 16), torch.randn(n, c, side // 2, side // 2)
    xd, wd, sd, gd = x.cuda(), logits.cuda(), sel.cuda(), gy.cuda()
    _, amax, _, _, idx = ops.convtree_fwd(xd, wd, sd, GEOM, W_SOFTMAX, want_indices=True)
    _lib.trace(True)
    gx, gw = ops.convtree_bwd(gd, xd, wd, sd, amax, GEOM, W_SOFTMAX)
    torch.cuda.synchronize()
    rep = _lib.trace_report()
    _lib.trace(False)
    assert "convtree_bwd_plane_kernel" in rep, rep
    xo, wo = x.clone().requires_grad_(True), logits.clone().requires_grad_(True)
    yf = oracle.full_convlogic(xo, oracle.gate_probabilities(wo, True), sel, forced_idx=idx.cpu())[0]
    gxo, gwo = torch.autograd.grad((yf * gy).sum(), (xo, wo))
    assert_close(gx, gxo, 1e-5, "gx vs oracle")
    assert_close(gw, gwo, 1e-5, "gw vs oracle")
    fm = gd.permute(1, 2, 3, 0).contiguous().permute(3, 0, 1, 2)
    gx2, gw2 = ops.convtree_bwd(fm, xd, wd, sd, amax, GEOM, W_SOFTMAX)
    assert torch.equal(gx, gx2) and torch.equal(gw, gw2)


def test_sliced_batch_equals_one_slice():
    """Gradient planes above 1 GB: the batch in two slices, the second ragged."""
    import convlogic_b200 as cb
    from convlogic_b200 import ops
    from convlogic_b200._lib import W_SOFTMAX

    torch.manual_seed(0)
    n, ci, c, side = 140, 8, 1000, 32   # 8.2 MB of planes per image
    sel = cb.ConvLogicLayer(ci, c, padding=1, complete=True).selection.clone().cuda()
    x, w = torch.rand(n, ci, side, side, device="cuda"), torch.randn(c, 7, 16, device="cuda")
    gy = torch.randn(n, c, side // 2, side // 2, device="cuda")
    _, amax, *_ = ops.convtree_fwd(x, w, sel, GEOM, W_SOFTMAX)
    gx, gw = ops.convtree_bwd(gy, x, w, sel, amax, GEOM, W_SOFTMAX)
    half = [ops.convtree_bwd(gy[s], x[s], w, sel, amax[s], GEOM, W_SOFTMAX) for s in (slice(0, 70), slice(70, n))]
    assert torch.equal(gx, torch.cat([g for g, _ in half]))
    assert_close(gw, half[0][1] + half[1][1], 2e-5, "gw")
