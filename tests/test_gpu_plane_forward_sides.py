"""The plane forward at 32, 28, 12 and 6 pixels (pairs of pooled rows of one image; rows of 28 or 24 of 32 lanes; a last turn that is
half empty) against the general kernel, bit for bit: ragged batches, one image, feature-major output, selections on three channels."""

import pytest
import torch

pytestmark = pytest.mark.gpu
GEOM = (1, 1, 1, 1, 3, 3)


@pytest.mark.parametrize("n,ci,c,side", [(1, 16, 5, 32), (9, 20, 3, 32), (300, 16, 2, 32), (7, 16, 4, 28), (1, 30, 2, 28), (1, 16, 7, 12), (35, 16, 3, 12),
                                         (130, 40, 9, 12), (1, 16, 3, 6), (37, 48, 10, 6), (300, 20, 4, 6)])
@pytest.mark.parametrize("spread", [False, True])
def test_plane_forward_sides(n, ci, c, side, spread):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib, ops
    from convlogic_b200._lib import W_SOFTMAX

    torch.manual_seed(n + side)
    sel = cb.ConvLogicLayer(ci, c, padding=1, complete=True).selection.clone().cuda()
    if spread:
        sel[0, 3] = (sel[0, 3] & 0xFFFF) | ((ci - 1) << 16)
        sel[0, 5] = (sel[0, 5] & 0xFFFF) | ((ci // 2) << 16)
    x, w = torch.rand(n, ci, side, side, device="cuda"), torch.randn(c, 7, 16, device="cuda")
    x = (x * 4).round() / 4  # ties between pooled positions
    want, amax_want, _, _, _ = ops.convtree_fwd(x, w, sel, GEOM, W_SOFTMAX, want_indices=True)
    _lib.trace(True)
    y, amax, _, _, _ = ops.convtree_fwd(x, w, sel, GEOM, W_SOFTMAX)
    torch.cuda.synchronize()
    rep = _lib.trace_report()
    _lib.trace(False)
    assert "convtree_fwd_plane_kernel" in rep, rep
    assert torch.equal(y, want) and torch.equal(amax, amax_want)
    fm = ops.convtree_fwd(x, w, sel, GEOM, W_SOFTMAX, y_feature_major=True)[0]
    assert torch.equal(fm, want)


@pytest.mark.parametrize("n,ci,c,side,plane", [(9, 9, 12, 32, False), (17, 5, 8, 28, False), (300, 8, 70, 12, False), (300, 4, 64, 16, False),
                                               (9, 18, 12, 32, True), (40, 8, 9, 6, True), (9, 15, 5, 28, True)])
def test_selections_on_many_channels_take_the_tiled_kernels_while_there_are_few(n, ci, c, side, plane):
    from convlogic_b200 import _lib, ops
    from convlogic_b200._lib import W_SOFTMAX

    torch.manual_seed(n + side)
    ch = torch.randint(0, ci, (c, 8))
    ch[:, :3] = torch.tensor([0, 1, 2])
    sel = ((ch << 16) | (torch.randint(0, 3, (c, 8)) << 8) | torch.randint(0, 3, (c, 8))).int().cuda()
    x, w = torch.rand(n, ci, side, side, device="cuda"), torch.randn(c, 7, 16, device="cuda")
    want, amax_want, _, _, _ = ops.convtree_fwd(x, w, sel, GEOM, W_SOFTMAX, want_indices=True)
    _lib.trace(True)
    y, amax, _, _, _ = ops.convtree_fwd(x, w, sel, GEOM, W_SOFTMAX)
    torch.cuda.synchronize()
    rep = _lib.trace_report()
    _lib.trace(False)
    assert ("convtree_fwd_plane_kernel" in rep) == plane, rep
    assert torch.equal(y, want) and torch.equal(amax, amax_want)
    assert torch.equal(ops.convtree_fwd(x, w, sel, GEOM, W_SOFTMAX, y_feature_major=True)[0], want)
