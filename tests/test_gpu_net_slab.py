"""The 3x3 slab block inside a compiled network (activations in split column order between the stages, feature rows written by the
last block) against the float model in eval mode: class counts, equal to the last one.

Image counts on both sides of a 128-sample slab and of a block's group of slabs (1, 4, 16 and 32 slabs), every side with the
block's input from a thermometer, from booleans and from the previous block; windows on one, two and more channels."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slabs", [1, 3, 4, 5, 16, 17, 33])
@pytest.mark.parametrize("side,ci", [(32, 1), (16, 4), (8, 3), (4, 2)])
def test_slab_blocks_equal_the_float_model(side, ci, slabs):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    torch.manual_seed(side + slabs)
    c = 6
    sel = torch.stack([torch.randint(0, n, (c, 8)) for n in (ci, 3, 3)], -1)
    sel[: c // 2, :, 0] %= 2  # half of the channels on at most two, the others on any
    words = ((sel[..., 0] << 16) | (sel[..., 1] << 8) | sel[..., 2]).int()
    layers = [cb.ConvLogicLayer(ci, c, padding=1, kernel=3, selection=words, complete=True)]
    if side >= 8:
        layers.append(cb.ConvLogicLayer(c, 4, padding=1, kernel=3, complete=True))
    feat = c * 4 if side == 4 else 4 * (side // 4) ** 2
    net = torch.nn.Sequential(*layers, torch.nn.Flatten(), cb.LogicLayer(feat, feat + -feat % 3), cb.GroupSum(3)).cuda()
    for p in net.parameters():
        p.data.normal_()
    compiled = cb.CompiledLogicNet(net.eval(), input_shape=(ci, side, side)).compile()
    batch = slabs * 128 - (slabs % 3) * 37
    px = torch.randint(0, 256, (batch, 1, side, side), device="cuda", dtype=torch.uint8)
    th = torch.rand(ci, device="cuda")
    bits = (px.float() / 255) > th.view(1, ci, 1, 1)
    with torch.no_grad():
        want = net(bits.float()).round().long()
    _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 0))
    try:
        for got in (compiled(bits), compiled.forward_pixels(px, th), compiled.forward_pixels(px.float() / 255, th)):
            assert torch.equal(got.long(), want)
    finally:
        _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 1))
