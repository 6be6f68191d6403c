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


def test_records_laid_out_on_every_call_equal_those_laid_out_once():
    """A caller of the C functions who gives no records memory."""
    import ctypes as C

    import convlogic_b200 as cb
    from convlogic_b200 import _lib
    from convlogic_b200.compiled_model import serialise

    torch.manual_seed(3)
    net = cb.ConvLogicCifarModel(k_param=4, input_channels=6).network.cuda()
    for p in net.parameters():
        p.data.normal_()
    x = torch.rand(300, 6, 32, 32, device="cuda") < 0.5
    lib = _lib.lib()
    _lib.check(lib.clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 0))
    try:
        want = cb.CompiledLogicNet(net.eval(), input_shape=(6, 32, 32)).compile()(x)
        blob = serialise(net, input_shape=(6, 32, 32))
        params, handle = torch.empty(len(blob), dtype=torch.uint8, device="cuda"), C.c_void_p()
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(lib.clb_net_create(blob, len(blob), C.c_void_p(params.data_ptr()), stream, C.byref(handle)))
        try:
            ws = torch.empty(lib.clb_net_workspace_bytes(handle, 300), dtype=torch.uint8, device="cuda")
            got = torch.empty_like(want)
            _lib.check(lib.clb_net_forward(handle, 0, C.c_void_p(x.data_ptr()), None, 0, 300, C.c_void_p(got.data_ptr()), C.c_void_p(ws.data_ptr()),
                                           ws.numel(), stream))
            torch.cuda.synchronize()
        finally:
            lib.clb_net_destroy(handle)
    finally:
        _lib.check(lib.clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 1))
    assert torch.equal(got, want)


@pytest.mark.parametrize("batch", [100, 1100])
@pytest.mark.parametrize("kind", ["one channel each", "one pair", "chain", "any pairs"])
@pytest.mark.parametrize("side,c", [(32, 40), (16, 70), (8, 300), (4, 700)])
def test_output_channels_in_an_order_that_shares_planes(side, c, kind, batch):
    """Trails through the graph of input channels: several runs of items per block, records with no, one or two new planes, a run that begins in the
    middle of a trail, output channels that read one input channel only."""
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    ci = 5
    torch.manual_seed(side + c)
    i = torch.arange(c)
    first, second = {"one channel each": (i % ci, i % ci), "one pair": (i * 0 + 1, i * 0 + 3), "chain": (i % ci, (i + 1) % ci),
                     "any pairs": tuple(torch.randint(0, ci, (2, c)))}[kind]
    ch = torch.where(torch.rand(c, 8) < 0.5, first[:, None], second[:, None])
    words = ((ch << 16) | (torch.randint(0, 3, (c, 8)) << 8) | torch.randint(0, 3, (c, 8))).int()
    feat = c * (side // 2) ** 2
    net = torch.nn.Sequential(cb.ConvLogicLayer(ci, c, padding=1, kernel=3, selection=words, complete=True), torch.nn.Flatten(),
                              cb.LogicLayer(feat, feat // 2 * 2), cb.GroupSum(2)).cuda()
    for p in net.parameters():
        p.data.normal_()
    bits = torch.rand(batch, ci, side, side, device="cuda") < 0.5
    with torch.no_grad():
        want = net.eval()(bits.float()).round().long()
    _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 0))
    try:
        assert torch.equal(cb.CompiledLogicNet(net, input_shape=(ci, side, side)).compile()(bits).long(), want)
    finally:
        _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 1))


@pytest.mark.parametrize("kind", ["chain", "any pairs"])
@pytest.mark.parametrize("side,c,batch", [(32, 40, 2300), (32, 40, 2450), (32, 40, 4900), (32, 40, 46000), (16, 70, 5300), (16, 70, 5500), (16, 70, 105000), (8, 300, 4700),
                                          (8, 300, 4900), (8, 300, 91000), (4, 700, 6000), (4, 700, 7000), (4, 700, 126000)])
def test_blocks_of_one_item_and_of_many(side, c, batch, kind):
    """On both sides of the line between a block per item and blocks that go on from item to item (148 SMs), and with several runs of items per block."""
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    ci = 5
    torch.manual_seed(side + c)
    i = torch.arange(c)
    first, second = (i % ci, (i + 1) % ci) if kind == "chain" else tuple(torch.randint(0, ci, (2, c)))
    ch = torch.where(torch.rand(c, 8) < 0.5, first[:, None], second[:, None])
    words = ((ch << 16) | (torch.randint(0, 3, (c, 8)) << 8) | torch.randint(0, 3, (c, 8))).int()
    feat = c * (side // 2) ** 2
    net = torch.nn.Sequential(cb.ConvLogicLayer(ci, c, padding=1, kernel=3, selection=words, complete=True), torch.nn.Flatten(),
                              cb.LogicLayer(feat, feat // 2 * 2), cb.GroupSum(2)).cuda()
    for p in net.parameters():
        p.data.normal_()
    bits = torch.rand(batch, ci, side, side, device="cuda") < 0.5
    net.eval()
    with torch.no_grad():
        want = torch.cat([net(part.float()).round().long() for part in bits.split(10000)])
    _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 0))
    try:
        assert torch.equal(cb.CompiledLogicNet(net, input_shape=(ci, side, side)).compile()(bits).long(), want)
    finally:
        _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 1))
