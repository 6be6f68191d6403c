"""The compiled network's one-launch kernel against the layer-by-layer launches: whole numbers, equal to the last one.

Sizes where it can go wrong: batches around a 128-sample slab and around the points where the cluster gets smaller, halos and
none, stride 2, features that are not a multiple of four, more than one flat layer, fused and not."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def one_launch():
    from convlogic_b200 import _lib

    def tune(v):
        _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, v))

    yield tune
    tune(1)


def _nets():
    import convlogic_b200 as cb

    yield "mnist", cb.ConvLogicMnistModel(k_param=2).network, (1, 28, 28), 1, True
    yield "cifar", cb.ConvLogicCifarModel(k_param=2, input_channels=6, input_size=16).network, (6, 16, 16), 2, True
    flat = torch.nn.Sequential(cb.LogicLayer(37, 90), cb.LogicLayer(90, 70), cb.LogicLayer(70, 70), cb.GroupSum(7))
    yield "flat", flat, None, 0, False
    odd = torch.nn.Sequential(cb.ConvLogicLayer(3, 5, stride=2, padding=1, complete=True), cb.ConvLogicLayer(5, 6, padding=0, kernel=2, complete=True),
                              torch.nn.Flatten(), cb.LogicLayer(54, 60), cb.LogicLayer(60, 30), cb.GroupSum(10))
    yield "odd", odd, (3, 28, 28), 3, False


@pytest.mark.parametrize("batch", [1, 31, 128, 129, 900, 2000, 5000])
def test_one_launch_equals_layer_launches(one_launch, batch):
    import convlogic_b200 as cb

    torch.manual_seed(batch)
    for name, net, shape, levels, fuse in _nets():
        for p in net.parameters():
            p.data.normal_()
        compiled = cb.CompiledLogicNet(net.eval(), input_shape=shape, fuse=fuse).compile()
        x = torch.rand(batch, *(shape or (37,)), device="cuda") < 0.4
        one_launch(0)
        want = compiled(x)
        one_launch(2)
        assert torch.equal(compiled(x), want), (name, batch)
        if levels:
            th = torch.tensor([0.5, 0.25, 0.75][:levels], device="cuda")
            px = torch.randint(0, 256, (batch, shape[0] // levels, *shape[1:]), device="cuda", dtype=torch.uint8)
            for pixels in (px, px.float() / 255):
                one_launch(0)
                want = compiled.forward_pixels(pixels, th)
                one_launch(2)
                assert torch.equal(compiled.forward_pixels(pixels, th), want), (name, batch, pixels.dtype)


def test_one_channel_image_of_more_than_65536_pixels():
    """The smallest square whose pixel count does not divide exactly by the kernel's multiplication runs layer by layer, whatever the switch."""
    import convlogic_b200 as cb

    torch.manual_seed(5)
    net = torch.nn.Sequential(cb.ConvLogicLayer(1, 3, stride=2, complete=True), torch.nn.Flatten(), cb.LogicLayer(3 * 65 * 65, 6400), cb.GroupSum(10))
    for p in net.parameters():
        p.data.normal_()
    x = torch.rand(40, 1, 260, 260, device="cuda") < 0.4
    got = cb.CompiledLogicNet(net.eval(), input_shape=(1, 260, 260)).compile()(x)
    with torch.no_grad():
        assert torch.equal(got, net.cuda()(cb.PackBitsTensor(x, 64)))


@pytest.mark.parametrize("batch", [32, 33, 64, 65, 96, 127, 224, 225, 256, 257, 448, 449, 512, 1025])
def test_slabs_of_every_size(one_launch, batch):
    """Batches around the slabs of 32, 64 and 128 samples and around the points where the choice between them changes."""
    import convlogic_b200 as cb

    torch.manual_seed(batch)
    net = cb.ConvLogicMnistModel(k_param=2).network
    for p in net.parameters():
        p.data.normal_()
    compiled = cb.CompiledLogicNet(net.eval(), input_shape=(1, 28, 28)).compile()
    x = torch.rand(batch, 1, 28, 28, device="cuda") < 0.4
    one_launch(0)
    want = compiled(x)
    one_launch(2)
    assert torch.equal(compiled(x), want)
