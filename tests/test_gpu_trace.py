"""The launch trace names every launch that the library counts, those that lay plans out included."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(batch):
    import convlogic_b200 as cb

    net = cb.fuse_logic_layers(cb.ConvLogicCifarModel(k_param=2, input_channels=3, tau=4.0).network).cuda().train()
    x, labels = torch.rand(batch, 3, 32, 32, device="cuda"), torch.randint(0, 10, (batch,), device="cuda")
    return lambda: net[-2].cross_entropy(net[:-2](x), labels, net[-1].k, net[-1].tau).backward()


def _flat():
    import convlogic_b200 as cb

    layer = cb.LogicLayer(100000, 100000).cuda().train()
    x = torch.rand(320, 100000, device="cuda", requires_grad=True)
    return lambda: layer(x).sum().backward()


def _packed():
    import convlogic_b200 as cb

    layer = cb.LogicLayer(30000, 30000).cuda().eval()
    x = cb.PackBitsTensor(torch.rand(2000, 30000, device="cuda") < 0.5, 32)
    return lambda: layer(x)


def _compiled():
    import convlogic_b200 as cb

    net = cb.ConvLogicCifarModel(k_param=64, input_channels=3, tau=4.0).network.eval()
    x = torch.rand(300, 3, 32, 32, device="cuda") < 0.5
    return lambda: cb.CompiledLogicNet(net, input_shape=(3, 32, 32)).compile()(x)


@pytest.mark.parametrize("call", [lambda: _step(32), lambda: _step(33), _flat, _packed, _compiled], ids=["step 32", "step 33", "flat", "packed", "compiled"])
def test_every_launch_is_traced(call):
    from convlogic_b200 import _lib

    torch.manual_seed(0)
    run = call()
    for _ in range(2):   # the first call lays out what it needs
        _lib.trace(True)
        before = _lib.lib().clb_kernel_launches()
        run()
        torch.cuda.synchronize()
        counted = _lib.lib().clb_kernel_launches() - before
        names = _lib.trace_report()
        _lib.trace(False)
        assert counted > 0 and sum(n for n, _ in names.values()) == counted, names
