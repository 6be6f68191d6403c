"""The layers inside what torch puts around a module: parametrized weights, traces, forward-mode AD, saved-tensor hooks, undefined
gradients, CUDA graph capture.  The autograd nodes are C++, so none of this comes by itself."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _flat():
    import convlogic_b200 as cb

    torch.manual_seed(0)
    return cb.LogicLayer(64, 96).cuda().train(), torch.rand(33, 64, device="cuda")


def _block():
    import convlogic_b200 as cb

    torch.manual_seed(0)
    return cb.ConvLogicLayer(3, 16, complete=True).cuda().train(), torch.rand(8, 3, 16, 16, device="cuda")


def _trees():
    import convlogic_b200 as cb

    torch.manual_seed(0)
    net = torch.nn.Sequential(cb.LogicLayer(64, 160), cb.LogicLayer(160, 80), cb.LogicLayer(80, 40))
    return cb.fuse_logic_layers(net.cuda())[0].train(), torch.rand(36, 64, device="cuda")


MADE = {"flat": _flat, "block": _block, "trees": _trees}


def _weights(m):
    return list(m.parameters())


def _step(m, x):
    x = x.detach().requires_grad_(True)
    y = m(x)
    g = torch.autograd.grad(y.sum(), [x] + _weights(m))
    return [y.detach(), *g]


class _Twice(torch.nn.Module):
    def forward(self, w):
        return w * 2


@pytest.mark.parametrize("kind", MADE)
def test_parametrized_weights(kind):
    import torch.nn.utils.parametrize as parametrize

    m, x = MADE[kind]()
    plain, _ = MADE[kind]()
    for p in plain.parameters():
        p.data *= 2
    want = _step(plain, x)
    for l in (m.layers if kind == "trees" else [m]):
        parametrize.register_parametrization(l, "weights", _Twice())
    got = _step(m, x)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    for a, b in zip(got[2:], want[2:]):
        assert torch.equal(a, 2 * b)
