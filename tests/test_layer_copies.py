"""Layers that have run can be copied, pickled and saved: the plans that the extension keeps on their connection buffers stay behind."""

import copy
import io
import pickle

import pytest
import torch


@pytest.mark.parametrize("kind", ["BlockPlan", "LogicPlan", "PackedOrder"])
def test_a_buffer_with_a_plan_is_copied_without_it(kind):
    from convlogic_b200 import _lib

    plan = getattr(_lib.native(), kind)
    t = torch.arange(6)
    t._clb_plan = plan()
    module = torch.nn.Module()
    module.register_buffer("t", t)

    def saved(obj, **how):
        f = io.BytesIO()
        torch.save(obj, f)
        f.seek(0)
        return torch.load(f, **how)

    for c in (copy.deepcopy(module).t, pickle.loads(pickle.dumps(module)).t, saved(module, weights_only=False).t, saved(t, weights_only=True)):
        assert torch.equal(c, t) and not isinstance(getattr(c, "_clb_plan", None), plan)
    assert isinstance(t._clb_plan, plan)


def _stacks():
    import convlogic_b200 as cb

    torch.manual_seed(0)
    yield cb.ConvLogicCifarModel(k_param=2, input_channels=3, tau=4.0).network, torch.rand(12, 3, 32, 32)
    yield cb.ConvLogicMnistModel(k_param=2, tau=4.0).network, torch.rand(12, 1, 28, 28)
    yield cb.fuse_logic_layers(cb.ConvLogicCifarModel(k_param=2, input_channels=3, tau=4.0).network), torch.rand(12, 3, 32, 32)


@pytest.mark.gpu
def test_stacks_are_copied_and_saved_after_a_training_step():
    for net, x in _stacks():
        net, x = net.cuda().train(), x.cuda()
        want = net(x)
        want.sum().backward()
        f = io.BytesIO()
        torch.save(net, f)
        f.seek(0)
        for other in (copy.deepcopy(net), torch.load(f, weights_only=False)):
            for p in other.parameters():
                p.grad = None
            y = other(x)
            y.sum().backward()
            assert torch.equal(y, want)
            for p, q in zip(net.parameters(), other.parameters()):
                assert torch.equal(p.grad, q.grad)
