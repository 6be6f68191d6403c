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


class _Loss(torch.nn.Module):
    def __init__(self, trees):
        super().__init__()
        self.trees = trees

    def forward(self, x):
        return self.trees.cross_entropy(x, torch.arange(x.shape[0], device="cuda") % 4, 4, 2.0)


def _followed_cases():
    import convlogic_b200 as cb

    for kind in MADE:
        m, x = MADE[kind]()
        yield kind, m, x
    m, x = _flat()
    yield "class sums", torch.nn.Sequential(m, cb.GroupSum(4, 2.0)), x
    m, x = _trees()
    yield "loss", _Loss(m), x


@pytest.mark.parametrize("train", [True, False])
def test_traces_follow_the_input(train):
    for name, m, x in _followed_cases():
        m.train(train)
        traced = torch.jit.trace(m, (x,), check_trace=False)
        other = 1 - x
        assert torch.equal(traced(other), m(other)), name
        assert not torch.equal(m(other), m(x)), name
        if train:
            a, b = (torch.autograd.grad(f(other).sum(), _weights(m)) for f in (traced, m))
            assert all(torch.allclose(p, q, rtol=1e-5, atol=1e-7) for p, q in zip(a, b)), name  # the general kernels' order of additions


def test_a_tangent_is_refused_and_not_dropped():
    import torch.autograd.forward_ad as fwad

    for name, m, x in _followed_cases():
        with fwad.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
            m(fwad.make_dual(x, torch.ones_like(x)))
    m, x = _flat()
    w = m.weights.detach()
    del m.weights
    with fwad.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
        m.weights = fwad.make_dual(w, torch.ones_like(w))
        m(x)


@pytest.mark.parametrize("kind", MADE)
def test_functorch_transforms_are_refused(kind):
    m, x = MADE[kind]()
    with pytest.raises(RuntimeError):
        torch.func.vmap(m)(torch.stack([x, x]))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: m(t).sum())(x)


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y):
        return y.sum()

    @staticmethod
    def backward(ctx, g):
        return None


def test_no_upstream_gradient_is_a_gradient_of_zeros():
    import convlogic_b200 as cb

    for name, m, x in _followed_cases():
        x.requires_grad_(True)
        _NoGradient.apply(m(x)).backward()
        for t in [x] + _weights(m):
            assert t.grad is not None and not t.grad.any(), name
        bucket = cb.GradBucket(m).direct()
        m(x).sum().backward()
        assert bucket.flat.any(), name
        _NoGradient.apply(m(x)).backward()
        assert not bucket.flat.any(), name   # not the step before's
        bucket.direct(False)


def test_saved_tensor_hooks_see_what_a_call_keeps():
    for name, m, x in _followed_cases():
        want = _step(m, x)
        kept = []

        def pack(t):
            kept.append((t.dtype, tuple(t.shape)))
            return t.cpu()

        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
            xr = x.detach().requires_grad_(True)
            y = m(xr)
        got = [y.detach(), *torch.autograd.grad(y.sum(), [xr] + _weights(m))]
        assert all(torch.equal(a, b) for a, b in zip(got, want)), name
        extra = {"block": (torch.uint8, (8, 16, 8, 8)), "loss": (torch.float32, (36, 4))}.get(name)   # arg-max bytes, score gradient
        assert extra is None or extra in kept, (name, kept)
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(y.sum(), _weights(m))


def test_the_first_step_of_a_flat_layer_may_be_captured():
    m, x = _flat()
    want = _step(_flat()[0], x)
    x.requires_grad_(True)
    go = torch.ones(33, 96, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = m(x)
        g = torch.autograd.grad(y, [x, m.weights], go)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want[0])
    # The separate kernels add in another order.  A basis sum has 33 terms of at most 1: any two orders agree to 2 * 32 * 33 * 2^-24 = 1.3e-4,
    # and a gate gradient, p (g - sum p g) with g of up to four basis sums, to 8 times that; in practice 2e-6.
    for a, b in zip(g, want[1:]):
        assert (a - b).abs().max() < 1e-3 and (a - b).norm() < 1e-5 * b.norm()
    again = _step(m, x)                                  # and the layer lays its lists out afterwards
    assert all(torch.equal(a, b) for a, b in zip(again, want))


def test_connections_made_in_inference_mode_get_no_plan():
    """Such a tensor has no version, so a plan of it could not be told from an outdated one."""
    with torch.inference_mode():
        flat, x = _flat()
        assert flat(x).shape == (33, 96)      # no plan needed
        block, img = _block()
        with pytest.raises(RuntimeError, match="[Ii]nference"):
            block(img)
    flat.weights = torch.nn.Parameter(flat.weights.clone())
    x = x.clone().requires_grad_(True)
    with pytest.raises(RuntimeError, match="[Ii]nference"):
        flat(x)
