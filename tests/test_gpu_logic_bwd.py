"""The flat layer's combined backward against autograd through the CPU oracle in fp64: batches around the 32- and 64-sample
stretches (rows of 16-byte units and odd ones), one and many consumers per feature, features nobody reads, a neuron that
reads one feature twice, and sizes on both sides of the dispatch (few and many feature groups)."""

import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fin,fout,batch", [(5, 9, 1), (33, 20, 31), (40, 700, 32), (257, 130, 33), (64, 64, 100), (300, 300, 65),
                                            (12, 4000, 36), (3000, 3100, 512), (3001, 2800, 511), (20000, 21000, 64), (19500, 19500, 3)])
def test_combined_backward_against_oracle(fin, fout, batch):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    g = torch.Generator().manual_seed(fin + batch)
    layer = cb.LogicLayer(fin, fout)
    a, b = torch.randint(0, fin, (fout,), generator=g), torch.randint(0, fin, (fout,), generator=g)
    b[0] = a[0]  # both inputs the same feature
    layer.indices_0, layer.indices_1 = a, b
    layer.given_x_indices_of_y_start, layer.given_x_indices_of_y = layer.build_consumer_lists(a, b, fin)
    w = torch.randn(fout, 16, generator=g)
    layer.weights.data = w.clone()
    x, gy = torch.rand(batch, fin, generator=g), torch.randn(batch, fout, generator=g)
    layer = layer.cuda().train()
    xd = x.cuda().requires_grad_(True)
    _lib.trace(True)
    y = layer(xd)
    y.backward(gy.cuda())
    kernels = _lib.trace_report()
    _lib.trace(False)
    assert "logic_bwd_kernel" in kernels, kernels
    xo, wo = x.double().requires_grad_(True), w.double().requires_grad_(True)
    yo = oracle.logic_layer(xo, a, b, oracle.gate_probabilities(wo, True))
    yo.backward(gy.double())

    def close(got, want):
        return float((got.cpu().double() - want).abs().max() / want.abs().max().clamp_min(1e-30)) <= 1e-5

    assert close(y.detach(), yo.detach()) and close(xd.grad, xo.grad) and close(layer.weights.grad, wo.grad)
    first = layer.weights.grad.clone(), xd.grad.clone()
    layer.weights.grad = xd.grad = None
    layer(xd).backward(gy.cuda())
    assert torch.equal(first[0], layer.weights.grad) and torch.equal(first[1], xd.grad)  # a fixed summation order


def test_large_activation_forward_walks_in_stretches():
    """Above the size at which the forward takes column stretches its values are those of the plain kernel."""
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    torch.manual_seed(0)
    layer = cb.LogicLayer(66000, 33001).cuda().train()
    x = torch.rand(260, 66000, device="cuda")
    _lib.trace(True)
    y = layer(x.clone().requires_grad_(True)).detach()
    assert "logic_fwd_cols_kernel" in _lib.trace_report()
    _lib.trace(False)
    small = layer(x[:128].contiguous())
    assert float((y[:128] - small).abs().max()) <= 1e-6


@pytest.mark.parametrize("fin,fout,batch,both,alone", [(1000, 1500, 512, False, False), (1000, 1500, 508, True, True), (500, 600, 512, True, True),
                                                       (1000, 1500, 514, True, True), (200, 6500, 128, True, True), (900, 30000, 512, False, False),
                                                       (3000, 97000, 256, True, False), (140000, 90000, 380, False, False), (140000, 90000, 384, True, False),
                                                       (140000, 140000, 300, True, False), (140000, 90000, 381, False, False)])
def test_combined_or_separate_backward_by_size(fin, fout, batch, both, alone):
    """Both sides of the lines of the choice, with and without a gate gradient, against the separate kernels."""
    import convlogic_b200 as cb
    from convlogic_b200 import _lib, ops
    from convlogic_b200._lib import W_SOFTMAX

    torch.manual_seed(batch)
    layer = cb.LogicLayer(fin, fout).cuda().train()
    layer.weights.data.normal_()
    x, gy = torch.rand(fin, batch, device="cuda"), torch.randn(fout, batch, device="cuda")
    tables = (layer.indices_0, layer.indices_1, layer.weights.detach())
    want_x = ops.logic_bwd_x(x, *tables, gy, layer.given_x_indices_of_y_start, layer.given_x_indices_of_y, W_SOFTMAX)
    want_w = ops.logic_bwd_w(x, *tables, gy, W_SOFTMAX)
    for gates, combined in ((True, both), (False, alone)):
        layer.weights.requires_grad_(gates)
        xd = x.t().detach().requires_grad_(True)
        y = layer(xd)
        _lib.trace(True)
        got = torch.autograd.grad(y, [xd] + ([layer.weights] if gates else []), gy.t())
        torch.cuda.synchronize()
        names = _lib.trace_report()
        _lib.trace(False)
        assert ("logic_bwd_kernel" in names) == combined and ("logic_bwd_x_kernel" in names) == (not combined), names
        # the same terms in another order: sums over a feature's readers, over the samples and of four basis sums
        assert (got[0].t() - want_x).norm() <= 1e-5 * want_x.norm()
        if gates:
            assert (got[1] - want_w).norm() <= 1e-5 * want_w.norm()
