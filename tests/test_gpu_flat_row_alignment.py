"""Flat layers on rows whose length leaves them 16-, 8- or 4-byte aligned, around the accesses that a lane has in flight, against a
double-precision restatement (outputs and both gradients, fp32)."""

import pytest
import torch

from tests.util import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 2, 31, 62, 63, 65, 66, 127, 128, 129, 130, 257, 258])
@pytest.mark.parametrize("in_dim,out_dim", [(40, 70), (3000, 5000)])
def test_flat_layer_rows_of_any_alignment(batch, in_dim, out_dim):
    import convlogic_b200 as cb

    torch.manual_seed(batch)
    first, layer = cb.LogicLayer(in_dim, out_dim).cuda(), cb.LogicLayer(out_dim, out_dim).cuda()
    x = torch.rand(batch, in_dim, device="cuda", requires_grad=True)
    gy = torch.randn(batch, out_dim, device="cuda")
    y = layer(first(x))
    gx, g1, g2 = torch.autograd.grad(y, (x, first.weights, layer.weights), gy)
    xo = x.detach().double().cpu().requires_grad_(True)
    h, ws = xo, []
    for m in (first, layer):
        w = m.weights.detach().double().cpu().requires_grad_(True)
        ws.append(w)
        a, b = h[:, m.indices_0.cpu()], h[:, m.indices_1.cpu()]
        h = sum(p * f for p, f in zip(torch.softmax(w, -1).unbind(-1), oracle_gates(a, b)))
    gxo, g1o, g2o = torch.autograd.grad(h, (xo, *ws), gy.double().cpu())
    assert_close(y, h, 1e-5, "y")
    assert_close(gx, gxo, 1e-5, "gx")
    assert_close(g1, g1o, 1e-5, "first gates")
    assert_close(g2, g2o, 1e-5, "second gates")


@pytest.mark.parametrize("batch", [1, 14, 68, 131])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float64, 1e-12)])
def test_gate_gradient_of_more_neurons_than_half_warps(batch, dtype, tol):
    """The first layer of a network (no input gradient); a half-warp takes two or three neurons in turn, the last ones none."""
    import convlogic_b200 as cb

    torch.manual_seed(batch)
    layer = cb.LogicLayer(50, 21001).to("cuda", dtype)
    x, gy = torch.rand(batch, 50, device="cuda", dtype=dtype), torch.randn(batch, 21001, device="cuda", dtype=dtype)
    (gw,) = torch.autograd.grad(layer(x), layer.weights, gy)
    w, xo = layer.weights.detach().double().cpu().requires_grad_(True), x.double().cpu()
    gates = oracle_gates(xo[:, layer.indices_0.cpu()], xo[:, layer.indices_1.cpu()])
    (gwo,) = torch.autograd.grad(sum(p * f for p, f in zip(torch.softmax(w, -1).unbind(-1), gates)), w, gy.double().cpu())
    assert_close(gw, gwo, tol, "gates")


@pytest.mark.parametrize("batch", [1, 2, 3, 5, 255, 1022, 1025, 4095, 4097])
@pytest.mark.parametrize("per_class", [1, 3, 5003])
def test_class_sum_gradient_rows_of_any_alignment(batch, per_class):
    """Rows that are not whole 16-byte words: every chunk's first words, its last ones and the wrap from a row to the next."""
    import convlogic_b200 as cb

    k = 3
    x = torch.zeros(k * per_class, batch, device="cuda").t().requires_grad_(True)
    g = torch.randn(batch, k, device="cuda")
    (gx,) = torch.autograd.grad(cb.GroupSum(k, tau=3.5)(x), x, g)
    assert torch.equal(gx, (g / torch.tensor(3.5, device="cuda")).repeat_interleave(per_class, 1))


def oracle_gates(a, b):
    """The sixteen gates as real-valued functions, in the order of their truth tables."""
    one, ab = torch.ones_like(a), a * b
    terms = [(0, 0, 0, 0), (0, 0, 0, 1), (0, 1, 0, -1), (0, 1, 0, 0), (0, 0, 1, -1), (0, 0, 1, 0), (0, 1, 1, -2), (0, 1, 1, -1)]
    half = [k * one + p * a + q * b + r * ab for k, p, q, r in terms]
    return half + [one - g for g in reversed(half)]


@pytest.mark.parametrize("n_in,n_out,batch,walk", [(66000, 66002, 256, True), (33000, 33300, 520, False), (75000, 65000, 256, False), (17000, 17008, 1004, True),
                                                   (35000, 35007, 500, False)])
@pytest.mark.parametrize("train", [False, True])
def test_large_forwards_without_a_gradient(n_in, n_out, batch, walk, train):
    """The walk in stretches is chosen by the layer's size, not by whether a gradient follows; both against the gate polynomial in 64 bits."""
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    torch.manual_seed(batch)
    layer = cb.LogicLayer(n_in, n_out).cuda().train(train)
    layer.weights.data.normal_()
    x = torch.rand(n_in, batch, device="cuda").t()
    assert (_lib.lib().clb_logic_fwd_scratch_bytes(n_in, n_out, batch, 0) > 0) == walk
    with torch.no_grad():
        _lib.trace(True)
        y = layer(x)
        torch.cuda.synchronize()
        names = _lib.trace_report()
        _lib.trace(False)
    assert ("logic_fwd_cols_kernel" in names) == walk, names
    pick = torch.randint(0, n_out, (500,), device="cuda")
    p = layer.weights[pick].detach().double()
    p = p.softmax(-1) if train else torch.nn.functional.one_hot(p.argmax(-1), 16).double()
    a, b = (x[:, i[pick]].double() for i in (layer.indices_0, layer.indices_1))
    want = torch.zeros(batch, 500, device="cuda", dtype=torch.float64)
    for g in range(16):
        f00, f01, f10, f11 = ((g >> s) & 1 for s in (3, 2, 1, 0))
        want += p[:, g] * (f00 * (1 - a) * (1 - b) + f01 * (1 - a) * b + f10 * a * (1 - b) + f11 * a * b)
    assert (y[:, pick] - want).abs().max() <= 64 * 2.0 ** -24   # 16 weights, four coefficients of up to 16 of them, three multiply-adds
