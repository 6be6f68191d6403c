"""Flat layers walked as paths, against autograd through the gates in fp64: batches around the 32- and 64-sample stretches, rows of
16-, 8- and 4-byte alignment, layers of a neuron to a few thousand, and connections whose graph is unlike the constructor's."""

import ctypes as C

import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _plan(a, b, fin):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    lib, fout = _lib.lib(), a.numel()
    start, cons = (t.cuda() for t in cb.LogicLayer.build_consumer_lists(a, b, fin))
    a, b = a.cuda(), b.cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    p = dict(a=a, b=b, start=torch.empty(fin + 1, **i32), entry=torch.empty(2 * fout, 2, **i32), rec=torch.empty(fout, 4, **i32),
             open=torch.empty(fin, **i32), count=torch.empty(2, **i32))
    assert lib.clb_logic_entries(_ptr(a), _ptr(b), _ptr(start), _ptr(cons), _ptr(p["start"]), _ptr(p["entry"]), fin, fout, _stream()) == 0
    n = lib.clb_logic_path_scratch_bytes(fin, fout)
    scratch = torch.empty(n, dtype=torch.uint8, device="cuda")
    assert lib.clb_logic_path(_ptr(a), _ptr(b), _ptr(p["start"]), _ptr(p["entry"]), _ptr(p["rec"]), _ptr(p["open"]), _ptr(p["count"]), _ptr(scratch), n,
                              fin, fout, _stream()) == 0
    return p


def _connections(kind, fin, fout):
    g = torch.Generator().manual_seed(fin + fout)
    if kind == "twice":      # every feature read exactly twice (fin = fout): what the constructor draws
        c = torch.randperm(2 * fout, generator=g) % fin
        return c[:fout].clone(), c[fout:].clone()
    if kind == "any":        # any number of readers, a neuron that reads one feature twice, features nobody reads
        a, b = torch.randint(0, fin, (fout,), generator=g), torch.randint(0, max(1, fin - 1), (fout,), generator=g)
        b[0] = a[0]
        return a, b
    if kind == "pairs":      # neurons 2i and 2i + 1 read the same two features: closed trails of two neurons
        a = torch.arange(fout) // 2 * 2 % fin
        return a, (a + 1) % fin
    a = torch.arange(fout) % fin   # one long trail
    return a, (a + 1) % fin


def _check_plan(p, fin, fout):
    laid, n_open = p["count"].tolist()
    rec = p["rec"].cpu().long()
    j, second = rec[:, 0] >> 1, (rec[:, 0] & 1).bool()
    a, b = p["a"].cpu()[j], p["b"].cpu()[j]
    assert laid == fout and torch.equal(j.sort().values, torch.arange(fout))
    assert torch.equal(torch.where(second, b, a), rec[:, 1]) and torch.equal(torch.where(second, a, b), rec[:, 2])
    linked, closes = (rec[:, 3] & 1).bool(), (rec[:, 3] & 2).bool()
    assert not linked[0] and torch.equal(rec[1:, 1][linked[1:]], rec[:-1, 2][linked[1:]])
    assert bool((linked | ~closes).all())
    both = torch.cat([rec[:, 1][closes], p["open"][:n_open].cpu().long()])
    assert torch.equal(both.sort().values, torch.arange(fin))
    return n_open


@pytest.mark.parametrize("kind,fin,fout,batch", [
    ("twice", 1, 1, 1), ("twice", 2, 2, 4), ("twice", 40, 40, 33), ("twice", 300, 300, 64), ("twice", 300, 300, 66), ("twice", 1000, 1000, 31),
    ("twice", 3000, 3000, 520), ("twice", 3000, 3000, 513), ("twice", 3001, 3001, 514), ("twice", 20000, 20000, 16), ("any", 7, 9, 5),
    ("any", 500, 900, 100), ("any", 900, 500, 36), ("pairs", 600, 600, 96), ("trail", 5000, 5000, 40), ("trail", 3, 200, 12)])
def test_path_passes_against_oracle(kind, fin, fout, batch):
    from convlogic_b200 import _lib

    lib = _lib.lib()
    a, b = _connections(kind, fin, fout)
    p = _plan(a, b, fin)
    n_open = _check_plan(p, fin, fout)
    g = torch.Generator().manual_seed(batch)
    w = torch.randn(fout, 16, generator=g)
    x, gy = torch.rand(fin, batch, generator=g), torch.randn(fout, batch, generator=g)
    xd, gyd, wd = x.cuda(), gy.cuda(), w.cuda()
    y, coef = torch.empty(fout, batch, device="cuda"), torch.empty(fout, 4, device="cuda")
    assert lib.clb_logic_path_fwd(_ptr(xd), _ptr(p["rec"]), _ptr(wd), _ptr(y), _ptr(coef), fin, fout, batch, _lib.W_SOFTMAX, _stream()) == 0
    n = lib.clb_logic_path_bwd_scratch_bytes(fout, batch)
    scratch = torch.empty(n, dtype=torch.uint8, device="cuda")

    def backward():
        gx, gw = torch.full_like(xd, float("nan")), torch.full_like(wd, float("nan"))
        assert lib.clb_logic_path_bwd(_ptr(xd), _ptr(wd), _ptr(coef), _ptr(gyd), _ptr(gx), _ptr(gw), _ptr(p["start"]), _ptr(p["entry"]), _ptr(p["rec"]),
                                      _ptr(p["open"]), n_open, _ptr(scratch), n, fin, fout, batch, _lib.W_SOFTMAX, _stream()) == 0
        return gx, gw

    gx, gw = backward()
    xo, wo = x.t().double().requires_grad_(True), w.double().requires_grad_(True)
    yo = oracle.logic_layer(xo, a, b, oracle.gate_probabilities(wo, True))
    yo.backward(gy.t().double())

    def close(got, want):
        # sums of up to 520 products of fp32 values: an error of a few roundings of the largest
        return float((got.cpu().double() - want).abs().max()) <= 1e-5 * float(want.abs().max())

    assert close(y, yo.detach().t()) and close(gx, xo.grad.t()) and close(gw, wo.grad)
    p2 = _plan(a, b, fin)    # the trails may be laid out in another order, the sums stay as they are
    p["rec"], p["open"], n_open = p2["rec"], p2["open"], _check_plan(p2, fin, fout)
    again = backward()
    assert torch.equal(gx, again[0]) and torch.equal(gw, again[1])


def test_lists_of_a_layer_with_the_same_number_of_readers():
    """Consistent tables of other connections: every neuron once all the same, linked only where it does read what the one before reads."""
    fin = fout = 64
    a, b = _connections("twice", fin, fout)
    p, other = _plan(a, b, fin), _plan(a.flip(0), b.flip(0), fin)
    rec, (laid, _) = _layout(p["a"], p["b"], other["start"], other["entry"], fin)
    rec = rec.cpu().long()
    assert laid == fout and torch.equal((rec[:, 0] >> 1).sort().values, torch.arange(fout))
    linked = (rec[1:, 3] & 1).bool()
    assert torch.equal(rec[1:, 1][linked], rec[:-1, 2][linked])


def test_a_layer_whose_lists_contradict_its_connections_does_not_walk():
    """Neurons listed twice, others not at all: no plan of paths, and outputs of the connections."""
    import convlogic_b200 as cb
    from convlogic_b200 import _lib, ops
    from convlogic_b200._lib import W_SOFTMAX

    n, batch = 100000, 320
    torch.manual_seed(0)
    layer = cb.LogicLayer(n, n).cuda().train()
    a, b = _connections("trail", n, n)
    layer.indices_0.copy_(a), layer.indices_1.copy_(b)
    start, cons = cb.LogicLayer.build_consumer_lists(a, b, n)
    cons[129:150000:128] = cons[131:150002:128]
    layer.given_x_indices_of_y_start.copy_(start), layer.given_x_indices_of_y.copy_(cons)
    x = torch.rand(n, batch, device="cuda")
    xd = x.t().detach().requires_grad_(True)
    _lib.trace(True)
    y = layer(xd)
    y.sum().backward()
    torch.cuda.synchronize()
    names = _lib.trace_report()
    _lib.trace(False)
    assert "path_walk_kernel" in names and not {"logic_path_fwd_kernel", "logic_path_bwd_kernel"} & set(names), names
    assert float((y.detach().t() - ops.logic_fwd(x, layer.indices_0, layer.indices_1, layer.weights.detach(), W_SOFTMAX)).abs().max()) <= 1e-5


@pytest.mark.parametrize("width,batch,path,forward", [(40000, 210, True, False), (40000, 200, False, False), (83400, 101, True, False), (83000, 101, False, False),
                                                      (28000, 900, True, False), (100000, 1024, True, True), (100000, 1022, True, True), (99001, 1021, True, True),
                                                      (99000, 318, True, True), (98000, 318, True, False),
                                                      (331000, 96, True, True), (331000, 97, True, False), (198000, 159, True, False), (198000, 160, True, True)])
def test_layers_take_the_path_by_size(width, batch, path, forward):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib, ops
    from convlogic_b200._lib import W_SOFTMAX

    torch.manual_seed(batch)
    layer = cb.LogicLayer(width, width).cuda().train()
    x, gy = torch.rand(width, batch, device="cuda"), torch.randn(width, batch, device="cuda")
    tables = (layer.indices_0, layer.indices_1, layer.weights.detach())
    xd = x.t().detach().requires_grad_(True)
    _lib.trace(True)
    y = layer(xd)
    y.backward(gy.t())
    torch.cuda.synchronize()
    names = _lib.trace_report()
    _lib.trace(False)
    assert ("logic_path_bwd_kernel" in names) == path and ("logic_path_fwd_kernel" in names) == forward, names
    # the same terms in another order
    for got, want in ((y.detach().t(), ops.logic_fwd(x, *tables, W_SOFTMAX)),
                      (xd.grad.t(), ops.logic_bwd_x(x, *tables, gy, layer.given_x_indices_of_y_start, layer.given_x_indices_of_y, W_SOFTMAX)),
                      (layer.weights.grad, ops.logic_bwd_w(x, *tables, gy, W_SOFTMAX))):
        assert (got - want).norm() <= 1e-5 * want.norm()
    # and a range of neurons and of features against the gates in fp64
    a, b = layer.indices_0, layer.indices_1
    some = torch.arange(width // 3, width // 3 + 50, device="cuda")
    xs = x.t().double()[:, torch.cat([a[some], b[some]])].cpu().requires_grad_(True)
    ws = layer.weights.detach()[some].double().cpu().requires_grad_(True)
    i = torch.arange(50)
    ys = oracle.logic_layer(xs, i, i + 50, oracle.gate_probabilities(ws, True))
    ys.backward(gy[some].t().double().cpu())
    assert (y.detach()[:, some].double().cpu() - ys).abs().max() <= 1e-5
    assert (layer.weights.grad[some].double().cpu() - ws.grad).abs().max() <= 1e-5 * ws.grad.abs().max()   # sums of 1024 products
    readers = [((a == f) | (b == f)).nonzero().flatten() for f in some[:10]]
    for f, js in zip(some[:10], readers):
        xs = x.t().double()[:, torch.cat([a[js], b[js]])].cpu()
        at = torch.cat([a[js], b[js]]).cpu() == int(f)
        col = x[f].double().cpu().requires_grad_(True)
        inputs = torch.where(at, col[:, None], xs)
        k = torch.arange(len(js))
        out = oracle.logic_layer(inputs, k, k + len(js), oracle.gate_probabilities(layer.weights.detach()[js].double().cpu(), True))
        out.backward(gy[js].t().double().cpu())
        assert (xd.grad[:, f].double().cpu() - col.grad).abs().max() <= 1e-5 * max(1.0, float(col.grad.abs().max()))


@pytest.mark.parametrize("kind,fin,fout,batch", [("twice", 1, 1, 1), ("twice", 300, 300, 66), ("any", 500, 900, 100), ("any", 900, 500, 33), ("pairs", 600, 600, 96),
                                                 ("trail", 5000, 5000, 40), ("twice", 3001, 3001, 514)])
def test_forward_in_the_order_of_other_connections(kind, fin, fout, batch):
    """The order of a plan, its own connections or not, and the connections of the call."""
    from convlogic_b200 import _lib

    lib = _lib.lib()
    g = torch.Generator().manual_seed(batch)
    a, b = _connections(kind, fin, fout)
    w, x = torch.randn(fout, 16, generator=g), torch.rand(fin, batch, generator=g)
    want = oracle.logic_layer(x.t().double(), a, b, oracle.gate_probabilities(w.double(), True)).t()
    other = torch.randint(0, fin, (2, fout), generator=g)
    a, b, w, x = a.cuda(), b.cuda(), w.cuda(), x.cuda()
    for p in (_plan(a.cpu(), b.cpu(), fin), _plan(other[0].contiguous(), other[1].contiguous(), fin)):
        y, coef, live = torch.empty(fout, batch, device="cuda"), torch.empty(fout, 4, device="cuda"), torch.empty_like(p["rec"])
        assert lib.clb_logic_path_fwd_live(_ptr(x), _ptr(a), _ptr(b), _ptr(p["rec"]), _ptr(live), _ptr(w), _ptr(y), _ptr(coef), fin, fout, batch,
                                           _lib.W_SOFTMAX, _stream()) == 0
        assert float((y.cpu().double() - want).abs().max()) <= 1e-5   # outputs in [0, 1], a dozen roundings


def test_large_layers_read_their_connections_on_every_call():
    import convlogic_b200 as cb
    from convlogic_b200 import ops
    from convlogic_b200._lib import W_SOFTMAX

    torch.manual_seed(0)
    layer = cb.LogicLayer(100000, 100000).cuda().train()
    x = torch.rand(100000, 320, device="cuda")
    xd = x.t().detach().requires_grad_(True)

    def same():
        want = ops.logic_fwd(x, layer.indices_0.clone(), layer.indices_1.clone(), layer.weights.detach(), W_SOFTMAX)
        return float((layer(xd).detach().t() - want).abs().max()) <= 1e-5

    assert same()
    layer.indices_0.data.copy_(layer.indices_0.flip(0))   # no version tells of this write
    assert same()
    layer.indices_1.copy_(layer.indices_1.flip(0))
    assert same()


@pytest.mark.parametrize("width,batch", [(100000, 320), (3000, 64)])
def test_a_captured_step_keeps_the_plan_it_reads(width, batch):
    """Connections written after a capture, a plan of the new ones in the old one's place, its memory asked for by others."""
    import convlogic_b200 as cb

    torch.manual_seed(0)
    layer = cb.LogicLayer(width, width).cuda().train()
    x, gy = torch.rand(batch, width, device="cuda", requires_grad=True), torch.randn(batch, width, device="cuda")

    def step():
        y = layer(x)
        return [y.detach(), *torch.autograd.grad(y, [x, layer.weights], gy)]

    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        want = step()
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    connections = layer.indices_0.clone()
    layer.indices_0.copy_(layer.indices_0.flip(0))
    step()
    layer.indices_0.copy_(connections)   # what the graph's plan was laid out for
    step()
    filler = [torch.full((width * 4,), 1 << 29, dtype=torch.int32, device="cuda") for _ in range(64)]
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    del filler


def _layout(a, b, start, entry, fin):
    from convlogic_b200 import _lib

    fout = a.numel()
    i32 = dict(dtype=torch.int32, device="cuda")
    rec, open_, count = torch.empty(fout, 4, **i32), torch.empty(fin, **i32), torch.empty(2, **i32)
    n = _lib.lib().clb_logic_path_scratch_bytes(fin, fout)
    scratch = torch.empty(n + 256, dtype=torch.uint8, device="cuda").fill_(77)
    assert _lib.lib().clb_logic_path(_ptr(a), _ptr(b), _ptr(start), _ptr(entry), _ptr(rec), _ptr(open_), _ptr(count), _ptr(scratch), n, fin, fout, _stream()) == 0
    assert bool((scratch[n:] == 77).all())
    return rec, count.tolist()


@pytest.mark.parametrize("kind", ["a neuron listed twice", "an end that runs into another trail", "values outside the tables", "starts outside the tables"])
def test_lists_of_other_connections_are_counted(kind):
    """What is outside the tables is not followed.  Either every neuron is laid out once, linked only where it does read what the one before reads, or
    the count is another than the number of neurons."""
    fin = fout = 40000
    a, b = _connections("trail", fin, fout)
    p = _plan(a, b, fin)
    start, entry = p["start"].clone(), p["entry"].clone()
    if kind == "a neuron listed twice":
        entry[2:20000:4, 0] = entry[0:19998:4, 0]
    elif kind == "an end that runs into another trail":
        entry[1001, 0] = entry[1003, 0]
    elif kind == "values outside the tables":
        entry[0::2, 0], entry[1::4, 0] = 1 << 30, -5
    else:
        start[1::2], start[0::2] = 1 << 30, -(1 << 30)
        start[:2] = 0
    rec, (laid, _) = _layout(p["a"], p["b"], start, entry, fin)
    if kind == "an end that runs into another trail":
        assert laid != fout
    else:
        code, linked = rec[:, 0].long(), (rec[1:, 3] & 1).bool()
        assert laid == fout and torch.equal((code >> 1).sort().values.cpu(), torch.arange(fout))
        a, b, second = p["a"][code >> 1], p["b"][code >> 1], (code & 1).bool()
        entered, left = torch.where(second, b, a), torch.where(second, a, b)
        assert torch.equal(entered[1:][linked], left[:-1][linked])


@pytest.mark.parametrize("packed", [False, True])
def test_a_plan_that_goes_while_another_stream_reads_it(packed):
    """Laid out on one stream, read on another that is behind, given back and its memory asked for on the first."""
    import convlogic_b200 as cb

    torch.manual_seed(0)
    n = 30000 if packed else 100000
    layer, side = cb.LogicLayer(n, n).cuda(), torch.cuda.Stream()
    layer.train(not packed)
    holder = layer.indices_0 if packed else layer.given_x_indices_of_y_start
    x = cb.PackBitsTensor(torch.rand(2000, n, device="cuda") < 0.5, 32) if packed else torch.rand(320, n, device="cuda", requires_grad=True)

    def call():
        return layer(x).rows() if packed else layer(x).detach()

    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        want = call()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)
    got = call()
    del holder._clb_plan
    with torch.cuda.stream(side):
        filler = [torch.full((size,), 1 << 29, dtype=torch.int32, device="cuda") for size in (n, n, n + 1, 2 * n, 4 * n, 4 * n) for _ in range(4)]
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    del filler
