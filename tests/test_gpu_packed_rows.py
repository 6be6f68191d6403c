"""Packing, flat layer and class counts on rows of every alignment, against the CPU oracle: batches around the 32-sample words,
the 256-sample tiles and the widths at which the number of lanes per neuron changes; feature counts around the 128-feature tiles."""

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 16, 32, 64])
@pytest.mark.parametrize("batch,features", [(1, 1), (7, 131), (33, 4), (129, 127), (256, 128), (257, 132), (1000, 37), (4104, 12), (2056, 9)])
def test_pack_logic_count_at_row_edges(bits, batch, features):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    g = torch.Generator().manual_seed(batch * 7 + bits)
    x = torch.rand(batch, features, generator=g) < 0.5
    packed, pad = _lib.native().pack_bits(x.cuda(), bits, True)
    want, want_pad = oracle.pack_bits(x.T.numpy(), bits)
    assert pad == want_pad and np.array_equal(packed.cpu().numpy().view(want.dtype), want)
    out = 530
    a, b = torch.randint(0, features, (out,), generator=g), torch.randint(0, features, (out,), generator=g)
    ops = torch.randint(0, 16, (out,), generator=g, dtype=torch.uint8)
    y = _lib.native().packed_logic(packed, a.cuda(), b.cuda(), ops.cuda())
    # truth-table bit of gate g for inputs (a, b): bit 3 - (2a + b)
    av, bv = x[:, a].long(), x[:, b].long()
    bit = (ops.long() >> (3 - (2 * av + bv))) & 1
    assert np.array_equal(y.cpu().numpy().view(want.dtype)[:, : want.shape[1]], oracle.pack_bits(bit.bool().T.numpy(), bits)[0] | _pad_bits(ops, want, batch, bits))
    counts = cb.PackBitsTensor.from_packed(y, pad).group_sum(10)
    assert torch.equal(counts.cpu().long(), bit.reshape(batch, 10, out // 10).sum(-1))


def _pad_bits(ops, like, batch, bits):
    """What a gate makes of the zero pad samples: f(0, 0)."""
    words = like.shape[1]
    mask = np.zeros((1, words), dtype=np.uint64)
    if batch % bits:
        mask[0, -1] = ((1 << bits) - 1) & ~((1 << (batch % bits)) - 1)
    on = ((ops.numpy() >> 3) & 1).astype(np.uint64)[:, None]
    return (on * mask).astype(np.uint64).astype(f"uint{bits}").view(like.dtype)


@pytest.mark.parametrize("rows_per_class", [1, 15, 128, 4096, 40000])
def test_class_counts_over_many_rows(rows_per_class):
    from convlogic_b200 import _lib

    x = torch.randint(-2**31, 2**31 - 1, (3 * rows_per_class, 33), device="cuda", dtype=torch.int32)
    want = torch.stack([(x.view(3, rows_per_class, 33).long() >> s) & 1 for s in range(32)], -1).sum(1)   # [3, 33, 32]
    got = _lib.native().group_popcount(x, 5, 3)
    assert torch.equal(got.long(), want.reshape(3, -1).t()[: 33 * 32 - 5])


@pytest.mark.parametrize("rows_per_class,row_bytes", [(1, 1), (15, 3), (127, 62), (128, 131), (2600, 257)])
def test_class_counts_over_rows_of_any_bytes(rows_per_class, row_bytes):
    from convlogic_b200 import _lib

    x = torch.randint(0, 256, (3 * rows_per_class, row_bytes), device="cuda", dtype=torch.uint8)
    want = torch.stack([(x.view(3, rows_per_class, row_bytes).long() >> s) & 1 for s in range(8)], -1).sum(1)   # [3, row_bytes, 8]
    got = _lib.native().group_popcount(x, 3, 3)
    assert torch.equal(got.long(), want.reshape(3, -1).t()[: 8 * row_bytes - 3])


@pytest.mark.parametrize("n,side,levels", [(1, 32, 64), (70, 9, 33), (300, 16, 100), (2000, 32, 40)])
@pytest.mark.parametrize("bytes_", [False, True])
def test_more_thermometer_levels_than_a_pass(n, side, levels, bytes_):
    """Passes over 32 levels at a time, each its own blocks where the grid is small (the last shape: in turn)."""
    from convlogic_b200 import ops

    torch.manual_seed(levels)
    px = torch.randint(0, 256, (n, 2, side, side), device="cuda", dtype=torch.uint8)
    th = torch.rand(levels, device="cuda")
    got, _ = ops.thermometer_pack(px if bytes_ else px.float() / 255, th)
    bits = torch.cat([px.float() / 255 > t for t in th], dim=1)
    want, _ = ops.pack_bits(bits.reshape(n, -1), 64, sample_major=True)
    assert torch.equal(got.reshape(want.shape), want)


@pytest.mark.parametrize("bits,words", [(8, 4), (8, 68), (16, 34), (32, 1), (32, 31), (32, 161), (64, 1), (64, 17), (64, 41), (64, 129), (32, 400)])
@pytest.mark.parametrize("fin,fout", [(1, 1), (300, 300), (50, 1000), (700, 400)])
def test_packed_layer_on_paths(bits, words, fin, fout):
    """Rows of 4-, 8- and 16-byte alignment, around the widths at which lanes and stretches change, against the neurons' own order."""
    import ctypes as C

    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    g = torch.Generator().manual_seed(words + fin)
    a, b = torch.randint(0, fin, (fout,), generator=g), torch.randint(0, fin, (fout,), generator=g)
    if fin == fout:
        c = torch.randperm(2 * fout, generator=g) % fin
        a, b = c[:fout].contiguous(), c[fout:].contiguous()
    start, cons = (t.cuda() for t in cb.LogicLayer.build_consumer_lists(a, b, fin))
    a, b, ops = a.cuda(), b.cuda(), torch.randint(0, 16, (fout,), generator=g, dtype=torch.uint8).cuda()
    x = torch.randint(0, 256, (fin, words * bits // 8), generator=g, dtype=torch.uint8).cuda().view({8: torch.int8, 16: torch.int16, 32: torch.int32, 64: torch.int64}[bits])
    lib, ptr, stream = _lib.lib(), lambda t: C.c_void_p(t.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    i32 = dict(dtype=torch.int32, device="cuda")
    s32, entry, rec, open_, count = (torch.empty(n, **i32) for n in (fin + 1, 4 * fout, 4 * fout, fin, 2))
    n = lib.clb_logic_path_scratch_bytes(fin, fout)
    scratch, y = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.empty(fout, words, dtype=x.dtype, device="cuda")
    assert lib.clb_logic_entries(ptr(a), ptr(b), ptr(start), ptr(cons), ptr(s32), ptr(entry), fin, fout, stream) == 0
    assert lib.clb_logic_path(ptr(a), ptr(b), ptr(s32), ptr(entry), ptr(rec), ptr(open_), ptr(count), ptr(scratch), n, fin, fout, stream) == 0
    assert lib.clb_packed_path(ptr(x), ptr(rec), ptr(ops), ptr(y), fin, fout, words, bits, stream) == 0
    assert torch.equal(y, _lib.native().packed_logic(x, a, b, ops))


def test_large_packed_layers_take_the_paths_by_themselves():
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    torch.manual_seed(0)
    layer = cb.LogicLayer(30000, 30000).cuda().eval()
    layer.weights.data.normal_()
    x = cb.PackBitsTensor(torch.rand(2000, 30000, device="cuda") < 0.5, 32)
    _lib.trace(True)
    y = layer(x)
    torch.cuda.synchronize()
    names = _lib.trace_report()
    _lib.trace(False)
    assert "packed_path_kernel" in names, names
    assert torch.equal(y.rows(), _lib.native().packed_logic(x.rows(), layer.indices_0, layer.indices_1, layer._gate_ids()))


@pytest.mark.parametrize("width,batch", [(300, 100), (30000, 2000)])
def test_packed_layers_need_no_consumer_lists(width, batch):
    """A deployed layer without the lists, which belong to the backward pass; with one of them; and with them."""
    import convlogic_b200 as cb

    torch.manual_seed(width)
    layer = cb.LogicLayer(width, width).cuda().eval()
    layer.weights.data.normal_()
    x = cb.PackBitsTensor(torch.rand(batch, width, device="cuda") < 0.5, 32)
    start, cons = layer.given_x_indices_of_y_start, layer.given_x_indices_of_y
    del layer.given_x_indices_of_y_start
    without_start = layer(x).rows()
    del layer.given_x_indices_of_y
    without = layer(x).rows()
    layer.register_buffer("given_x_indices_of_y_start", start)
    layer.register_buffer("given_x_indices_of_y", cons)
    assert torch.equal(without, layer(x).rows()) and torch.equal(without, without_start)


def _walk(x, a, b, ops, order):
    import ctypes as C

    from convlogic_b200 import _lib

    ptr = lambda t: C.c_void_p(t.data_ptr())
    y = torch.empty(a.numel(), x.shape[1], dtype=x.dtype, device="cuda")
    assert _lib.lib().clb_packed_walk(ptr(x), ptr(a), ptr(b), ptr(order), ptr(ops), ptr(y), x.shape[0], a.numel(), x.shape[1], x.element_size() * 8,
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return y


def _order(a, b, fin):
    import ctypes as C

    from convlogic_b200 import _lib

    ptr, lib = lambda t: C.c_void_p(t.data_ptr()), _lib.lib()
    n = lib.clb_packed_order_scratch_bytes(fin, a.numel())
    scratch, order = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.full((a.numel(),), -1, dtype=torch.int32, device="cuda")
    assert lib.clb_packed_order(ptr(a), ptr(b), ptr(order), ptr(scratch), n, fin, a.numel(), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return order


@pytest.mark.parametrize("bits,words", [(8, 4), (16, 34), (32, 31), (32, 161), (64, 1), (64, 17), (64, 41), (64, 129), (32, 400)])
@pytest.mark.parametrize("kind,fin,fout", [("twice", 1, 1), ("twice", 300, 300), ("twice", 20000, 20000), ("any", 50, 1000), ("any", 700, 400), ("pairs", 600, 600),
                                           ("one", 3, 5000)])
def test_packed_layer_in_any_order(kind, fin, fout, bits, words):
    """The order of the layer's own connections, and one that has nothing to do with them: every neuron once, the same bits."""
    from convlogic_b200 import _lib

    g = torch.Generator().manual_seed(words + fin)
    i = torch.arange(fout)
    if kind == "twice":
        c = torch.randperm(2 * fout, generator=g) % fin
        a, b = c[:fout].contiguous(), c[fout:].contiguous()
    elif kind == "any":
        a, b = torch.randint(0, fin, (fout,), generator=g), torch.randint(0, fin, (fout,), generator=g)
    else:   # closed trails of two neurons; one feature that every neuron reads, some of them twice
        a, b = (i // 2 * 2 % fin, (i // 2 * 2 + 1) % fin) if kind == "pairs" else (i * 0 + 1, i % fin)
    a, b, ops = a.cuda(), b.cuda(), torch.randint(0, 16, (fout,), generator=g, dtype=torch.uint8).cuda()
    x = torch.randint(0, 256, (fin, words * bits // 8), generator=g, dtype=torch.uint8).cuda().view({8: torch.int8, 16: torch.int16, 32: torch.int32, 64: torch.int64}[bits])
    want = _lib.native().packed_logic(x, a, b, ops)
    own = _order(a, b, fin)
    other = (2 * torch.randperm(fout, generator=g) + torch.randint(0, 2, (fout,), generator=g)).int().cuda()
    for order in (own, other):
        assert torch.equal((order >> 1).sort().values.cpu(), i.int())
        assert torch.equal(_walk(x, a, b, ops, order), want)
    if fout == 20000:   # pairs apart and closed trails aside, the next neuron reads what the last one read second
        j, second = (own >> 1).long(), (own & 1).bool()
        entered, left = torch.where(second, b[j], a[j]), torch.where(second, a[j], b[j])
        assert (entered[1:] == left[:-1]).float().mean() > 0.9


def _large(width=30000):
    import convlogic_b200 as cb

    torch.manual_seed(0)
    layer = cb.LogicLayer(width, width).cuda().eval()
    layer.weights.data.normal_()
    x = cb.PackBitsTensor(torch.rand(2000, width, device="cuda") < 0.5, 32)
    from convlogic_b200 import _lib

    def want():
        return _lib.native().packed_logic(x.rows(), layer.indices_0.clone(), layer.indices_1.clone(), layer._gate_ids())

    return layer, x, want


def test_large_packed_layers_read_their_connections_on_every_call():
    """Connections written in ways that leave their version as it is, and in ways that do not."""
    layer, x, want = _large()
    assert torch.equal(layer(x).rows(), want())
    layer.indices_0.data.copy_(layer.indices_0.flip(0))
    assert torch.equal(layer(x).rows(), want())
    layer.indices_1.copy_(torch.randint(0, 30000, (30000,), device="cuda"))
    assert torch.equal(layer(x).rows(), want())
    with torch.inference_mode():
        layer.indices_0 = layer.indices_0.clone()
        assert layer.indices_0.is_inference() and torch.equal(layer(x).rows(), want())


def test_large_packed_layers_do_not_read_their_lists():
    layer, x, want = _large()
    layer.given_x_indices_of_y.fill_(1 << 40)
    layer.given_x_indices_of_y_start.fill_(-(1 << 40))
    assert torch.equal(layer(x).rows(), want())


def test_a_captured_packed_layer_follows_its_connections():
    layer, x, want = _large()
    layer(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer(x).rows()
    for _ in range(2):
        layer.indices_0.copy_(torch.randint(0, 30000, (30000,), device="cuda"))
        layer(x)
        filler = [torch.full((30000,), 1 << 30, dtype=torch.int32, device="cuda") for _ in range(64)]   # (the order's memory is not among it)
        graph.replay()
        assert torch.equal(y, want())
        del filler
