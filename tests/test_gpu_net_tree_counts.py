"""Flat trees with their class sums in one pass, against the same network launched layer by layer: whole numbers, equal to the last one.

Sizes where it can go wrong: classes of as few trees as walkers, of about sixteen for each, which is what the register planes hold, and
of many; one part and several; walkers of 8, 16 and 32 lanes, all of them in use or not; input rows walked in pieces."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [2, 3])
@pytest.mark.parametrize(
    "classes, size, batch, features",
    [(7, 33, 726401, 50), (3, 127, 442000, 50), (3, 128, 441985, 50), (10, 129, 131000, 50), (2, 513, 163700, 50), (10, 1999, 9088, 50),
     (10, 2560, 8001, 50), (5, 9000, 3800, 50), (5, 9000, 5999, 50), (1, 170001, 1000, 50), (10, 640, 184325, 50), (2, 20000, 204800, 50),
     (2, 2000, 614400, 50), (10, 2000, 30720, 30000)],
)
def test_counts_equal_layer_launches(levels, classes, size, batch, features):
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    torch.manual_seed(size)
    dims = [features] + [classes * size * 2 ** i for i in reversed(range(levels))]
    net = torch.nn.Sequential(*[cb.LogicLayer(i, o) for i, o in zip(dims[:-1], dims[1:])], cb.GroupSum(classes)).cuda().eval()
    for p in net.parameters():
        p.data.normal_()
    x = torch.rand(batch, features, device="cuda") < 0.4
    want = cb.CompiledLogicNet(net, fuse=False).compile()(x)
    fused = cb.CompiledLogicNet(net, fuse=True).compile()
    _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 0))
    try:
        _lib.trace(True)
        got = fused(x)
        torch.cuda.synchronize()
        names = _lib.trace_report()
    finally:
        _lib.trace(False)
        _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 1))
    assert "packed_tree_count_kernel" in names and "group_popcount_kernel" not in names
    assert torch.equal(got, want)


@pytest.mark.parametrize("classes, size, batch, fused_counts", [(50, 500, 12288, False), (200, 500, 3000, False), (100, 500, 16384, True), (150, 2000, 4096, True), (31, 500, 12288, True),
                                                                (32, 500, 6000, False), (10, 2000, 30720, True), (100, 1000, 8192, True)])
def test_many_classes_on_both_sides_of_their_line(classes, size, batch, fused_counts):
    """One part and several, one wave of blocks and several (148 SMs); apart where too few blocks would be left."""
    import convlogic_b200 as cb
    from convlogic_b200 import _lib

    torch.manual_seed(size)
    net = torch.nn.Sequential(cb.LogicLayer(50, classes * size * 4), cb.LogicLayer(classes * size * 4, classes * size * 2),
                              cb.LogicLayer(classes * size * 2, classes * size), cb.GroupSum(classes)).cuda().eval()
    for p in net.parameters():
        p.data.normal_()
    x = torch.rand(batch, 50, device="cuda") < 0.4
    want = cb.CompiledLogicNet(net, fuse=False).compile()(x)
    fused = cb.CompiledLogicNet(net, fuse=True).compile()
    _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 0))
    try:
        _lib.trace(True)
        got = fused(x)
        torch.cuda.synchronize()
        names = _lib.trace_report()
    finally:
        _lib.trace(False)
        _lib.check(_lib.lib().clb_tune(_lib.TUNE_NET_ONE_LAUNCH, 1))
    assert ("packed_tree_count_kernel" in names) == fused_counts, names
    assert torch.equal(got, want)
