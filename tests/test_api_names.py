"""The function-level interface on the host: names that callers of ``ops`` and ``functional`` use, and the Functions as torch Functions."""

import pytest
import torch


def test_functions_and_ops():
    import convlogic_b200 as cb
    from convlogic_b200 import functional, ops

    for name in ("FullConvLogicFunction", "LogicLayerCudaFunction", "ConvLogicFunction", "TreeLogicFunction", "GradFactor"):
        assert issubclass(getattr(cb, name), torch.autograd.Function), name
    for name in ("GroupSumFunction", "GroupSumCrossEntropyFunction", "LogicTreeFunction", "LogicTreeCrossEntropyFunction", "FeatureMajorFunction"):
        assert issubclass(getattr(functional, name), torch.autograd.Function), name
    for name in ("convtree_fwd", "convtree_bwd", "convtree_bwd_x", "convtree_bwd_w", "plane_lists", "conv_groups", "logic_fwd", "logic_bwd_w", "logic_bwd_x",
                 "pack_bits", "packed_logic", "group_popcount", "packed_convtree", "packed_convtree_slab", "thermometer_pack", "group_sum_fwd",
                 "group_sum_bwd", "group_sum_ce", "logic_tree_fwd", "logic_tree_bwd", "logic_tree_fwd_ce", "transpose2d", "adam_step"):
        assert callable(getattr(ops, name)), name


@pytest.mark.parametrize("k", [0, -4])
def test_class_counts_that_are_not_positive_raise(k):
    """k = 0 was an integer division by zero in C++, which ends the process."""
    from convlogic_b200 import _lib, ops

    with pytest.raises(ValueError, match="positive"):
        ops.group_popcount(torch.zeros(4, 2, dtype=torch.int32), 0, k)
    with pytest.raises(ValueError, match="positive"):
        _lib.native().group_sum_ce(torch.zeros(3, 8), torch.zeros(3, dtype=torch.int64), k, 1.0)
    lib = _lib.lib()
    assert lib.clb_group_sum_scratch_bytes(8, 4, k, 0) == 0   # the C interface takes no such count either
    assert lib.clb_group_popcount(1 << 20, 1 << 20, 8, 2, 32, 0, k, None) == -1   # before any pointer is looked at
