"""The function-level interface: names that callers of ``ops`` and ``functional`` use, and the Functions as torch Functions."""

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
