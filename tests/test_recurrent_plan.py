"""What a recurrent layer plans for a step: the portions' split into long and short, and nothing that grows with their lengths."""

import numpy as np
import pytest

from lalamo_b200 import ops
from lalamo_b200.parts.base import HostSegments
from lalamo_b200.parts.gated_delta import GatedDelta
from lalamo_b200.parts.linear_attention import LinearAttention


@pytest.mark.parametrize("layer", [GatedDelta, LinearAttention])
@pytest.mark.parametrize("lengths", [(), (1, 1, 1), (191,), (192,), (1, 193, 5, 2048, 224)])
def test_plans(layer, lengths):
    starts = tuple(sum(lengths[:i]) for i in range(len(lengths)))
    plan = layer.plan_step(None, HostSegments(starts, lengths, (0,) * len(lengths)))
    long = [i for i, n in enumerate(lengths) if n >= ops.GDR_LONG_PORTION]
    assert set(plan) == {"direct", "long_table"} and all(array.dtype == np.int32 for array in plan.values())
    assert plan["direct"].tolist() == [i for i in range(len(lengths)) if i not in long]
    blocks = [-(-lengths[i] // 32) for i in long]
    assert plan["long_table"].tolist() == [x for j, i in enumerate(long) for x in (i, sum(blocks[:j]), blocks[j])]
    other = ops.gated_delta_chunk_plan(starts, lengths)   # the plan of numbered chunks says the same
    assert all(np.array_equal(plan[name], other[name]) for name in plan)
