"""Long portions of the recurrences in a bounded scratch: what a call takes beside its inputs does not grow with the step, and a smaller bound changes no bit."""

import numpy as np
import pytest
import torch

from test_recurrent_blocks_gpu import make, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("delta", [True, False])
def test_scratch_of_a_large_step(delta):
    from lalamo_b200 import ops

    tokens, heads, dk, dv = 16384, 16, 128, 128
    generator = torch.Generator(device="cuda").manual_seed(1)
    random = lambda *shape: torch.randn(*shape, generator=generator, device="cuda")  # noqa: E731
    q, k, v = random(tokens, heads, dk), torch.nn.functional.normalize(random(tokens, heads, dk), dim=-1), random(tokens, heads, dv)
    decay, beta, state = torch.sigmoid(2 + random(tokens, heads, dk)), torch.sigmoid(random(tokens, heads)) if delta else None, random(1, heads, dk, dv)
    ints = lambda values: torch.tensor(np.asarray(values), dtype=torch.int32, device="cuda")  # noqa: E731
    plan = ops.gated_delta_chunk_plan([0], [tokens])
    chunk_plan = {**{name: ints(values) for name, values in plan.items()}, "num_chunks": plan["chunk_start"].size, "num_long": 1, "num_direct": 0}
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = ops._recurrence(q, k, decay, v, beta, state, num_groups=heads, segment_start=ints([0]), segment_length=ints([tokens]), segment_slot=ints([0]), segments=1, status=status,
                          chunk_plan=chunk_plan)
    taken = torch.cuda.max_memory_allocated() - before - out.numel() * 4
    assert int(status.item()) == 0 and bool(out.isfinite().all())
    assert taken <= (260 << 20), taken


@pytest.mark.parametrize("delta", [True, False])
@pytest.mark.parametrize("blocks", [1, 2, 3, 5])
def test_a_smaller_bound_gives_the_same_bits(blocks, delta, monkeypatch):
    from lalamo_b200 import ops

    lengths, heads, groups, dk, dv = [33, 5, 96, 31, 130], 4, 2, 64, 40
    inputs = make(lengths, heads, groups, dk, dv, delta)
    whole, whole_state, _ = run(*inputs, lengths, 32)
    block = heads * 4 * (ops._lib().lb_recurrent_pack_floats(dk, dv, int(delta)) + ops._lib().lb_recurrent_value_floats(dv, int(delta)))
    monkeypatch.setattr(ops, "RECURRENT_SCRATCH_BYTES", blocks * block)
    got, state, _ = run(*inputs, lengths, 32)
    assert torch.equal(got, whole) and torch.equal(state, whole_state)
