"""Long portions in blocks of 32 tokens against the recurrence itself in 64 bits: portions that end at, before and behind a block's end,
key and value sizes with padding, decays of exactly zero, plans of other chunks; and a token without a number reaches none before it."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(lengths, heads, groups, dk, dv, delta):
    generator = torch.Generator().manual_seed(dk + dv)
    random = lambda *shape: torch.randn(*shape, generator=generator)  # noqa: E731
    tokens = sum(lengths)
    q, k, v = random(tokens, groups, dk), torch.nn.functional.normalize(random(tokens, groups, dk), dim=-1), random(tokens, heads, dv)
    decay = torch.sigmoid(4 * random(tokens, heads, dk))
    decay[decay < 0.01] = 0.0
    beta = torch.sigmoid(random(tokens, heads)) if delta else None
    return q, k, v, decay, beta, random(len(lengths) + 1, heads, dk, dv)


def run(q, k, v, decay, beta, state, lengths, chunk):
    from lalamo_b200 import ops

    starts, slots = np.cumsum([0] + list(lengths[:-1])), list(range(len(lengths)))[::-1]
    ints = lambda values: torch.tensor(np.asarray(values), dtype=torch.int32, device="cuda")  # noqa: E731
    plan = ops.gated_delta_chunk_plan(starts.tolist(), lengths, chunk_tokens=chunk, long_portion=16)
    chunk_plan = {**{name: ints(values) for name, values in plan.items()}, "num_chunks": plan["chunk_start"].size, "num_long": plan["long_table"].size // 3,
                  "num_direct": plan["direct"].size}
    status, on_device = torch.zeros(1, dtype=torch.int32, device="cuda"), state.cuda()
    out = ops._recurrence(q.cuda(), k.cuda(), decay.cuda(), v.cuda(), None if beta is None else beta.cuda(), on_device, num_groups=q.shape[1], segment_start=ints(starts),
                          segment_length=ints(lengths), segment_slot=ints(slots), segments=len(lengths), status=status, chunk_plan=chunk_plan)
    assert int(status.item()) == 0
    return out.cpu(), on_device.cpu(), slots


@pytest.mark.parametrize("delta", [True, False])
@pytest.mark.parametrize("dk,dv,chunk", [(20, 8, 32), (32, 130, 64), (66, 7, 40), (64, 128, 32), (128, 72, 256), (256, 40, 32)])
def test_blocks(dk, dv, chunk, delta):
    lengths, heads, groups = [33, 5, 96, 31, 130], 4, 2
    q, k, v, decay, beta, state = make(lengths, heads, groups, dk, dv, delta)
    got, new_state, slots = run(q, k, v, decay, beta, state, lengths, chunk)
    want, want_state, at = torch.zeros_like(got, dtype=torch.float64), state.double(), 0
    for length, slot in zip(lengths, slots):
        S = want_state[slot].clone()
        for t in range(at, at + length):
            key, query = (x[t].double().repeat_interleave(heads // groups, dim=0) for x in (k, q))
            S = S * decay[t].double()[:, :, None]
            u = v[t].double() if beta is None else beta[t].double()[:, None] * (v[t].double() - torch.einsum("hkv,hk->hv", S, key))
            S = S + key[:, :, None] * u[:, None, :]
            want[t] = torch.einsum("hkv,hk->hv", S, query)
        want_state[slot] = S
        at += length
    # a few hundred products in 32 bits on the way to every number, their errors in no common direction: below 16 roundings of it
    assert float((got - want).norm() / want.norm()) < 16 * 2 ** -24
    assert float((new_state - want_state).norm() / want_state.norm()) < 16 * 2 ** -24


@pytest.mark.parametrize("delta", [True, False])
def test_a_token_without_a_number_reaches_none_before_it(delta):
    lengths = [70]
    q, k, v, decay, beta, state = make(lengths, 2, 2, 64, 24, delta)
    clean, _, _ = run(q, k, v, decay, beta, state, lengths, 32)
    v[41], k[45] = float("nan"), float("inf")
    got, _, _ = run(q, k, v, decay, beta, state, lengths, 32)
    assert torch.equal(got[:41], clean[:41]) and bool(torch.isnan(got[41:]).any())
