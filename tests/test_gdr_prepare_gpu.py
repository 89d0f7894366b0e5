"""The delta rule's inputs (convolutions, unit queries and keys, beta, decays) against the same in 64 bits: portions that begin and end anywhere in a
run of eight tokens, tokens around a warp's runs and a block's, heads narrower than a warp's piece, projections whose rows come in no fours, one
decay a channel and one a head, a slot that is none; and a token's numbers are the same bits alone and beside other portions."""

import pytest
import torch

pytestmark = pytest.mark.gpu

TAPS = 4


def make(heads, groups, dk, dv, tokens, slots, dtype, per_head, pad):
    generator = torch.Generator().manual_seed(heads * dk + dv + tokens)
    random = lambda *shape: torch.randn(*shape, generator=generator)  # noqa: E731
    channels, decays = 2 * groups * dk + heads * dv, heads if per_head else heads * dk
    return {"proj": random(tokens, -(-(channels + heads) // pad) * pad).to(dtype), "low": random(tokens, -(-decays // pad) * pad).to(dtype),
            "conv_state": random(slots, TAPS - 1, channels).to(dtype), "conv": random(channels, TAPS) * 0.6, "a_log": random(heads), "dt_bias": random(decays)}


def run(inputs, heads, groups, dk, dv, lengths, slots, per_head):
    """q, k, v, beta, decays and the state's rows as the launch leaves them, rows that it does not write as NaN; and the status."""
    from lalamo_b200 import ops

    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    ints = lambda values: torch.as_tensor(values, dtype=torch.int32).cuda()  # noqa: E731
    on = {name: tensor.cuda() for name, tensor in inputs.items()}
    tokens, single = on["proj"].shape[0], all(length == 1 for length in lengths)
    empty = lambda *shape: torch.full(shape, float("nan"), device="cuda")  # noqa: E731
    q, k, v, beta, decay = empty(tokens, groups, dk), empty(tokens, groups, dk), empty(tokens, heads, dv), empty(tokens, heads), empty(tokens, heads, dk)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    code = ops._lib().lb_gdr_prepare(on["proj"], on["proj"].shape[1], on["low"], on["low"].shape[1], on["conv_state"], on["conv"], on["a_log"], on["dt_bias"], q, k, v, beta, decay,
                                     ints([i for i, n in enumerate(lengths) for _ in range(n)]), ints(starts), ints(slots), tokens, heads, groups, dk, dv, TAPS,
                                     on["conv_state"].shape[0], 1e-6, dk ** -0.5, ops.dtype_code(on["proj"].dtype), status, ops._stream(), int(single), int(per_head))
    assert code == 0
    return [tensor.cpu() for tensor in (q, k, v, beta, decay)], int(status.item())


def wanted(inputs, heads, groups, dk, dv, lengths, slots, per_head):
    proj, low, conv = inputs["proj"].double(), inputs["low"].double(), inputs["conv"].double()
    channels, tokens, at, mixed = 2 * groups * dk + heads * dv, proj.shape[0], 0, []
    for length, slot in zip(lengths, slots):
        rows = torch.cat([inputs["conv_state"][slot].double(), proj[at: at + length, :channels]])
        mixed.append(torch.nn.functional.silu(sum(rows[j: j + length] * conv[:, j] for j in range(TAPS))))
        at += length
    q, k, v = torch.cat(mixed).split([groups * dk, groups * dk, heads * dv], dim=1)
    unit = lambda x: x.view(tokens, groups, dk) * torch.rsqrt((x.view(tokens, groups, dk) ** 2).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    z = low[:, : heads if per_head else heads * dk] + inputs["dt_bias"].double()
    decay = torch.exp(-torch.exp(inputs["a_log"].double())[:, None] * torch.nn.functional.softplus(z).view(tokens, heads, -1)).expand(tokens, heads, dk)
    return unit(q) * dk ** -0.5, unit(k), v.view(tokens, heads, dv), torch.sigmoid(proj[:, channels: channels + heads]), decay


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,groups,dk,dv,per_head,pad", [(4, 2, 8, 8, False, 8), (4, 2, 8, 8, True, 8), (3, 3, 20, 64, False, 4), (3, 3, 20, 64, True, 4), (2, 1, 64, 128, False, 8),
                                                             (2, 2, 128, 20, True, 8), (2, 2, 128, 128, False, 8), (1, 1, 4, 4, False, 4), (3, 1, 20, 8, False, 1), (2, 2, 18, 30, True, 1)])
@pytest.mark.parametrize("lengths", [[7], [8], [9], [31], [32], [33], [1, 2, 1, 5, 1, 1, 3, 12, 1, 8], [30, 1, 2, 70]])
def test_inputs(lengths, heads, groups, dk, dv, per_head, pad, dtype):
    tokens, slots = sum(lengths), [len(lengths) - i for i in range(len(lengths))]
    inputs = make(heads, groups, dk, dv, tokens, len(lengths) + 1, dtype, per_head, pad)
    sizes = (heads, groups, dk, dv, lengths, slots, per_head)
    got, status = run(inputs, *sizes)
    assert status == 0
    for name, one, other in zip(("q", "k", "v", "beta", "decay"), got, wanted(inputs, *sizes)):
        # 32-bit throughout: a convolution's four products, an exponential and a quotient; a unit norm's sum of dk squares and its root; a decay's
        # exponent (of size below 16 where the decay is not nothing) is off by a few roundings, which is the decay's relative error
        assert float((one - other).norm() / other.norm()) < 32 * 2 ** -24, name


@pytest.mark.parametrize("heads,groups,dk,dv,per_head", [(4, 2, 8, 8, False), (3, 3, 20, 64, True), (2, 1, 64, 128, False), (2, 2, 128, 128, False), (2, 2, 100, 36, False)])
def test_a_token_alone_and_beside_other_portions(heads, groups, dk, dv, per_head):
    """Every sum is in one order whatever else is in the step."""
    lengths, slots = [1, 5, 1, 9, 1, 1, 17, 1], [7, 1, 2, 3, 4, 5, 6, 0]
    inputs = make(heads, groups, dk, dv, sum(lengths), len(slots), torch.bfloat16, per_head, 8)
    beside, _ = run(inputs, heads, groups, dk, dv, lengths, slots, per_head)
    alone = [i for i, n in enumerate(lengths) if n == 1]
    rows = [sum(lengths[:i]) for i in alone]
    only = {**inputs, "proj": inputs["proj"][rows].contiguous(), "low": inputs["low"][rows].contiguous()}
    single, _ = run(only, heads, groups, dk, dv, [1] * len(alone), [slots[i] for i in alone], per_head)
    for name, one, other in zip(("q", "k", "v", "beta", "decay"), beside, single):
        assert torch.equal(one[rows], other), name


def test_a_slot_that_is_none():
    """Its portion is left out and reported, the ones beside it are what they are without it."""
    lengths, sizes = [5, 6, 9], (2, 2, 64, 32)
    inputs = make(*sizes, sum(lengths), 3, torch.float32, False, 8)
    clean, _ = run(inputs, *sizes, lengths, [2, 0, 1], False)
    got, status = run(inputs, *sizes, lengths, [2, 3, 1], False)
    assert status != 0
    for one, other in zip(got[:3], clean[:3]):
        assert torch.equal(one[:5], other[:5]) and torch.equal(one[11:], other[11:]) and bool(torch.isnan(one[5:11]).all())
