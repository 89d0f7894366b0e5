"""The grouped experts' products where tiles end: experts without a pair, with one, with a row more or less than a box of 32 or a
tile of 128; matrices whose rows and columns end inside a tile; pairs whose expert is no expert."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated,weigh", [(True, False), (True, True), (False, False)])
@pytest.mark.parametrize("counts,width,ff", [((0, 1, 31, 33, 0, 127), 72, 40), ((129, 128, 0, 257), 256, 264), ((5, 0, 3), 1032, 136), ((700, 9), 64, 520),
                                             # as many pairs as one launch sorts and gathers, two more, and several thousand: two launches
                                             ((0, 511, 1, 0, 380, 128, 0), 72, 40), ((300, 0, 722, 0), 64, 72), ((0, 1900, 1, 257, 0, 1843, 0), 40, 64)])
def test_ragged_experts(counts, width, ff, gated, weigh):
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(sum(counts))
    experts, missing = len(counts), 4   # four pairs more whose expert is none
    chosen = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)] + [torch.tensor([-1, experts, -1, experts + 7])])
    chosen = chosen[torch.randperm(chosen.numel(), generator=generator)]
    if chosen.numel() % 2:
        chosen = torch.cat([chosen, torch.tensor([-1])])
    chosen = chosen.view(-1, 2).to(torch.int32)
    tokens = chosen.shape[0]
    assert tokens * 2 >= sum(counts) + missing
    random = lambda *shape: torch.randn(*shape, generator=generator)  # noqa: E731
    x = random(tokens, width).bfloat16()
    gate, up, down = (random(experts, *shape).mul(shape[1] ** -0.5).bfloat16() for shape in ((ff, width), (ff, width), (width, ff)))
    weights = torch.rand(tokens, 2, generator=generator) + 0.5
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.moe_experts(x.cuda(), gate.cuda() if gated else None, up.cuda(), down.cuda(), chosen.cuda(), weights.cuda(), "silu" if gated else "gelu", path="grouped",
                          weigh_input=weigh, status=status).double().cpu()
    want = torch.zeros(tokens, width, dtype=torch.float64)
    for t in range(tokens):
        for k in range(2):
            e = int(chosen[t, k])
            if not 0 <= e < experts:
                continue
            before, after = (weights[t, k].double(), 1.0) if weigh else (1.0, weights[t, k].double())
            u = up[e].double() @ x[t].double() * before
            hidden = torch.nn.functional.silu(gate[e].double() @ x[t].double() * before) * u if gated else torch.nn.functional.gelu(u)
            want[t] += after * (down[e].double() @ hidden)
    # Rounded to bfloat16 on the way: both sides, the activated gate, the hidden value, the result, each by at most 2**-8 of itself, by less than
    # 2**-9 in the root mean square, and in no common direction: sqrt(5) * 2**-9 of the norm at the most.
    assert float((got - want).norm() / want.norm()) < 5 ** 0.5 * 2 ** -9
    assert int(status.item()) == 0


@pytest.mark.parametrize("tokens", [1, 297, 593, 1187])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_router_at_every_number_of_tokens_a_block(tokens, dtype):
    """One, two, four and eight tokens a block (the last block partly filled), an odd number of router rows."""
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(tokens)
    x, router = torch.randn(tokens, 516, generator=generator).to(dtype), torch.randn(11, 516, generator=generator) * 0.05
    chosen, weights, gates = ops.moe_route(x.cuda(), router.cuda(), top=3, extra=1)
    logits = x.double() @ router.double().T
    scores = torch.sigmoid(logits[:, :10])
    want = torch.gather(scores, 1, chosen.long().cpu())
    # a lane adds 20 products at the most, then five sums are added: 25 roundings of the products' sizes (together below 20), the
    # sigmoid's slope a quarter; and the sigmoid's own roundings
    bound = 25 * 2 ** -24 * 20 / 4 + 4 * 2 ** -24
    assert float((weights.double().cpu() - want).abs().max()) < bound and float((gates.double().cpu() - torch.sigmoid(logits[:, 10:])).abs().max()) < bound
    assert float((scores.topk(3).values - want).abs().max()) < 2 * bound   # the best ones, but for ties within the rounding
