"""The experts' weighted sum four columns at a time and one at a time: the same bits, at widths that come in fours and widths that do not, one to nine
experts a token, pairs whose expert is none (whatever their rows hold), with and without weights."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [4, 10, 1020, 1024, 1028, 2049])
@pytest.mark.parametrize("top,weighted", [(1, True), (4, True), (4, False), (8, True), (9, True)])
def test_sums(top, weighted, width, dtype):
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(top * width)
    tokens, experts = 5, 6
    rows, weights = torch.randn(tokens * top, width, generator=generator), torch.rand(tokens, top, generator=generator)
    chosen = torch.randint(-1, experts + 1, (tokens, top), generator=generator, dtype=torch.int32)
    chosen[0] = -1   # a token of no expert at all
    real = (chosen >= 0) & (chosen < experts)
    rows[~real.view(-1)] = float("nan")   # nothing was computed there
    put = lambda pairs: ops.ExpertSum(pairs.cuda(), weights.cuda() if weighted else None, chosen.cuda(), experts, dtype).sum().cpu()  # noqa: E731
    got = put(rows)
    # rows that start off 16 bytes go a column at a time
    shifted = torch.empty(rows.numel() + 1, device="cuda")[1:].view(rows.shape)
    shifted.copy_(rows)
    narrow = ops.ExpertSum(shifted, weights.cuda() if weighted else None, chosen.cuda(), experts, dtype).sum().cpu()
    assert torch.equal(got, narrow)
    factors = (weights if weighted else torch.ones(tokens, top)).double() * real
    want = (torch.nan_to_num(rows).double().view(tokens, top, width) * factors[:, :, None]).sum(1)
    # `top` products and sums in 32 bits, and the rounding to the result's type
    size = (torch.nan_to_num(rows).double().abs().view(tokens, top, width) * factors[:, :, None]).sum(1)
    assert bool(((got.double() - want).abs() <= size * top * 2 ** -23 + want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 0)).all())
