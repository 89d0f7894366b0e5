"""Latent attention in runs of twice as many tokens: the same sums in the same order as in single runs, bit for bit, for runs that end
anywhere, more heads than a CTA's rows, windows, several cached rows' blocks, shares of the rows merged."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,latent,rope", [(16, 256, 32), (3, 64, 16), (70, 144, 32)])
@pytest.mark.parametrize("window,splits", [(None, 1), (50, 1), (None, 2)])
def test_double_runs(heads, latent, rope, window, splits):
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(heads)
    lengths, contexts, page, blocks = [37, 1, 9, 130], [0, 70, 129, 5], 16, 16
    tokens = sum(lengths)
    q = torch.randn(tokens, heads, latent + rope, generator=generator).bfloat16().cuda()
    pages = torch.randn(len(lengths) * blocks, page, 1, latent + rope, generator=generator).bfloat16().cuda()
    ints = lambda x: torch.as_tensor(x, dtype=torch.int32).reshape(-1).cuda()  # noqa: E731
    table = torch.randperm(len(lengths) * blocks, generator=generator).view(len(lengths), blocks).to(torch.int32).cuda()
    positions = ints(torch.cat([torch.arange(c, c + n) for n, c in zip(lengths, contexts)]))
    segment = ints(torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)))
    found = []
    for double in (False, True):
        run = ops.latent_attention_tiling(heads)[1] * (2 if double else 1)
        items, start = [], 0
        for n in lengths:
            items += [(i, min(run, start + n - i)) for i in range(start, start + n, run)]
            start += n
        out, status = torch.empty(tokens, heads, latent, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.latent_attention(q, pages, out, items=ints(items), num_items=len(items), positions=positions, token_segment=segment, block_table=table, num_heads=heads,
                             latent=latent, rope=rope, scale=0.1, window=window, status=status, splits=splits, double=double)
        assert int(status.item()) == 0
        found.append(out)
    if splits == 1:
        assert torch.equal(found[0], found[1])
    else:   # a run's shares begin elsewhere: the same sums, cut at other blocks; the result's and the weights' roundings to bfloat16
        assert float((found[0].float() - found[1].float()).norm() / found[0].float().norm()) < 2 * 2 ** -8
    plain = torch.empty_like(found[0])
    ops.latent_attention_plain(q, pages, plain, positions=positions, token_segment=segment, block_table=table, num_heads=heads, latent=latent, rope=rope, scale=0.1,
                               window=window, status=status)
    assert float((found[1].float() - plain.float()).norm() / plain.float().norm()) < 2 * 2 ** -8
