"""The plain attention's kernel that shares keys among rows, against dense softmax in 64 bits: several requests within a block's tokens, one
to sixteen query heads a key head, chunks' ends, windows with and without kept keys, pages whose rows come in no fours, positions that
nobody has written."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,groups,dim,vdim,value_groups", [(4, 4, 64, 64, 4), (6, 2, 20, 36, 2), (16, 1, 128, 128, 1), (4, 2, 64, 128, 1)])
@pytest.mark.parametrize("window,keep,page", [(0, 0, 16), (70, 3, 8), (33, 0, 5)])
def test_rows(heads, groups, dim, vdim, value_groups, window, keep, page):
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(heads * dim)
    random = lambda *shape: torch.randn(*shape, generator=generator)  # noqa: E731
    lengths, contexts = [3, 1, 62, 2, 40], [0, 130, 1, 64, 99]
    blocks = -(-max(n + c for n, c in zip(lengths, contexts)) // page)
    table = torch.randperm(len(lengths) * blocks, generator=generator).view(len(lengths), blocks).to(torch.int32)
    keys, values = random(len(lengths), blocks * page, groups, dim), random(len(lengths), blocks * page, value_groups, vdim)
    tokens = sum(lengths)
    positions = torch.cat([torch.arange(c, c + n) for n, c in zip(lengths, contexts)])
    segment = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths))
    for i, (n, c) in enumerate(zip(lengths, contexts)):
        values[i, c + n:] = float("nan")   # positions that nobody has written
    k_pages, v_pages = torch.zeros(table.numel(), page, groups, dim), torch.zeros(table.numel(), value_groups, vdim, page)
    for i in range(len(lengths)):
        k_pages[table[i].long()] = keys[i].view(blocks, page, groups, dim)
        v_pages[table[i].long()] = values[i].view(blocks, page, value_groups, vdim).permute(0, 2, 3, 1)
    if window:   # pages that the window has passed are given back
        for i, c in enumerate(contexts):
            table[i, -(-keep // page): max(-(-keep // page), max(0, c - window + 1) // page)] = -1
    q, out, status = random(tokens, heads * dim), torch.empty(tokens, heads * vdim, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ints = lambda x: x.to(torch.int32).cuda()  # noqa: E731
    ops.paged_attention_plain(q.cuda(), k_pages.cuda(), v_pages.cuda(), out, positions=ints(positions), token_segment=ints(segment), block_table=table.cuda(),
                              num_heads=heads, num_groups=groups, head_dim=dim, scale=dim ** -0.5, window=window or None, status=status, value_dim=vdim,
                              keep_first=keep, value_groups=value_groups)
    assert int(status.item()) == 0
    want = torch.empty(tokens, heads, vdim, dtype=torch.float64)
    for t in range(tokens):
        p, i = int(positions[t]), int(segment[t])
        j = torch.arange(p + 1)
        j = j[(p - j < window) | (j < keep)] if window else j
        for h in range(heads):
            g = h // (heads // groups)
            scores = keys[i, j, g].double() @ q[t, h * dim: (h + 1) * dim].double() * dim ** -0.5
            want[t, h] = torch.softmax(scores, 0) @ values[i, j, g // (groups // value_groups)].double()
    # scores of size below 6 from sums of `dim` products in 32 bits: off by about sqrt(dim) roundings of 6, which is the weights' relative error
    assert float((out.cpu().view_as(want) - want).norm() / want.norm()) < 6 * dim ** 0.5 * 2 ** -24 + 2 ** -21


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,groups,dim,window,page", [(16, 16, 64, 0, 16), (16, 16, 128, 0, 16), (16, 8, 64, 40, 16), (8, 8, 64, 0, 6)])
def test_a_request_alone_and_beside_many(heads, groups, dim, window, page, dtype):
    """The same bits whatever else is in the step, which decides a block's tokens and stages; few keys, and what nobody has written is no number."""
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(dim + page)
    random = lambda *shape: torch.randn(*shape, generator=generator)  # noqa: E731
    lengths = [1, 2, 1, 5, 1, 1, 30] + [1] * 60
    contexts = [0, 0, 15, 64, 127, 200, 3] + [(7 * i) % 140 for i in range(60)]
    blocks = -(-max(n + c for n, c in zip(lengths, contexts)) // page)
    table = torch.randperm(len(lengths) * blocks, generator=generator).view(len(lengths), blocks).to(torch.int32)
    k_pages, v_pages = torch.empty(table.numel(), page, groups, dim), torch.empty(table.numel(), groups, dim, page)
    for i, (n, c) in enumerate(zip(lengths, contexts)):
        keys, values = random(blocks * page, groups, dim), random(blocks * page, groups, dim)
        keys[n + c:] = values[n + c:] = float("nan")
        k_pages[table[i].long()], v_pages[table[i].long()] = keys.view(blocks, page, groups, dim), values.view(blocks, page, groups, dim).permute(0, 2, 3, 1)
    q = random(sum(lengths), heads * dim).to(dtype).cuda()
    k_pages, v_pages = k_pages.to(dtype).cuda(), v_pages.to(dtype).cuda()

    def attend(requests):
        rows = [row for i in requests for row in range(sum(lengths[:i]), sum(lengths[:i]) + lengths[i])]
        ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")  # noqa: E731
        out, status = torch.empty(len(rows), heads * dim, dtype=dtype, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        ops.paged_attention_plain(q[rows].contiguous(), k_pages, v_pages, out, positions=ints([c for i in requests for c in range(contexts[i], contexts[i] + lengths[i])]),
                                  token_segment=ints([s for s, i in enumerate(requests) for _ in range(lengths[i])]), block_table=table[requests].contiguous().cuda(), num_heads=heads,
                                  num_groups=groups, head_dim=dim, scale=dim ** -0.5, window=window or None, status=status)
        assert int(status.item()) == 0
        return out.cpu()

    every, k_held, v_held = attend(list(range(len(lengths)))), k_pages.cpu(), v_pages.cpu()
    assert bool(every.isfinite().all())
    at = 0
    for i in range(9):
        assert torch.equal(attend([i]), every[at: at + lengths[i]]), i
        at += lengths[i]
    for t, (i, position) in enumerate((i, c) for i in range(9) for c in range(contexts[i], contexts[i] + lengths[i])):
        keys = torch.arange(max(0, position - window + 1) if window else 0, position + 1)
        k, v = k_held[table[i, keys // page].long(), keys % page].double(), v_held[table[i, keys // page].long(), :, :, keys % page].double()
        query = q[t].cpu().double().view(groups, heads // groups, dim)
        weights = torch.softmax(torch.einsum("gpd,kgd->gpk", query, k) * dim ** -0.5, -1)
        want = torch.einsum("gpk,kgd->gpd", weights, v).reshape(-1)
        # as above; in bfloat16 the result's rounding
        assert float((every[t].double() - want).norm() / want.norm()) < 6 * dim ** 0.5 * 2 ** -24 + 2 ** -21 + (2 ** -8 if dtype == torch.bfloat16 else 0)
