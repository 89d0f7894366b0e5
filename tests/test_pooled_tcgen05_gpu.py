"""Pooled attention on the fifth-generation tensor cores (heads of 64 + 64 channels) against the plain attention over the whole sequence: one to eight query heads
a K/V head, tiles of 64 rows begun and ended by windows, blocks and portions, no cap, caps that scores stay within and that they pass, shares of the rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shares", [1, None, 5])
@pytest.mark.parametrize("case", [
    dict(heads=8, groups=2, window=100, pool=8, rot_dims=64, page_size=16, contexts=[0, 99, 111, 700], lengths=[130, 2, 33, 17], cap=30.0),
    dict(heads=3, groups=1, window=7, pool=24, rot_dims=8, page_size=16, contexts=[22, 23, 54], lengths=[3, 2, 40], cap=5.0),
    dict(heads=2, groups=2, window=128, pool=5, rot_dims=64, page_size=48, contexts=[0, 330], lengths=[150, 70], cap=0.0),
    dict(heads=6, groups=1, window=1, pool=3, rot_dims=0, page_size=16, contexts=[0, 1, 200], lengths=[2, 3, 65], cap=400.0),
    dict(heads=4, groups=2, window=64, pool=16, rot_dims=32, page_size=32, contexts=[63, 64, 1100], lengths=[64, 2, 31], cap=28.0),
])
def test_every_edge(case, shares):
    from test_zozenex_gpu import pooled_case

    assert pooled_case(torch.bfloat16, dk=64, dv=64, seed=7, tensor_cores=True, shares=shares, alone=False, **case) < 2e-2


def test_a_token_without_numbers_reaches_no_earlier_one():
    """A key that is no number, within a tile of rows and within the pair of weights that share a reciprocal."""
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(3)
    tokens, bad, ints = 200, 101, lambda x: torch.as_tensor(x, dtype=torch.int32).reshape(-1).cuda()  # noqa: E731
    q = torch.randn(tokens, 4 * 64, generator=generator).bfloat16().cuda()
    pages = torch.randn(13, 16, 1, 128, generator=generator).bfloat16().cuda()
    table, status = torch.arange(13, dtype=torch.int32).view(1, 13).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for spoilt in (False, True):
        if spoilt:
            pages.view(208, 128)[bad, :64] = float("nan")
        found = torch.empty(tokens, 4 * 64, dtype=torch.bfloat16, device="cuda")
        ops.pooled_attention(q, pages, None, found, tiles=ints([(i, min(32, tokens - i)) for i in range(0, tokens, 32)]), num_tiles=7, positions=ints(range(tokens)),
                             token_segment=ints([0] * tokens), block_table=table, pool_table=None, num_heads=4, num_groups=1, head_dim=64, value_dim=64, scale=0.125, softcap=30.0,
                             head_bias=None, window=150, pool=0, value_freq=None, status=status)
        out.append(found)
    assert int(status.item()) == 0 and torch.equal(out[0][:bad], out[1][:bad]) and bool(out[1][bad:].isnan().all())


def _prompt(heads, tokens, seed, width=128):
    """Queries, pages and what the kernels take beside them, for one prompt of ``tokens`` over one K/V head."""
    generator = torch.Generator().manual_seed(seed)
    ints = lambda x: torch.as_tensor(x, dtype=torch.int32).reshape(-1).cuda()  # noqa: E731
    blocks = -(-tokens // 16)
    q = torch.randn(tokens, heads * 64, generator=generator).bfloat16().cuda()
    pages = torch.randn(blocks, 16, 1, width, generator=generator).bfloat16().cuda()
    common = dict(positions=ints(range(tokens)), token_segment=ints([0] * tokens), block_table=torch.arange(blocks, dtype=torch.int32).view(1, blocks).cuda(), pool_table=None,
                  num_heads=heads, num_groups=1, head_dim=64, value_dim=64, window=150, pool=0, status=torch.zeros(1, dtype=torch.int32, device="cuda"))
    run = 16 * (8 // min(heads, 4))
    tiles = [(i, min(run, tokens - i)) for i in range(0, tokens, run)]
    return q, pages, dict(tiles=ints(tiles), num_tiles=len(tiles)), common


# exponents that a pair of weights shares a reciprocal for, that it does not, and both within a head's scores
@pytest.mark.parametrize("cap,scale", [(0.0, 0.125), (0.0, 1.0), (30.0, 0.125), (30.0, 1.0), (55.0, 1.0)])
def test_closed_heads(cap, scale):
    """Heads that a bias all but closes: weights down to 2 ** -115, as the 32-bit kernel has them."""
    from lalamo_b200 import ops

    tokens, heads = 200, 4
    q, pages, tiles, common = _prompt(heads, tokens, 5)
    common.update(scale=scale, softcap=cap, head_bias=torch.tensor([-2.0, -41.0, -45.0, -72.0 if scale < 1 else -47.0]).cuda(), value_freq=None)
    found, plain = (torch.empty(tokens, heads * 64, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.pooled_attention(q, pages, None, found, **tiles, **common)
    ops.pooled_attention_plain(q, pages, None, plain, **common)
    assert int(common["status"].item()) == 0
    difference, size = ((x.double().view(tokens, heads, 64)).norm(dim=-1) for x in (found.double() - plain.double(), plain))
    # the results' and the weights' roundings to bfloat16, of 2 ** -9 of a value each at most
    assert float((difference / size).max()) < 2 * 2 ** -8


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("shares", [1, 3])
@pytest.mark.parametrize("heads", [1, 2, 3, 6])
def test_sums_turned_back(heads, shares, interleaved):
    """Both pairings of the channels that the sums are turned back by, in the epilogue and in the kernel that adds up shares, against the 32-bit sums turned back in 64 bits."""
    from lalamo_b200 import ops

    tokens = 131
    q, pages, tiles, common = _prompt(heads, tokens, heads)
    freq = (200.0 ** (-torch.arange(32, dtype=torch.float64) / 32)).float().cuda()
    common.update(scale=0.125, softcap=30.0, head_bias=torch.linspace(-2, 1, heads).cuda())
    found, sums = torch.empty(tokens, heads * 64, dtype=torch.bfloat16, device="cuda"), torch.empty(tokens, heads * 64, device="cuda")
    ops.pooled_attention(q, pages, None, found, value_freq=freq, interleaved=interleaved, shares=shares, **tiles, **common)
    ops.pooled_attention_plain(q.float(), pages.float(), None, sums, value_freq=None, **common)
    sums = sums.double().view(tokens, heads, 64)
    first, second = (sums[..., 0::2], sums[..., 1::2]) if interleaved else (sums[..., :32], sums[..., 32:])
    angle = torch.arange(tokens, device="cuda", dtype=torch.float64)[:, None, None] * freq.double()
    turned = first * angle.cos() + second * angle.sin(), second * angle.cos() - first * angle.sin()
    want = torch.stack(turned, dim=-1).flatten(2) if interleaved else torch.cat(turned, dim=-1)
    assert int(common["status"].item()) == 0
    # the result's and the weights' roundings to bfloat16, of 2 ** -9 of a value each at most
    assert float(((found.double().view_as(want) - want).norm(dim=-1) / want.norm(dim=-1)).max()) < 2 * 2 ** -8


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("pool", [1, 8, 63, 64, 65, 72, 100, 129])
def test_means_of_long_blocks(pool, dtype):
    """Blocks of as many positions as a block of threads looks up at once, and of more; begun and ended within pages, several completed by one step."""
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(pool)
    groups, page, contexts, lengths = 2, 16, [0, pool // 2, 3 * pool - 1], [2 * pool + 5, pool, 1]
    blocks = -(-max(c + n for c, n in zip(contexts, lengths)) // page)
    ints = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()  # noqa: E731
    table = torch.randperm(len(lengths) * blocks, generator=generator).view(len(lengths), blocks)
    pages = torch.randn(len(lengths) * blocks, page, groups, 24, generator=generator).to(dtype)
    columns = max(c + n for c, n in zip(contexts, lengths)) // pool + 1
    means = torch.full((len(lengths) * columns, 1, groups, 24), float("nan"), dtype=dtype, device="cuda")   # a block a page
    pool_table = torch.arange(means.shape[0]).view(len(lengths), columns)
    status = ints([0])
    ops.pooled_means(pages.cuda(), means, segment_length=ints(lengths), segment_context=ints(contexts), block_table=ints(table), pool_table=ints(pool_table), segments=len(lengths),
                     max_length=max(lengths), num_groups=groups, head_dim=16, value_dim=8, pool=pool, status=status)
    assert int(status.item()) == 0
    written = torch.zeros(means.shape[0], dtype=torch.bool)
    for i, (n, c) in enumerate(zip(lengths, contexts)):
        rows = pages[table[i]].reshape(blocks * page, groups, 24).double()
        for block in range(c // pool, (c + n) // pool):
            written[pool_table[i, block]] = True
            want = rows[block * pool : (block + 1) * pool].mean(0)
            # `pool` additions in 32-bit of values of size one, and the rounding of the mean: half of the last of bfloat16's eight bits
            bound = pool * 2.0 ** -24 * 4 + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24) * want.abs().max()
            assert float((means[pool_table[i, block], 0].double().cpu() - want).abs().max()) <= bound
    assert written.sum() >= 3 and bool(means[~written.cuda()].isnan().all())
