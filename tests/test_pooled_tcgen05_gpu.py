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
