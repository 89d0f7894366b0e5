"""Latent attention on the fifth-generation tensor cores against the plain kernel (all sums in 32-bit): runs that end anywhere, tiles of cached rows
begun and ended within a page, windows that cut a tile, rows nobody sees that hold no numbers, shares of the rows merged, sinks, every width taken."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,latent,rope,page", [(16, 256, 32, 16), (3, 64, 16, 32), (64, 128, 64, 16), (1, 192, 64, 48), (5, 256, 16, 16)])
@pytest.mark.parametrize("window,splits,sink", [(None, 1, False), (50, 1, True), (200, 1, False), (None, 3, True), (300, 2, False)])
def test_against_plain(heads, latent, rope, page, window, splits, sink):
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(heads + latent)
    lengths, contexts = [37, 1, 9, 130, 128], [0, 70, 129, 500, 127]
    tokens, blocks = sum(lengths), -(-700 // page)
    q = torch.randn(tokens, heads, latent + rope, generator=generator).bfloat16().cuda()
    table = torch.randperm(len(lengths) * blocks, generator=generator).view(len(lengths), blocks)
    pages = torch.full((len(lengths) * blocks, page, 1, latent + rope), float("nan"))
    for i, (n, c) in enumerate(zip(lengths, contexts)):
        first = max(0, c - window + 1) if window else 0   # pages that the window has passed hold no numbers either
        for position in range(first, c + n):
            pages[table[i, position // page], position % page, 0] = torch.randn(latent + rope, generator=generator) * (3.0 if position % 50 == 49 else 1.0)
    pages = pages.bfloat16().cuda()
    ints = lambda x: torch.as_tensor(x, dtype=torch.int32).reshape(-1).cuda()  # noqa: E731
    common = dict(positions=ints(torch.cat([torch.arange(c, c + n) for n, c in zip(lengths, contexts)])),
                  token_segment=ints(torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths))), block_table=table.to(torch.int32).cuda(), num_heads=heads,
                  latent=latent, rope=rope, scale=0.1, window=window, status=torch.zeros(1, dtype=torch.int32, device="cuda"),
                  sink=torch.linspace(-3, 9, heads).cuda() if sink else None)
    run = ops.latent_attention_tiling(heads)[1] * 2
    items, start = [], 0
    for n in lengths:
        items += [(i, min(run, start + n - i)) for i in range(start, start + n, run)]
        start += n
    found, plain = (torch.empty(tokens, heads, latent, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.latent_attention(q, pages, found, items=ints(items), num_items=len(items), splits=splits, tcgen05=True, **common)
    ops.latent_attention_plain(q, pages, plain, **common)
    assert int(common["status"].item()) == 0
    # the result's and the weights' roundings to bfloat16, of 2 ** -9 of a value each at most
    difference = (found.float() - plain.float()).norm(dim=-1) / plain.float().norm(dim=-1)
    assert float(difference.max()) < 2 * 2 ** -8


def test_sizes_not_taken():
    from lalamo_b200 import ops

    supported = ops.latent_attention_tcgen05_supported
    assert supported(torch.bfloat16, 256, 32, 16, 16, 0.1)
    assert not supported(torch.bfloat16, 256, 64, 16, 16, 0.1) and not supported(torch.bfloat16, 144, 32, 16, 16, 0.1) and not supported(torch.bfloat16, 256, 12, 16, 16, 0.1)
    assert not supported(torch.float32, 256, 32, 16, 16, 0.1) and not supported(torch.bfloat16, 256, 32, 8, 16, 0.1) and not supported(torch.bfloat16, 256, 32, 16, 65, 0.1)
    assert not supported(torch.bfloat16, 256, 32, 16, 16, 0.0) and not supported(torch.bfloat16, 256, 32, 16, 16, -0.1)


@pytest.mark.parametrize("counts,few", [([1] * 200, True), ([4] * 150, True), ([1] * 140 + [5] * 20, False), ([1] * 100, False)])
def test_which_kernel_a_layer_takes(counts, few, monkeypatch):
    """More items than multiprocessors behind next to nothing go to the mma.sync kernel where its runs are long enough; both give the same layer."""
    from lalamo_b200 import ops
    from lalamo_b200.cache import CacheManager
    from lalamo_b200.config import plan
    from lalamo_b200.engine import StepEntry
    from lalamo_b200.engine.executor import BatchBuilder
    from lalamo_b200.parts import Runtime, build_part

    heads, dim, rope, rank, width = 16, 64, 32, 256, 64
    spec = plan.LatentAttentionSpec(model_dim=width, num_heads=heads, head_dim=dim, rope_dim=rope, value_dim=dim, latent_dim=rank, latent_norm=plan.RMSNormSpec(dim=rank, eps=1e-6, exact=True),
                                    position=plan.RopeSpec(rotary_dim=rope, theta=10000.0), window=2048)
    generator = torch.Generator().manual_seed(4)
    matrix = lambda *shape: (torch.randn(*shape, generator=generator) * shape[1] ** -0.5).bfloat16().cuda()  # noqa: E731
    tensors = {"q_proj": matrix(heads * (dim + rope), width), "down_proj": matrix(rank + rope, width), "latent_norm": torch.ones(rank).cuda(), "key_up_proj": matrix(heads * dim, rank),
               "value_up_proj": matrix(heads * dim, rank), "out_proj": matrix(width, heads * dim)}
    runtime = Runtime(device=torch.device("cuda:0"), dtype=torch.bfloat16)
    part = build_part(spec, tensors, runtime)
    cache = CacheManager([part.cache_need()], [None], runtime, page_size=16, num_pages=len(counts), num_slots=len(counts))
    for i in range(len(counts)):
        cache.admit(i)
    built = BatchBuilder(cache, runtime.device, 100, planners=[part]).build([StepEntry(i, [0] * n) for i, n in enumerate(counts)])
    view = cache.views(built.block_tables, built.inputs.segment_slot)[0]
    x = torch.randn(sum(counts), width, generator=generator).bfloat16().cuda()
    taken, real = [], ops.latent_attention
    monkeypatch.setattr(ops, "latent_attention", lambda *arguments, **keywords: (taken.append(keywords["tcgen05"]), real(*arguments, **keywords)))
    out = part.forward(x, built.inputs, view)
    monkeypatch.setattr(ops, "latent_attention_few_rows", lambda *arguments: not few)
    other = part.forward(x, built.inputs, view)
    assert taken == ([False, True] if few else [True, max(counts) > 4]) and int(runtime.status.item()) == 0
    # the weights' and the sums' roundings to bfloat16, of 2 ** -8 of a value each at most, and the layer's rounding
    assert float((out.float() - other.float()).norm() / other.float().norm()) < 3 * 2 ** -8
