"""A layer's launches in one call against the same kernels launched one binding after the other: the same bits."""

import pytest
import torch

from lalamo_b200 import ops

pytestmark = pytest.mark.gpu


def _values(*shape, seed, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to("cuda", dtype)


@pytest.mark.parametrize("tokens,width,hidden,rows", [(1, 64, 32, 8), (3, 96, 160, 40), (16, 1024, 4608, 1024)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_gated_mlp_step(tokens, width, hidden, rows, accumulate):
    x, up_gate, down = _values(tokens, width, seed=1), _values(2 * hidden, width, seed=2, scale=width**-0.5), _values(rows, hidden, seed=3, scale=hidden**-0.5)
    stream = _values(tokens, rows, seed=4, dtype=torch.float32) if accumulate else None
    expected = stream.clone() if accumulate else None
    inner = ops.gated_linear(x, up_gate, "silu")
    if accumulate:
        assert ops.linear_accumulate(inner, down, expected) is None
    else:
        expected = ops.linear(inner, down)
    out = ops.gated_mlp_step(x, up_gate, down, "silu", 0.0, stream)
    assert (out is stream) == accumulate and torch.equal(out, expected)


def test_gated_mlp_step_leaves_other_forms():
    x, up_gate, down = _values(2, 64, seed=1), _values(64, 64, seed=2), _values(8, 32, seed=3)
    assert ops.gated_mlp_step(x, up_gate, down, "silu", 0.0, None) is not None
    for changed in ((x.float(), up_gate, down), (x.t(), up_gate, down), (_values(17, 64, seed=1), up_gate, down), (x, up_gate[:62], down), (x, up_gate, _values(9, 32, seed=3)),
                    (_values(2 * 64 + 1, seed=1)[1:].view(2, 64), up_gate, down)):   # (the last: rows that start 2 bytes past a multiple of 16)
        assert ops.gated_mlp_step(*changed, "silu", 0.0, None) is None
    assert ops.gated_mlp_step(x, up_gate, down, "silu", 0.0, _values(2, 8, seed=4)) is None   # the stream is 32-bit
    assert ops.gated_mlp_step(x, up_gate, down, "unknown", 0.0, None) is None


# (tokens of each request, context of each, query heads, groups, head size, rotated channels, window, norms)
@pytest.mark.parametrize("lengths,contexts,heads,groups,hd,rotary,window,norms", [
    ([1], [0], 1, 1, 32, 0, None, False),
    ([1, 1, 1], [700, 5, 16], 8, 2, 64, 64, None, True),
    ([2, 5, 1, 8], [33, 0, 1000, 127], 6, 2, 80, 32, 64, True),
    ([16], [2000], 8, 8, 128, 128, None, False),
])
@pytest.mark.parametrize("accumulate", [False, True])
def test_attention_step(lengths, contexts, heads, groups, hd, rotary, window, norms, accumulate):
    tokens, width, page = sum(lengths), 96, 16
    blocks = max((c + n + page - 1) // page for c, n in zip(contexts, lengths))
    pages = blocks * len(lengths)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(5)).to("cuda", torch.int32).view(len(lengths), blocks)
    positions = torch.tensor([c + i for c, n in zip(contexts, lengths) for i in range(n)], dtype=torch.int32, device="cuda")
    segment = torch.tensor([s for s, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32, device="cuda")
    k_pages, v_pages = _values(pages, page, groups, hd, seed=6), _values(pages, groups, hd, page, seed=7)
    x = _values(tokens, width, seed=8)
    qkv = _values((heads + 2 * groups) * hd, width, seed=9, scale=width**-0.5)
    out_weight = _values(width, heads * hd, seed=10, scale=(heads * hd) ** -0.5)
    norm = [_values(hd, seed=11 + i, dtype=torch.float32) for i in range(2)] if norms else [None, None]
    inv_freq = 10000.0 ** -(torch.arange(rotary // 2, device="cuda", dtype=torch.float32) / max(rotary // 2, 1)) if rotary else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    max_context = max(c + n for c, n in zip(contexts, lengths))
    stream = _values(tokens, width, seed=13, dtype=torch.float32) if accumulate else None

    keys, values, expected = k_pages.clone(), v_pages.clone(), stream.clone() if accumulate else None
    queries, mixed = x.new_empty(tokens, heads * hd), x.new_empty(tokens, heads * hd)
    common = dict(positions=positions, token_segment=segment, block_table=table, num_heads=heads, num_groups=groups, head_dim=hd, status=status)
    ops.qk_norm_rope_write(ops.linear(x, qkv), queries, keys, values, q_weight=norm[0], k_weight=norm[1], eps=1e-5, scale_offset=0.0, inv_freq=inv_freq, rotary_dim=rotary,
                           write_kv=True, **common)
    ops.attention_decode(queries, keys, values, mixed, scale=hd**-0.5, window=window, max_context=max_context, fresh_keys=16, **common)
    if accumulate:
        assert ops.linear_accumulate(mixed, out_weight, expected) is None
    else:
        expected = ops.linear(mixed, out_weight)

    def step(first=x, table=table, dim=hd):
        return ops.attention_step(first, qkv, out_weight, stream, k_pages, v_pages, table, positions, segment, norm[0], norm[1], 1e-5, 0.0, inv_freq, rotary, 1.0, heads, groups, dim,
                                  hd**-0.5, window, 0, 0.0, 0, True, max_context, 16, status)

    for other in (dict(first=x.float()), dict(first=x.repeat(17, 1)), dict(table=table.long()), dict(table=table[0]), dict(dim=hd + 1)):
        assert step(**other) is None
    out = step()
    assert (out is stream) == accumulate and torch.equal(out, expected)
    assert torch.equal(k_pages, keys) and torch.equal(v_pages, values) and status.item() == 0


class _Step:
    """An attention layer of two tokens, each of a request of its own."""

    def __init__(self):
        self.ints = lambda *values: torch.tensor(values, dtype=torch.int32, device="cuda")
        self.x, self.qkv, self.out_weight = _values(2, 64, seed=1), _values(6 * 32, 64, seed=2), _values(64, 2 * 32, seed=3)
        self.k_pages, self.v_pages = _values(2, 16, 2, 32, seed=4), _values(2, 2, 32, 16, seed=5)
        self.table, self.status = self.ints(0, 1).view(2, 1), self.ints(0)

    def run(self, scale=0.1, keep_first=0, every=0, window=None, out_weight=None, positions=None, segment=None):
        return ops.attention_step(self.x, self.qkv, self.out_weight if out_weight is None else out_weight, None, self.k_pages, self.v_pages, self.table,
                                  self.ints(3, 4) if positions is None else positions, self.ints(0, 1) if segment is None else segment, None, None, 1e-5, 0.0, None, 0, 1.0, 2, 2, 32, scale,
                                  window, keep_first, 0.0, every, True, 16, 16, self.status)


def test_a_refused_step_launches_nothing():
    """What one of a step's kernels would refuse is refused before the first of them: no page, no row of the workspace is written."""
    step = _Step()
    keys, values = step.k_pages.clone(), step.v_pages.clone()
    apart = _values(64 * 64 + 1, seed=3)[1:].view(64, 64)   # rows that start 2 bytes past a multiple of 16
    for refused in (dict(scale=0.0), dict(scale=-1.0), dict(keep_first=-1, window=8), dict(every=-1), dict(out_weight=apart)):
        assert step.run(**refused) is None
        assert torch.equal(step.k_pages, keys) and torch.equal(step.v_pages, values), refused
    assert step.run() is not None and not torch.equal(step.k_pages, keys) and step.status.item() == 0
    up_gate, down, work = _values(64, 64, seed=6), _values(64 * 32 + 1, seed=7)[1:].view(64, 32), torch.full((2, 32), float("nan"), dtype=torch.bfloat16, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert ops._lib().lb_gated_mlp_step(step.x, up_gate, down, torch.empty_like(step.x), work, 2 * 2 * 32, 2, 64, 32, 64, 1, 0.0, 0, stream) == -2
    assert bool(work.isnan().all())


def test_fewer_positions_than_tokens():
    step = _Step()
    assert step.run(positions=step.ints(3)) is None and step.run(segment=step.ints(0)) is None
    for wrong in (dict(positions=step.ints(3), token_segment=step.ints(0, 1)), dict(positions=step.ints(3, 4), token_segment=step.ints(0))):
        with pytest.raises(ops.KernelError):
            ops.qk_norm_rope_write(ops.linear(step.x, step.qkv), step.x.new_empty(2, 64), step.k_pages, step.v_pages, q_weight=None, k_weight=None, eps=1e-5, scale_offset=0.0,
                                   inv_freq=None, rotary_dim=0, block_table=step.table, num_heads=2, num_groups=2, head_dim=32, write_kv=True, status=step.status, **wrong)
