"""Which steps of latent attention run in runs of twice as many tokens: none in which tokens that decode are most of the items."""

from types import SimpleNamespace

import pytest

from lalamo_b200 import ops
from lalamo_b200.parts.base import HostSegments
from lalamo_b200.parts.latent_attention import LatentAttention


@pytest.mark.parametrize("heads,lengths,double", [
    (16, [1] * 64, False), (16, [4] * 9, False), (16, [9] + [1] * 40, False), (16, [33] + [1] * 64, False), (16, [300] + [1] * 40, False), (16, [1000] + [1] * 40, False),
    (16, [5] + [1] * 8, True), (16, [9], False), (16, [33], False), (16, [64], False), (16, [65], True), (16, [5] + [1] * 15, False), (16, [300] + [1] * 8, True), (16, [2000] + [1] * 64, True), (16, [1023], True), (16, [200], True), (16, [700] * 5, True), (16, [6] * 20, True),
    (32, [300] + [1] * 40, False), (32, [300], True), (64, [2] + [1] * 40, False), (64, [40], True), (130, [4], False), (130, [12], True), (16, [], False)])
def test_runs(heads, lengths, double):
    starts = tuple(sum(lengths[:i]) for i in range(len(lengths)))
    layer = SimpleNamespace(spec=SimpleNamespace(num_heads=heads), takes_double=True)
    items = LatentAttention.plan_step(layer, HostSegments(starts, tuple(lengths), (0,) * len(lengths)))["items"].reshape(-1, 2).tolist()
    run = ops.latent_attention_tiling(heads)[1]
    assert (max((count for _, count in items), default=0) > run) == double
    # all rows, in order, each portion cut by itself
    assert [row for first, count in items for row in range(first, first + count)] == list(range(sum(lengths)))
    assert all(count <= run * (2 if double else 1) for _, count in items) and not any(first < start < first + count for first, count in items for start in starts)


def test_shares_of_runs_of_twice_as_many_tokens():
    """Few items behind many rows fill one round of multiprocessors, not a round and a third."""
    for items in range(1, 149):
        shares = ops.latent_attention_splits(items, 16, 256, 2048, 4096, sms=148, double=True)
        assert shares >= 1 and (shares == 1 or items * shares <= 222) and (shares <= 5 or items * shares <= 166)


@pytest.mark.parametrize("items,context,few", [(149, 64, True), (149, 16, True), (148, 16, False), (149, 65, False), (600, 1, True), (0, 0, False)])
def test_items_of_few_rows(items, context, few):
    """More items than multiprocessors, behind next to nothing."""
    assert ops.latent_attention_few_rows(items, context, sms=148) == few
