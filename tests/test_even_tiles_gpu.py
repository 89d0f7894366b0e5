"""The walking product's tiles of equal numbers of tokens: numbers that end inside 32, in one, two and several tiles, halves of unequal size,
every epilogue that leaves by bulk stores or by the threads' own, cut into slices of K."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [129, 257, 300, 513, 777])
@pytest.mark.parametrize("rows,width,epilogue,slices", [(4096, 72, "gated", 1), (1100, 200, "store", 1), (1101, 64, "store_float", 1), (640, 2048, "residual_add", 1),
                                                        (384, 1024, "store", 3), (20480, 64, "gated", 1)])
def test_products(tokens, rows, width, epilogue, slices):
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(tokens + rows)
    x, w = torch.randn(tokens, width, generator=generator).bfloat16().cuda(), (torch.randn(rows, width, generator=generator) * width ** -0.5).bfloat16().cuda()
    residual = torch.randn(tokens, rows, generator=generator).cuda() if epilogue == "residual_add" else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x.double() @ w.double().T
    if epilogue == "gated":
        up, gate = want.chunk(2, dim=1)
        want = up * torch.nn.functional.silu(gate)
    if residual is not None:
        want = want + residual.double()
    got = ops.linear_tcgen05(x, w, epilogue, residual, slices=slices, activation="silu" if epilogue == "gated" else "identity", status=status)
    assert int(status.item()) == 0
    # Rounded to bfloat16, each time by at most 2**-8 of the value, over a row by less than 2**-9 in the root mean square: a stored sum once, a float one not at all (its sums are 32-bit); a gated
    # result four times, both sides, the activated gate and itself, of which the gate's own is passed on times g silu'(g) / silu(g), about one
    # where the result is not small: four times 2**-9 if all four went the same way.
    bound = {"gated": 4, "store": 1, "residual_add": 1, "store_float": 2 ** -10}[epilogue] * 2 ** -9
    worst = ((got.double() - want).norm(dim=1) / want.norm(dim=1)).max()   # every token's row
    assert float(worst) < bound
