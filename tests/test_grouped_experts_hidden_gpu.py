"""The grouped experts' hidden values bit for bit as the streaming kernels make them, over bfloat16 arguments of every size: inputs are unit
vectors, so that a sum is one element of the matrix, and `down` is the unit matrix, so that the output is the hidden value."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated,activation,limit", [(False, "gelu", 0.0), (False, "silu", 0.0), (True, "silu", 0.0), (True, "gelu", 0.0), (True, "sigmoid_limit", 7.0)])
def test_hidden_values(gated, activation, limit):
    from lalamo_b200 import ops

    size, tokens = 1024, 64
    # token t with the matrix's column t sees 1,024 arguments: all 65,536 patterns of 16 bits, but those beyond 2**40 and below 2**-40 and no numbers
    patterns = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).view(size, tokens).float()
    arguments = torch.where(patterns.isfinite() & (patterns.abs() < 2.0 ** 40) & (patterns.abs() > 2.0 ** -40), patterns, torch.zeros(()))
    arguments[0, :3] = torch.tensor([7.0, -7.0, 7.03125])   # at the limit and just beyond
    matrix = torch.zeros(1, size, size)
    matrix[0, :, :tokens] = arguments
    other = torch.zeros(1, size, size)
    other[0, :, :tokens] = 1.0 + torch.rand(size, tokens, generator=torch.Generator().manual_seed(1))
    x, down = torch.eye(size)[:tokens], torch.eye(size)[None]
    on = lambda tensor: tensor.bfloat16().cuda()  # noqa: E731
    chosen, weights, status = torch.zeros(tokens, 1, dtype=torch.int32, device="cuda"), torch.ones(tokens, 1, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    gate, up = (on(matrix), on(other)) if gated else (None, on(matrix))
    got = {path: ops.moe_experts(on(x), gate, up, on(down), chosen, weights, activation, path=path, limit=limit, status=status) for path in ("grouped", "stream")}
    assert int(status.item()) == 0
    assert torch.equal(got["grouped"], got["stream"])
    z = arguments.double()
    want = torch.nn.functional.silu(z) if activation == "silu" else torch.nn.functional.gelu(z) if activation == "gelu" else z.clamp(max=limit) * torch.sigmoid(1.702 * z.clamp(max=limit))
    if gated:
        want = want * (other[0, :, :tokens].bfloat16().double() + (1 if activation == "sigmoid_limit" else 0))
    # one rounding (2**-8 of the value at most) of the hidden value and, gated, one of the activated gate; what the functions themselves are off by (below 2**-18 of a gelu's
    # argument where it is nearly nothing) is far below
    assert bool(((got["grouped"].double().cpu().T - want).abs() <= 2.02 * 2 ** -8 * want.abs() + 2 ** -18).all())
