"""A product of some of a matrix's columns: bit for bit that of a copy of them, on every kernel the numbers of tokens lead to, and where rows do not start on
16 bytes."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [0, 1, 8, 16, 17, 128, 129, 300])
@pytest.mark.parametrize("columns,first,width,rows", [(3208, 3080, 128, 2048), (104, 8, 32, 40), (64, 0, 64, 8), (72, 4, 64, 16), (61, 8, 32, 24)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_as_a_copy(tokens, columns, first, width, rows, dtype):
    from lalamo_b200 import ops

    ops.configure_matmul_precision()
    generator = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, columns, generator=generator).to(dtype).cuda()
    weight = torch.randn(rows, width, generator=generator).to(dtype).cuda()
    found, copied = ops.linear_of_columns(x, first, weight), ops.linear(x[:, first : first + width].clone(memory_format=torch.contiguous_format), weight)
    if dtype == torch.bfloat16:
        assert torch.equal(found, copied)
    else:   # the library may add up in another order: 2 ** -24 a sum, of `width` terms
        assert torch.allclose(found, copied, rtol=0.0, atol=width * 2.0 ** -24 * 8 * width ** 0.5)


def test_what_is_refused():
    from lalamo_b200 import ops

    x, weight = torch.zeros(4, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(8, 32, dtype=torch.bfloat16, device="cuda")
    for first, matrix in ((40, x), (-8, x), (0, x.t())):
        with pytest.raises(ops.KernelError):
            ops.linear_of_columns(matrix, first, weight)
