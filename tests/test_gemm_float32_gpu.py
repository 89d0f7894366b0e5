"""The 32-bit path's own products against 64 bits: tiles of 16, 32 and 64 rows begun and ended, columns that end inside a block, every number of slices, rows of X that
lie apart."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,rows,width,apart", [(2, 8, 4, 0), (2, 65, 1024, 0), (15, 64, 36, 4), (16, 200, 516, 0), (17, 63, 128, 0), (32, 130, 1028, 8), (33, 129, 132, 0), (64, 4096, 260, 0),
                                                     (300, 1000, 1024, 12), (320, 2048, 96, 0), (257, 512, 4608, 0)])
@pytest.mark.parametrize("slices", [0, 1, 2, 4, 8])
def test_against_64_bits(tokens, rows, width, apart, slices):
    from lalamo_b200 import ops

    generator = torch.Generator().manual_seed(tokens + width)
    x = torch.randn(tokens, width + apart, generator=generator).cuda()
    weight = torch.randn(rows, width, generator=generator).cuda()
    out = torch.full((tokens, rows), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert ops._lib().lb_gemm_float32(x, weight, out, tokens, rows, width, width + apart, slices, stream) == 0
    want = x[:, :width].double() @ weight.double().T
    # each of `width` additions rounds by 2 ** -24 of a sum at most; as a random walk, with room for its tail
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -24 * (width ** 0.5 + 4)


def test_which_products():
    from lalamo_b200 import ops

    ops.configure_matmul_precision()
    takes = ops.float32_product_supported
    assert takes(8, 9216, 1024) and takes(300, 1024, 1024) and not takes(1, 2048, 1024) and not takes(300, 16384, 2048) and not takes(24, 8, 30)
    x, weight = torch.randn(24, 64, device="cuda"), torch.randn(40, 64, device="cuda")
    assert torch.allclose(ops.linear(x, weight), torch.mm(x, weight.T), rtol=1e-5, atol=1e-5)
    assert ops._lib().lb_gemm_float32(x, weight, x, 24, 40, 62, 64, 0, None) == -2 and ops._lib().lb_gemm_float32(x, weight, x, 24, 40, 64, 62, 0, None) == -2
