"""fp32 operands on both sides of the lines between one rounding kernel and two: the same call on operands that were rounded
beforehand, and an output that holds something else before the call."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,S,D", [(1, 2, 2048, 64), (1, 2, 2049, 64), (1, 1, 5, 64), (2, 4, 256, 64), (3, 3, 301, 80),
                                     (1, 8, 512, 64), (1, 8, 513, 64),
                                     (1, 2, 1024, 64), (1, 2, 1025, 64), (1, 1, 512, 128), (1, 1, 513, 128)])
@pytest.mark.parametrize("factor", [1.0, 1e5])
def test_one_rounding_kernel_or_two(B, H, S, D, factor):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    gen = torch.Generator().manual_seed(S)
    q, k = (torch.randn(B, H, S, D, generator=gen).cuda() for _ in range(2))
    q[0, 0, 0, 0] = factor                  # one value past fp16's range takes both operands to bf16
    half = torch.bfloat16 if factor > 65504 else torch.float16
    want = fc.flash_colsum(q.to(half), k.to(half))
    torch.full((B * S,), 7.0, device="cuda")     # (what the allocator hands out next need not be zero)
    got = fc.flash_colsum(q, k)
    assert fc.device_status() == 0
    # the same operands and kernels; adds into the output in another order
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
