"""Host-memory calls: chunks of batch entries and of heads, against the call on device tensors."""

import pytest
import torch

from flash_colsum_b200.inputs import Workload, make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Sq,Sk,D,dtype,causal,cls", [
    (8, 6, 700, 700, 64, "fp16", False, None),       # entries, then heads of the last one
    (2, 16, 1024, 1024, 128, "bf16", False, None),
    (1, 12, 2000, 2000, 64, "fp16", False, None),    # one entry by heads
    (1, 9, 300, 9000, 128, "bf16", True, None),      # a causal call by heads
    (5, 7, 90, 90, 40, "fp16", False, None),         # one chunk
    (6, 8, 1500, 1500, 64, "fp32", False, 1),        # few rows, fp32
    (3, 5, 1000, 1000, 80, "bf16", False, 3),
])
@pytest.mark.parametrize("pinned", [True, False])
def test_host_call_matches_the_device_call(B, H, Sq, Sk, D, dtype, causal, cls, pinned):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    w = Workload("host", B, H, Sq, Sk, D, dtype, is_causal=causal, cls_len=cls, seed=B + H + Sk)
    q, k = make_inputs(w)
    if pinned:
        q, k = q.pin_memory(), k.pin_memory()
    want = fc.flash_colsum(q.cuda(), k.cuda(), is_causal=causal, cls_len=cls).cpu()
    for _ in range(2):
        got = fc.flash_colsum_host(q, k, is_causal=causal, cls_len=cls)
        assert got.device.type == "cpu" and got.shape == want.shape
        torch.testing.assert_close(got, want, rtol=3e-4, atol=1e-8)
    with pytest.raises(ValueError):
        fc.flash_colsum_host(q, k[:, :, :, :8], is_causal=causal)
    assert fc.device_status() == 0
