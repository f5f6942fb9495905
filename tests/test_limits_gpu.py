"""Calls at the limits of what the operator takes, against the plain float64 evaluation."""

import pytest
import torch

from conftest import REL_L2_TOL
from flash_colsum_b200.inputs import Workload, make_inputs
from oracle.naive_colsum import naive_colsum_f64, parity_errors

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fc():
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200
    return flash_colsum_b200


@pytest.mark.parametrize("Sq", [1, 2, 4, 5, 130])
@pytest.mark.parametrize("D,dtype", [(64, "fp16"), (80, "bf16"), (128, "fp32")])
def test_the_largest_k_past_shows_every_key(fc, Sq, D, dtype):
    """k_past + row is past 32 bits: every row sees every key, in the few-row forms, the one-kernel form and the
    streaming passes alike."""
    q, k = make_inputs(Workload("k_past", 1, 4, Sq, 700, D, dtype, is_causal=True, seed=Sq + D))
    ref = [t.half() if dtype == "fp32" else t for t in (q, k)]
    want = naive_colsum_f64(*ref, is_causal=True, k_past=700)
    for k_past in (2 ** 31 - 1, 2 ** 31 - 3, 2 ** 31 - 200, 700):
        got = fc.flash_colsum_causal(q.cuda(), k.cuda(), k_past=k_past).cpu().numpy()
        assert fc.device_status() == 0
        rel, mx = parity_errors(got, want)
        assert rel <= REL_L2_TOL, (k_past, rel, mx)
