"""Partly visible tiles of the streaming kernels, which are walked in runs of 32 columns dealt over the consumer groups:
diagonals and ragged ends on, before and behind the edges of runs, halves and blocks."""

import numpy as np
import pytest
import torch

from flash_colsum_b200.inputs import Workload, make_inputs
from oracle import c_oracle
from oracle.naive_colsum import parity_errors

pytestmark = pytest.mark.gpu

# exps of relative accuracy 1e-4 in the statistics and in the columns
REL_TOL = 2e-4


def direct(q, k, k_past):
    """The column means in double, the scores materialised."""
    s = q.double() @ k.double().transpose(-1, -2) * q.shape[-1] ** -0.5
    hidden = torch.arange(k.shape[2])[None, :] > k_past + torch.arange(q.shape[2])[:, None]
    return s.masked_fill_(hidden, float("-inf")).softmax(-1).mean((1, 2)).numpy()


@pytest.mark.parametrize("Sq,Sk,k_past", [
    (257, 257, 0), (300, 300, 0), (384, 640, 256), (511, 1023, 512), (640, 640, 31), (640, 700, 32), (640, 700, 33),
    (1000, 1100, 95), (300, 3000, 2700), (300, 3000, 2687), (130, 2600, 1000), (600, 900, 900), (2000, 2000, 0)])
@pytest.mark.parametrize("D", [64, 128])
def test_causal_diagonals(Sq, Sk, k_past, D):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    from flash_colsum_b200 import _cabi
    q, k = make_inputs(Workload("v", 2, 3, Sq, Sk, D, "fp16", is_causal=True, seed=Sq + k_past))
    want = direct(q, k, k_past)
    _cabi.set_short_fused(_cabi.SHORT_FUSED_NEVER)
    try:
        got = fc.flash_colsum_causal(q.cuda(), k.cuda(), k_past=k_past).cpu().numpy()
    finally:
        _cabi.set_short_fused(_cabi.SHORT_FUSED_AUTO)
    assert fc.device_status() == 0
    assert np.isfinite(got).all()
    rel, _ = parity_errors(got, want)
    assert rel <= REL_TOL, rel


@pytest.mark.parametrize("S", [257, 287, 289, 383, 385, 450, 511, 545])
def test_ragged_ends(S):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    q, k = make_inputs(Workload("v", 2, 3, S, S, 128, "bf16", seed=S))
    got = fc.flash_colsum(q.cuda(), k.cuda()).cpu().numpy()
    assert fc.device_status() == 0
    rel, _ = parity_errors(got, c_oracle.colsum_c(q, k))
    assert rel <= REL_TOL, rel
