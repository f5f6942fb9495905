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


# Calls in which no quarter of a tile is visible as a whole: no exp in them may be a polynomial's.  One key stands out, and
# all others are `below` it in powers of two, near where the polynomial is off by most (9.4e-5).
# Exps good to 2^-22, arguments of up to 15 rounded twice to 24 bits (1.3e-6), sums of 64 terms (2e-7):
EXACT_TOL = 2e-6


@pytest.mark.parametrize("Sq,Sk,causal", [(64, 64, True), (50, 64, True), (40, 64, True), (63, 63, False), (40, 63, False)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("below", [0.25, 0.75, 14.25, 14.75])
@pytest.mark.parametrize("short", [True, False])
def test_cut_tiles_take_no_polynomial(Sq, Sk, causal, D, below, short):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    from flash_colsum_b200 import _cabi
    scale = float(np.float32(np.log(2.0)))
    q, k = torch.zeros(1, 1, Sq if causal else Sk, D), torch.zeros(1, 1, Sk, D)
    q[..., 0] = 1.0
    k[..., 1:, 0] = -below
    s = (q.double() @ k.double().transpose(-1, -2)) * scale
    if causal:
        s.masked_fill_(torch.arange(Sk)[None, :] > Sk - Sq + torch.arange(Sq)[:, None], float("-inf"))
    want = s[:, :, :Sq].softmax(-1).mean((1, 2)).numpy()
    _cabi.set_single_pass(_cabi.SINGLE_PASS_NEVER)       # (whose exps are rounded to fp16)
    _cabi.set_short_fused(_cabi.SHORT_FUSED_AUTO if short else _cabi.SHORT_FUSED_NEVER)
    try:
        qd, kd = q.bfloat16().cuda(), k.bfloat16().cuda()     # (exact; fp16's way of subtracting the log-sum is good to 5e-6)
        got = (fc.flash_colsum_causal(qd, kd, scale=scale) if causal else fc.flash_colsum(qd, kd, scale=scale, cls_len=Sq)).cpu().numpy()
    finally:
        _cabi.set_short_fused(_cabi.SHORT_FUSED_AUTO)
        _cabi.set_single_pass(_cabi.SINGLE_PASS_AUTO)
    assert fc.device_status() == 0
    worst = float(np.max(np.abs(got - want) / want))
    assert worst <= EXACT_TOL, worst
