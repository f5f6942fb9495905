"""Masks decided per warp and ragged key groups: diagonals, groups without keys, extreme scores."""

import pytest
import torch

from conftest import REL_L2_TOL
from flash_colsum_b200.inputs import Workload, make_inputs
from oracle import c_oracle
from oracle.naive_colsum import parity_errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Sq,Sk,D,causal", [
    (1, 2, 900, 900, 64, False),       # statistics and column passes
    (1, 2, 900, 900, 128, True),       # ... with a causal diagonal
    (2, 2, 577, 577, 64, False),       # single-pass cluster kernel: groups of 64, 1 and no keys
    (1, 2, 128, 1500, 64, True),       # one-kernel form
])
@pytest.mark.parametrize("jump,scale", [(30.0, None), (1.0e4, None), (1.0, 0.0)])
def test_extreme_scores_and_a_scale_of_zero(B, H, Sq, Sk, D, causal, jump, scale):
    """Keys further on that lift the scores by hundreds and by hundreds of thousands of powers of two, and a
    scale of zero (every visible key counts the same)."""
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    w = Workload("jump", B, H, Sq, Sk, D, "bf16", is_causal=causal, seed=Sk + D)
    q, k = make_inputs(w)
    k[:, :, Sk // 3::7] *= jump
    got = fc.flash_colsum(q.cuda(), k.cuda(), scale=scale, is_causal=causal).cpu().numpy()
    assert fc.device_status() == 0
    want = c_oracle.colsum_c(q, k, scale=scale, is_causal=causal)
    rel, mx = parity_errors(got, want)
    # (scores in the hundreds of thousands: an fp32 score has no more than a percent of a unit)
    assert rel <= (REL_L2_TOL if jump <= 30 else 0.1), (jump, rel, mx)


@pytest.mark.parametrize("B,H,S,D,cls", [(50, 8, 150, 64, 1), (38, 12, 33, 128, 4), (45, 10, 280, 40, 3), (20, 16, 300, 64, 2)])
def test_few_rows_over_many_pairs(B, H, S, D, cls):
    """Clusters per batch entry with four CTAs per SM, contiguous and strided."""
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    q, k = make_inputs(Workload("few", B, H, S, S, D, "bf16", cls_len=cls, seed=B + S))
    want = c_oracle.colsum_c(q, k, cls_len=cls)
    for strided in (False, True):
        a, b = (t.transpose(1, 2).contiguous().cuda().transpose(1, 2) if strided else t.cuda() for t in (q, k))
        got = fc.flash_colsum(a, b, cls_len=cls).cpu().numpy()
        assert fc.device_status() == 0
        rel, mx = parity_errors(got, want)
        assert rel <= REL_L2_TOL and mx <= REL_L2_TOL, (strided, rel, mx)


@pytest.mark.parametrize("B,H,Sq,Sk,D", [(1, 16, 4000, 4000, 64), (2, 16, 4000, 4100, 128), (1, 15, 6100, 20000, 64)])
def test_causal_statistics_longest_tiles_first(B, H, Sq, Sk, D):
    """Calls whose statistics items go by rounds of heads (24 query tiles and more, few items; the last shape in
    rounds of 13 and 2), against a materialising evaluation in double precision."""
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    q, k = (t.cuda() for t in make_inputs(Workload("rounds", B, H, Sq, Sk, D, "bf16", is_causal=True, seed=Sq)))
    got = fc.flash_colsum_causal(q, k).cpu().numpy()
    assert fc.device_status() == 0
    hidden = torch.arange(Sk, device="cuda")[None, :] > (Sk - Sq + torch.arange(Sq, device="cuda"))[:, None]
    want = torch.zeros(B, Sk, dtype=torch.float64, device="cuda")
    for b in range(B):
        for h in range(H):
            s = (q[b, h].double() @ k[b, h].double().T) / D ** 0.5
            want[b] += torch.softmax(s.masked_fill_(hidden, float("-inf")), dim=-1).sum(dim=0) / (H * Sq)
    rel, mx = parity_errors(got, want.cpu().numpy())
    assert rel <= REL_L2_TOL and mx <= REL_L2_TOL, (rel, mx)
