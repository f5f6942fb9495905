"""fp32 operands, rounded on the device: every kernel choice, inside fp16's range and outside it, from
strided memory, without a synchronisation (a call is captured in a CUDA graph)."""

import numpy as np
import pytest
import torch

from conftest import MAX_ABS_TOL, REL_L2_TOL
from flash_colsum_b200.inputs import Workload, make_inputs
from oracle import c_oracle
from oracle.naive_colsum import parity_errors

pytestmark = pytest.mark.gpu

CASES = [  # B, H, Sq, Sk, D, causal, cls
    (2, 4, 256, 256, 64, False, None),      # single pass
    (2, 3, 300, 300, 80, False, None),      # streaming passes
    (1, 4, 128, 1500, 128, True, None),     # one-kernel form
    (1, 4, 300, 5000, 128, True, None),     # two resident query blocks, key ranges merged
    (2, 3, 700, 700, 64, False, 40),        # a CLS prefix of more than four rows
    (2, 4, 185, 185, 64, False, 1),         # one row: a cluster per batch entry
    (2, 5, 500, 500, 40, False, 3),
    (1, 4, 4, 9000, 128, True, None),       # four rows: two kernels
    (1, 20, 1, 3000, 96, True, None),
    (50, 8, 60, 60, 64, False, 2),          # many pairs: four CTAs of a cluster per SM
]


def _wide(t, strided):
    return t.transpose(1, 2).contiguous().cuda().transpose(1, 2) if strided else t.cuda()


@pytest.mark.parametrize("B,H,Sq,Sk,D,causal,cls", CASES)
@pytest.mark.parametrize("factor,strided", [(1.0, False), (1.0, True), (1e5, False)])
def test_fp32_operands(B, H, Sq, Sk, D, causal, cls, factor, strided):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    w = Workload("f", B, H, Sq, Sk, D, "fp32", is_causal=causal, cls_len=cls, seed=Sk + D)
    q, k = make_inputs(w)
    q = q * factor
    few = (cls or Sq) <= 4
    # out of fp16's range both are rounded to bf16; the few-row forms leave such values as they are
    if factor == 1.0:
        ref = [t.half() for t in (q, k)]
    elif few:
        ref = [torch.where(t.abs() < 60000, t.half().float(), t) for t in (q, k)]
    else:
        ref = [t.bfloat16() for t in (q, k)]
    scale = D ** -0.5 / factor
    got = fc.flash_colsum(_wide(q, strided), _wide(k, strided), scale=scale, is_causal=causal, cls_len=cls)
    assert fc.device_status() == 0
    want = c_oracle.colsum_c(*ref, scale=scale, is_causal=causal, cls_len=cls)
    rel, mx = parity_errors(got.cpu().numpy(), want)
    assert rel <= REL_L2_TOL and mx <= MAX_ABS_TOL, (rel, mx)


def test_an_fp32_call_can_be_captured():
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    w = Workload("f", 2, 4, 256, 256, 64, "fp32", seed=5)
    q, k = (t.cuda() for t in make_inputs(w))
    want = fc.flash_colsum(q, k)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fc.flash_colsum(q, k)
    for _ in range(2):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_allclose(out.cpu().numpy(), want.cpu().numpy(), rtol=1e-5, atol=1e-9)
