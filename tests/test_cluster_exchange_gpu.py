"""The single-pass kernel's exchange, score accumulators and late write-out at the sizes where they change: every cluster
size, halves and groups of a slice without keys, batch entries of one tile (written out one tile after the other), odd
numbers of tiles per cluster."""

import numpy as np
import pytest
import torch

from flash_colsum_b200.inputs import Workload, make_inputs
from oracle import c_oracle
from oracle.naive_colsum import parity_errors

pytestmark = pytest.mark.gpu

# exps as fp16 (2^-11 relative each) of scores whose exps are good to 1e-4: a mean of such terms is off by no more
REL_TOL = 6e-4


@pytest.mark.parametrize("B,H,S", [
    (300, 1, 128), (5, 1, 60), (3, 1, 129),          # one or two tiles per batch entry, more entries than clusters
    (2, 3, 256), (2, 3, 257), (2, 3, 384), (2, 3, 385), (2, 3, 512),       # a second slice with 1, 128, 129, 256 keys
    (7, 2, 513), (1, 5, 640), (2, 2, 769), (2, 3, 1024), (2, 2, 1025), (1, 3, 1536), (1, 2, 1793), (1, 2, 2048)])
def test_every_cluster_size_and_ragged_halves(B, H, S):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    from flash_colsum_b200 import _cabi
    w = Workload("x", B, H, S, S, 64, "fp16", seed=B + S)
    q, k = make_inputs(w)
    want = c_oracle.colsum_c(q, k)
    _cabi.set_single_pass(_cabi.SINGLE_PASS_ALWAYS)
    try:
        outs = [fc.flash_colsum(q.cuda(), k.cuda()).cpu().numpy() for _ in range(2)]
    finally:
        _cabi.set_single_pass(_cabi.SINGLE_PASS_AUTO)
    assert fc.device_status() == 0
    for got in outs:
        assert np.isfinite(got).all()
        rel, _ = parity_errors(got, want)
        assert rel <= REL_TOL, rel
        assert abs(float(got.sum()) - B) <= REL_TOL * B
