"""The single-pass kernel's exchange, score accumulators and late write-out at the sizes where they change: every cluster
size, halves and groups of a slice without keys, batch entries of one tile (written out one tile after the other), odd
numbers of tiles per cluster, sums written out in the middle of a batch entry."""

import numpy as np
import pytest
import torch

from flash_colsum_b200.inputs import Workload, make_inputs
from oracle import c_oracle
from oracle.naive_colsum import parity_errors

pytestmark = pytest.mark.gpu

# exps as fp16 (2^-11 relative each) of scores whose exps are good to 1e-4: a mean of such terms is off by no more
REL_TOL = 6e-4


@pytest.fixture
def forced():
    """The single pass wherever its shape allows, also where the one-kernel form for few rows would take the call."""
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    from flash_colsum_b200 import _cabi
    _cabi.set_single_pass(_cabi.SINGLE_PASS_ALWAYS)
    _cabi.set_short_fused(_cabi.SHORT_FUSED_NEVER)
    try:
        yield
    finally:
        _cabi.set_single_pass(_cabi.SINGLE_PASS_AUTO)
        _cabi.set_short_fused(_cabi.SHORT_FUSED_AUTO)


def check(q, k, want, cls_len=None):
    import flash_colsum_b200 as fc
    from flash_colsum_b200 import _cabi
    B, H, S, _ = q.shape
    rows = cls_len or S
    assert _cabi.single_pass_applies(B, H, S, sq_rows=rows) and _cabi.short_fused_applies(B, H, rows, S, False, D=64) is None
    for _ in range(2):
        got = fc.flash_colsum(q.cuda(), k.cuda(), cls_len=cls_len).cpu().numpy()
        assert fc.device_status() == 0
        assert np.isfinite(got).all()
        rel, _ = parity_errors(got, want)
        assert rel <= REL_TOL, rel
        # (the tensor core's accumulations truncate; half a unit in the last place each, 1024 at most)
        np.testing.assert_allclose(got.sum(axis=1, dtype=np.float64), 1.0, atol=2e-4)


@pytest.mark.parametrize("B,H,S", [
    (300, 1, 128), (5, 1, 60), (3, 1, 129),          # one or two tiles per batch entry, more entries than clusters
    (2, 3, 256), (2, 3, 257), (2, 3, 384), (2, 3, 385), (2, 3, 512),       # a second slice with 1, 128, 129, 256 keys
    (7, 2, 513), (1, 5, 640), (2, 2, 769), (2, 3, 1024), (2, 2, 1025), (1, 3, 1536), (1, 2, 1793), (1, 2, 2048)])
def test_every_cluster_size_and_ragged_halves(forced, B, H, S):
    q, k = make_inputs(Workload("x", B, H, S, S, 64, "fp16", seed=B + S))
    check(q, k, c_oracle.colsum_c(q, k))


@pytest.mark.parametrize("S", [60, 64, 300, 512, 577, 1024, 1500, 2000, 2048])
def test_batch_entries_of_one_tile_one_after_the_other(forced, S):
    """Padded and not, with and without an exchange: two to three entries per cluster, each written out while the next
    one's sums wait for it."""
    from flash_colsum_b200 import _cabi
    B = _cabi.single_pass_info(S)[1] * 5 // 2
    rows = min(S, 100)
    q, k = make_inputs(Workload("x", B, 1, S, S, 64, "fp16", cls_len=rows, seed=S))
    check(q, k, c_oracle.colsum_c(q, k, cls_len=rows), cls_len=rows)


@pytest.mark.parametrize("S", [120, 128, 577, 1024, 2048])
def test_sums_written_out_inside_a_batch_entry(forced, S):
    """One entry of so many heads that every cluster's share is longer than an accumulation may be (128 query tiles)."""
    from flash_colsum_b200 import _cabi
    tiles = -(-S // 128)
    H = _cabi.single_pass_info(S)[1] * (128 // tiles) * 9 // 8
    gen = torch.Generator(device="cuda").manual_seed(S)
    q, k = (torch.randn(1, H, S, 64, generator=gen, device="cuda", dtype=torch.float16) for _ in range(2))
    want = torch.zeros(1, S, dtype=torch.float64, device="cuda")
    for h in range(0, H, 32):
        s = q[:, h:h + 32].double() @ k[:, h:h + 32].double().transpose(-1, -2) / 8
        want += s.softmax(-1).sum((1, 2)) / (H * S)
    check(q, k, want.cpu().numpy())
