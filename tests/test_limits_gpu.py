"""Calls at the limits of what the operator takes, against the plain float64 evaluation."""

import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import REL_L2_TOL, ROOT
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


@pytest.mark.parametrize("B,H,Sq,Sk,D,causal,cls", [
    (2, 16, 2000, 2000, 64, False, 1),      # 16 MB an entry: several chunks
    (1, 12, 1500, 1500, 128, False, 4),
    (1, 16, 2, 9000, 64, True, None),
])
def test_host_calls_with_few_rows_outside_the_range_of_fp16(fc, B, H, Sq, Sk, D, causal, cls):
    """Every chunk of an fp32 call takes the few-row forms, which leave values past fp16's range as they are."""
    q, k = make_inputs(Workload("host_fp32", B, H, Sq, Sk, D, "fp32", is_causal=causal, cls_len=cls, seed=Sk))
    q = q * 1e5
    scale = D ** -0.5 / 1e5
    rows = cls or Sq
    ref = [torch.where(t.abs() < 60000, t.half().float(), t) for t in (q[:, :, :rows], k)]
    want = naive_colsum_f64(*ref, scale=scale, is_causal=causal)
    got = fc.flash_colsum_host(q.pin_memory(), k.pin_memory(), scale=scale, is_causal=causal, cls_len=cls)
    assert fc.device_status() == 0
    rel, mx = parity_errors(got.numpy(), want)
    assert rel <= REL_L2_TOL, (rel, mx)


OUT_OF_MEMORY = """
import torch
import flash_colsum_b200 as fc
from flash_colsum_b200.inputs import Workload, make_inputs
q, k = (t.pin_memory() for t in make_inputs(Workload("oom", 8, 16, 2048, 2048, 64, "fp16", seed=5)))
want = fc.flash_colsum_host(q, k)                   # (32 MB an operand; the first chunk's scratch is 7 MB)
torch.cuda.synchronize()
torch.cuda.empty_cache()
total = torch.cuda.get_device_properties(0).total_memory
torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (70 << 20)) / total)
try:
    fc.flash_colsum_host(q, k)
    raise SystemExit("the call found memory after all")
except torch.OutOfMemoryError:
    pass
# the operands' memory comes back for these, and nothing writes to it any more
again = [torch.full((8 << 20,), 1.0, device="cuda") for _ in range(2)]
torch.cuda.synchronize()
torch.cuda.set_per_process_memory_fraction(1.0)
assert all(bool((t == 1.0).all()) for t in again)
del again
torch.testing.assert_close(fc.flash_colsum_host(q, k), want, rtol=3e-4, atol=1e-8)
assert fc.device_status() == 0
"""


def test_a_host_call_that_runs_out_of_memory_leaves_nothing_in_flight(fc):
    """The scratch of the first chunk cannot be had while two chunks are being copied: the call raises torch's
    error after the copies have ended, so that the memory they went to can be used at once.  (In a process of its
    own, whose allocator holds nothing that would serve after all.)"""
    done = subprocess.run([sys.executable, "-c", OUT_OF_MEMORY], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr


def masked_inputs(B, H, Sq, Sk, D, dtype, causal, where, value):
    """Keys that a mask in the first feature takes out: the query's is 1 there, theirs `value`, the others' 0."""
    q, k = make_inputs(Workload("masked", B, H, Sq, Sk, D, dtype, is_causal=causal, seed=Sq + Sk + D))
    q[..., 0], k[..., 0] = 1.0, 0.0
    value = torch.finfo(q.dtype).min if value == "lowest" else float("-inf")
    if where == "tail":
        k[:, :, Sk * 2 // 3:, 0] = value
    elif where == "group":
        k[:, :, 64:128, 0] = value
    else:
        k[:, :, -1, 0] = value
    return q, k


@pytest.mark.parametrize("Sq,Sk,causal", [
    (128, 128, False), (150, 150, False), (200, 200, False), (330, 330, False), (700, 700, False),
    (513, 513, False), (577, 577, False), (1024, 1024, False),           # non-causal (to 64 columns: the single pass)
    (128, 200, True), (128, 700, True), (60, 1500, True),                # one-kernel form
    (200, 200, True), (129, 130, True), (900, 900, True), (300, 5000, True),      # streaming passes
])
@pytest.mark.parametrize("D,dtype,scale", [(128, "fp16", None), (72, "bf16", 1.0), (64, "fp16", None), (40, "bf16", 1.0)])
@pytest.mark.parametrize("where,value", [("tail", "-inf"), ("group", "-inf"), ("last", "-inf"), ("tail", "lowest")])
def test_masked_keys(fc, Sq, Sk, causal, D, dtype, scale, where, value):
    """Scores of -inf weigh nothing, wherever a tile's visible columns begin with a run of them."""
    q, k = masked_inputs(2 if not causal else 1, 3, Sq, Sk, D, dtype, causal, where, value)
    got = fc.flash_colsum(q.cuda(), k.cuda(), scale=scale, is_causal=causal).cpu().numpy()
    assert fc.device_status() == 0
    rel, mx = parity_errors(got, naive_colsum_f64(q, k, scale=scale, is_causal=causal))
    assert rel <= REL_L2_TOL and mx <= REL_L2_TOL, (rel, mx)


@pytest.mark.parametrize("S,D", [(200, 128), (700, 128), (150, 64), (577, 64), (1024, 64)])
def test_a_head_without_a_key_left_gives_nan(fc, S, D):
    """The softmax of nothing but -inf: the batch entry's means are NaN, the other entry's are not."""
    q, k = masked_inputs(2, 3, S, S, D, "fp16", False, "tail", "-inf")
    k[0, 1, :, 0] = float("-inf")
    got = fc.flash_colsum(q.cuda(), k.cuda()).cpu()
    assert torch.isnan(got[0]).all()
    rel, _ = parity_errors(got[1:].numpy(), naive_colsum_f64(q[1:], k[1:]))
    assert rel <= REL_L2_TOL


@pytest.mark.parametrize("S", [150, 256, 577, 1000])
@pytest.mark.parametrize("scale", [1e-36, -1e-36, 0.0])
def test_scales_at_the_end_of_the_range(fc, S, scale):
    """bf16 scores of 1e36 under a scale of 1e-36 are ordinary; under a scale of zero every key counts the same."""
    q, k = make_inputs(Workload("scale", 2, 3, S, S, 64, "fp32", seed=S))
    q, k = (q * 1e18).bfloat16(), (k * 1e17).bfloat16()
    got = fc.flash_colsum(q.cuda(), k.cuda(), scale=scale).cpu().numpy()
    assert fc.device_status() == 0
    rel, mx = parity_errors(got, naive_colsum_f64(q, k, scale=scale))
    assert rel <= REL_L2_TOL, (rel, mx)
    if scale == 0.0 and S % 64 == 0:
        assert (got == 1.0 / S).all()        # (every exp is one, every sum exact)


def with_nan(q, k, what, at):
    t = (q if what == "query" else k).clone()
    t[0, 0, at, 3] = float("nan")
    return (t, k) if what == "query" else (q, t)


@pytest.mark.parametrize("B,H,Sk,D,R,dtype", [
    (2, 4, 577, 64, 1, "fp16"),        # a cluster per batch entry
    (1, 20, 577, 104, 4, "bf16"),      # two kernels
    (2, 4, 5000, 128, 2, "fp16"),
    (50, 8, 60, 64, 2, "fp16"),        # four CTAs of a cluster per SM
    (2, 4, 700, 80, 3, "fp32"),
])
def test_few_rows_pass_nan_on(fc, B, H, Sk, D, R, dtype):
    """A NaN in a key makes its head's rows NaN, and so the batch entry's means; the other entries' stay."""
    q, k = make_inputs(Workload("nan", B, H, R, Sk, D, dtype, is_causal=True, seed=Sk + D))
    want = fc.flash_colsum_causal(q.cuda(), k.cuda(), k_past=Sk).cpu()
    for at in (0, 1, 7, Sk // 2, Sk - 2, Sk - 1):
        qn, kn = with_nan(q, k, "key", at)
        got = fc.flash_colsum_causal(qn.cuda(), kn.cuda(), k_past=Sk).cpu()
        assert torch.isnan(got[0]).all(), at
        torch.testing.assert_close(got[1:], want[1:])


@pytest.mark.parametrize("Sq,Sk,causal", [
    (65, 65, False), (150, 150, False), (256, 256, False), (577, 577, False), (700, 700, False), (1024, 1024, False),
    (128, 200, True), (128, 700, True),                                     # one-kernel form
    (129, 130, True), (300, 300, True), (300, 5000, True), (900, 900, True),     # streaming passes
])
@pytest.mark.parametrize("D,dtype", [(64, "fp16"), (128, "bf16"), (80, "fp32")])
@pytest.mark.parametrize("what,value", [("key", "nan"), ("query", "nan"), ("key", "inf")])
def test_nan_is_passed_on(fc, Sq, Sk, causal, D, dtype, what, value):
    """A NaN in a key that every row sees, or in a query row, makes the batch entry's means NaN (the keys the row
    sees, under a causal mask) and no other's, whichever exp unit its column falls to; so does a score of +inf."""
    q, k = make_inputs(Workload("nan", 2, 2, Sq, Sk, D, dtype, is_causal=causal, seed=Sk + D))
    if value == "inf":
        q = q.abs()
    # (fp32 operands with an infinite value are rounded to bf16, all of them: outside fp16's range)
    qw, kw = (q.bfloat16(), k.bfloat16()) if dtype == "fp32" and value == "inf" else (q, k)
    want = fc.flash_colsum_causal(qw.cuda(), kw.cuda()) if causal else fc.flash_colsum(qw.cuda(), kw.cuda())
    rows = Sq if what == "query" else Sk - Sq + 1 if causal else Sk
    for at in sorted({0, 1, 2, 3, 6, 14, 31, rows // 2, rows - 2, rows - 1} & set(range(rows))):
        qn, kn = with_nan(q, k, what, at)
        if value == "inf":
            kn[0, 0, at, 3] = float("inf")
        got = fc.flash_colsum_causal(qn.cuda(), kn.cuda()) if causal else fc.flash_colsum(qn.cuda(), kn.cuda())
        seen = Sk if not causal or what == "key" else Sk - Sq + at + 1
        assert torch.isnan(got[0, :seen]).all(), (at, int(torch.isnan(got[0]).sum()))
        torch.testing.assert_close(got[1:], want[1:])


def test_number_arguments_of_other_types(fc):
    """What int() takes is a k_past, whether or not the native path has been loaded; only a whole number of
    any integer type is a k."""
    q, k = (t.cuda() for t in make_inputs(Workload("args", 1, 2, 40, 300, 64, "fp16", is_causal=True, seed=3)))
    want = fc.flash_colsum_causal(q, k, k_past=100)
    for k_past in (100.0, 100.9, np.int64(100), np.float32(100), torch.tensor(100)):
        assert torch.equal(fc.flash_colsum_causal(q, k, k_past=k_past) > 0, want > 0)
    everything = fc.flash_colsum_causal(q, k, k_past=300)
    torch.testing.assert_close(fc.flash_colsum_causal(q, k, k_past=2 ** 70), everything)
    for k_top in (5, np.int32(5), torch.tensor(5)):
        assert fc.topk_columns(want, k_top)[1].shape == (1, 5)
    for k_top in (5.0, 5.5, "5"):
        with pytest.raises(TypeError):
            fc.topk_columns(want, k_top)


def test_the_single_sample_launcher_takes_the_first_entry(fc):
    from flash_colsum_b200.ops import _flash_colsum_causal
    q, k = (t.cuda() for t in make_inputs(Workload("first", 3, 2, 40, 300, 64, "fp16", is_causal=True, seed=4)))
    got = _flash_colsum_causal(q, k, 0.125)
    assert got.shape == (1, 300)
    torch.testing.assert_close(got, fc.flash_colsum(q[:1], k[:1], scale=0.125, is_causal=True))
