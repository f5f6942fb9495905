"""The pruning step at the edges of its launch shapes: rows of one CTA, of a cluster of CTAs, and
rows whose slices are read again by every pass."""

import numpy as np
import pytest
import torch

from oracle.naive_colsum import topk_positions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 33, 1024, 1025, 4096, 4097, 8193, 16385, 32769, 65537, 131072, 131073, 300001])
@pytest.mark.parametrize("B,ties", [(1, False), (2, True), (10, True)])    # (one row, and several at once)
def test_selection_at_the_edges_of_the_launch_shapes(S, B, ties):
    if not torch.cuda.is_available():
        pytest.fail("the gpu-marked tests need a CUDA device")
    import flash_colsum_b200 as fc
    g = torch.Generator().manual_seed(S)
    x = torch.randn(B, S, generator=g).exp()
    if ties:
        x = (x * 2).round() / 4
    d = x.cuda()
    for k in sorted({1, (S + 7) // 8, S // 2 + 1, S}):
        val, idx = fc.topk_columns(d, k)
        want = topk_positions(x.numpy(), k)
        np.testing.assert_array_equal(idx.cpu().numpy(), want)
        np.testing.assert_array_equal(val.cpu().numpy(), np.take_along_axis(x.numpy(), want, axis=1))
    for thr in (0.5, 1.5, 1e9):
        idx, cnt = fc.threshold_columns(d, thr)
        for b in range(B):
            keep = np.nonzero(x[b].numpy() >= np.float32(thr))[0]
            assert int(cnt[b]) == len(keep)
            np.testing.assert_array_equal(idx[b, :len(keep)].cpu().numpy(), keep)
            assert (idx[b, len(keep):] == -1).all()
    # the relative form adds the row up in one fixed order: 1024 strided partial sums, a tree, a run
    part = np.zeros((B, 1024), np.float32)
    for i in range(0, S, 1024):
        part[:, :min(1024, S - i)] += x[:, i:i + 1024].numpy()
    tree = part.reshape(B, 32, 32)
    for o in (16, 8, 4, 2, 1):
        tree = tree + tree[:, :, np.arange(32) ^ o]
    total = np.zeros(B, np.float32)
    for w in range(32):
        total += tree[:, w, 0]
    idx, cnt = fc.threshold_columns(d, 1.0, relative=True)
    for b in range(B):
        keep = np.nonzero(x[b].numpy() >= total[b] / np.float32(S))[0]
        assert int(cnt[b]) == len(keep)
        np.testing.assert_array_equal(idx[b, :len(keep)].cpu().numpy(), keep)
