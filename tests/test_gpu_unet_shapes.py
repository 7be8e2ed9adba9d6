"""The convolutions on volumes whose rows fill no block, one, or several strips: weight
gradients against the CUDA-core reduction, and the forward pass against itself on a crop."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_unet import layout

pytestmark = pytest.mark.gpu


def _net(ib3d, seed=3):
    net = ib3d.Net(seed=seed)
    _, head = layout()
    p = net.get_params()
    p[head:head + 16] = np.random.default_rng(seed).standard_normal(16) * 0.3
    net.set_params(p)
    return net


# levels of 4, 2 and 1 voxels; a batch whose planes share blocks; 20 and 36: rows of no power of two;
# 132: rows of several strips at the first level
@pytest.mark.parametrize("batch,size", [(1, 4), (5, 8), (2, 20), (1, 36), (1, 132)])
def test_weight_gradients_match_the_cuda_core_reduction(ib3d, batch, size):
    """Both sum the same BF16 products in FP32 in different orders: relative norm 1e-4 a block, as
    for the batch of 16^3 voxels."""
    net = _net(ib3d)
    rng = np.random.default_rng(size)
    x = rng.standard_normal((batch, size, size, size, 4)).astype(np.float32)
    t = rng.standard_normal((batch, size, size, size)).astype(np.float32)
    _, tc, out = net.loss_grad(x, t)
    net.set_wgrad_tensor_cores(False)
    _, cc, out2 = net.loss_grad(x, t)
    assert np.array_equal(out, out2)
    for w, b, n, k in layout()[0]:
        assert np.linalg.norm(tc[w:b] - cc[w:b]) <= 1e-4 * np.linalg.norm(cc[w:b]), (n, k)
    net.close()


def test_strips_give_the_bits_of_whole_rows(ib3d):
    """An output depends on the 32 voxels around it; a crop that holds them all, cut at a multiple
    of the pooling, sums the same products in the same order, across the strips' ends too."""
    net = _net(ib3d)
    x = np.random.default_rng(1).standard_normal((1, 132, 132, 132, 4)).astype(np.float32)
    _, _, whole = net.loss_grad(x, np.zeros(x.shape[:4], np.float32))
    c = np.s_[20:116]
    _, _, crop = net.loss_grad(np.ascontiguousarray(x[:, c, c, c]), np.zeros((1, 96, 96, 96), np.float32))
    a, b = np.s_[52:84], np.s_[32:64]
    assert np.array_equal(whole[:, a, a, a], crop[:, b, b, b])
    net.close()


# several voxels a thread; the smallest; a batch
@pytest.mark.parametrize("batch,size", [(1, 4), (1, 108), (3, 64)])
def test_loss_adds_voxels_in_fp64(ib3d, batch, size):
    """A zero head gives an output of 0, so a constant target t leaves one FP32 square, t * t rounded,
    a voxel: their mean is that square. The FP64 additions of at most 150 terms a thread, 5 + 8 a
    block and one a block into the total (1,024 blocks at most), and the quotients, are off by less
    than 2,000 * 2^-53 of it."""
    net = ib3d.Net(seed=3)
    _, head = layout()
    p = net.get_params()
    p[head:head + 17] = 0.0
    net.set_params(p)
    x = np.random.default_rng(0).standard_normal((batch, size, size, size, 4)).astype(np.float32)
    t = np.float32(0.7)
    loss, _, out = net.loss_grad(x, np.full(x.shape[:4], t, np.float32))
    net.close()
    assert not out.any()
    square = float(t * t)
    assert abs(loss - square) <= 2000 * 2.0 ** -53 * square
