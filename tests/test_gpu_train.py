"""The fused training kernel (one kernel per 128-row tile, forward and backward)
and the fixed-order reduction with Adam, at the edges of its tiles: a partial
tile, one row past a tile, and more tiles than blocks resident at once."""
import numpy as np
import pytest
import torch

from oracle import mlp_oracle as M
from pbf_b200 import learned

from test_gpu_mlp import random_params, random_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [127, 129, 148 * 128 + 5])
def test_gradients_at_tile_edges(n):
    feat, target = random_rows(n, 11)
    w, b = random_params(11, feat, target)
    tr = learned.Trainer(w, b, max_batch=n)
    gw, gb, loss = tr.gradients(torch.from_numpy(feat).cuda(), torch.from_numpy(target).cuda())
    rw, rb, rloss = M.gradients(w, b, feat, target)
    assert abs(loss - rloss) <= 2e-2 * rloss
    for g, r in ((gw[M.W1:M.W2], rw[M.W1:M.W2]), (gw[M.W2:M.W3], rw[M.W2:M.W3]), (gw[M.W3:M.W4], rw[M.W3:M.W4]),
                 (gw[M.W4:], rw[M.W4:]), (gb[:193], rb[:193])):
        # BF16 weights and activations: the bounds of the other gradient tests
        assert np.linalg.norm(g - r) <= 4e-2 * np.linalg.norm(r)
        assert np.dot(g, r) >= 0.999 * np.linalg.norm(g) * np.linalg.norm(r)
    tr.close()


def test_padding_rows_add_nothing():
    """One row gives the mean over 128 copies of it: the factor 1/128 commutes with
    every BF16 rounding, so only the FP32 sums' order differs (128 equal terms:
    128 * 2^-24 = 8e-6 relative)."""
    feat, target = random_rows(200, 12)
    w, b = random_params(12, feat, target)
    tr = learned.Trainer(w, b, max_batch=128)
    one = torch.from_numpy(feat[:1]).cuda(), torch.from_numpy(target[:1]).cuda()
    gw1, gb1, l1 = tr.gradients(*one)
    gw2, gb2, l2 = tr.gradients(one[0].repeat(128, 1).contiguous(), one[1].repeat(128).contiguous())
    assert abs(l1 - l2) <= 8e-6 * abs(l1)
    assert np.abs(gw1 - gw2).max() <= 8e-6 * np.abs(gw1).max()
    assert np.abs(gb1 - gb2).max() <= 8e-6 * np.abs(gb1).max()
    tr.close()


def test_step_is_adam_on_the_gradients():
    """Two steps equal Adam on the gradients of the same batches: the parameter's
    own rounding (2^-23 of it), and 1 - beta2^k in float32 (2^-24 / 1e-3 = 6e-5
    relative, half of that under the root) on the step."""
    feat, target = random_rows(600, 13)
    w, b = random_params(13, feat, target)
    f, t = torch.from_numpy(feat).cuda(), torch.from_numpy(target).cuda()
    tr = learned.Trainer(w, b, max_batch=600)
    lr = 1e-3
    p = np.concatenate([w, b[:193]]).astype(np.float64)
    m, v = np.zeros_like(p), np.zeros_like(p)
    for k in (1, 2):
        gw, gb, _ = tr.gradients(f, t)
        g = np.concatenate([gw, gb[:193]]).astype(np.float64)
        tr.step(f, t, lr)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p -= lr * (m / (1 - 0.9 ** k)) / (np.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
        w32, b32, w16 = tr.params()
        got = np.concatenate([w32, b32[:193]])
        big = np.abs(g) > 1e-6  # where the denominator is above its epsilon's reach
        assert np.abs(got - p)[big].max() <= 2e-4 * lr + 2.0 ** -23 * np.abs(p).max()
        assert np.array_equal(w16, learned.bf16_bits(w32))
        assert np.array_equal(b32[193:], b[193:])
    tr.close()
