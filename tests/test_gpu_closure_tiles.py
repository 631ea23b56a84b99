"""Closure convolutions at the edges of their tiles, against the FP64 numpy
restatement of the network (oracle/orc_nn.py).

A block of the convolution kernels takes 4 x 4 (forward) or 2 x 4 (weight
gradient) rows by segments of 64 voxels, a warp 32 (or 16) of those: N = 16 is
one part-filled segment, 32 a half, 48 one and a half warps, 80 a whole segment
and a remainder whose halo wraps.  Activations and gradients are BF16 between
layers on both sides, so outputs agree to 1e-2 and gradients to 3e-2 relative
rms, the loss to 1e-3.
"""
import numpy as np
import pytest

import mgpicola as M
from oracle import orc_nn as NN

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


@pytest.mark.parametrize("N", [16, 32, 48, 80])
def test_convolutions_at_tile_edges(N):
    rng = np.random.default_rng(N)
    w = rng.normal(0, 0.15, (4, 27, 16, 16)).astype(np.float32)
    b = rng.normal(0, 0.05, (4, 16)).astype(np.float32)
    w[3, :, 3:, :] = 0.0  # the last layer has three outputs
    b[3, 3:] = 0.0
    x = rng.normal(0, 1, (N ** 3, 3)).astype(np.float32)
    t = rng.normal(0, 1, (N ** 3, 3)).astype(np.float32)
    with M.Closure(N) as cl:
        cl.set_weights(w, b, 2.0)
        cl.set_sample(x, t)
        loss, gw, gb = cl.gradients()
        out = cl.forward()
    X = np.zeros((N, N, N, 16))
    X[..., :3] = x.reshape(N, N, N, 3)
    w64, b64 = w.astype(np.float64), b.astype(np.float64)
    lr, _, gwr, gbr = NN.loss_and_grads(X, w64, b64, t.reshape(N, N, N, 3).astype(np.float64), 2.0)
    _, ref = NN.forward(X, w64, b64)
    assert rel_rms(out, ref[..., :3].reshape(-1, 3)) < 1e-2
    assert abs(loss - lr) / lr < 1e-3
    for l in range(4):
        assert rel_rms(gw[l], gwr[l]) < 3e-2, l
        assert rel_rms(gb[l], gbr[l]) < 3e-2, l
