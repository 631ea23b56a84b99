"""Precision of the closure's bias gradients, sums of one value a voxel over the mesh.

Weights and biases are zero, so the last layer's output gradient is -2 t / (3 V) in BF16
and its bias gradient the sum of that.  Half of the targets are 1, the others s = 2^-14:
both have the same BF16 mantissa, so the gradient with s is 1 + 2^-14 times the one with
zeros in their place, which is exact (8 bits times a count).  What becomes of the
2^-14 shows how many FP32 additions the sum went through:
- sums over a tile (eight products of 16 voxels, at most 64 ones): a tensor core drops what
  lies below 2^-24 of the largest term, 2^-18, a 16th of s, and rounds within a 32nd;
- sums over tiles keep what they round away;
- the blocks' sums add at most 27 roundings of half an ulp below 2^20 ones, 2^-4 each, to the 64
  that all s make up: a 32nd.
Bound: an eighth of the 2^-14.  Without the sums over tiles keeping theirs, a block has up to
1728 ones in a sum, which an s no longer reaches.
"""
import numpy as np
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu


def test_small_terms_survive_in_the_bias_gradient():
    N = 128
    w, b = np.zeros((4, 27, 16, 16), np.float32), np.zeros((4, 16), np.float32)
    t = np.zeros((N ** 3, 3), np.float32)
    t[0::2] = 1.0
    got = []
    with M.Closure(N) as cl:
        cl.set_weights(w, b, 1.0)
        for small in (0.0, 2.0 ** -14):
            t[1::2] = small
            cl.set_sample(np.zeros((N ** 3, 3), np.float32), t)
            got.append(cl.gradients()[2][3, :3].astype(np.float64))
    ratio = got[1] / got[0] - 1.0
    assert np.all(got[0] < 0)
    assert np.all(np.abs(ratio - 2.0 ** -14) < 2.0 ** -17)
