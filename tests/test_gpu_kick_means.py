"""Precision of the means of a kick: each thread sums its particles in FP32, the
threads' sums are added in FP64.

All particles have one velocity c, an integer = 1 mod 4 of b bits, and the kick has no
width, so the velocities stay c.  FP32 sums of up to 2^(24-b) such numbers are
exact and the mean is c; past that every addition rounds down by 1 (the sum
stays a multiple of 4), which a thread with twice the particles shows: an
error of about 1e-6 c.  The particles move by c dt, and the drift subtracts the mean
in the offset of all particles, so what is left of the displacement is the
mean's error times dt, and the rounding of two FP32 numbers of that size and of
their FP32 factor: 3 2^-24 c dt, plus the rounding of positions, 2^-24 box.

2^24 particles on 152 SMs: in lattice order, with four blocks of 256 threads an SM, a
thread has 108 particles and puts its sums aside half-way (b = 18: exact up to 64); in tile
order, with two blocks and tiles of 512 particles on this uniform lattice, it has 216
and does the same (b = 17: exact up to 128).
"""
import numpy as np
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu


def _residual(ctx, pos, vel):
    """Displacement of every particle by a drift without a kick, and the box."""
    zero = np.zeros_like(pos)
    ctx.set_particles(pos, vel, zero, zero)
    ctx.get_displacements(0.5)
    ctx.kick_drift(0.5, 0.5, 0.5, 0.6)
    dx = ctx.get_particles()[0].astype(np.float64) - pos
    return dx - ctx.params.Box * np.round(dx / ctx.params.Box)


@pytest.mark.parametrize("order,bits", [(0, 18), (2, 17)])
def test_mean_of_equal_velocities_is_exact(order, bits):
    N, Ns, box, c = 512, 256, 512.0, 2 ** bits - 3
    q = np.stack(np.meshgrid(*(np.arange(Ns, dtype=np.float32),) * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (q * np.float32(box / Ns)).astype(np.float32)
    pos += np.float32(0.25 * box / N)  # no particle on a face of the box or of a tile
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=box, Seed=1, Init_Redshift=19.0, pofk_nbins=8)
    with M.Context(p) as ctx:
        ctx.set_particle_order(order)
        sign = np.where(np.arange(Ns ** 3) % 2 == 0, 1.0, -1.0).astype(np.float32)
        dt = np.abs(_residual(ctx, pos, np.repeat(sign[:, None], 3, 1))).mean()  # unit velocities of mean zero
        left = _residual(ctx, pos, np.full_like(pos, c))
    assert dt > 1e-3
    assert np.abs(left).max() < 3 * 2.0 ** -24 * c * dt + 2.0 ** -24 * box
