"""The particle order that a single box starts with, and the means of a kick.

Default order: the density, the velocities and the positions of one step against
both explicit orders, up to the order of float sums: a cell adds up to 16 weights
(16 2^-24 of the largest cell, bound 2e-6); forces of the two densities agree to
about 1e-6 rms as the transforms' own error is 5e-7 (bound 1e-5, also of the
lattice spacing for positions).  Sizes on either side of the line (Nmesh 512 in
multiples of 64), the smallest mesh with tiles and one without.

Means: Drift subtracts the mean velocity (src/main.c:747-787).  Particles with a
large common velocity keep their mean position: positions are FP32 numbers below
the box size, so the mean moves by no more than a few roundings of 2^-25 box
(bound 1e-6 box, the common velocity would give above 1e-2 box).  Particle counts
below one warp, a ragged count over a few blocks, and more blocks than are resident
when the particles are taken by lattice order.
"""
import numpy as np
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu


def params(N, Ns):
    return M.default_params(Nmesh=N, Nsample=Ns, Box=2.0 * N, Seed=5001, Init_Redshift=19.0, pofk_nbins=8)


@pytest.mark.parametrize("N,Ns", [(16, 8), (20, 10), (64, 32), (496, 32), (512, 32), (520, 26)])
def test_default_order_matches_explicit_orders(N, Ns):
    box = 2.0 * N
    rng = np.random.default_rng(N)
    q = np.stack(np.meshgrid(*(np.arange(Ns),) * 3, indexing="ij"), -1).reshape(-1, 3) * (box / Ns)
    pos = np.mod(q + rng.normal(0, 0.3 * box / Ns, q.shape), box).astype(np.float32)
    pos[pos >= box] = 0.0
    vel = rng.normal(0, 1.0, q.shape).astype(np.float32)
    d1, d2 = (rng.normal(0, 1.0, q.shape).astype(np.float32) for _ in range(2))
    out = []
    for order in (None, 0, 2):
        with M.Context(params(N, Ns)) as ctx:
            ctx.set_particles(pos, vel, d1, d2)
            if order is not None:
                ctx.set_particle_order(order)
            ctx.get_displacements(0.5)
            rho = ctx.grid(0)[:, :, :N].astype(np.float64)
            ctx.kick_drift(0.45, 0.55, 0.5, 0.6)
            out.append((rho, *(x.astype(np.float64) for x in ctx.get_particles()[:2])))
    rho0, x0, v0 = out[0]
    for rho1, x1, v1 in out[1:]:
        assert np.abs(rho0 - rho1).max() < 2e-6 * np.abs(rho0).max()
        assert np.sqrt(np.mean((v0 - v1) ** 2)) < 1e-5 * np.sqrt(np.mean(v0 ** 2))
        dx = x0 - x1
        dx -= box * np.round(dx / box)
        assert np.sqrt(np.mean(dx ** 2)) < 1e-5 * box / Ns


@pytest.mark.parametrize("N,Ns,size", [(64, 32, (10, 10, 36)), (40, 24, (9, 9, 20)), (512, 64, (20, 20, 72))])
def test_crowded_tiles_match_lattice_order(N, Ns, size):
    """All particles in one corner: tiles with several thousand beside empty ones,
    more than a block reads ahead.  A cell adds about 75 weights, at most 128
    (bound 128 2^-24 of the largest cell)."""
    box = 2.0 * N
    rng = np.random.default_rng(Ns)
    scale = 2.0 * (Ns ** 3 / 9.0 / np.prod(size)) ** (1 / 3)  # nine particles a cell
    pos = (rng.random((Ns ** 3, 3)) * np.array(size) * scale + 5.0).astype(np.float32)
    assert pos.max() < box
    vel, d1, d2 = (rng.normal(0, 1.0, pos.shape).astype(np.float32) for _ in range(3))
    out = []
    for order in (0, 2):
        with M.Context(params(N, Ns)) as ctx:
            ctx.set_particle_order(order)
            ctx.set_particles(pos, vel, d1, d2)
            ctx.get_displacements(0.5)
            rho = ctx.grid(0)[:, :, :N].astype(np.float64)
            ctx.kick_drift(0.45, 0.55, 0.5, 0.6, drift=False)
            out.append((rho, ctx.get_particles()[1].astype(np.float64)))
    assert np.abs(out[0][0] - out[1][0]).max() < 128 * 2.0 ** -24 * np.abs(out[0][0]).max()
    assert np.sqrt(np.mean((out[0][1] - out[1][1]) ** 2)) < 1e-5 * np.sqrt(np.mean(out[0][1] ** 2))


@pytest.mark.parametrize("order", [0, 2])
@pytest.mark.parametrize("N,Ns", [(16, 2), (32, 17), (64, 64)])
def test_drift_subtracts_mean_velocity(N, Ns, order):
    box = 2.0 * N
    rng = np.random.default_rng(Ns)
    pos = (rng.random((Ns ** 3, 3)) * box).astype(np.float32)
    vel = (rng.normal(0, 5, (Ns ** 3, 3)) + [100.0, -50.0, 75.0]).astype(np.float32)
    zero = np.zeros_like(pos)
    with M.Context(params(N, Ns)) as ctx:
        ctx.set_particles(pos, vel, zero, zero)
        ctx.set_particle_order(order)
        for _ in range(2):  # the second finds the block counter as the first left it
            before = ctx.get_particles()[0].astype(np.float64)
            ctx.get_displacements(0.5)
            ctx.kick_drift(0.5, 0.5, 0.5, 0.6)
            dx = ctx.get_particles()[0].astype(np.float64) - before
            dx -= box * np.round(dx / box)
            rms = np.sqrt(np.mean(dx ** 2))
            assert np.abs(dx.mean(0)).max() < 1e-6 * box
            assert rms < 0.2 * box  # no displacement near half the box: the nearest image is the right one
