"""Meshes that start in lattice order, put in tile order (mgp_set_particle_order 2): the
particles that a call hands out, the redshift-space multipoles of arrays in tile order, and
short runs against the same runs in lattice order.

Particles read from tile order are the same bits as after the arrays were put back in
lattice order.  Multipoles: the deposits' float sums differ in their order, 2e-5 of max |P0|
for P0 and up to 100 times that for P4, whose combination amplifies it.  Runs: as for one
step, density sums differ at 1e-7 and forces at 1e-6 rms; 1e-5 of the rms velocity and of
the lattice spacing after three steps.
"""
import numpy as np
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu

SIZES = [(16, 8), (32, 16), (64, 32), (64, 64), (72, 30), (90, 45)]


def _params(N, Ns, **kw):
    return M.default_params(Nmesh=N, Nsample=Ns, Box=2.0 * Ns, Seed=11, Init_Redshift=9.0, WhichSpectrum=2,
                            pofk_nbins=N // 2, pofk_bintype=0, pofk_kmin=0.0, pofk_kmax=0.0, **kw)


@pytest.mark.parametrize("N,Ns", SIZES)
def test_particles_from_tile_order(N, Ns):
    with M.Context(_params(N, Ns)) as ctx:
        ctx.set_particle_order(2)
        ctx.displacement_fields()
        ctx.step(0.1, 0.1, 0.25, 0.4)
        tile = ctx.get_particles()
        ctx.get_displacements(0.4)
        mid = ctx.get_particles()  # between the density and the kick
        ctx.set_particle_order(0)
        lat = ctx.get_particles()
    for a, b, c in zip(tile, mid, lat):
        np.testing.assert_array_equal(a, c)
        np.testing.assert_array_equal(b, c)


@pytest.mark.parametrize("N,Ns,nbins,sd", [(16, 8, 8, 0), (64, 32, 32, 0), (72, 30, 40, 0), (128, 64, 1100, 0),
                                           (128, 64, 64, 1)])
def test_rsd_from_tile_order(N, Ns, nbins, sd):
    p = _params(N, Ns, scaledependent=sd)
    p.pofk_nbins = nbins
    with M.Context(p) as ctx:
        ctx.set_particle_order(2)
        ctx.displacement_fields()
        A = 0.1
        for _ in range(2):
            ctx.step(A, A, A + 0.15, A + 0.3)
            A += 0.3
        tiles = ctx.pofk_rsd(A)
        again = ctx.pofk_rsd(A)
        ctx.set_particle_order(0)
        ref = ctx.pofk_rsd(A)
    top = np.max(np.abs(ref[1]))
    for got in (tiles, again):
        np.testing.assert_array_equal(got[7], ref[7])
        for c, tol in ((1, 2e-5), (2, 4e-4), (3, 2e-3)):
            assert np.max(np.abs(got[c] - ref[c])) < tol * top, c


@pytest.mark.parametrize("N,Ns", SIZES)
@pytest.mark.parametrize("model", ["lcdm", "dgp"])
def test_runs_match_lattice_order(N, Ns, model):
    kw = dict(model=M.MODEL_DGP, modified_gravity_active=1, include_screening=1, rcH0_DGP=1.0, Rsmooth=2.0,
              smoothing_filter=M.FILTER_GAUSSIAN) if model == "dgp" else {}
    out = []
    for order in (0, 2):
        with M.Context(_params(N, Ns, **kw)) as ctx:
            ctx.set_particle_order(order)
            ctx.displacement_fields()
            for i in range(3):
                A = 0.1 + 0.2 * i
                ctx.step(A, A, A + 0.1, A + 0.2)
            out.append([a.astype(np.float64) for a in ctx.get_particles()[:2]])
    (x0, v0), (x1, v1) = out
    dx = x0 - x1
    dx -= 2.0 * Ns * np.round(dx / (2.0 * Ns))
    assert np.sqrt(np.mean(dx ** 2)) < 1e-5 * 2.0
    assert np.sqrt(np.mean((v0 - v1) ** 2)) < 1e-5 * np.sqrt(np.mean(v0 ** 2))
