"""Redshift-space multipoles and particle read-out from the tile order.

The tile deposit of the redshift-space displacements (meshes that split into
tiles; particle arrays in lattice or in tile order) against the
lattice-order deposit of the same particles (mgp_set_particle_order 0), over
both tile shapes' edges, meshes without own transforms, lattices that are no
power of two, bins below, at and above what shared memory holds with its
tables, and log bins.  Both are FP32 sums of the same weights with the
positions rounded at another point: 2e-5 of max |P0| for P0, and 100 times
that for P4, whose combination 35 p4 - 30 p2 + 3 p0 amplifies it.
Particles read from tile order are the same bits as after the arrays were
put back in lattice order.
"""
import numpy as np
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu


def _params(N, Ns, nbins, bintype, **kw):
    return M.default_params(Nmesh=N, Nsample=Ns, Box=2.0 * Ns, Seed=11, Init_Redshift=9.0, WhichSpectrum=2,
                            pofk_nbins=nbins, pofk_bintype=bintype, pofk_kmin=0.0 if bintype == 0 else 2 * np.pi / Ns,
                            pofk_kmax=np.pi * N / (2.0 * Ns), pofk_subtract_shotnoise=1, **kw)


@pytest.mark.parametrize("N,Ns,nbins,bintype,sd", [
    (16, 8, 8, 0, 0), (64, 32, 32, 0, 0), (64, 32, 20, 1, 0), (72, 30, 40, 0, 0), (128, 64, 1100, 0, 0),
    (64, 64, 8000, 0, 0), (64, 32, 9000, 0, 0), (512, 128, 256, 0, 0), (576, 96, 64, 0, 0), (128, 64, 64, 0, 1)])
def test_rsd_tiles_match_lattice_order(N, Ns, nbins, bintype, sd):
    with M.Context(_params(N, Ns, nbins, bintype, scaledependent=sd)) as ctx:
        ctx.displacement_fields()
        A = 0.1
        for q in range(2):
            ctx.step(A, A, A + 0.15, A + 0.3)
            A += 0.3
        tiles = ctx.pofk_rsd(A)  # arrays in tile order (but for sd)
        again = ctx.pofk_rsd(A)
        ctx.set_particle_order(1)  # lattice order, tile deposit
        lattice_tiles = ctx.pofk_rsd(A)
        ctx.set_particle_order(0)
        ref = ctx.pofk_rsd(A)
    top = np.max(np.abs(ref[1]))
    assert top > 0
    for got in (tiles, again, lattice_tiles):
        np.testing.assert_array_equal(got[0], ref[0])
        np.testing.assert_array_equal(got[7], ref[7])
        for c, tol in ((1, 2e-5), (2, 4e-4), (3, 2e-3)):
            assert np.max(np.abs(got[c] - ref[c])) < tol * top, c


@pytest.mark.parametrize("N,Ns", [(16, 8), (64, 32), (72, 30), (512, 96)])
def test_particles_from_tile_order(N, Ns):
    with M.Context(_params(N, Ns, 8, 0)) as ctx:
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
