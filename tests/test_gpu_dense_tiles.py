"""The tile kick of lattices with more than 768 particles in a tile of 8 x 8 x 64 cells
(all of a tile's particles no longer fit what the threads read ahead), against the
kick in lattice order: the density after one step of both, for a lattice that is a
power of two and one that is none.

The two deposits add a cell's weights in another order, so the forces agree to about
1e-6 rms and the drifted positions to a few roundings; a cell's density moves by
that fraction of its weights: 1e-5 of the density's rms.
"""
import numpy as np
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Ns", [(512, 310), (512, 512), (576, 340)])
def test_dense_tiles_match_lattice_order(N, Ns):
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=1.0 * N, Seed=7, Init_Redshift=9.0, WhichSpectrum=2, pofk_nbins=8)
    rho = []
    for order in (0, 2):
        with M.Context(p) as ctx:
            ctx.set_particle_order(order)
            ctx.displacement_fields()
            ctx.step(0.1, 0.1, 0.3, 0.5)
            ctx.get_displacements(0.5)
            rho.append(ctx.grid(0)[:, :, :N])
    d = rho[0] - rho[1]
    assert np.sqrt(np.mean(d ** 2, dtype=np.float64)) < 1e-5 * np.sqrt(np.mean(rho[0] ** 2, dtype=np.float64))
