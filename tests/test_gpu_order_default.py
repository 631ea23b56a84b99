"""Which particle order a single box starts with: tile order (the step sorts its
particles) where the mesh splits into tiles and is large, else lattice order."""
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Ns,tiles", [(448, 32, False), (512, 32, True), (592, 32, False), (656, 32, True),
                                        (720, 32, True), (648, 32, False), (648, 648, True), (650, 32, False)])
def test_default_order(N, Ns, tiles):
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=2.0 * N, Seed=1, Init_Redshift=9.0, WhichSpectrum=2, pofk_nbins=8)
    with M.Context(p) as ctx:
        ctx.set_timing(True)
        ctx.displacement_fields()
        ctx.step(0.1, 0.1, 0.15, 0.2)
        assert (ctx.kernel_ms("sort") >= 0) == tiles
