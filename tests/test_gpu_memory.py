"""Device memory of contexts on this library's transforms, in grids of one box: what a run
holds beside its particles.  Past 256 MB of scratch a batch takes none of its own for the
transforms, a single box one grid, and two more for the initial conditions.

Counted: density, delta(k), three force grids and, for f(R), the solver's; twelve floats a
particle.  Bound: 0.3 grids more for tables, power spectrum sums and allocation steps (the
grids are 539 MB, those of the other mesh 67, an allocation step 2 MB).
"""
import pytest

import mgpicola as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, NS = 512, 256
GRID = 4.0 * N * N * (N + 2)


def _params(**kw):
    return M.default_params(Nmesh=N, Nsample=NS, Box=512.0, Seed=1, Init_Redshift=9.0, WhichSpectrum=2, pofk_nbins=64,
                            **kw)


def _used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_batch_keeps_no_scratch_grids():
    p = _params(model=M.MODEL_FOFR, modified_gravity_active=1, include_screening=1, fofr0=1e-5, nfofr=1.0,
                input_pofk_is_for_lcdm=0)
    before = _used()
    with M.Batch(p, [dict(Seed=1 + i) for i in range(4)]) as b:
        b.run(1)
        grids = (_used() - before) / GRID / 4
    assert grids < 6 + 12 * (NS / N) ** 3 + 0.3


def test_single_box_scratch():
    before = _used()
    with M.Context(_params()) as ctx:
        base = 5 + 12 * (NS / N) ** 3 + 0.3
        ctx.set_particle_order(0)  # no arrays of the tile order
        ctx.get_displacements(0.5)  # particles at the lattice points
        assert (_used() - before) / GRID < base + 1
        ctx.displacement_fields()
        assert (_used() - before) / GRID < base + 3


@pytest.mark.parametrize("n,ns,more", [(256, 128, 0.0), (256, 256, 3.0)])
def test_rsd_multipoles_reuse_the_force_grids(n, ns, more):
    """The redshift-space displacements (three floats a particle) lie in a force grid where they
    fit, else in one staging array; bound 0.2 grids for the bins' sums."""
    p = M.default_params(Nmesh=n, Nsample=ns, Box=256.0, Seed=1, Init_Redshift=9.0, WhichSpectrum=2, pofk_nbins=64)
    with M.Context(p) as ctx:
        ctx.displacement_fields()
        before = _used()
        ctx.pofk_rsd(0.1)
        assert (_used() - before) / (4.0 * n * n * (n + 2)) < more + 0.2
