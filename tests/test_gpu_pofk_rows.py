"""P(k) binning at the edges of its rows: a warp takes 64 modes along kz, two a
lane, and kz = N/2 apart.  N/2 = 8 and 32 fill part of a warp, 45 and 65 leave a
lane one mode (65 in a second pass), 64 is one whole pass; both layouts of the
spectrum (powers of two from 64 on are planar).

Against the FP64 oracle's binning of the same delta(k): a term is rounded at most
17 times on its way to its bin (modulus 2, four rows 3, window 5, lanes and scan 7),
17 2^-24 = 1.0e-6, and all terms are positive (bound 1.2e-6).
"""
import numpy as np
import pytest

import mgpicola as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bintype,nbins,kmin,kmax", [(0, 0, 0.0, 0.0), (1, 12, 0.05, 1.5), (0, 200, 0.1, 0.9)])
@pytest.mark.parametrize("N", [16, 64, 90, 128, 130])
def test_binning_matches_oracle(N, bintype, nbins, kmin, kmax):
    Ns, box = 16, 2.0 * N
    nbins = nbins or N // 2
    rng = np.random.default_rng(N)
    pos = (rng.random((Ns ** 3, 3)) * box * 0.999).astype(np.float32)
    zero = np.zeros_like(pos)
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=box, Seed=1, pofk_nbins=nbins, pofk_bintype=bintype, pofk_kmin=kmin,
                         pofk_kmax=kmax, pofk_subtract_shotnoise=0)
    with M.Context(p) as ctx:
        ctx.set_particles(pos, zero, zero, zero)
        ctx.get_displacements(0.5)
        _, pk, _, n = ctx.pofk()
        dk = ctx.grid(1).astype(np.float64)
    _, ref, _, nref = O.pofk(np.ascontiguousarray(dk), N, Ns, box, nbins, bintype, 0, kmin, kmax)
    np.testing.assert_array_equal(n, nref)
    m = (nref > 0) & (ref > 1e-6 * ref.max())  # not the bin of the k = 0 mode alone
    assert np.max(np.abs(pk[m] / ref[m] - 1)) < 1.2e-6
