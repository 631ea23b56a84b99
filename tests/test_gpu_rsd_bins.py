"""Redshift-space multipoles of meshes with many modes a bin against the FP64 oracle:
planar spectra (128, 256) and cuFFT's (90, 130), linear and log bins.

Tolerances, as fractions of P0 with its shot noise, or of the shot noise where a displaced
lattice has less power than that.  A mode's power carries the FP32 transform's error (a
fraction of the field's rms) and the FP32 cell fractions', about 1e-6 together; P2 = 5/2 (3 p2 - p0)
and P4 = 9/8 (35 p4 - 30 p2 + 3 p0) multiply it by at most 10 and 77.  Five times that
bounds every bin.  Beyond |k| = 32 a bin holds 1e4 modes and more, whose errors
average to a hundredth of it: 1e-5 for all three, which FP32 sums over the modes of
a bin, in error by a few 1e-6 times 77, would not meet.
"""
import ctypes as C

import numpy as np
import pytest

import mgpicola as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Ns,nbins,log", [(128, 64, 48, 0), (128, 64, 40, 1), (256, 128, 128, 0), (90, 45, 40, 0),
                                            (130, 52, 50, 1)])
def test_rsd_bins_match_oracle(N, Ns, nbins, log):
    box, A = 2.0 * N, 0.6
    kf = 2 * np.pi / box
    kmin, kmax = (kf, kf * N / 2) if log else (0.0, 0.0)
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=box, Seed=1, Init_Redshift=19.0, WhichSpectrum=2, pofk_nbins=nbins,
                         pofk_bintype=log, pofk_kmin=kmin, pofk_kmax=kmax, pofk_subtract_shotnoise=1)
    rng = np.random.default_rng(N)
    q = np.stack(np.meshgrid(*(np.arange(Ns),) * 3, indexing="ij"), -1).reshape(-1, 3) * (box / Ns)
    pos = np.mod(q + rng.normal(0, 0.5 * box / Ns, q.shape), box).astype(np.float32)
    pos[pos >= box] = 0.0
    # redshift-space shifts of about a cell (the reference wraps them once)
    vel = rng.normal(0, 1.0, pos.shape).astype(np.float32)
    d1, d2 = (rng.normal(0, 1.0, pos.shape).astype(np.float32) for _ in range(2))
    with M.Context(p) as ctx:
        ctx.set_particles(pos, vel, d1, d2)
        k, P0, P2, P4, s0, s2, s4, n = ctx.pofk_rsd(A)
        extra = d1.astype(np.float64) * ctx.growth(1, A) + d2.astype(np.float64) * ctx.growth(4, A)
    H = O.lib().orc_hubble(C.byref(O.make_mg(O.LCDM, p.Omega)), A)
    vnorm = 3.2407789e-18 * (3.085678e24 / 1e5) / A / (100.0 * A * H) * N / box
    res = []
    for axis in (1, 2):
        out = [np.zeros(max(N, nbins)) for _ in range(5)]
        nb = C.c_int(nbins)
        O.lib().orc_pofk_rsd_axis(pos.astype(np.float64), vel.astype(np.float64), extra.ctypes.data, Ns ** 3, axis, N,
                                  Ns, box, vnorm, C.byref(nb), log, 1, kmin, kmax, *out)
        assert nb.value == nbins
        res.append([o[:nbins] for o in out])
    (ky, y0, y2, y4, ny), (_, z0, z2, z4, _) = res
    np.testing.assert_array_equal(n, ny)
    m = ny > 0
    m[0] = False  # bin 0 may hold the k = 0 mode alone
    np.testing.assert_allclose(k[m], ky[m], rtol=1e-13)
    shot = (box / Ns) ** 3
    scale = np.maximum(np.abs(0.5 * (y0 + z0) + shot), shot)
    far = m & (k > 36.0 * kf)
    assert far.sum() >= 4
    for got, a, b, amp in ((P0, y0, z0, 1.0), (P2, y2, z2, 10.0), (P4, y4, z4, 77.0)):
        err = np.abs(got - 0.5 * (a + b)) / scale
        assert err[m].max() < 5e-6 * amp
        assert err[far].max() < 1e-5
