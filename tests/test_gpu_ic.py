"""2LPT initial conditions at the edges of the IC kernels' ranges: lattices
and meshes from the smallest up, every ratio Nmesh / Nsample they tell apart
(1, whole, fractional, below 1), rows that are no multiple of a warp, both
amplitude modes and both mode cuts, against the FP64 oracle.

Tolerances: delta(k) is an FP64 amplitude times an FP32 sine or cosine and
rounded to FP32, 1e-6 relative rms; the displacements pass FP32 transforms,
1e-5 (ZA) and 1e-4 (2LPT) relative rms as for the larger sizes.
"""
import numpy as np
import pytest

import mgpicola as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


@pytest.mark.parametrize("N,Ns", [(8, 4), (8, 8), (12, 4), (30, 15), (20, 8), (66, 33), (24, 36), (64, 16), (96, 96)])
@pytest.mark.parametrize("fixed,inverted,sphere", [(0, 0, 0), (1, 1, 0), (0, 0, 1)])
def test_ic_matches_oracle(N, Ns, fixed, inverted, sphere):
    box, seed = 50.0, 4242
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=box, Seed=seed, Init_Redshift=19.0, WhichSpectrum=2,
                         amplitude_fixed_initial_condition=fixed, inverted_initial_condition=inverted,
                         SphereMode=sphere)
    with M.Context(p) as ctx:
        ctx.displacement_fields()
        dk = ctx.grid(1)
        pos, vel, d1, d2 = ctx.get_particles()
    pw = O.make_power(omega=p.Omega, omega_b=p.OmegaBaryon, h=p.HubbleParam, ns=p.PrimordialIndex, sigma8=p.Sigma8)
    D1, D2, odk, _ = O.ic_2lpt(N, Ns, box, seed, pw, fixed=fixed, inverted=inverted, sphere=sphere, want_k=True)
    assert rel_rms(dk.reshape(-1), odk.reshape(-1)) < 1e-6
    assert rel_rms(d1, D1) < 1e-5
    assert rel_rms(d2, D2) < 1e-4
    assert np.all(vel == 0)
