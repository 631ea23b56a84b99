"""Fields of the initial conditions on this library's transforms (Nmesh and Nsample
powers of two from 64 on), where the smaller sizes of the other tests take cuFFT's:
D1 and D2 of the Gaussian draw against the FP64 oracle for Nmesh = Nsample, 2 and 4
Nsample, every draw mode and mode cut; start velocities without COLA; the IC of given
particles; the scale-dependent fields; the total matter field with massive neutrinos; and
batches, whose boxes share the work grids.

Tolerances as where the sizes are smaller: delta(k) 1e-6 (ZA 1e-5, 2LPT 1e-4) relative
rms; the IC of particles 1e-4 and 1e-3; scale-dependent fields 1e-4; the neutrino sum
1e-5 of cuFFT's in the same context; batches 1e-4 of cuFFT's velocities.
"""
import numpy as np
import pytest

import mgpicola as M
from golden import camb_tables
from oracle import oracle as O
from test_gpu_icfile import gaussian_particles, make, oracle_ic
from test_gpu_nu import params as nu_params
from test_gpu_sd import oracle_fields
from test_gpu_sd import params as sd_params

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


@pytest.mark.parametrize("N,Ns,fixed,inverted,sphere", [
    (64, 64, 0, 0, 0), (64, 64, 1, 1, 0), (64, 64, 0, 0, 1), (128, 64, 0, 1, 0), (128, 64, 1, 0, 0), (128, 64, 0, 0, 1),
    (256, 64, 0, 0, 0), (256, 64, 0, 0, 1), (128, 128, 0, 0, 0)])
def test_ic_matches_oracle(N, Ns, fixed, inverted, sphere):
    box, seed = 100.0, 4242
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


@pytest.mark.parametrize("N,Ns", [(64, 64), (128, 64)])
def test_start_velocities_without_cola(N, Ns):
    """v = D1 dD/dy + D2 dD2/dy at the start (FP32 products of the returned fields)."""
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=100.0, Seed=3, Init_Redshift=19.0, WhichSpectrum=2, UseCOLA=0)
    with M.Context(p) as ctx:
        ctx.displacement_fields()
        _, vel, d1, d2 = ctx.get_particles()
        g1, g2 = ctx.growth(1, 0.05), ctx.growth(4, 0.05)
    ref = d1.astype(np.float64) * g1 + d2.astype(np.float64) * g2
    assert rel_rms(vel, ref) < 1e-6


@pytest.mark.parametrize("N,Ns,model", [(64, 64, "lcdm"), (64, 64, "fofr"), (128, 64, "fofr")])
def test_ic_from_positions_matches_oracle(N, Ns, model):
    p, mg = make(N, Ns, 4.0 * Ns, model)
    pos = gaussian_particles(p)
    with M.Context(p) as c:
        c.displacement_fields_from_positions(pos)
        _, _, d1, d2 = c.get_particles()
    u = pos / p.Box
    u -= np.floor(u)
    D1, D2 = oracle_ic(p, mg, u)
    assert rel_rms(d1, D1) < 1e-4
    assert rel_rms(d2, D2) < 1e-3


@pytest.mark.parametrize("N,Ns", [(64, 64), (128, 64), (256, 64)])
def test_scale_dependent_fields_match_oracle(N, Ns):
    box, A, AFF = 256.0, 0.4, 0.45
    p = sd_params("fofr", N, Ns, box)
    with M.Context(p) as ctx:
        ctx.displacement_fields()
        pos, vel, ic, _ = ctx.get_particles()
        ctx.assign_fields(A, AFF, M.FIELD_ddDddy, M.FIELD_deltaD)  # both fields of a call
        _, _, kick, drift = ctx.get_particles()
        ctx.assign_fields(A, AFF, M.FIELD_D)  # one
        _, _, one, _ = ctx.get_particles()
    D = oracle_fields("fofr", N, Ns, box, 0.05, 0.05, O.FIELD_D)
    q = np.stack(np.meshgrid(*(np.arange(Ns),) * 3, indexing="ij"), -1).reshape(-1, 3) * (box / Ns)
    dx = pos - (q + D)
    dx -= box * np.round(dx / box)
    assert np.abs(dx).max() < 1e-4 * box / Ns
    assert np.all(vel == 0)
    assert rel_rms(ic, D) < 1e-4
    assert rel_rms(kick, oracle_fields("fofr", N, Ns, box, A, AFF, O.FIELD_ddDddy)) < 1e-4
    assert rel_rms(drift, oracle_fields("fofr", N, Ns, box, A, AFF, O.FIELD_deltaD)) < 1e-4
    assert rel_rms(one, oracle_fields("fofr", N, Ns, box, A, AFF, O.FIELD_D)) < 1e-4


@pytest.mark.parametrize("model", ["lcdm", "fofr"])
@pytest.mark.parametrize("Ns", [64, 32])
def test_neutrinos_match_cufft(tmp_path, model, Ns):
    info = camb_tables.write_tables(str(tmp_path))
    with M.Context(nu_params(info, model, N=64, Ns=Ns)) as ctx:
        out = []
        for ic in (0, 1):  # the stored IC field in either layout
            ctx.set_fft_mode(ic)
            ctx.displacement_fields()
            for mode in (0, 1):
                ctx.set_fft_mode(mode)
                ctx.get_displacements(0.6)
                out.append([ctx.grid(1), ctx.pofk(total=True)[1]] + [ctx.grid(2 + a)[:, :, :64] for a in range(3)])
    for got in out[1:]:
        for i, (a, b) in enumerate(zip(got, out[0])):
            # the screened forces amplify rounding as in the FFT size tests
            assert rel_rms(a, b) < (1e-4 if model == "fofr" and i >= 2 else 1e-5), i


@pytest.mark.parametrize("N,Ns,boxes", [(64, 64, 2), (64, 64, 3), (128, 64, 5), (64, 32, 7)])
@pytest.mark.parametrize("model", ["lcdm", "fofr"])
def test_batch_matches_single_boxes(N, Ns, boxes, model):
    """Every box of a batch against a single box of the same seed with cuFFT's transforms:
    groups of the IC that do not divide the batch, and the work grids shared by the boxes."""
    kw = dict(model=M.MODEL_FOFR, modified_gravity_active=1, include_screening=1, fofr0=1e-5, nfofr=1.0,
              input_pofk_is_for_lcdm=0) if model == "fofr" else {}
    p = M.default_params(Nmesh=N, Nsample=Ns, Box=2.0 * Ns, Seed=1, Init_Redshift=9.0, WhichSpectrum=2, pofk_nbins=8,
                         **kw)
    with M.Batch(p, [dict(Seed=10 + i, fofr0=1e-5) for i in range(boxes)]) as b:
        b.run(2)
        got = [b.particles(i) for i in range(boxes)]
    for i in range(boxes):
        with M.Batch(p, [dict(Seed=10 + i, fofr0=1e-5)]) as b:
            M._check(M.lib().mgp_set_fft_mode(b.h, 0))
            b.run(2)
            pos, vel = b.particles(0)
        dx = got[i][0].astype(np.float64) - pos
        dx -= p.Box * np.round(dx / p.Box)
        assert np.sqrt(np.mean(dx ** 2)) < 1e-5 * p.Box / Ns
        assert rel_rms(got[i][1], vel) < 1e-4
