"""This library's power-of-two transforms and the passes fused into them
(mgp_set_fft_mode 1) against cuFFT's 3D plans with the separate k-space and
screening passes (mode 0), at every mesh size they cover below 1024 (which
tests/test_gpu_fft.py covers), for every form of the field passes: the force
pass straight from the density, a multiple of delta(k), the screened
density-plus-source spectrum with each smoothing filter, potential screening
with the separate source spectrum, no screening, a user's screening function,
the closure's force spectra, and batches.

Both are FP32 transforms of the same fields, which agree to a few 1e-7
relative rms; the bound is 1e-5 of each grid's rms, and 1e-4 for the fields
that pass a screening function (its slope amplifies the rounding of the
smoothed field).
"""
import numpy as np
import pytest

import mgpicola as M

pytestmark = pytest.mark.gpu

MODELS = {
    "lcdm": dict(),
    "dgp": dict(model=M.MODEL_DGP, modified_gravity_active=1, include_screening=1, rcH0_DGP=1.0, Rsmooth=2.0,
                smoothing_filter=M.FILTER_GAUSSIAN, input_pofk_is_for_lcdm=0),
    "dgp_tophat": dict(model=M.MODEL_DGP, modified_gravity_active=1, include_screening=1, rcH0_DGP=1.0, Rsmooth=2.0,
                       smoothing_filter=M.FILTER_TOPHAT, input_pofk_is_for_lcdm=0),
    "dgp_linear": dict(model=M.MODEL_DGP, modified_gravity_active=1, include_screening=0, rcH0_DGP=1.0, Rsmooth=2.0,
                       smoothing_filter=M.FILTER_GAUSSIAN, input_pofk_is_for_lcdm=0),
    "fofr": dict(model=M.MODEL_FOFR, modified_gravity_active=1, include_screening=1, fofr0=1e-5, nfofr=1.0,
                 input_pofk_is_for_lcdm=0),
    "fofr_linear": dict(model=M.MODEL_FOFR, modified_gravity_active=1, include_screening=0, fofr0=1e-5, nfofr=1.0,
                        input_pofk_is_for_lcdm=0),
}


def _params(N, model, **kw):
    return M.default_params(Nmesh=N, Nsample=N // 2, Box=2.0 * N, Seed=5003, Init_Redshift=9.0, pofk_nbins=N // 2,
                            pofk_bintype=0, pofk_kmin=0.0, pofk_kmax=0.0, pofk_compute_every_step=1,
                            pofk_subtract_shotnoise=0, **dict(MODELS[model], **kw))


def _rel_rms(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


def _fields(ctx, N, mode, A):
    ctx.set_fft_mode(mode)
    ctx.get_displacements(A)
    out = {"pk": ctx.pofk()[1], "dk": ctx.grid(1)}
    for i, f in enumerate(("fx", "fy", "fz")):
        out[f] = ctx.grid(2 + i)[:, :, :N]
    if ctx.params.modified_gravity_active and (ctx.params.model == M.MODEL_FOFR or ctx.params.include_screening):
        out["source"] = ctx.grid(0)
    if ctx.params.modified_gravity_active and ctx.params.include_screening:
        out["solver"] = ctx.grid(6)[:, :, :N]
    return out


def _compare(own, ref, screened):
    assert own.keys() == ref.keys()
    for f in ref:
        tol = 1e-4 if screened and f in ("fx", "fy", "fz", "source") else 1e-5
        assert _rel_rms(own[f], ref[f]) < tol, f


@pytest.mark.parametrize("N", [64, 128, 256, 512])
@pytest.mark.parametrize("model", list(MODELS))
def test_fields_match_cufft(N, model):
    p = _params(N, model)
    with M.Context(p) as ctx:
        ctx.displacement_fields()
        ref = _fields(ctx, N, 0, 0.5)
        own = _fields(ctx, N, 1, 0.5)
    # the tile deposit's float sums differ from call to call at 1e-7
    _compare(own, ref, p.include_screening and p.modified_gravity_active)


@pytest.mark.parametrize("model", ["dgp", "fofr"])
def test_user_screening_matches_cufft(model):
    N = 64
    hooks = (M.ModelHooks.from_functions(screening_factor_density=lambda a, d: 1.0 / (1.0 + max(0.0, 1.0 + d)))
             if model == "dgp" else
             M.ModelHooks.from_functions(screening_factor_potential=lambda a, u: 0.7 if u < 0 else 1.0))
    with M.Context(_params(N, model), hooks=hooks) as ctx:
        ctx.displacement_fields()
        ref = _fields(ctx, N, 0, 0.5)
        own = _fields(ctx, N, 1, 0.5)
    for f in ("dk", "solver"):
        assert _rel_rms(own[f], ref[f]) < 1e-5, f
    # a potential within rounding of zero may take either side of the step function
    for f in ("fx", "fy", "fz", "source"):
        assert _rel_rms(own[f], ref[f]) < 1e-3, f


@pytest.mark.parametrize("model", ["lcdm", "dgp", "fofr"])
def test_closure_forces_match_cufft(model):
    N = 64
    rng = np.random.default_rng(3)
    w = rng.normal(0, 0.07, (4, 27, 16, 16)).astype(np.float32)
    w[3, :, 3:, :] = 0.0
    with M.Context(_params(N, model)) as ctx, M.Closure(N) as cl:
        cl.set_weights(w, np.zeros((4, 16), np.float32), 1e-3)
        cl.attach(ctx)
        ctx.displacement_fields()
        ref = _fields(ctx, N, 0, 0.5)
        own = _fields(ctx, N, 1, 0.5)
        M.Closure.detach(ctx)
    _compare(own, ref, True)  # the network's BF16 activations round differently


@pytest.mark.parametrize("N,boxes", [(64, 1), (64, 5), (128, 3)])
@pytest.mark.parametrize("model", ["lcdm", "dgp", "fofr", "dgp_linear"])
def test_batch_matches_cufft(N, boxes, model):
    p = _params(N, model)
    lst = [dict(Seed=10 + i, inverted=i % 2, fofr0=1e-5 * (i + 1), rcH0=1.0 + i) for i in range(boxes)]
    out = {}
    for mode in (0, 1):
        with M.Batch(p, lst) as b:
            M._check(M.lib().mgp_set_fft_mode(b.h, mode))
            b.run(3)
            out[mode] = [(b.pofk(i, 3)[1], b.particles(i)[1]) for i in range(boxes)]
    for (pk0, v0), (pk1, v1) in zip(out[0], out[1]):
        assert _rel_rms(pk1, pk0) < 1e-5
        assert _rel_rms(v1, v0) < 1e-4
