"""Synthetic seismic at the edges of its kernel: two- and three-stage z
lengths, one without a compiled kernel, one and eight angles (at 512 layers
eight take the narrow tiles), tiles without a filtered trace, pairs with one,
no padding and one kept layer, against the formulas in float64.

Tolerance on the filtered traces: a forward and an inverse transform of N
points (each eps log2(N) / 2, eps = 2^-24) and a handful of roundings of the
combination and the filter, relative to lines that differ from their first
sample by as much as the output's scale: 1e-6 covers 2 x 2.7e-7 at N = 512 and
the output's factor of the wavelet's pass band."""
import numpy as np
import pytest
import torch

from crava_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,nt,used", [
    ((20, 6, 24), 3, (17, 5, 20)), ((16, 5, 64), 1, (16, 5, 64)), ((18, 7, 300), 5, (3, 2, 250)),
    ((15, 4, 343), 2, (14, 4, 343)), ((16, 3, 375), 3, (13, 2, 300)), ((10, 3, 512), 8, (9, 3, 460)),
    ((35, 9, 512), 5, (33, 1, 1)), ((16, 4, 525), 2, (16, 4, 500)),
])
def test_synthetic_seismic_at_the_edges(shape, nt, used):
    nx, ny, nz = shape
    ux, uy, uz = used
    rng = np.random.default_rng(sum(shape) + nt)
    ang = list(np.linspace(0.0, 40.0, nt))
    wav = np.stack([synth.ricker_fft_order(nz, 4.0, 25.0, 81, 1.0 + 0.1 * l) for l in range(nt)])
    case = synth.Case(nxp=nx, nyp=ny, nzp=nz, angles_deg=ang, dt=4.0, low_cut=5.0, high_cut=55.0, wnc=0.1, nz=uz,
                      lz=uz * 4.0, min_rel_thick=1.0, wavelet=wav, A=synth.aki_richards_pp(ang),
                      theta_cov=np.eye(nt), var0=synth.prior_var0(), mu=[], data=[], cov=[], err_corr=None)
    full = (nz, ny, 2 * (nx // 2 + 1))
    m = [(8.0 - q + 0.1 * rng.standard_normal(full)).astype(np.float32) for q in range(3)]
    ctx = api.Context(case)
    outs = [torch.full(full, 7.0, device="cuda") for _ in range(nt)]
    ctx.synt_seismic(*[api.to_device(g) for g in m], outs, ux, uy)
    k = np.arange(nz)
    D = np.exp(2j * np.pi * k / nz) - 1.0
    z = np.arange(uz, nz)[:, None, None].astype(np.float64)
    for l in range(nt):
        got = outs[l].cpu().numpy()
        A = case.A[l]
        raw = np.float32(0) + m[0] * A[0]
        raw = raw + m[1] * A[1]
        raw = raw + m[2] * A[2]
        imp = sum(np.float64(A[q]) * m[q].astype(np.float64) for q in range(3))[:, :uy, :ux]
        rel = imp - imp[:1]  # H[0] = 0: constants do not pass
        if uz < nz:  # the taper ((z - uz) imp[0] + (nz - z - 1) imp[uz - 1]) / (nz - uz - 1), relative to imp[0]
            rel[uz:] = (nz - z - 1) * rel[uz - 1] / (nz - uz - 1)
        H = D * np.conj(np.fft.fft(wav[l].astype(np.float64)))
        ref = np.fft.ifft(np.fft.fft(rel, axis=0) * H[:, None, None], axis=0).real
        err = np.linalg.norm(got[:, :uy, :ux] - ref)
        assert err <= 1e-6 * max(np.linalg.norm(ref), np.abs(H).max() * np.linalg.norm(rel)), (l, err)
        mask = np.ones(full, bool)
        mask[:, :uy, :ux] = False
        assert np.array_equal(got[mask], raw[mask])
