"""The FP32 unit at the headline size and at the uneven vintage grids without
the reference's build: the transforms by torch in 64 bits, rounded to float32,
and between them the per-bin solve of the repository's own C statement of the
reference's loop (float, its order of operations).

Tolerance: the FP32 solve passes the rounding of its input spectra on, up to
4e-5 on the residuals (d - K mu cancels); 1e-4 bounds the two sides' together.
"""
import numpy as np
import pytest
import torch

from crava_b200 import api, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ANGLES5 = (0.0, 10.0, 20.0, 30.0, 40.0)


def _case(name):
    if name == "full":
        return synth.config_full(seed=2, noise_frac=0.10)
    return synth.make_case(*map(int, name.split("x")), ANGLES5, 0.10, seed=43, wavelet_scale_range=(0.8, 1.2))


def _forward(g, nx, scale):
    s = torch.fft.rfftn(torch.from_numpy(g[..., :nx]).cuda().double()) * scale
    return torch.view_as_real(s.to(torch.complex64)).reshape(g.shape).cpu().numpy()


def _inverse(g, nx, scale):
    s = torch.view_as_complex(torch.from_numpy(g).cuda().reshape(g.shape[:2] + (-1, 2))).to(torch.complex128)
    return torch.fft.irfftn(s, s=g.shape[:2] + (nx,), norm="forward") * scale


@pytest.mark.parametrize("name", ["full", "96x200x300", "192x160x384"])
def test_fp32_unit_vs_restated_loop(name):
    case = _case(name)
    nx, n = case.nxp, case.nxp * case.nyp * case.nzp
    ctx = api.Context(case)
    d = lambda gs: [api.to_device(g) for g in gs]
    mu, data, cov, err = d(case.mu), d(case.data), d(case.cov), d([case.err_corr])[0]
    ctx.posterior_unit(mu, data, cov, err, api.FP32)
    st = ctx.stats()
    r = n ** -0.5
    spectra = {"mu": [_forward(g, nx, r) for g in case.mu], "data": [_forward(g, nx, r) for g in case.data],
               "cov": [_forward(g, nx, 1.0) for g in case.cov], "err": _forward(case.err_corr, nx, 1.0)}
    omu, ores, ocov, ofail = O.posterior_fp32(case, spectra)
    assert st.chol_fail_bins == ofail
    assert st.nonfinite_bins == 0
    for g, o, scale in zip(mu + data + cov, omu + ores + ocov, [r] * (3 + len(data)) + [1.0 / n] * 6):
        ref = _inverse(np.ascontiguousarray(o), nx, scale)
        e = float((g[..., :nx].double() - ref).norm() / ref.norm())
        assert e < 1e-4, e
