"""Realisations drawn several per pass, whose generator joins a part formed
once per bin with a part formed once per stream, against the same noise
drawn one stream at a time (noise_fill), filtered (sim_filter), transformed
and added to the mean.  The indices put the streams 3 (first_index + r) + p
below, across and above 2^32, where the parts cannot be joined and where the
high word enters."""
import pytest
import torch

from crava_b200 import api, synth

pytestmark = pytest.mark.gpu

EDGE = 1431655765  # 3 EDGE = 2^32 - 1

# Both sides draw the same words and hold them in FP32; they differ by the
# order of the FP32 transform and of the mean's addition alone, below
# log2(12 * 16 * 36) * 2^-24 = 8e-7 of the largest value.  Another noise is off
# by about the largest value itself.
TOL = 5e-6


@pytest.mark.parametrize("shape", [(16, 12, 32), (15, 9, 32)])
@pytest.mark.parametrize("first", [0, EDGE - 10, EDGE - 3, EDGE + 1])
def test_joined_streams_equal_single_streams(shape, first):
    case = synth.make_case(*shape, (10.0, 25.0), 0.1, seed=3)
    ctx = api.Context(case)
    mu, cov = [[api.to_device(g) for g in gs] for gs in (case.mu, case.cov)]
    for g in cov:
        ctx.fft_r2c(g, api.COVARIANCE)
    count = 9
    outs = [torch.zeros_like(mu[0]) for _ in range(3 * count)]
    ctx.simulate(cov, mu, (7 << 33) + 77, first, outs)
    nx = case.nxp
    for r in range(count):
        one = [torch.zeros_like(mu[0]) for _ in range(3)]
        for p in range(3):
            ctx.noise_fill(one[p], (7 << 33) + 77, 3 * (first + r) + p)
        ctx.sim_filter(cov, one)
        for p in range(3):
            ctx.fft_c2r(one[p], api.PARAMETER)
            want = (one[p] + mu[p])[..., :nx]
            got = outs[3 * r + p][..., :nx]
            top = want.abs().max()
            assert top > 0 and (got - want).abs().max() <= TOL * top, (r, p)
