"""The unit and realisations through the built-in passes where several grids
share a launch and where the z pass applies the band-gated covariance rule,
against the same work grid by grid: a z pass named by the tuning (16) takes one
grid per launch and leaves the rule to the solve.  At z lengths that are powers
of two both z passes have the same arithmetic, so the results agree bit for
bit; at others to the rounding of the transforms, which the solve passes on
(relative L2 < 1e-5, as for the other choices of a pass)."""
import numpy as np
import pytest
import torch

from crava_b200 import api, synth

pytestmark = pytest.mark.gpu

A3 = (0.0, 15.0, 30.0)


def _dev(case):
    d = lambda gs: [api.to_device(g) for g in gs]
    return d(case.mu), d(case.data), d(case.cov), d([case.err_corr])[0]


def _unit(ctx, src, tile_z, prec):
    ctx.set_tuning(-1, tile_z, 0, 3, -1)
    dst = [torch.empty_like(g) for g in src[0]], [torch.empty_like(g) for g in src[1]], \
          [torch.empty_like(g) for g in src[2]], torch.empty_like(src[3])
    n = api.launch_count()
    ctx.posterior_unit_oop(src, dst, prec)
    st = ctx.stats()
    return dst[0] + dst[1] + dst[2], (st.nonfinite_bins, st.chol_fail_bins), api.launch_count() - n


def _rel(a, b):
    return float((a - b).double().norm() / b.double().norm())


def test_split_planes_of_many_grids_in_one_launch():
    """256x256x256, above what the L2 holds: all grids of a unit, and all of a
    call's realisations with their means, in one launch per pass."""
    case = synth.make_case(256, 256, 256, (10.0,), 0.1, seed=21)
    ctx = api.Context(case)
    src = _dev(case)
    got, counts, few = _unit(ctx, src, -1, api.FP64)
    ref, counts_ref, many = _unit(ctx, src, 16, api.FP64)
    assert few < 12 < 2 * 21 < many  # 11 grids forward and 10 back, two passes each
    assert counts == counts_ref
    for a, b in zip(got, ref):
        assert torch.equal(a[..., :256], b[..., :256])
    cov = src[2]
    for g in cov:
        ctx.fft_r2c(g, api.COVARIANCE)
    gen = torch.Generator(device="cuda").manual_seed(4)
    mean = [p + torch.randn(got[0].shape, device="cuda", generator=gen) for p in range(3)]
    outs = {}
    for tile_z in (-1, 16):
        ctx.set_tuning(-1, tile_z, 0, 3, -1)
        outs[tile_z] = [torch.empty_like(mean[0]) for _ in range(6)]
        ctx.simulate(cov, mean, 9, 2, outs[tile_z])
    for a, b in zip(outs[-1], outs[16]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("shape", [(48, 40, 60), (45, 27, 75), (30, 32, 343), (256, 256, 64)])
@pytest.mark.parametrize("prec", [api.FP64, api.MIXED])
def test_gated_rule_at_other_lengths_and_split_planes(shape, prec):
    """The rule's values, and with NaNs planted in two of the six prior grids
    its counting (every bin once)."""
    case = synth.make_case(*shape, A3, 0.1, seed=33)
    ctx = api.Context(case)
    src = _dev(case)
    got, counts, _ = _unit(ctx, src, -1, prec)
    ref, counts_ref, _ = _unit(ctx, src, 16, prec)
    assert counts == counts_ref and counts[0] == 0
    nx = shape[0]
    for a, b in zip(got, ref):
        if shape[2] & (shape[2] - 1):
            assert _rel(a[..., :nx], b[..., :nx]) < 1e-5
        else:
            assert torch.equal(a[..., :nx], b[..., :nx])
    src[2][1][5, 7, 9] = np.nan
    src[2][4][20, 3, 2] = np.nan
    got, counts, _ = _unit(ctx, src, -1, prec)
    ref, counts_ref, _ = _unit(ctx, src, 16, prec)
    assert counts == counts_ref and counts[0] == (nx // 2 + 1) * shape[1] * shape[2]
    for a, b in zip(got, ref):
        assert torch.equal(a.isnan(), b.isnan())
