"""The built-in x, y and z passes at the edges of their ranges: the shortest
and longest compiled lengths and their neighbours that are not compiled, two-
and three-stage lengths, odd rows (two per line; an odd number of them),
ragged last tiles of rows and of columns, the fused planes of one and of two
parts with and without the z pass that completes them, and grids that share
a launch.

Tolerance: a transform of N points in float32 has a relative L2 error below
about eps log2(N) / 2 with eps = 2^-24 (each of the log2(N) levels adds at
most two roundings of independent sign): 7.6e-7 at 2^25.5 cells."""
import numpy as np
import pytest
import torch

from crava_b200 import api, synth

pytestmark = pytest.mark.gpu

TOL = 7.6e-7

SHAPES = [
    (32, 24, 24),      # the shortest rows and columns
    (30, 21, 20),      # below them: the other passes
    (512, 24, 25),     # the longest even rows
    (24, 512, 27),     # the longest columns
    (70, 35, 512),
    (25, 25, 49),      # odd rows, 25 x 49 rows: an odd number
    (245, 27, 28), (27, 245, 30), (63, 81, 50),
    (50, 243, 343), (96, 200, 300), (40, 360, 400),  # three stages; radix 20
    (64, 64, 24), (128, 64, 35), (64, 128, 45), (128, 128, 64), (256, 64, 54),  # one-part planes
    (256, 256, 64), (256, 256, 128),  # two parts
    (256, 256, 60),    # no z pass for two parts: separate passes
    (525, 28, 32), (28, 525, 32), (48, 25, 525),  # one dimension beyond the range
]


def _numpy(g, nx):
    n = g.shape[0] * g.shape[1] * nx
    return np.fft.rfftn(g[..., :nx].astype(np.float64)) / np.sqrt(n)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _params(nx, ny, nz):
    return synth.Case(nxp=nx, nyp=ny, nzp=nz, angles_deg=[10.0], dt=4.0, low_cut=5.0, high_cut=55.0, wnc=0.1,
                      nz=nz, lz=nz * 4.0, min_rel_thick=1.0, wavelet=synth.ricker_fft_order(nz, 4.0)[None],
                      A=synth.aki_richards_pp([10.0]), theta_cov=np.eye(1), var0=synth.prior_var0(),
                      mu=[], data=[], cov=[], err_corr=None)


@pytest.mark.parametrize("shape", [s for s in SHAPES if all(_smooth(n) for n in s)])
def test_passes_at_the_edges(shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx * 7 + ny * 3 + nz)
    g = np.full((nz, ny, 2 * (nx // 2 + 1)), np.float32(1e9))
    g[..., :nx] = rng.standard_normal((nz, ny, nx), dtype=np.float32)
    ctx = api.Context(_params(nx, ny, nz))
    t = api.to_device(g)
    ctx.fft_r2c(t, api.PARAMETER)
    spec = t.clone()
    assert _rel(api.complex_view(t.cpu().numpy(), nx), _numpy(g, nx)) < TOL
    ctx.fft_c2r(t, api.PARAMETER)
    back = t.cpu().numpy()
    assert _rel(back[..., :nx], g[..., :nx]) < 2 * TOL
    assert np.all(back[..., nx:] == 0.0)
    # the x and y passes alone, then the z pass: the same values
    s = api.to_device(g)
    ctx.fft_xy(s, -1, api.PARAMETER)
    ctx.fft_z(s, -1)
    assert torch.equal(s, spec)
    ctx.fft_z(s, 1)
    ctx.fft_xy(s, 1, api.PARAMETER)
    assert torch.equal(s, t)


@pytest.mark.parametrize("shape", [(32, 24, 24), (25, 27, 49), (64, 64, 30), (256, 256, 64)])
def test_grids_of_one_launch_and_addend(shape):
    """Eleven realisations (33 grids, more than a launch takes) with the mean
    added equal single calls; the constant mean of a unit transforms to zero
    off its DC value."""
    nx, ny, nz = shape
    ctx = api.Context(_params(nx, ny, nz))
    full = (nz, ny, 2 * (nx // 2 + 1))
    gen = torch.Generator(device="cuda").manual_seed(3)
    cov = [torch.zeros(full, device="cuda") for _ in range(6)]
    for c in cov[:3]:
        c[..., 0::2] = 0.5 + torch.rand(full[:2] + (full[2] // 2,), device="cuda", generator=gen)
    mean = [torch.randn(full, device="cuda", generator=gen) for _ in range(3)]
    many = [torch.empty(full, device="cuda") for _ in range(33)]
    ctx.simulate(cov, mean, 5, 0, many)
    for r in (0, 7, 10):
        one = [torch.empty(full, device="cuda") for _ in range(3)]
        ctx.simulate(cov, mean, 5, r, one)
        for a, b in zip(one, many[3 * r:3 * r + 3]):
            assert torch.equal(a[..., :nx], b[..., :nx])
    if all(n & (n - 1) == 0 for n in (nx, ny, nz)):
        c = torch.full(full, 8.006, device="cuda")
        ctx.fft_r2c(c, api.PARAMETER)
        c[0, 0, 0] = 0.0
        assert float(c.abs().max()) == 0.0
