"""The x and y passes of slabs, and the planes they work on.

256x256 planes, which the fused x + y pass splits over two CTAs: the last y
step over the two parts is the z pass's first butterfly where that z pass
follows, and the plane kernel's own where it does not (the x and y passes of a
slab, a z pass that the tuning names).  Both are one pass over the plane and
give the same values.  Slab by slab the passes give the whole grid's values."""
import numpy as np
import pytest
import torch

from crava_b200 import api, synth

pytestmark = pytest.mark.gpu


def _context(nx, ny, nz):
    return api.Context(synth.Case(
        nxp=nx, nyp=ny, nzp=nz, angles_deg=[10.0], dt=4.0, low_cut=5.0, high_cut=55.0, wnc=0.1, nz=nz, lz=nz * 4.0,
        min_rel_thick=1.0, wavelet=synth.ricker_fft_order(nz, 4.0)[None], A=synth.aki_richards_pp([10.0]),
        theta_cov=np.eye(1), var0=synth.prior_var0(), mu=[], data=[], cov=[], err_corr=None))


def _grid(nx, ny, nz, seed=1):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((nz, ny, 2 * (nx // 2 + 1)), device="cuda", generator=gen)


def _launches(f):
    n = api.launch_count()
    f()
    torch.cuda.synchronize()
    return api.launch_count() - n


@pytest.mark.parametrize("nz", [64, 128])
def test_x_and_y_of_a_slab_in_one_pass(nz):
    ctx = _context(256, 256, nz)
    g = _grid(256, 256, nz)
    assert _launches(lambda: ctx.fft_xy(g, -1, api.DATA)) == 1
    assert _launches(lambda: ctx.fft_xy(g, 1, api.DATA)) == 1


@pytest.mark.parametrize("tile_z", [16, 1, 2])
def test_named_z_pass_follows_the_whole_plane_pass(tile_z):
    """Two passes, and the values of the z pass that completes y itself."""
    ctx = _context(256, 256, 64)
    a, b = _grid(256, 256, 64), _grid(256, 256, 64)
    ctx.fft_r2c(a, api.PARAMETER)
    ctx.set_tuning(-1, tile_z, 0, 3, -1, None, 1)
    assert _launches(lambda: ctx.fft_r2c(b, api.PARAMETER)) == 2
    assert torch.equal(a, b)
    assert _launches(lambda: ctx.fft_c2r(b, api.PARAMETER)) == 2
    ctx.set_tuning(-1, -1, 0, 3, -1, None, -1)
    ctx.fft_c2r(a, api.PARAMETER)
    assert torch.equal(a, b)


@pytest.mark.parametrize("nz,tile_z", [(16, -1), (60, -1), (60, 2), (96, 8)])
def test_fused_pass_on_at_any_depth(nz, tile_z):
    """xy_fused = 1 is one pass over the planes whatever the z length, 0 two;
    a float32 transform of N points is within eps log2(N) / 2, eps = 2^-24."""
    ctx = _context(256, 256, nz)
    g = _grid(256, 256, nz)
    ref = torch.fft.rfftn(g[..., :256].double()) / np.sqrt(256 * 256 * nz)
    for xy, passes in ((1, 2), (0, 3)):
        ctx.set_tuning(-1, tile_z, 0, 3, -1, None, xy)
        t = g.clone()
        assert _launches(lambda: ctx.fft_r2c(t, api.PARAMETER)) == passes
        spec = torch.view_as_complex(t.view(nz, 256, 129, 2)).to(ref.dtype)
        assert float((spec - ref).norm() / ref.norm()) < 7.6e-7
        assert _launches(lambda: ctx.fft_c2r(t, api.PARAMETER)) == passes
        assert float((t - g)[..., :256].norm() / g[..., :256].norm()) < 2 * 7.6e-7
        assert float(t[..., 256:].abs().max()) == 0.0


@pytest.mark.parametrize("shape,slabs", [
    ((256, 256, 128), (32, 96)),   # the whole grid has the two-part planes, a slab's depth alone would not
    ((256, 256, 192), (64, 128)),  # the other way round
    ((128, 128, 54), (24, 30)),
    ((64, 48, 50), (25, 25)),
    ((25, 27, 50), (25, 25)),      # odd rows, an odd number of them in a slab
])
def test_slabs_equal_the_whole_transform(shape, slabs):
    """The x and y passes slab by slab and the z pass are the 3-D transform of
    the whole grid bit for bit, forward and inverse."""
    nx, ny, nz = shape
    whole = _context(nx, ny, nz)
    parts, z0 = [], 0
    for n in slabs:
        parts.append((_context(nx, ny, n), slice(z0, z0 + n)))
        z0 += n
    a = _grid(nx, ny, nz)
    b = a.clone()
    whole.fft_r2c(a, api.PARAMETER)
    for ctx, s in parts:
        ctx.fft_xy(b[s], -1, api.PARAMETER, nz)
    whole.fft_z(b, -1)
    assert torch.equal(a, b)
    whole.fft_c2r(a, api.PARAMETER)
    whole.fft_z(b, 1)
    for ctx, s in parts:
        ctx.fft_xy(b[s], 1, api.PARAMETER, nz)
    assert torch.equal(a, b)


@pytest.mark.parametrize("direction", [-1, 1])
def test_odd_rows_keep_to_their_plane(direction):
    """Odd rows are transformed two per line: the last row of a plane of an odd
    number of them is not paired with the next plane's first, so a plane that
    is not finite leaves the others' values alone, bit for bit."""
    nx, ny, nz = 25, 27, 24
    ctx = _context(nx, ny, nz)
    a = _grid(nx, ny, nz)
    b = a.clone()
    b[11] = float("nan")
    for g in (a, b):
        ctx.fft_xy(g, direction, api.PARAMETER)
    assert bool(torch.isnan(b[11][..., :nx]).all())
    rest = [z for z in range(nz) if z != 11]
    assert torch.equal(a[rest], b[rest])


def test_whole_planes_of_several_grids_in_one_launch():
    """Realisations with their means through the pass that completes y, three
    grids per launch, against the separate passes (float32 rounding of one
    inverse transform each, and of the mean's addition)."""
    nx, ny, nz = 256, 256, 24
    ctx = _context(nx, ny, nz)
    gen = torch.Generator(device="cuda").manual_seed(6)
    full = (nz, ny, 2 * (nx // 2 + 1))
    cov = [torch.zeros(full, device="cuda") for _ in range(6)]
    for c in cov[:3]:
        c[..., 0::2] = 0.5 + torch.rand(full[:2] + (full[2] // 2,), device="cuda", generator=gen)
    mean = [torch.randn(full, device="cuda", generator=gen) for _ in range(3)]
    outs = {}
    for xy in (1, 0):
        ctx.set_tuning(-1, -1, 0, 3, -1, None, xy)
        outs[xy] = [torch.empty(full, device="cuda") for _ in range(12)]
        ctx.simulate(cov, mean, 5, 0, outs[xy])
    for a, b in zip(outs[1], outs[0]):
        a, b = a[..., :nx].double(), b[..., :nx].double()
        assert float((a - b).norm() / b.norm()) < 2 * 7.6e-7
