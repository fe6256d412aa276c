"""Workloads of the inversion path, one per call that a program makes.

Each case is one call (or one short sequence of calls) of the public binding
crava_b200.api on one GPU, over the sizes that surveys have in earnest: from
64x64x128 test cubes to the 256x256x512 headline grid, with ragged padded
sizes, three to seven angles, the three solve precisions, device and host
buffers.  The inputs are seeded synthetic surveys made on the GPU with the
formulas of crava_b200/synth.py (prior covariance from correlation functions,
truth = mean + prior realisation, Ricker seismic plus noise).

  listed()             the fixed cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  the inputs and the context a program holds before the call
  run(state)           one pass
  exact(case, seed)    what run returns, from plain torch in 64 bits
  work(case)           bytes and flops a pass cannot do without
"""
import math

import numpy as np
import torch

from crava_b200 import api, synth

PRECISION = {"fp64": api.FP64, "mixed": api.MIXED, "fp32": api.FP32}
PAIRS = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))  # covariance grid order
# State4D's order of the upper triangle and its slot in the grid order above
P4, Q4, SLOT4 = (0, 0, 0, 1, 1, 2), (0, 1, 2, 1, 2, 2), (0, 3, 4, 1, 5, 2)
LOW_CUT, HIGH_CUT, WNC, DT = 5.0, 55.0, 0.1, 4.0
MU = (math.log(3000.0), math.log(1500.0), math.log(2.3))


# ------------------------------------------------------------------ the cases
def _case(name, kind, nx, ny, nz, **more):
    return dict({"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz}, **more)


def listed():
    return [
        # a small test cube: one inversion is many short launches
        _case("unit_small", "unit", 64, 64, 128, ntheta=3, precision="fp64"),
        # a padded survey whose sides are no powers of two, plain FP64 solves
        _case("unit_ragged", "unit", 96, 200, 300, ntheta=5, precision="fp64"),
        # a middle-sized survey with the mixed-precision solve, the binding's default
        _case("unit_mixed", "unit", 192, 160, 384, ntheta=5, precision="mixed"),
        # the headline inversion
        _case("unit_full", "unit", 256, 256, 512, ntheta=5, precision="fp64"),
        # drop-in use from a program with host grids, the reference's FP32 arithmetic
        _case("unit_host", "host", 128, 128, 256, ntheta=3, precision="fp32"),
        # single-grid transforms (FFTGrid::fftInPlace / invFFTInPlace), the large grid
        _case("fft_full", "fft", 256, 256, 512, type=api.PARAMETER),
        # single-grid transforms of a grid with odd sides
        _case("fft_odd", "fft", 125, 150, 225, type=api.COVARIANCE),
        # posterior realisations, a batch of eight (Crava::simulate)
        _case("simulate_full", "simulate", 256, 256, 512, count=8),
        # synthetic seismic of a padded model, all angles (Crava::computeSyntSeismic)
        _case("synth_full", "synth", 256, 256, 512, ntheta=5),
        # wavelet and noise calibration: value and gradients of the likelihood
        _case("likelihood", "likelihood", 192, 160, 384, ntheta=5),
        # time-lapse step between surveys (ModelGeneral::advanceTime)
        _case("advance_time", "advance", 128, 128, 256),
        # two vintages of uneven size, inverted by one graph launch
        _case("vintages", "vintages", 128, 128, 256, nx2=96, ny2=200, nz2=300, ntheta=5, precision="mixed"),
    ]


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _side(rng, lo, hi, even=False):
    """A side that the transforms take (2, 3, 5, 7-smooth), log-uniform."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while not _smooth(n) or (even and n % 2):
        n -= 1
    return n


def draw(rng):
    kind = rng.choice(["unit", "unit", "unit", "fft", "fft", "simulate", "synth", "likelihood", "advance",
                       "host", "vintages"])
    c = {"kind": kind, "nx": _side(rng, 48, 256), "ny": _side(rng, 40, 256), "nz": _side(rng, 64, 512)}
    if kind in ("unit", "synth", "likelihood", "vintages"):
        c["ntheta"] = rng.randint(3, 5 if kind == "likelihood" else 7)
    if kind == "unit":
        c["precision"] = rng.choice(["fp64", "fp64", "mixed", "fp32"])
        if c["nx"] * c["ny"] * c["nz"] > 16e6:
            c["ntheta"] = min(c["ntheta"], 5)
    if kind == "host":
        c = {"kind": kind, "nx": _side(rng, 48, 128), "ny": _side(rng, 40, 128), "nz": _side(rng, 64, 256),
             "ntheta": rng.randint(3, 5), "precision": rng.choice(["mixed", "fp32"])}
    if kind == "fft":
        c["type"] = rng.choice([api.DATA, api.PARAMETER, api.COVARIANCE])
    if kind == "simulate":
        c["count"] = rng.randint(1, 8)
    if kind == "advance":
        c.update(nx=_side(rng, 48, 160), ny=_side(rng, 40, 160), nz=_side(rng, 64, 256))
    if kind == "vintages":
        c.update(nx=_side(rng, 48, 128), ny=_side(rng, 40, 200), nz=_side(rng, 64, 300), nx2=_side(rng, 48, 128),
                 ny2=_side(rng, 40, 200), nz2=_side(rng, 64, 300), precision=rng.choice(["fp64", "mixed"]))
    return c


# ------------------------------------------------------------------ inputs
def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _angles(nt):
    return [40.0 * l / max(nt - 1, 1) for l in range(nt)]


def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 16 + salt)


def _padded(real):
    """[nz, ny, nx] -> the padded layout [nz, ny, 2 (nx / 2 + 1)], padding 0."""
    nx = real.shape[-1]
    out = torch.zeros(real.shape[:2] + (2 * (nx // 2 + 1),), dtype=real.dtype, device=real.device)
    out[..., :nx] = real
    return out


def _grid(spectrum):
    """Complex [nz, ny, nx / 2 + 1] -> the float layout of a transformed grid."""
    return torch.view_as_real(spectrum.contiguous()).reshape(spectrum.shape[:2] + (-1,)).clone()


def _prior_base(nx, ny, nz):
    circ = torch.from_numpy(synth.circ_corr_t(nz, DT, 20.0, LOW_CUT)).cuda()
    lateral = torch.from_numpy(synth.corr_xy(nx, ny, 25.0, 25.0, 500.0)).cuda()
    return circ[:, None, None] * lateral[None], lateral


def _prior_fields(base, gen):
    """Three independent fields with the prior's correlation, in float32."""
    size = tuple(base.shape)
    filt = torch.fft.rfftn(base).real.abs().sqrt()
    return [torch.fft.irfftn(filt * torch.fft.rfftn(torch.randn(size, device="cuda", generator=gen)), s=size)
            for _ in range(3)]


def _survey(nx, ny, nz, nt, seed):
    """The seeded survey: (synth.Case with the parameters, mu, data, cov, err),
    the grids on the GPU in the padded layout."""
    gen = _generator(seed)
    rng = np.random.default_rng(int(seed))
    angles = _angles(nt)
    var0 = synth.prior_var0()
    base, lateral = _prior_base(nx, ny, nz)
    cov = [_padded(base * float(np.float32(var0[p, q]))) for p, q in PAIRS]
    err = torch.zeros_like(base)
    err[0] = lateral
    L0 = np.linalg.cholesky(var0)
    fields = _prior_fields(base, gen)
    truth = [MU[p] + sum(float(L0[p, q]) * fields[q] for q in range(p + 1)) for p in range(3)]
    A = synth.aki_richards_pp(angles)
    wav = np.stack([synth.ricker_fft_order(nz, DT, 25.0, 81, s) for s in rng.uniform(0.8, 1.2, nt)])
    k = torch.arange(nz // 2 + 1, device="cuda", dtype=torch.float64)
    dop = torch.polar(torch.ones_like(k), 2 * math.pi * k / nz) - 1.0
    data, var = [], []
    for l in range(nt):
        imp = sum(float(A[l, p]) * truth[p] for p in range(3))
        W = torch.fft.rfft(torch.from_numpy(wav[l]).cuda().double()).conj() * dop
        sig = torch.fft.irfft(torch.fft.rfft(imp, dim=0) * W.to(torch.complex64)[:, None, None], n=nz, dim=0)
        noise = math.sqrt(0.1 * float(sig.double().square().mean()))
        d = sig + noise * torch.randn(sig.shape, device="cuda", generator=gen)
        var.append(float(d.double().square().mean()) * 0.1 / 1.1)
        data.append(_padded(d))
    theta = np.radians(angles)
    theta_cov = np.sqrt(np.outer(var, var)) * np.exp(-3.0 * np.abs(theta[:, None] - theta[None]) / math.radians(10.0))
    params = synth.Case(nxp=nx, nyp=ny, nzp=nz, angles_deg=angles, dt=DT, low_cut=LOW_CUT, high_cut=HIGH_CUT,
                        wnc=WNC, nz=nz, lz=nz * DT, min_rel_thick=1.0, wavelet=wav, A=A,
                        theta_cov=theta_cov.astype(np.float32).astype(np.float64), var0=var0,
                        mu=[], data=[], cov=[], err_corr=None)
    mu = [_padded(torch.full((nz, ny, nx), MU[p], device="cuda")) for p in range(3)]
    return params, mu, data, cov, _padded(err)


def _like(src):
    mu, data, cov, err = src
    new = lambda gs: [torch.empty_like(g) for g in gs]  # noqa: E731
    return new(mu), new(data), new(cov), torch.empty_like(err)


def _context(params, precision="mixed"):
    return api.Context(params, precision=PRECISION[precision])


def _bare(nx, ny, nz, nt=3):
    """Parameters of a context that is used for its transforms alone."""
    return synth.Case(nxp=nx, nyp=ny, nzp=nz, angles_deg=_angles(nt), dt=DT, low_cut=LOW_CUT, high_cut=HIGH_CUT,
                      wnc=WNC, nz=nz, lz=nz * DT, min_rel_thick=1.0,
                      wavelet=np.stack([synth.ricker_fft_order(nz, DT)] * nt), A=synth.aki_richards_pp(_angles(nt)),
                      theta_cov=np.eye(nt), var0=synth.prior_var0(), mu=[], data=[], cov=[], err_corr=None)


def _decay(nx, ny, nz):
    """A positive spectrum in the layout of a transformed grid."""
    f = lambda n, m: torch.minimum(torch.arange(m), n - torch.arange(m)).double() / n  # noqa: E731
    r2 = (f(nz, nz)[:, None, None] ** 2 * 9 + f(ny, ny)[None, :, None] ** 2 * 25
          + f(nx, nx // 2 + 1)[None, None] ** 2 * 25)
    return (1.0 / (1.0 + r2)).float().cuda()


def _seeded_spd(rng, n):
    g = rng.standard_normal((n, n))
    return g @ g.T / n + 0.5 * np.eye(n)


def _fft_inputs(case, seed):
    """A real grid and the spectrum of another one."""
    nx, ny, nz = _dims(case)
    a, b = (torch.randn((nz, ny, nx), device="cuda", generator=_generator(seed, s)) for s in (1, 2))
    return _padded(a), _grid(torch.fft.rfftn(b) * _scale(case["type"], nx * ny * nz))


def _simulate_inputs(case, seed):
    nx, ny, nz = _dims(case)
    lam = _decay(nx, ny, nz)
    S = _seeded_spd(np.random.default_rng(int(seed)), 3) * 0.01
    cov = [_grid(torch.complex(lam * float(S[p, q]), torch.zeros_like(lam))) for p, q in PAIRS]
    mean = [_padded(MU[p] + 0.1 * torch.randn((nz, ny, nx), device="cuda", generator=_generator(seed, p)))
            for p in range(3)]
    return cov, mean, int(seed) + 17


def _synth_inputs(case, seed):
    """A model padded in every direction (about a tenth), as simboxes are."""
    nx, ny, nz = _dims(case)
    used = max(1, int(0.9 * nx)), max(1, int(0.9 * ny)), max(1, int(0.9 * nz))
    base, _ = _prior_base(nx, ny, nz)
    fields = _prior_fields(base, _generator(seed))
    params = _bare(nx, ny, nz, case["ntheta"])
    params.nz, params.lz = used[2], used[2] * DT
    rng = np.random.default_rng(int(seed))
    params.wavelet = np.stack([synth.ricker_fft_order(nz, DT, 25.0, 81, s) for s in rng.uniform(0.8, 1.2, case["ntheta"])])
    return params, [_padded(MU[p] + 0.1 * fields[p]) for p in range(3)], used


def _likelihood_inputs(case, seed):
    nx, ny, nz = _dims(case)
    nt = case["ntheta"]
    params, mu, data, cov, err = _survey(nx, ny, nz, nt, seed)
    f = lambda g, t: _grid(torch.fft.rfftn(g[..., :nx]) * _scale(t, nx * ny * nz))  # noqa: E731
    src = ([f(g, api.PARAMETER) for g in mu], [f(g, api.DATA) for g in data],
           [f(g, api.COVARIANCE) for g in cov], f(err, api.COVARIANCE))
    rng = np.random.default_rng(int(seed) + 1)
    scale = rng.uniform(0.9, 1.1, nt)
    var = np.diag(params.theta_cov) * rng.uniform(0.8, 1.2, nt)
    spec = np.fft.rfft(params.wavelet.astype(np.float64), axis=-1).T.copy()
    return params, src, scale, var, spec


def _advance_inputs(case, seed):
    nx, ny, nz = _dims(case)
    n = nx * ny * nz
    rng = np.random.default_rng(int(seed))
    gen = _generator(seed)
    lam = _decay(nx, ny, nz)
    zero = torch.zeros_like(lam)
    flat = lambda s: _grid(torch.complex(lam * float(s), zero))  # noqa: E731
    field = lambda: torch.randn((nz, ny, nx), device="cuda", generator=gen)  # noqa: E731
    spec = lambda: _grid(torch.fft.rfftn(field()) / math.sqrt(n))  # noqa: E731
    S = _seeded_spd(rng, 6)
    state = {"ms": [spec() for _ in range(3)], "md": [spec() for _ in range(3)],
             "ss": [flat(S[P4[r], Q4[r]]) for r in range(6)],
             "dd": [flat(S[P4[r] + 3, Q4[r] + 3]) for r in range(6)],
             "sd": [flat(S[l, k + 3]) for l in range(3) for k in range(3)]}
    C = S[:3, :3] + S[3:, 3:] + S[:3, 3:] + S[3:, :3]
    # the inverted survey in the time domain
    mu = [_padded(field()) for _ in range(3)]
    corr = torch.fft.irfftn(lam, s=(nz, ny, nx))
    cov = [_padded(corr * float(0.6 * C[p, q])) for p, q in PAIRS]
    # a contracting transition, so that a long series of steps stays bounded
    E = 0.9 * np.eye(6) + 0.02 * rng.standard_normal((6, 6))
    return state, mu, cov, E, 0.01 * rng.standard_normal(6), _seeded_spd(rng, 6) * 1e-4


# ------------------------------------------------------------------ one pass
def prepare(case, seed):
    kind = case["kind"]
    nx, ny, nz = _dims(case)
    s = {"kind": kind}
    if kind == "unit":
        params, *src = _survey(nx, ny, nz, case["ntheta"], seed)
        s.update(ctx=_context(params, case["precision"]), src=src, dst=_like(src))
    elif kind == "host":
        params, *src = _survey(nx, ny, nz, case["ntheta"], seed)
        host = lambda g: torch.empty(g.shape, pin_memory=True).copy_(g)  # noqa: E731
        mu, data, cov, err = src
        src = [[host(g) for g in mu], [host(g) for g in data], [host(g) for g in cov], host(err)]
        blank = lambda gs: [torch.zeros(g.shape, pin_memory=True) for g in gs]  # noqa: E731
        s.update(ctx=_context(params, case["precision"]), src=src,
                 dst=[blank(src[0]), blank(src[1]), blank(src[2]), blank(src[3:])[0]])
    elif kind == "fft":
        real, spectrum = _fft_inputs(case, seed)
        s.update(ctx=_context(_bare(nx, ny, nz)), real=real, spectrum=spectrum, type=case["type"])
    elif kind == "simulate":
        cov, mean, noise_seed = _simulate_inputs(case, seed)
        s.update(ctx=_context(_bare(nx, ny, nz)), cov=cov, mean=mean, seed=noise_seed,
                 outs=[torch.empty_like(mean[0]) for _ in range(3 * case["count"])])
    elif kind == "synth":
        params, model, used = _synth_inputs(case, seed)
        s.update(ctx=_context(params), model=model, used=used,
                 outs=[torch.empty_like(model[0]) for _ in range(case["ntheta"])])
    elif kind == "likelihood":
        params, src, scale, var, spec = _likelihood_inputs(case, seed)
        s.update(ctx=_context(params), src=src, scale=scale, var=var, spec=spec)
    elif kind == "advance":
        state, mu, cov, E, cm, cc = _advance_inputs(case, seed)
        s.update(ctx=_context(_bare(nx, ny, nz)), state=state, mu=mu, cov=cov, step=(E, cm, cc),
                 work=torch.empty_like(mu[0]), nx=nx, ny=ny)
    elif kind == "vintages":
        s["jobs"] = []
        for k, (a, b, c) in enumerate(((nx, ny, nz), (case["nx2"], case["ny2"], case["nz2"]))):
            params, *src = _survey(a, b, c, case["ntheta"], seed * 2 + k)
            s["jobs"].append({"ctx": _context(params, case["precision"]), "src": src, "dst": _like(src)})
        s["batch"] = api.Batch(s["jobs"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "unit":
        s["ctx"].posterior_unit_oop(s["src"], s["dst"])
        return s["dst"][:3]
    if kind == "host":
        s["ctx"].posterior_unit_host_async(s["src"], s["dst"])
        s["ctx"].host_wait()
        return s["dst"][:3]
    if kind == "fft":
        # both directions in place; the two buffers change roles
        s["ctx"].fft_r2c(s["real"], s["type"])
        s["ctx"].fft_c2r(s["spectrum"], s["type"])
        s["real"], s["spectrum"] = s["spectrum"], s["real"]
        return s["spectrum"], s["real"]
    if kind == "simulate":
        s["ctx"].simulate(s["cov"], s["mean"], s["seed"], 0, s["outs"])
        return s["outs"]
    if kind == "synth":
        s["ctx"].synt_seismic(*s["model"], s["outs"], s["used"][0], s["used"][1])
        return s["outs"]
    if kind == "likelihood":
        return s["ctx"].loglik_grad(*s["src"], s["scale"], s["var"], s["spec"])
    if kind == "advance":
        # the inverted survey to the Fourier domain, then the step, which
        # leaves the next prior in the time domain
        for g in s["mu"]:
            s["ctx"].fft_r2c(g, api.PARAMETER)
        for g in s["cov"]:
            s["ctx"].fft_r2c(g, api.COVARIANCE)
        failed = s["ctx"].advance_time(s["state"], 1, s["nx"], s["ny"], *s["step"], s["mu"], s["cov"], s["work"])
        return s["state"], s["mu"], s["cov"], failed
    s["batch"].run()
    return [job["dst"][:3] for job in s["jobs"]]


# ------------------------------------------------------------------ 64 bits
def _scale(kind, n):
    """FFTGrid's forward scaling."""
    return 1.0 if kind == api.COVARIANCE else 1.0 / math.sqrt(n)


def _forward(grid, nx, kind):
    n = grid.shape[0] * grid.shape[1] * nx
    return torch.fft.rfftn(grid[..., :nx].cuda().double()) * _scale(kind, n)


def _inverse(spec, nx, kind):
    """Real grid in the padded layout; imaginary parts of the x DC and Nyquist
    values are ignored, as a complex-to-real transform does."""
    nz, ny, _ = spec.shape
    s = torch.fft.ifftn(spec, dim=(0, 1))
    s[..., 0].imag = 0.0
    if nx % 2 == 0:
        s[..., -1].imag = 0.0
    real = torch.fft.irfft(s, n=nx, dim=-1)
    return _padded(real if kind == api.COVARIANCE else real * math.sqrt(nx * ny * nz))


def _operators(p):
    """Per-kz operator w, error multipliers and band of the constant-thickness
    inversion, complex128 [nz, ntheta]."""
    nz = p.nzp
    wav = p.wavelet.astype(np.float64)
    back = lambda a: a - np.roll(a, 1, -1)  # noqa: E731
    ahead = lambda a: np.roll(a, -1, -1) - a  # noqa: E731
    g = back(ahead(wav))
    g = 0.5 * (np.roll(g, -1, -1) - np.roll(g, 1, -1))
    W, G = np.fft.fft(wav, axis=-1).T, np.fft.fft(g, axis=-1).T
    k = np.arange(nz)
    D = np.exp(2j * np.pi * k / nz) - 1.0
    freq = (p.nz * 1000.0) / (p.lz * nz) * np.minimum(k, nz - k)
    freq = freq.astype(np.float32)
    band = (freq > np.float32(p.low_cut * p.min_rel_thick)) & (freq < np.float32(p.high_cut))
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return (up(D[:, None] * W.conj()), up(W.conj() / np.linalg.norm(wav, axis=-1)),
            up(G.conj() / np.linalg.norm(g, axis=-1)), band, up(D), up(W))


def _cholesky(M, n):
    """Lower factors of n x n Hermitian matrices, each entry a tensor."""
    L = {}
    for i in range(n):
        for j in range(i + 1):
            v = M[i, j]
            for k in range(j):
                v = v - L[i, k] * L[j, k].conj()
            L[i, j] = v.real.sqrt().to(v.dtype) if i == j else v / L[j, j]
    return L


def _ahead(L, b, n):
    """L^-1 b for one right-hand side (a list of tensors)."""
    x = []
    for i in range(n):
        v = b[i]
        for k in range(i):
            v = v - L[i, k] * x[k]
        x.append(v / L[i, i])
    return x


def _model(p, ops, k, mu, data, cov, err, theta):
    """The Gaussian model of one kz plane: prior S, K S, M and d - K mu."""
    w, e1, e2 = (o[k] for o in ops[:3])
    nt, A = len(p.angles_deg), p.A.astype(np.float64)
    var0 = {}
    S = {}
    for (i, j), c in zip(PAIRS, cov):
        var0[i, j] = float(p.var0[i, j])
        S[i, j] = S[j, i] = (c.real / var0[i, j]).abs() * var0[i, j]
    AS = [[sum(A[l, i] * S[i, j] for i in range(3)) for j in range(3)] for l in range(nt)]
    lam = 0.5 * (1.0 - float(np.float32(p.wnc))) * err.real.abs()
    M = {}
    for l in range(nt):
        for m in range(l + 1):
            B = sum(AS[l][j] * A[m, j] for j in range(3))
            M[l, m] = w[l] * w[m].conj() * B + lam * theta[l, m] * (e1[l] * e1[m].conj() + e2[l] * e2[m].conj())
            if l == m:
                M[l, m] = M[l, m] + float(np.float32(p.wnc)) * theta[l, l]
    KS = [[w[l] * AS[l][j] for l in range(nt)] for j in range(3)]
    r = [data[l] - w[l] * sum(A[l, j] * mu[j] for j in range(3)) for l in range(nt)]
    return S, KS, M, r, A


def _exact_unit(params, src):
    mu, data, cov, err = src
    nx, nt = params.nxp, len(params.angles_deg)
    fm = [_forward(g, nx, api.PARAMETER) for g in mu]
    fd = [_forward(g, nx, api.DATA) for g in data]
    fc = [_forward(g, nx, api.COVARIANCE) for g in cov]
    fe = _forward(err, nx, api.COVARIANCE)
    ops = _operators(params)
    theta = torch.from_numpy(params.theta_cov).cuda()
    for k in range(params.nzp):
        m, d, c = [g[k] for g in fm], [g[k] for g in fd], [g[k] for g in fc]
        S, KS, M, r, A = _model(params, ops, k, m, d, c, fe[k], theta)
        if not ops[3][k]:
            for t, (i, j) in enumerate(PAIRS):
                fc[t][k] = S[i, j].to(fc[t].dtype)
            continue
        L = _cholesky(M, nt)
        Y, z = [_ahead(L, col, nt) for col in KS], _ahead(L, r, nt)
        for j in range(3):
            fm[j][k] = m[j] + sum(y.conj() * v for y, v in zip(Y[j], z))
        for l in range(nt):
            fd[l][k] = d[l] - ops[0][k, l] * sum(A[l, j] * fm[j][k] for j in range(3))
        for t, (i, j) in enumerate(PAIRS):
            fc[t][k] = S[i, j] - sum(a.conj() * b for a, b in zip(Y[i], Y[j]))
    return ([_inverse(g, nx, api.PARAMETER) for g in fm], [_inverse(g, nx, api.DATA) for g in fd],
            [_inverse(g, nx, api.COVARIANCE) for g in fc])


def _normals(seed, stream, counter):
    """Philox-4x32-10 (Salmon et al., SC 2011) and Box-Muller, complex128."""
    lo32 = 0xFFFFFFFF

    def mul(a, m):  # high and low words of a 32 x 32 bit product
        a0, a1, m0, m1 = a & 0xFFFF, a >> 16, m & 0xFFFF, m >> 16
        mid = a1 * m0 + ((a0 * m0) >> 16)
        mid2 = a0 * m1 + (mid & 0xFFFF)
        return a1 * m1 + (mid >> 16) + (mid2 >> 16), ((mid2 & 0xFFFF) << 16) | ((a0 * m0) & 0xFFFF)

    x, y = counter & lo32, counter >> 32
    z, w = torch.full_like(x, stream & lo32), torch.full_like(x, stream >> 32)
    k0, k1 = seed & lo32, seed >> 32
    for _ in range(10):
        h0, l0 = mul(x, 0xD2511F53)
        h1, l1 = mul(z, 0xCD9E8D57)
        x, y, z, w = h1 ^ y ^ k0, l1, h0 ^ w ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & lo32, (k1 + 0xBB67AE85) & lo32
    u1, u2 = ((x >> 8).double() + 1.0) / 2.0 ** 24, (y >> 8).double() / 2.0 ** 24
    return torch.polar((-2.0 * u1.log()).sqrt(), 2.0 * math.pi * u2)


def _noise(seed, stream, nx, ny, nz):
    """Complex white noise under FFTGrid::fillInComplexNoise's rules."""
    cnx = nx // 2 + 1
    i = torch.arange(cnx * ny * nz, device="cuda")
    x, jk = i % cnx, i // cnx
    partner = ((ny - jk % ny) % ny) + ((nz - jk // ny) % nz) * ny
    plane = (x == 0) | ((x == cnx - 1) & (i % 2 == 1))
    alone, mirrored = plane & (partner == jk), plane & (partner < jk)
    v = _normals(seed, stream, torch.where(mirrored, partner * cnx + x, i))
    v = torch.where(alone, torch.complex(v.real, torch.zeros_like(v.real)), v * math.sqrt(0.5))
    return torch.where(mirrored, v.conj(), v).reshape(nz, ny, cnx)


def _exact_simulate(case, seed):
    nx, ny, nz = _dims(case)
    cov, mean, noise_seed = _simulate_inputs(case, seed)
    c = {p: torch.view_as_complex(g.reshape(g.shape[:2] + (-1, 2))).to(torch.complex128) for p, g in zip(PAIRS, cov)}
    L = _cholesky({(q, p): v.conj() if p != q else v for (p, q), v in c.items()}, 3)
    out = []
    for r in range(case["count"]):
        z = [_noise(noise_seed, 3 * r + q, nx, ny, nz) for q in range(3)]
        for p in range(3):
            real = _inverse(sum(L[p, q] * z[q] for q in range(p + 1)), nx, api.PARAMETER)
            out.append(real + mean[p].double())
    return out


def _exact_synth(case, seed):
    p, model, (ux, uy, uz) = _synth_inputs(case, seed)
    nx, ny, nz = _dims(case)
    model = [m.double() for m in model]
    _, _, _, _, D, W = _operators(p)
    z = torch.arange(uz, nz, device="cuda", dtype=torch.float64)[:, None, None]
    out = []
    for l in range(case["ntheta"]):
        imp = sum(float(p.A[l, q]) * model[q] for q in range(3))
        box = imp[:, :uy, :ux].clone()
        if uz < nz:
            box[uz:] = ((z - uz) * box[0] + (nz - z - 1) * box[uz - 1]) / (nz - uz - 1)
        filt = (D * W[:, l].conj())[:, None, None]
        imp[:, :uy, :ux] = torch.fft.ifft(torch.fft.fft(box, dim=0) * filt, dim=0).real
        out.append(imp)
    return out


def _exact_likelihood(case, seed):
    p, src, scale, var, spec = _likelihood_inputs(case, seed)
    nx, ny, nz = _dims(case)
    nt, cn = case["ntheta"], nz // 2 + 1
    cpx = lambda g: torch.view_as_complex(g.reshape(g.shape[:2] + (-1, 2))).to(torch.complex128)  # noqa: E731
    mu, data, cov, err = [cpx(g) for g in src[0]], [cpx(g) for g in src[1]], [cpx(g) for g in src[2]], cpx(src[3])
    ops = list(_operators(p))
    s = torch.from_numpy(scale).cuda().requires_grad_()
    v = torch.from_numpy(var).cuda().requires_grad_()
    W = torch.from_numpy(spec).cuda().requires_grad_()
    weight = torch.full((nx // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
    weight[0] = 1.0
    if nx % 2 == 0:
        weight[-1] = 1.0
    base = torch.from_numpy(p.theta_cov).cuda()
    ratio = v / base.diagonal()
    theta = base * (ratio[:, None] * ratio[None]).sqrt()
    full = torch.cat([W, W[1:nz - cn + 1].flip(0).conj()])
    w_all = s * ops[4][:, None] * full.conj()
    # the gradient of the whole sum plane by plane, through leaf copies
    w_leaf, t_leaf = w_all.detach().requires_grad_(), theta.detach().requires_grad_()
    total = 0.0
    for k in range(nz):
        if not ops[3][k]:
            continue
        ops[0] = w_leaf
        _, _, M, r, _ = _model(p, ops, k, [g[k] for g in mu], [g[k] for g in data], [g[k] for g in cov], err[k], t_leaf)
        L = _cholesky(M, nt)
        term = sum(-2.0 * L[l, l].real.log() for l in range(nt)) - sum(y.abs().square() for y in _ahead(L, r, nt))
        part = (term * weight).sum()
        part.backward()
        total += float(part)
    torch.autograd.backward([w_all, theta], [w_leaf.grad, t_leaf.grad])
    host = lambda t: t.detach().cpu().numpy()  # noqa: E731
    return total, host(s.grad), host(v.grad), host(W.grad), None


def _exact_advance(case, seed):
    state, mu, cov, E, cm, cc = _advance_inputs(case, seed)
    nx, ny, nz = _dims(case)
    n = nx * ny * nz
    cpx = lambda g: torch.view_as_complex(g.reshape(g.shape[:2] + (-1, 2))).to(torch.complex128)  # noqa: E731
    F = {}
    for r in range(6):
        for o, key in ((0, "ss"), (3, "dd")):
            F[P4[r] + o, Q4[r] + o] = cpx(state[key][r])
    for l in range(3):
        for m in range(3):
            F[l, m + 3] = cpx(state["sd"][3 * l + m])
    for i in range(6):
        for j in range(i + 1, 6):
            F[j, i] = F[i, j].conj()
    m = [cpx(g) for g in state["ms"] + state["md"]]
    post_mu = [_forward(g, nx, api.PARAMETER) for g in mu]
    post = {}
    for (i, j), g in zip(PAIRS, cov):
        post[i, j] = post[j, i] = _forward(g, nx, api.COVARIANCE)
    # split: the current state's update spread over the static and dynamic parts
    V = {(i, j): F[i, j] + F[i, j + 3] for i in range(6) for j in range(3)}
    C = {(i, j): V[i, j] + V[i + 3, j] for i in range(3) for j in range(3)}
    L = _cholesky(C, 3)
    B = {}
    for i in range(6):
        y = _ahead(L, [V[i, j].conj() for j in range(3)], 3)
        x = [None] * 3
        for j in (2, 1, 0):
            x[j] = (y[j] - sum(L[t, j].conj() * x[t] for t in range(j + 1, 3))) / L[j, j]
        for j in range(3):
            B[j, i] = x[j]
    H = {(i, j): sum((post[i, t] - C[i, t]) * B[t, j] for t in range(3)) for i in range(3) for j in range(6)}
    dm = [post_mu[t] - (m[t] + m[t + 3]) for t in range(3)]
    m = [m[i] + sum(B[t, i].conj() * dm[t] for t in range(3)) for i in range(6)]
    for i in range(6):
        for j in range(i, 6):
            F[i, j] = F[i, j] + sum(B[t, i].conj() * H[t, j] for t in range(3))
            F[j, i] = F[i, j]  # evolve takes both parts unchanged
    # the time increment's correlation (FFTGrid::fillInGenExpCorr)
    fold = lambda k: torch.minimum(torch.arange(k), k - torch.arange(k)).double().cuda()  # noqa: E731
    ranges = [float(np.float32(v)) / 3.0 for v in (nx, ny)] + [5.0]
    q = ((fold(nz) / ranges[2]).square()[:, None, None] + (fold(ny) / ranges[1]).square()[None, :, None]
         + (fold(nx) / ranges[0]).square()[None, None])
    lam = torch.fft.rfftn(torch.exp(-3.0 * q.sqrt())).real
    m = [sum(E[i, j] * m[j] for j in range(6)) for i in range(6)]
    for i in range(6):
        m[i][0, 0, 0] += cm[i] * math.sqrt(n)
    T = {(i, j): sum(E[i, k] * F[k, j] for k in range(6)) for i in range(6) for j in range(6)}
    F = {(i, j): sum(T[i, k] * E[j, k] for k in range(6)) + cc[i, j] * lam for i in range(6) for j in range(i, 6)}
    new = {"ms": [_grid(g) for g in m[:3]], "md": [_grid(g) for g in m[3:]],
           "ss": [_grid(F[P4[r], Q4[r]]) for r in range(6)],
           "dd": [_grid(F[P4[r] + 3, Q4[r] + 3]) for r in range(6)],
           "sd": [_grid(F[l, k + 3]) for l in range(3) for k in range(3)]}
    merged = [F[i, j] + F[i + 3, j + 3] + F[j, i + 3].conj() + F[i, j + 3] for i, j in PAIRS]
    return (new, [_inverse(m[l] + m[l + 3], nx, api.PARAMETER) for l in range(3)],
            [_inverse(g, nx, api.COVARIANCE) for g in merged], None)


def exact(case, seed):
    kind = case["kind"]
    nx, ny, nz = _dims(case)
    if kind in ("unit", "host"):
        params, *src = _survey(nx, ny, nz, case["ntheta"], seed)
        return _exact_unit(params, src)
    if kind == "fft":
        real, spectrum = _fft_inputs(case, seed)
        spec = torch.view_as_complex(spectrum.reshape(nz, ny, -1, 2)).to(torch.complex128)
        return _grid(_forward(real, nx, case["type"])), _inverse(spec, nx, case["type"])
    if kind == "simulate":
        return _exact_simulate(case, seed)
    if kind == "synth":
        return _exact_synth(case, seed)
    if kind == "likelihood":
        return _exact_likelihood(case, seed)
    if kind == "advance":
        return _exact_advance(case, seed)
    out = []
    for k, (a, b, c) in enumerate(((nx, ny, nz), (case["nx2"], case["ny2"], case["nz2"]))):
        params, *src = _survey(a, b, c, case["ntheta"], seed * 2 + k)
        out.append(_exact_unit(params, src))
    return out


# ------------------------------------------------------------------ what a pass needs
def work(case):
    kind = case["kind"]

    def grid(nx, ny, nz):  # bytes of a grid, flops of its transform
        n = nx * ny * nz
        return 4.0 * 2 * (nx // 2 + 1) * ny * nz, 2.5 * n * math.log2(n)

    def unit(nx, ny, nz):  # all grids in and out; transforms and the solve of the band
        g, f = grid(nx, ny, nz)
        nt = case["ntheta"]
        band = min(1.0, 2 * (HIGH_CUT - LOW_CUT) * DT / 1000.0)
        return np.array([(19 + 2 * nt) * g, (19 + 2 * nt) * f + band * g / 8 * (8 * nt * nt + 87 * nt + 403)])

    g, f = grid(*_dims(case))
    if kind in ("unit", "host"):
        b, w = unit(*_dims(case))
    elif kind == "vintages":
        b, w = unit(*_dims(case)) + unit(case["nx2"], case["ny2"], case["nz2"])
    elif kind == "fft":
        b, w = 4 * g, 2 * f
    elif kind == "simulate":
        b, w = (6 + 3 + 3 * case["count"]) * g, 3 * case["count"] * f
    elif kind == "synth":
        n = g / 4
        b, w = (3 + case["ntheta"]) * g, case["ntheta"] * n * (5 * math.log2(case["nz"]) + 8)
    elif kind == "likelihood":
        nt = case["ntheta"]
        band = min(1.0, 2 * (HIGH_CUT - LOW_CUT) * DT / 1000.0)
        b, w = band * (10 + nt) * g, band * g / 8 * (20 * nt * nt * nt / 3 + 60 * nt * nt)
    else:  # advance: 27 state and 9 survey grids both ways
        b, w = 72 * g, 19 * f
    return {"bytes": float(b), "flops": float(w)}
