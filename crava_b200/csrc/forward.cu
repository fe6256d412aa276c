// forward.cu -- synthetic seismic (forward modelling) on the device.
//
// Replaces Crava::computeSyntSeismic (src/crava.cpp:1666-1719) with
// Crava::computeSeismicImpedance (:1632-1663), constant thickness (relative
// thickness and local stretch 1, no local shift or gain).  For angle l:
//   imp = A_l0 alpha + A_l1 beta + A_l2 rho           (every real cell)
//   per trace x < nx, y < ny: imp[z] for z >= nz replaced by the linear
//   taper fac ((z - nz) imp[0] + (nzp - z - 1) imp[nz - 1]),
//   fac = 1 / (nzp - nz - 1); then the cyclic forward difference, the
//   unnormalised FFT, multiplication by conj(W_l(kz)) and the inverse FFT
//   scaled by 1/nzp.
// The difference and the wavelet are applied as one spectral factor
//   H_l(kz) = (exp(2 pi i kz / nzp) - 1) conj(W_l(kz)) / nzp,
// Hermitian in kz (both factors are spectra of real sequences), so two
// adjacent real traces x = 2p, 2p + 1 are filtered together as one complex
// line a + i b: the real grid viewed as complex pairs is exactly the
// complex layout the z column transforms work on.  The compiled lengths do all
// of it in one pass (synt_pass.cuh).  Traces outside
// x < nx, y < ny keep imp, as in the reference.
#include <math.h>

#include <vector>

#include "context.cuh"
#include "synt_pass.cuh"

using namespace crava;

namespace {

constexpr int kThreads = 256;

struct SyntArgs {
  const float2 *m[3];     // alpha, beta, rho as float2 pairs
  float2 *out;            // one angle's output grid as float2 pairs
  const float2 *H;        // [nzp] filter of this angle
  float A[3];
  int cnxp, nyp, nzp, nx, ny, nz;
};

__device__ __forceinline__ float2 imp_at(const SyntArgs &a, long long idx) {
  const float2 x = a.m[0][idx], y = a.m[1][idx], z = a.m[2][idx];
  return make_float2(imp1(x.x, y.x, z.x, a.A), imp1(x.y, y.y, z.y, a.A));
}

// Generic lengths, step 1: impedance and taper written to the output grid.
__global__ void __launch_bounds__(kThreads) k_synt_imp(const __grid_constant__ SyntArgs a) {
  const long long plane = (long long)a.cnxp * a.nyp;
  const long long n = plane * a.nzp;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const int m = (int)(idx / plane);
  const long long col = idx - (long long)m * plane;
  const int y = (int)(col / a.cnxp);
  // relative to the line's first sample: the filter takes constants to zero,
  // and what follows then rounds at the size of the line's variation; below
  // nz the taper fac ((z - nz) imp[0] + (nzp - z - 1) imp[nz - 1])
  const bool tapered = y < a.ny && m >= a.nz;
  const long long from = tapered ? col + (long long)(a.nz - 1) * plane : idx;
  float2 d[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) d[q] = csub(a.m[q][from], a.m[q][col]);
  float2 v = make_float2(imp1(d[0].x, d[1].x, d[2].x, a.A), imp1(d[0].y, d[1].y, d[2].y, a.A));
  if (tapered) v = cscale(v, (1.0f / (float)(a.nzp - a.nz - 1)) * (float)(a.nzp - m - 1));
  a.out[idx] = v;
}

// Generic lengths, step 3: multiply the z spectra by H(kz).
__global__ void __launch_bounds__(kThreads) k_synt_filter(const __grid_constant__ SyntArgs a) {
  const long long plane = (long long)a.cnxp * a.nyp;
  const long long n = plane * a.nzp;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  a.out[idx] = cmul(a.out[idx], __ldg(a.H + idx / plane));
}

// Generic lengths, step 5: traces outside x < nx, y < ny get imp back.
__global__ void __launch_bounds__(kThreads) k_synt_fixup(const __grid_constant__ SyntArgs a) {
  const long long plane = (long long)a.cnxp * a.nyp;
  const long long n = plane * a.nzp;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const long long col = idx % plane;
  const int y = (int)(col / a.cnxp), p = (int)(col % a.cnxp);
  const bool fx = 2 * p < a.nx, fy = 2 * p + 1 < a.nx;
  if (y < a.ny && fx && fy) return;
  const float2 raw = imp_at(a, idx);
  float2 v = a.out[idx];
  if (y >= a.ny || !fx) v.x = raw.x;
  if (y >= a.ny || !fy) v.y = raw.y;
  a.out[idx] = v;
}

// H_l(kz) = D(kz) conj(W_l(kz)) / nzp in double, stored as float2 [nt][nzp];
// the upper half is the exact conjugate mirror of the lower, and the kz = 0
// and Nyquist entries are real (a real-to-complex inverse drops their
// imaginary parts).
std::vector<float2> synt_filters(const crava_gpu_ctx *c) {
  const int nzp = c->p.nzp, nt = c->p.ntheta;
  std::vector<float2> H((size_t)nt * nzp);
  std::vector<double> cs(nzp), sn(nzp);  // e^{-2 pi i m / nzp}
  for (int m = 0; m < nzp; ++m) {
    const double ang = -2.0 * M_PI * (double)m / nzp;
    cs[m] = cos(ang);
    sn[m] = sin(ang);
  }
  for (int l = 0; l < nt; ++l) {
    const float *w = c->wavelet.data() + (size_t)l * nzp;
    for (int k = 0; 2 * k <= nzp; ++k) {
      double wr = 0.0, wi = 0.0;
      for (int n = 0, m = 0; n < nzp; ++n, m = m + k < nzp ? m + k : m + k - nzp) {
        wr += w[n] * cs[m];
        wi += w[n] * sn[m];
      }
      const double ang = 2.0 * M_PI * (double)k / nzp;
      const double dr = cos(ang) - 1.0, di = sin(ang);
      double hr = (dr * wr + di * wi) / nzp, hi = (di * wr - dr * wi) / nzp;
      if (k == 0 || 2 * k == nzp) hi = 0.0;
      H[(size_t)l * nzp + k] = make_float2((float)hr, (float)hi);
      if (k > 0 && 2 * k < nzp) H[(size_t)l * nzp + nzp - k] = make_float2((float)hr, -(float)hi);
    }
  }
  return H;
}

// Synthetic seismic with local wavelets, first step: every angle's
// impedance imp_l = A_l0 alpha + A_l1 beta + A_l2 rho on every cell (the
// reference's float sequence), and on the simbox traces (x < nx, y < ny)
// the tapered trace differenced forward in z (cyclic), the time-domain
// input of the per-trace wavelet filter (src/crava.cpp:1674-1694).  One
// thread per padded trace, x fastest; the three parameter grids are read
// once for all angles.
struct DiffArgs {
  const float *m[3];
  float *out[CRAVA_GPU_MAX_THETA];
  float A[CRAVA_GPU_MAX_THETA][3];
  int rnxp, nyp, nzp, nx, ny, nz;
};

template <int NT>
__global__ void __launch_bounds__(kThreads) k_synt_diff(const __grid_constant__ DiffArgs a) {
  const long long plane = (long long)a.rnxp * a.nyp;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= plane) return;
  const int i = (int)(t % a.rnxp), j = (int)(t / a.rnxp);
  auto imp = [&](int z, int l) {
    const long long o = t + (long long)z * plane;
    return imp1(a.m[0][o], a.m[1][o], a.m[2][o], a.A[l]);
  };
  if (!(i < a.nx && j < a.ny)) {
    for (int z = 0; z < a.nzp; ++z) {
      const long long o = t + (long long)z * plane;
      const float x = a.m[0][o], y = a.m[1][o], w = a.m[2][o];
#pragma unroll
      for (int l = 0; l < NT; ++l) a.out[l][o] = imp1(x, y, w, a.A[l]);
    }
    return;
  }
  // fac ((k - nz) imp[0] + (nzp - k - 1) imp[nz - 1]), fac = 1 / (nzp - nz - 1)
  const float fac = a.nz < a.nzp ? __fdiv_rn(1.0f, (float)(a.nzp - a.nz - 1)) : 0.0f;
  float v0[NT], vl[NT], prev[NT];
#pragma unroll
  for (int l = 0; l < NT; ++l) {
    v0[l] = imp(0, l);
    vl[l] = imp(a.nz - 1, l);
    prev[l] = v0[l];
  }
  for (int z = 0; z + 1 < a.nzp; ++z) {
    const int k = z + 1;
    float x = 0.f, y = 0.f, w = 0.f;
    if (k < a.nz) {
      const long long o = t + (long long)k * plane;
      x = a.m[0][o]; y = a.m[1][o]; w = a.m[2][o];
    }
    const long long oz = t + (long long)z * plane;
#pragma unroll
    for (int l = 0; l < NT; ++l) {
      const float next = k < a.nz ? imp1(x, y, w, a.A[l])
                                  : __fmul_rn(fac, __fadd_rn(__fmul_rn((float)(k - a.nz), v0[l]),
                                                             __fmul_rn((float)(a.nzp - k - 1), vl[l])));
      a.out[l][oz] = __fsub_rn(next, prev[l]);
      prev[l] = next;
    }
  }
  const long long ol = t + (long long)(a.nzp - 1) * plane;
#pragma unroll
  for (int l = 0; l < NT; ++l) a.out[l][ol] = __fsub_rn(v0[l], prev[l]);
}

}  // namespace

extern "C" int crava_gpu_synt_seismic(crava_gpu_ctx *c, const float *alpha, const float *beta,
                                      const float *rho, int nx, int ny, float *const *out) {
  if (!c || !alpha || !beta || !rho || !out) return CRAVA_GPU_ERR_ARG;
  const int nt = c->p.ntheta;
  auto mis = [](const void *p) { return !p || (reinterpret_cast<uintptr_t>(p) & 7u) != 0; };
  if (mis(alpha) || mis(beta) || mis(rho)) return CRAVA_GPU_ERR_ARG;
  for (int l = 0; l < nt; ++l) if (mis(out[l])) return CRAVA_GPU_ERR_ARG;
  if (nx == 0) nx = c->g.nxp;
  if (ny == 0) ny = c->g.nyp;
  const int nz = c->p.nz;
  if (nx < 1 || nx > c->g.nxp || ny < 1 || ny > c->g.nyp || nz < 1 || nz > c->g.nzp) return CRAVA_GPU_ERR_ARG;
  // the taper factor 1 / (nzp - nz - 1) is undefined with one padding layer
  if (nz == c->g.nzp - 1) return CRAVA_GPU_ERR_ARG;
  DeviceGuard guard(c->device);
  if (!c->synt_H) {
    std::vector<float2> H = synt_filters(c);
    if (cudaMalloc(&c->synt_H, H.size() * sizeof(float2)) != cudaSuccess) { c->synt_H = nullptr; return CRAVA_GPU_ERR_ALLOC; }
    CRAVA_CUDA_TRY(cudaMemcpy(c->synt_H, H.data(), H.size() * sizeof(float2), cudaMemcpyHostToDevice));
  }
  const cudaStream_t s = c->stream;
  if (c->plans.pass.synt) {
    // compiled z lengths: all angles in one pass
    SyntPassArgs b;
    b.m[0] = reinterpret_cast<const float2 *>(alpha);
    b.m[1] = reinterpret_cast<const float2 *>(beta);
    b.m[2] = reinterpret_cast<const float2 *>(rho);
    for (int l = 0; l < nt; ++l) {
      b.out[l] = reinterpret_cast<float2 *>(out[l]);
      for (int q = 0; q < 3; ++q) b.A[l][q] = c->A[3 * l + q];
    }
    b.H = c->synt_H;
    b.tw = c->plans.pass.synt;
    b.nt = nt; b.nx = nx; b.ny = ny; b.nz = nz;
    b.cnxp = (uint32_t)c->g.cnxp;
    b.plane = (uint32_t)(c->g.cnxp * c->g.nyp);
    b.fcnxp = make_fastdiv(b.cnxp);
    return synt_launch(c->g.nzp)(b, s);
  }
  SyntArgs a{};
  a.m[0] = reinterpret_cast<const float2 *>(alpha);
  a.m[1] = reinterpret_cast<const float2 *>(beta);
  a.m[2] = reinterpret_cast<const float2 *>(rho);
  a.cnxp = c->g.cnxp; a.nyp = c->g.nyp; a.nzp = c->g.nzp;
  a.nx = nx; a.ny = ny; a.nz = nz;
  const long long n = c->g.csize;
  const dim3 eg((unsigned)((n + kThreads - 1) / kThreads));
  int rc;
  for (int l = 0; l < nt; ++l) {
    a.out = reinterpret_cast<float2 *>(out[l]);
    a.H = c->synt_H + (size_t)l * c->g.nzp;
    for (int q = 0; q < 3; ++q) a.A[q] = c->A[3 * l + q];
    k_synt_imp<<<eg, kThreads, 0, s>>>(a);
    CRAVA_LAUNCH_CHECK();
    if ((rc = fft_cols_z(c->plans, a.out, -1, s))) return rc;
    k_synt_filter<<<eg, kThreads, 0, s>>>(a);
    CRAVA_LAUNCH_CHECK();
    if ((rc = fft_cols_z(c->plans, a.out, 1, s))) return rc;
    k_synt_fixup<<<eg, kThreads, 0, s>>>(a);
    CRAVA_LAUNCH_CHECK();
  }
  return CRAVA_GPU_OK;
}

extern "C" int crava_gpu_synt_seismic_local(crava_gpu_ctx *c, const float *alpha, const float *beta,
                                            const float *rho, int nx, int ny, const double *rel_thick,
                                            float dz, const float *shift, const float *gain, float *const *out) {
  if (!c || !alpha || !beta || !rho || !out || !rel_thick || !(dz > 0.0f)) return CRAVA_GPU_ERR_ARG;
  const int nt = c->p.ntheta;
  auto mis = [](const void *p) { return !p || (reinterpret_cast<uintptr_t>(p) & 7u) != 0; };
  if (mis(alpha) || mis(beta) || mis(rho)) return CRAVA_GPU_ERR_ARG;
  for (int l = 0; l < nt; ++l) if (mis(out[l])) return CRAVA_GPU_ERR_ARG;
  if (nx == 0) nx = c->g.nxp;
  if (ny == 0) ny = c->g.nyp;
  const int nz = c->p.nz;
  if (nx < 1 || nx > c->g.nxp || ny < 1 || ny > c->g.nyp || nz < 1 || nz > c->g.nzp) return CRAVA_GPU_ERR_ARG;
  if (nz == c->g.nzp - 1) return CRAVA_GPU_ERR_ARG;  // the taper divides by nzp - nz - 1
  DeviceGuard guard(c->device);
  DiffArgs a{};
  a.m[0] = alpha; a.m[1] = beta; a.m[2] = rho;
  for (int l = 0; l < nt; ++l) {
    a.out[l] = out[l];
    for (int q = 0; q < 3; ++q) a.A[l][q] = c->A[3 * l + q];
  }
  a.rnxp = c->g.rnxp; a.nyp = c->g.nyp; a.nzp = c->g.nzp; a.nx = nx; a.ny = ny; a.nz = nz;
  const long long ntr = (long long)a.rnxp * a.nyp;
  const dim3 grd((unsigned)((ntr + kThreads - 1) / kThreads));
  const cudaStream_t s = c->stream;
  switch (nt) {
#define CRAVA_DIFF_CASE(N) case N: k_synt_diff<N><<<grd, kThreads, 0, s>>>(a); break;
    CRAVA_DIFF_CASE(1) CRAVA_DIFF_CASE(2) CRAVA_DIFF_CASE(3) CRAVA_DIFF_CASE(4)
    CRAVA_DIFF_CASE(5) CRAVA_DIFF_CASE(6) CRAVA_DIFF_CASE(7) CRAVA_DIFF_CASE(8)
#undef CRAVA_DIFF_CASE
    default: return CRAVA_GPU_ERR_ARG;
  }
  CRAVA_LAUNCH_CHECK();
  // resultVec.fft1DInPlace(), times conj(localWavelet->getCAmp(k, sf)),
  // invFFT1DInPlace() (1 / nzp): the per-trace filter of the multiply-back
  // with no pre-scale and 1 / nzp after
  return multiply_local_wavelet(c, out, rel_thick, nx, ny, dz, shift, gain, 1.0f, (float)c->g.nzp, false);
}
