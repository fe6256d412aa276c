// synt_pass.cuh -- synthetic seismic of all angles in one pass over HBM.
//
// Impedance, taper, difference and wavelet are linear in the three parameters
// and the angle enters only through the coefficients A_l and the filter H_l, so
// a trace pair is transformed once per parameter and back once per angle:
//   out_l = IDFT( H_l(k) sum_p A_lp DFT(m_p)(k) ),
// 3 + nt transforms instead of 2 nt.  A CTA holds kTX trace pairs (adjacent
// complex columns) of the three parameters in shared memory; the lines are
// transformed in place stage by stage (fft_line.cuh); the last forward stage
// keeps its butterflies' outputs in registers, forms each angle's filtered
// combination there and does the first inverse butterfly on it.  The inverse
// stages undo the forward ones in reverse order on the same slots (inverse
// butterfly, then the conjugate twiddles), so its first stage needs the very
// values the last forward stage has, and its last leaves in natural order.
//
// H_l(0) = 0: a constant does not reach the output, so every line is taken
// relative to its first sample, which keeps the transforms' rounding at the
// size of the trace's variation instead of its level.
//
// 256x256x512, five angles: 415 us (1.08 GB, 2.6 TB/s; one 512-thread CTA per SM
// with 160 KB of lines: bound by the latency of its phases) against 847 us for
// the earlier kernel (forward and inverse transform per angle, 32-byte runs, two
// buffers per stage); error against 64 bits 5e-8 instead of 3e-7.  A first form
// that read its twiddles and filters from L2 in the angle loop and the
// unfiltered traces one value at a time took 801 us.
#pragma once

#include "common.cuh"
#include "fft_line.cuh"

namespace crava {

// Radices up to 10 (the last forward stage holds three lines' butterflies),
// the largest first.
__host__ __device__ constexpr LineList synt_list(int n) {
  LineList best{};
  for (int c = 2; c <= 10; ++c)
    for (int b = c; b >= 2; --b) {
      if (n % c || (n / c) % b) continue;
      const int a = n / c / b;
      if (a < 1 || a > b || a > 10) continue;
      best.n = a == 1 ? 2 : 3;
      best.r[0] = c;
      best.r[1] = b;
      best.r[2] = a;
      return best;
    }
  return best;
}
template <int N, class I>
struct SyntLineImpl;
template <int N, size_t... I>
struct SyntLineImpl<N, std::index_sequence<I...>> {
  using type = CtLine<0, synt_list(N).r[I]...>;
};

// ((0 + alpha A0) + beta A1) + rho A2 with separate roundings, the
// reference's float sequence (no fused multiply-add), so the traces the
// reference leaves unfiltered match it bit for bit.
__device__ __forceinline__ float imp1(float x, float y, float z, const float *A) {
  float r = __fadd_rn(0.0f, __fmul_rn(x, A[0]));
  r = __fadd_rn(r, __fmul_rn(y, A[1]));
  return __fadd_rn(r, __fmul_rn(z, A[2]));
}

struct SyntPassArgs {
  const float2 *m[3];
  float2 *out[CRAVA_GPU_MAX_THETA];
  const float2 *H;   // [nt][nzp]
  const float2 *tw;  // stage tables of the line
  float A[CRAVA_GPU_MAX_THETA][3];
  int nt, nx, ny, nz;
  uint32_t cnxp, plane;  // complex columns of a row, of a plane
  FastDiv fcnxp;
};

// TX trace pairs per CTA: 8 (64-byte runs), 4 where eight angles' buffers would
// not fit.
template <int N, int TX>
struct SyntCfg {
  using L = typename SyntLineImpl<N, std::make_index_sequence<synt_list(N).n>>::type;
  static constexpr int NTH = N > 256 ? 512 : 256;
  // an even last radix: the low slot bit takes the parity of the digit above,
  // so that the two slots of an access lie in different halves of the banks
  static constexpr int RL = L::R(L::nst() - 1);
  static __device__ __forceinline__ int at(int slot, int c) {
    return (RL % 2 == 0 ? slot ^ ((slot / RL) & 1) : slot) * TX + c;
  }
  static constexpr size_t smem(int nt) {
    return sizeof(float2) * ((size_t)N * TX * (nt < 3 ? 3 : nt) + (size_t)nt * N + L::entries());
  }
};

// Butterfly j of stage s, the fastest-varying digit the one next to the
// stage's own (adjacent slots).
template <class L, int S>
__device__ __forceinline__ int synt_task(int u) {
  if constexpr (S == 0) return u;
  constexpr int HI = L::M(S) / L::NS(S);  // rest digits (1 in the last stage)
  if constexpr (HI > 1) return u / HI + (u % HI) * L::NS(S);
  if constexpr (S == 1) return u;
  // last of three: the second digit fastest
  return u / L::R(1) + (u % L::R(1)) * L::R(0);
}

// The stage's twiddles from the tables in shared memory.
template <int R, int DIR, class L>
__device__ __forceinline__ void synt_twiddle(const L &l, int s, int j, float2 *v, const float2 *tw) {
  const float2 *t = tw + l.T(s) + line_base(l, s, j);
#pragma unroll
  for (int q = 1; q < R; ++q) v[q] = cmul(v[q], DIR > 0 ? cconj(t[q * l.NS(s)]) : t[q * l.NS(s)]);
}

template <int N, int TX>
__global__ void __launch_bounds__(SyntCfg<N, TX>::NTH, 65536 / 128 / SyntCfg<N, TX>::NTH)
    k_synt_pass(const __grid_constant__ SyntPassArgs a) {
  using C = SyntCfg<N, TX>;
  using L = typename C::L;
  constexpr L l{};
  constexpr int NTH = C::NTH, LAST = L::nst() - 1, BUF = N * TX, STEP = NTH / TX;
  constexpr int R0 = L::R(0), M0 = L::M(0);
  extern __shared__ float4 sm4[];
  float2 *B = reinterpret_cast<float2 *>(sm4);  // [max(3, nt)][N][TX]
  float2 *H = B + (a.nt < 3 ? 3 : a.nt) * BUF;  // [nt][N]
  float2 *tw = H + a.nt * N;
  const int tid = threadIdx.x, c = tid % TX, u0 = tid / TX;
  const uint32_t f0 = blockIdx.x * TX;
  const bool ok = f0 + c < a.plane;
  const uint32_t f = ok ? f0 + c : a.plane - 1;  // this thread's column of a plane
  const uint32_t y = fdiv(f, a.fcnxp), p = f - y * a.cnxp;
  const bool row = ok && (int)y < a.ny;
  const bool fx = row && (int)(2 * p) < a.nx, fy = row && (int)(2 * p + 1) < a.nx;  // filtered traces

  // a line's impedances where a trace is not filtered (the reference's float
  // sequence): element j + i M0 of every angle
  auto raw_out = [&](int j, auto put) {
    float2 r[3][R0];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int i = 0; i < R0; ++i) r[q][i] = a.m[q][f + (size_t)(j + i * M0) * a.plane];
#pragma unroll 1
    for (int k = 0; k < a.nt; ++k) {
      const float *A = a.A[k];
#pragma unroll
      for (int i = 0; i < R0; ++i)
        put(k, j + i * M0, make_float2(imp1(r[0][i].x, r[1][i].x, r[2][i].x, A), imp1(r[0][i].y, r[1][i].y, r[2][i].y, A)));
    }
  };
  if (!__syncthreads_or(fx || fy)) {  // no trace of this tile is filtered
    if (!ok) return;
#pragma unroll 1
    for (int j = u0; j < M0; j += STEP)
      raw_out(j, [&](int k, int z, float2 v) { a.out[k][f + (size_t)z * a.plane] = v; });
    return;
  }
  for (int i = tid; i < a.nt * N; i += NTH) H[i] = __ldg(a.H + i);
  for (int i = tid; i < L::entries(); i += NTH) tw[i] = __ldg(a.tw + i);

  // forward, first stage: below nz the taper
  // fac ((z - nz) imp[0] + (nzp - z - 1) imp[nz - 1])
  {
    const float fac = a.nz < N ? 1.0f / (float)(N - a.nz - 1) : 0.0f;
#pragma unroll 1
    for (int j = u0; j < M0; j += STEP) {
      float2 v[3][R0], v0[3], vl[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const float2 *m = a.m[q] + f;
        v0[q] = m[0];
        vl[q] = m[(size_t)(a.nz - 1) * a.plane];
#pragma unroll
        for (int i = 0; i < R0; ++i) {
          const int z = j + i * M0;
          v[q][i] = m[(size_t)(z < a.nz ? z : a.nz - 1) * a.plane];
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        vl[q] = csub(vl[q], v0[q]);
#pragma unroll
        for (int i = 0; i < R0; ++i) {
          const int z = j + i * M0;
          float2 x = z < a.nz ? csub(v[q][i], v0[q]) : cscale(vl[q], fac * (float)(N - z - 1));
          v[q][i] = make_float2(fx ? x.x : 0.f, fy ? x.y : 0.f);
        }
        Dft<R0, -1>::run(v[q]);
#pragma unroll
        for (int i = 0; i < R0; ++i) B[q * BUF + C::at(j + i * M0, c)] = v[q][i];
      }
    }
  }
  __syncthreads();
  if constexpr (L::nst() > 2) {
    constexpr int R = L::R(1), M = L::M(1), ST = L::S(1);
#pragma unroll 1
    for (int t = u0; t < 3 * M; t += STEP) {
      const int q = t / M, j = synt_task<L, 1>(t % M), s = line_slot(l, 1, j);
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = B[q * BUF + C::at(s + i * ST, c)];
      synt_twiddle<R, -1>(l, 1, j, v, tw);
      Dft<R, -1>::run(v);
#pragma unroll
      for (int i = 0; i < R; ++i) B[q * BUF + C::at(s + i * ST, c)] = v[i];
    }
    __syncthreads();
  }
  // forward, last stage; per angle the combination, its filter and the first
  // inverse butterfly
  {
    constexpr int R = L::R(LAST), M = L::M(LAST), ST = L::S(LAST);
#pragma unroll 1
    for (int u = u0; u < M; u += STEP) {
      const int j = synt_task<L, LAST>(u), s = line_slot(l, LAST, j);
      float2 v[3][R], t[R];
#pragma unroll
      for (int i = 1; i < R; ++i) t[i] = tw[L::T(LAST) + j + i * L::NS(LAST)];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[q][i] = B[q * BUF + C::at(s + i * ST, c)];
#pragma unroll
        for (int i = 1; i < R; ++i) v[q][i] = cmul(v[q][i], t[i]);
        Dft<R, -1>::run(v[q]);
      }
#pragma unroll 1
      for (int k = 0; k < a.nt; ++k) {
        const float A0 = a.A[k][0], A1 = a.A[k][1], A2 = a.A[k][2];
        float2 w[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float2 x = make_float2(A0 * v[0][i].x + A1 * v[1][i].x + A2 * v[2][i].x,
                                       A0 * v[0][i].y + A1 * v[1][i].y + A2 * v[2][i].y);
          w[i] = cmul(x, H[k * N + j + i * M]);
        }
        Dft<R, 1>::run(w);
#pragma unroll
        for (int i = 1; i < R; ++i) w[i] = cmul(w[i], cconj(t[i]));
#pragma unroll
        for (int i = 0; i < R; ++i) B[k * BUF + C::at(s + i * ST, c)] = w[i];
      }
    }
  }
  __syncthreads();
  // inverse of the middle stage
  if constexpr (L::nst() > 2) {
    constexpr int R = L::R(1), M = L::M(1), ST = L::S(1);
#pragma unroll 1
    for (int t = u0; t < a.nt * M; t += STEP) {
      const int k = t / M, j = synt_task<L, 1>(t % M), s = line_slot(l, 1, j);
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = B[k * BUF + C::at(s + i * ST, c)];
      Dft<R, 1>::run(v);
      synt_twiddle<R, 1>(l, 1, j, v, tw);
#pragma unroll
      for (int i = 0; i < R; ++i) B[k * BUF + C::at(s + i * ST, c)] = v[i];
    }
    __syncthreads();
  }
  // inverse of the first stage, natural order, to HBM
  if (!ok) return;
#pragma unroll 1
  for (int j = u0; j < M0; j += STEP) {
#pragma unroll 1
    for (int k = 0; k < a.nt; ++k) {
      float2 v[R0];
#pragma unroll
      for (int i = 0; i < R0; ++i) v[i] = B[k * BUF + C::at(j + i * M0, c)];
      Dft<R0, 1>::run(v);
      float *o = reinterpret_cast<float *>(a.out[k] + f);
#pragma unroll
      for (int i = 0; i < R0; ++i) {
        float *e = o + 2 * (size_t)(j + i * M0) * a.plane;
        if (fx && fy) *reinterpret_cast<float2 *>(e) = v[i];
        else if (fx) e[0] = v[i].x;
        else if (fy) e[1] = v[i].y;
      }
    }
    if (!(fx && fy))
      raw_out(j, [&](int k, int z, float2 v) {
        float *e = reinterpret_cast<float *>(a.out[k] + f + (size_t)z * a.plane);
        if (!fx) e[0] = v.x;
        if (!fy) e[1] = v.y;
      });
  }
}

template <int N, int TX>
int launch_synt_pass(const SyntPassArgs &a, cudaStream_t s) {
  using C = SyntCfg<N, TX>;
  int rc = func_smem((const void *)k_synt_pass<N, TX>, C::smem(a.nt));
  if (rc) return rc;
  k_synt_pass<N, TX><<<(a.plane + TX - 1) / TX, C::NTH, C::smem(a.nt), s>>>(a);
  CRAVA_LAUNCH_CHECK();
  return CRAVA_GPU_OK;
}
template <int N>
int run_synt_pass(const SyntPassArgs &a, cudaStream_t s) {
  return SyntCfg<N, 8>::smem(a.nt) <= 220 * 1024 ? launch_synt_pass<N, 8>(a, s) : launch_synt_pass<N, 4>(a, s);
}
// The compiled lengths (fft_len.cu); null: none.
using SyntLaunch = int (*)(const SyntPassArgs &, cudaStream_t);
SyntLaunch synt_launch(int n);

}  // namespace crava
