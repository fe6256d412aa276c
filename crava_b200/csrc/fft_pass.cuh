// fft_pass.cuh -- the built-in x, y and z passes of a 3-D transform: device
// code of a tile and the kernels over all grids of a batch.
//
// Rows (x): a CTA transforms kB rows of nxp reals.  Even nxp: the packed
// nxp / 2-point complex line; the split into the half spectrum (forward) or
// out of it (inverse) pairs position k with nh - k, one thread doing both.
// Odd nxp: two rows of a plane at a time as real and imaginary part of one
// nxp-point line (the last of an odd nyp alone), so that a plane's values do not
// hang on its neighbours', nor on which planes are in the grid.
// Columns (y and z): a CTA transforms 16 adjacent lines, 128 bytes of every
// row it touches; lanes run along the lines, so a shared-memory row is one
// 128-byte access whatever the stage and a warp reads two twiddles.
// Each pass reads and writes HBM (or L2, where the grids of a launch fit it)
// once, in the layout of FFTGrid, in place or (forward rows) from a source
// grid; the scalings and an addend are fused.  A launch takes several grids:
// a pass over one small grid is shorter than a launch.
//
// Replaces FFTGrid::fftInPlace / invFFTInPlace (src/fftgrid.cpp:1803-1862).
#pragma once

#include "fft.cuh"
#include "fft_banks.cuh"
#include "fft_line.cuh"
#include "synt_pass.cuh"

namespace crava {

struct PassGrids {
  const float *src[kGridBatch];
  float *dst[kGridBatch];
  const float *add[kGridBatch];
  float scale[kGridBatch];
};

// ------------------------------------------------------------------ rows
struct RowPassArgs {
  PassGrids g;
  uint32_t nlines;    // rows, nyp nzp (odd nxp: pairs, ceil(nyp / 2) nzp)
  uint32_t odd;       // nyp mod 2
  FastDiv fpairs;     // ceil(nyp / 2)
  const float2 *tw;   // stage tables of the direction's line
  const float2 *post; // W_nxp^k, k <= nxp / 2 (even nxp)
};

// Small CTAs, about 1024 points on 128 threads and eight resident per SM: one's
// barriers then wait for few warps while the others load and store.  256 threads
// with 4096 points and four per SM took longer in every pass that is not launch
// bound, and longer than the register-resident pass of fft.cu at 64 and 256
// points inverse: us forward / inverse, 128 x 64 x 64 rows 8.6 / 8.6 -> 6.6 / 6.8,
// 512 x 256 x 256 54 / 66 -> 52 / 62, 96 x 200 x 300 18.7 / 16.7 -> 15.2 / 14.7, 200 x
// 200 x 192 22.9 / 20.9 -> 22.8 / 18.8; with 2048 points 7.6 / 8.5 at the first, 16.9 /
// 14.7 at the third and the same at the others.
constexpr int kRowThreads = 128, kRowMinBlocks = 8;

template <int NX>
struct RowCfg {
  static constexpr bool ODD = NX % 2 != 0;
  static constexpr int N = ODD ? NX : NX / 2;   // line length
  static constexpr int CX = NX / 2 + 1, RX = 2 * CX;
  static constexpr RowBanks kBanks = row_banks(N);
  using F = LineOf<N, kBanks.sf, false>;  // forward: first radix small (long runs of loads)
  using I = LineOf<N, kBanks.si, true>;   // inverse: last radix small (long runs of stores)
  static constexpr int PF = kBanks.pf, PI = kBanks.pi;
  static_assert(PF >= F::R(0) * F::S(0) && PI >= I::R(0) * I::S(0), "a row holds its line");
  // lines per CTA: about 1024 points
  static constexpr int kB = 1024 / N < 8 ? 8 : 1024 / N > 32 ? 32 : 1024 / N / 8 * 8;
  static constexpr int NP = N / 2 + N % 2;  // position pairs of an even row
  static constexpr size_t smem(int dir) { return sizeof(float2) * (size_t)kB * (dir < 0 ? PF : PI); }
};

// Tasks of a stage spread over the CTA's threads in rounds, G rounds' loads
// issued before the first of them computes.
template <int TASKS, int NTH, int G, class Load, class Finish>
__device__ __forceinline__ void rounds(int tid, Load load, Finish finish) {
  constexpr int K = (TASKS + NTH - 1) / NTH;
#pragma unroll 1
  for (int rd = 0; rd < K; rd += G) {
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const int t = tid + (rd + u) * NTH;
      if ((K % G == 0 && TASKS % NTH == 0) || t < TASKS) load(u, t);
    }
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const int t = tid + (rd + u) * NTH;
      if ((K % G == 0 && TASKS % NTH == 0) || t < TASKS) finish(u, t);
    }
  }
}
// Rounds whose R values a thread holds at once.
__host__ __device__ constexpr int rounds_group(int r, int budget, int rounds) {
  const int g = budget / r < 1 ? 1 : budget / r;
  return g > rounds ? rounds : g;
}
__host__ __device__ constexpr int ceil_div(int a, int b) { return (a + b - 1) / b; }

// One stage of the rows of a tile in shared memory, in place (TW: with
// twiddles).
template <class L, int S, int DIR, int B, int P, int NTH>
__device__ __forceinline__ void row_stage(float2 *A, const float2 *tw, int tid) {
  constexpr int R = L::R(S), M = L::M(S), ST = L::S(S);
  constexpr L l{};
#pragma unroll 1
  for (int t = tid; t < B * M; t += NTH) {
    const int q = t / M, j = t % M;
    float2 *o = A + q * P + line_slot(l, S, j);
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = o[i * ST];
    if constexpr (S > 0) line_twiddle<R, DIR>(l, S, j, v, tw);
    Dft<R, DIR>::run(v);
#pragma unroll
    for (int i = 0; i < R; ++i) o[i * ST] = v[i];
  }
}

// The packed line's values at k and nh - k to the half spectrum's:
// X_k = E + W^k O, X_{nh-k} = conj(E - W^k O) with E = (z_k + conj z_{nh-k}) / 2,
// O = -i (z_k - conj z_{nh-k}) / 2; and back (a factor 2 left in):
// Z_k = e + i o, Z_{nh-k} = conj(e - i o) with e = X_k + conj X_{nh-k},
// o = conj(W^k) (X_k - conj X_{nh-k}).  Same operations as the other x passes.
__device__ __forceinline__ void split_pair(float2 zk, float2 zm, float2 w, float2 *xk, float2 *xm) {
  zm.y = -zm.y;
  const float2 e = cscale(cadd(zk, zm), 0.5f);
  const float2 d = csub(zk, zm);
  const float2 t = cmul(w, make_float2(0.5f * d.y, -0.5f * d.x));
  *xk = cadd(e, t);
  *xm = cconj(csub(e, t));
}
__device__ __forceinline__ void merge_pair(float2 xk, float2 xm, float2 w, float2 *zk, float2 *zm) {
  xm.y = -xm.y;
  const float2 e = cadd(xk, xm);
  const float2 o = cmul(csub(xk, xm), cconj(w));
  *zk = make_float2(e.x - o.y, e.y + o.x);
  *zm = make_float2(e.x + o.y, o.x - e.y);
}

// Forward rows row0 .. row0 + B of an even nxp: src -> dst (half spectrum).
template <int NX, int NTH>
__device__ __forceinline__ void rows_fwd_even(const float *src, float *dst, long long row0, int nrows, float scale,
                                              const float2 *tw, const float2 *post, float2 *A, int tid) {
  using C = RowCfg<NX>;
  using L = typename C::F;
  constexpr L l{};
  constexpr int B = C::kB, P = C::PF, NH = C::N, CX = C::CX, NP = C::NP;
  {
    constexpr int R = L::R(0), M = L::M(0), S = L::S(0), G = rounds_group(R, 16, ceil_div(B * M, NTH));
    float2 v[G][R];
    rounds<B * M, NTH, G>(
        tid,
        [&](int u, int t) {
          const int q = t / M, j = t % M;
          const float2 *row = reinterpret_cast<const float2 *>(src) + (row0 + (q < nrows ? q : 0)) * CX + j;
#pragma unroll
          for (int i = 0; i < R; ++i) v[u][i] = row[i * M];
        },
        [&](int u, int t) {
          const int q = t / M, j = t % M;
          Dft<R, -1>::run(v[u]);
          float2 *o = A + q * P + j;
#pragma unroll
          for (int i = 0; i < R; ++i) o[i * S] = v[u][i];
        });
  }
  __syncthreads();
  row_stage<L, 1, -1, B, P, NTH>(A, tw, tid);
  if constexpr (L::nst() > 2) {
    __syncthreads();
    row_stage<L, 2, -1, B, P, NTH>(A, tw, tid);
  }
  __syncthreads();
#pragma unroll 2
  for (int t = tid; t < B * NP; t += NTH) {
    const int q = t / NP, k = t % NP;
    if (q >= nrows) continue;
    const float2 *z = A + q * P;
    float2 *o = reinterpret_cast<float2 *>(dst) + (row0 + q) * CX;
    const float2 zk = z[line_out(l, k)];
    if (k > 0) {
      const float2 zm = z[line_out(l, NH - k)];
      float2 xk, xm;
      split_pair(zk, zm, __ldg(post + k), &xk, &xm);
      o[k] = cscale(xk, scale);
      o[NH - k] = cscale(xm, scale);
    } else {
      o[0] = make_float2(scale * (zk.x + zk.y), 0.f);
      o[NH] = make_float2(scale * (zk.x - zk.y), 0.f);
      if constexpr (NH % 2 == 0) {
        const float2 zc = z[line_out(l, NH / 2)];  // its own partner: conj z
        o[NH / 2] = make_float2(scale * zc.x, -(scale * zc.y));
      }
    }
  }
}

// Inverse rows: src half spectrum -> dst real row (scale, addend, zero pad).
template <int NX, int NTH>
__device__ __forceinline__ void rows_inv_even(const float *src, float *dst, const float *add, long long row0, int nrows,
                                              float scale, const float2 *tw, const float2 *post, float2 *A, int tid) {
  using C = RowCfg<NX>;
  using L = typename C::I;
  constexpr L l{};
  constexpr int B = C::kB, P = C::PI, NH = C::N, CX = C::CX, NP = C::NP;
  // the imaginary parts of the DC and Nyquist values are ignored
  constexpr int G = rounds_group(2, 8, ceil_div(B * NP, NTH));
  float2 xk[G], xm[G], xc[G];
  rounds<B * NP, NTH, G>(
      tid,
      [&](int u, int t) {
        const int q = t / NP, k = t % NP;
        const float2 *X = reinterpret_cast<const float2 *>(src) + (row0 + (q < nrows ? q : 0)) * CX;
        xk[u] = X[k];
        xm[u] = X[NH - k];
        if constexpr (NH % 2 == 0)
          if (k == 0) xc[u] = X[NH / 2];
      },
      [&](int u, int t) {
        const int q = t / NP, k = t % NP;
        float2 *z = A + q * P;
        if (k > 0) {
          merge_pair(xk[u], xm[u], __ldg(post + k), z + line_in(l, k), z + line_in(l, NH - k));
        } else {
          z[0] = make_float2(xk[u].x + xm[u].x, xk[u].x - xm[u].x);
          if constexpr (NH % 2 == 0) z[line_in(l, NH / 2)] = make_float2(2.f * xc[u].x, -2.f * xc[u].y);
        }
      });
  __syncthreads();
  row_stage<L, 0, 1, B, P, NTH>(A, tw, tid);
  __syncthreads();
  if constexpr (L::nst() > 2) {
    row_stage<L, 1, 1, B, P, NTH>(A, tw, tid);
    __syncthreads();
  }
  constexpr int S = L::nst() - 1, R = L::R(S), M = L::M(S), ST = L::S(S);
#pragma unroll 1
  for (int t = tid; t < B * M; t += NTH) {
    const int q = t / M, j = t % M;
    if (q >= nrows) continue;
    const float2 *o = A + q * P + line_slot(l, S, j);
    float2 v[R], w[R];
    if (add) {  // its loads run under the butterfly
      const float2 *arow = reinterpret_cast<const float2 *>(add) + (row0 + q) * CX + j;
#pragma unroll
      for (int i = 0; i < R; ++i) w[i] = arow[i * M];
    }
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = o[i * ST];
    line_twiddle<R, 1>(l, S, j, v, tw);
    Dft<R, 1>::run(v);
    float2 *orow = reinterpret_cast<float2 *>(dst) + (row0 + q) * CX + j;
    if (add) {
#pragma unroll
      for (int i = 0; i < R; ++i) orow[i * M] = cadd(cscale(v[i], scale), w[i]);
    } else {
#pragma unroll
      for (int i = 0; i < R; ++i) orow[i * M] = cscale(v[i], scale);
    }
    if (j == 0) orow[NH] = make_float2(0.f, 0.f);
  }
}

// Odd nxp: the first row of pair l, and whether the pair has a second one.
struct RowPair {
  uint32_t row;
  bool two;
};
__device__ __forceinline__ RowPair row_pair(const RowPassArgs &a, uint32_t l) {
  if (!a.odd) return RowPair{2 * l, true};
  const uint32_t plane = fdiv(l, a.fpairs);
  return RowPair{2 * l - plane, l - plane * a.fpairs.d + 1 != a.fpairs.d};
}

// Odd nxp: the pairs line0 .. line0 + B of rows.
template <int NX, int NTH>
__device__ __forceinline__ void rows_fwd_odd(const RowPassArgs &a, const float *src, float *dst, uint32_t line0,
                                             int nlines, float scale, const float2 *tw, float2 *A, int tid) {
  using C = RowCfg<NX>;
  using L = typename C::F;
  constexpr L l{};
  constexpr int B = C::kB, P = C::PF, N = C::N, CX = C::CX, RX = C::RX;
  {
    constexpr int R = L::R(0), M = L::M(0), S = L::S(0);
#pragma unroll 1
    for (int t = tid; t < B * M; t += NTH) {
      const int q = t / M, j = t % M;
      const RowPair pr = row_pair(a, line0 + (q < nlines ? q : 0));
      const float *ra = src + (size_t)pr.row * RX + j;
      const bool two = pr.two;
      const float *rb = two ? ra + RX : ra;
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = make_float2(ra[i * M], two ? rb[i * M] : 0.f);
      Dft<R, -1>::run(v);
      float2 *o = A + q * P + j;
#pragma unroll
      for (int i = 0; i < R; ++i) o[i * S] = v[i];
    }
  }
  __syncthreads();
  row_stage<L, 1, -1, B, P, NTH>(A, tw, tid);
  if constexpr (L::nst() > 2) {
    __syncthreads();
    row_stage<L, 2, -1, B, P, NTH>(A, tw, tid);
  }
  __syncthreads();
  // X_a = (Z_k + conj Z_{n-k}) / 2, X_b = -i (Z_k - conj Z_{n-k}) / 2
  const float h = 0.5f * scale;
#pragma unroll 1
  for (int t = tid; t < B * CX; t += NTH) {
    const int q = t / CX, k = t % CX;
    if (q >= nlines) continue;
    const RowPair pr = row_pair(a, line0 + q);
    const float2 *z = A + q * P;
    const float2 zk = z[line_out(l, k)], zm = k == 0 ? zk : z[line_out(l, N - k)];
    float2 *o = reinterpret_cast<float2 *>(dst) + (size_t)pr.row * CX + k;
    o[0] = make_float2(h * (zk.x + zm.x), h * (zk.y - zm.y));
    if (pr.two) o[CX] = make_float2(h * (zk.y + zm.y), h * (zm.x - zk.x));
  }
}

template <int NX, int NTH>
__device__ __forceinline__ void rows_inv_odd(const RowPassArgs &a, const float *src, float *dst, const float *add,
                                             uint32_t line0, int nlines, float scale, const float2 *tw, float2 *A,
                                             int tid) {
  using C = RowCfg<NX>;
  using L = typename C::I;
  constexpr L l{};
  constexpr int B = C::kB, P = C::PI, N = C::N, CX = C::CX, RX = C::RX;
  // Z_k = X_a + i X_b, Z_{n-k} = conj X_a + i conj X_b; the imaginary parts
  // of the DC values are ignored
#pragma unroll 1
  for (int t = tid; t < B * CX; t += NTH) {
    const int q = t / CX, k = t % CX;
    const RowPair pr = row_pair(a, line0 + (q < nlines ? q : 0));
    const float2 *X = reinterpret_cast<const float2 *>(src) + (size_t)pr.row * CX + k;
    const float2 xa = X[0], xb = pr.two ? X[CX] : make_float2(0.f, 0.f);
    float2 *z = A + q * P;
    if (k == 0) {
      z[0] = make_float2(xa.x, xb.x);
    } else {
      z[line_in(l, k)] = make_float2(xa.x - xb.y, xa.y + xb.x);
      z[line_in(l, N - k)] = make_float2(xa.x + xb.y, xb.x - xa.y);
    }
  }
  __syncthreads();
  row_stage<L, 0, 1, B, P, NTH>(A, tw, tid);
  __syncthreads();
  if constexpr (L::nst() > 2) {
    row_stage<L, 1, 1, B, P, NTH>(A, tw, tid);
    __syncthreads();
  }
  constexpr int S = L::nst() - 1, R = L::R(S), M = L::M(S), ST = L::S(S);
#pragma unroll 1
  for (int t = tid; t < B * M; t += NTH) {
    const int q = t / M, j = t % M;
    if (q >= nlines) continue;
    const RowPair pr = row_pair(a, line0 + q);
    const bool two = pr.two;
    const float2 *o = A + q * P + line_slot(l, S, j);
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = o[i * ST];
    line_twiddle<R, 1>(l, S, j, v, tw);
    Dft<R, 1>::run(v);
    const size_t e = (size_t)pr.row * RX + j;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      v[i] = cscale(v[i], scale);
      if (add) v[i] = cadd(v[i], make_float2(add[e + i * M], two ? add[e + RX + i * M] : 0.f));
      dst[e + i * M] = v[i].x;
      if (two) dst[e + RX + i * M] = v[i].y;
    }
    if (j == 0) {
      dst[e + N] = 0.f;
      if (two) dst[e + RX + N] = 0.f;
    }
  }
}

template <int NX, int DIR>
__global__ void __launch_bounds__(kRowThreads, kRowMinBlocks) k_row_pass(const __grid_constant__ RowPassArgs a) {
  using C = RowCfg<NX>;
  extern __shared__ float4 sm4[];
  float2 *A = reinterpret_cast<float2 *>(sm4);
  const uint32_t line0 = blockIdx.x * C::kB;
  const int g = blockIdx.y;
  const int n = (int)(a.nlines - line0 < C::kB ? a.nlines - line0 : C::kB);
  const float *src = a.g.src[g];
  float *dst = a.g.dst[g];
  const float s = a.g.scale[g];
  if constexpr (C::ODD) {
    if constexpr (DIR < 0) rows_fwd_odd<NX, kRowThreads>(a, src, dst, line0, n, s, a.tw, A, threadIdx.x);
    else rows_inv_odd<NX, kRowThreads>(a, src, dst, a.g.add[g], line0, n, s, a.tw, A, threadIdx.x);
  } else {
    if constexpr (DIR < 0) rows_fwd_even<NX, kRowThreads>(src, dst, line0, n, s, a.tw, a.post, A, threadIdx.x);
    else rows_inv_even<NX, kRowThreads>(src, dst, a.g.add[g], line0, n, s, a.tw, a.post, A, threadIdx.x);
  }
}

// ------------------------------------------------------------------ columns
constexpr int kColLines = 16;

// Line f starts at (f mod inner) + (f div inner) outer, elements es apart:
//   z pass: inner = the lines of a plane, es = the plane;
//   y pass: inner = cnxp, outer = the plane, es = cnxp.
struct ColPassArgs {
  float2 *dst[kGridBatch];
  long long nlines;
  uint32_t inner, outer, es;  // a grid has fewer than 2^32 complex values
  FastDiv finner;
  const float2 *tw;
  // band-gated rule of the forward z pass, per grid (mode 0: none)
  double v[kGridBatch];
  int mode[kGridBatch];
  const int *inv;
  unsigned *nf_bits, *nf_any;
  uint32_t ahead;  // z pass of split planes: tiles ahead whose input is fetched into L2
};

template <int N>
struct ColCfg {
  using L = LineOf<N, 0, true>;
  static constexpr int max_m() {
    int m = 0;
    for (int s = 0; s < L::nst(); ++s) m = L::M(s) > m ? L::M(s) : m;
    return m;
  }
  static constexpr int max_r() {
    int m = 0;
    for (int s = 0; s < L::nst(); ++s) m = L::R(s) > m ? L::R(s) : m;
    return m;
  }
  static constexpr int min_m() {
    int m = N;
    for (int s = 0; s < L::nst(); ++s) m = L::M(s) < m ? L::M(s) : m;
    return m;
  }
  // butterflies of a line that run at once: those of a stage in one round
  // where at most 20, else in equal rounds.  Where one stage has half of the
  // other's (128 = 16 x 8, 162, 200 = 20 x 10) the smaller number, so that no
  // thread idles in that stage: a unit of 256x128x128, three angles, 486 -> 466 us
  // (480 with the register-resident passes), of 96x200x300 727 -> 709.  Two rounds
  // where the stages are alike cost instead: 128x256x256 931 -> 1139.
  static constexpr bool kHalf = min_m() >= 8 && max_m() <= 20 && max_m() == 2 * min_m();
  static constexpr int kRounds = kHalf ? 2 : ceil_div(max_m(), 20);
  static constexpr int TPB = (ceil_div(max_m(), kRounds) + 1) / 2 * 2;
  static constexpr int NTH = kColLines * TPB;
  static constexpr int kHold = 16;  // points a thread's loads in flight cover (at least a radix)
  static constexpr int kRegs = 64;
  static constexpr int kMinB = 65536 / (NTH * kRegs) < 1 ? 1 : 65536 / (NTH * kRegs) > 16 ? 16 : 65536 / (NTH * kRegs);
  static constexpr size_t smem() { return sizeof(float2) * (size_t)N * kColLines; }
};

template <int N, int S, int DIR>
__device__ __forceinline__ void col_mid(float2 *B, const float2 *tw, int p, int t) {
  using C = ColCfg<N>;
  using L = typename C::L;
  constexpr L l{};
  constexpr int R = L::R(S), M = L::M(S), ST = L::S(S);
#pragma unroll 1
  for (int j = t; j < M; j += C::TPB) {
    float2 *o = B + line_slot(l, S, j) * kColLines + p;
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = o[i * ST * kColLines];
    line_twiddle<R, DIR>(l, S, j, v, tw);
    Dft<R, DIR>::run(v);
#pragma unroll
    for (int i = 0; i < R; ++i) o[i * ST * kColLines] = v[i];
  }
}

// One tile: the line that starts at data[line] (ok: it exists), elements es
// apart; p: its column in the tile, t: the thread's butterfly.  zp.mode 0: no
// rule.
template <int N, int DIR>
__device__ __forceinline__ void col_tile(float2 *data, uint32_t line, bool ok, uint32_t es, const float2 *tw, float2 *B,
                                         int p, int t, const ZPrior &zp) {
  using C = ColCfg<N>;
  using L = typename C::L;
  constexpr L l{};
  {
    constexpr int R = L::R(0), M = L::M(0), K = ceil_div(M, C::TPB), G = rounds_group(R, C::kHold, K);
    const uint32_t step = M * es;
#pragma unroll 1
    for (int rd = 0; rd < K; rd += G) {
      float2 v[G][R];
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int j = t + (rd + u) * C::TPB;
        if (ok && ((K % G == 0 && M % C::TPB == 0) || j < M)) {
          const uint32_t o = line + j * es;
#pragma unroll
          for (int i = 0; i < R; ++i) v[u][i] = data[o + i * step];
        }
      }
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int j = t + (rd + u) * C::TPB;
        if (ok && ((K % G == 0 && M % C::TPB == 0) || j < M)) {
          Dft<R, DIR>::run(v[u]);
          float2 *o = B + j * kColLines + p;
#pragma unroll
          for (int i = 0; i < R; ++i) o[i * L::S(0) * kColLines] = v[u][i];
        }
      }
    }
  }
  __syncthreads();
  if constexpr (L::nst() > 2) {
    if (ok) col_mid<N, 1, DIR>(B, tw, p, t);
    __syncthreads();
  }
  constexpr int S = L::nst() - 1, R = L::R(S), M = L::M(S), ST = L::S(S);
  const uint32_t step = M * es;
#pragma unroll 1
  for (int j = t; j < M; j += C::TPB) {
    if (!ok) break;
    unsigned gated = 0u;  // bit i: output i lies on a band-gated plane
    if (DIR < 0 && zp.mode) {
#pragma unroll
      for (int i = 0; i < R; ++i) gated |= __ldg(zp.inv + j + i * M) == 0 ? 1u << i : 0u;
    }
    const float2 *o = B + line_slot(l, S, j) * kColLines + p;
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = o[i * ST * kColLines];
    line_twiddle<R, DIR>(l, S, j, v, tw);
    Dft<R, DIR>::run(v);
    const uint32_t d = line + j * es;
    if (DIR < 0 && gated) {
#pragma unroll
      for (int i = 0; i < R; ++i)
        if ((gated >> i) & 1u) v[i] = zprior_apply(zp, v[i], d + i * step);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) data[d + i * step] = v[i];
  }
}

template <int N, int DIR>
__global__ void __launch_bounds__(ColCfg<N>::NTH, ColCfg<N>::kMinB) k_col_pass(const __grid_constant__ ColPassArgs a) {
  extern __shared__ float4 sm4[];
  float2 *B = reinterpret_cast<float2 *>(sm4);  // [N][kColLines]
  const int p = threadIdx.x % kColLines, t = threadIdx.x / kColLines, g = blockIdx.y;
  const long long f = (long long)blockIdx.x * kColLines + p;
  const bool ok = f < a.nlines;
  const uint32_t q = ok ? fdiv((uint32_t)f, a.finner) : 0u;
  const uint32_t line = ok ? (uint32_t)f - q * a.inner + q * a.outer : 0u;
  ZPrior zp;
  if (DIR < 0) {
    zp.mode = a.mode[g];
    zp.v = a.v[g];
    zp.inv = a.inv;
    zp.nf_bits = a.nf_bits;
    zp.nf_any = a.nf_any;
  }
  col_tile<N, DIR>(a.dst[g], line, ok, a.es, a.tw, B, p, t, zp);
}

// ------------------------------------------------------------------ launch
template <int NX, int DIR>
int launch_rows(const RowPassArgs &a, int ngrids, cudaStream_t s) {
  using C = RowCfg<NX>;
  const size_t sm = C::smem(DIR);
  int rc = func_smem((const void *)k_row_pass<NX, DIR>, sm);
  if (rc) return rc;
  k_row_pass<NX, DIR><<<dim3((a.nlines + C::kB - 1) / C::kB, (unsigned)ngrids), kRowThreads, sm, s>>>(a);
  CRAVA_LAUNCH_CHECK();
  return CRAVA_GPU_OK;
}

template <int N, int DIR>
int launch_cols(const ColPassArgs &a, int ngrids, cudaStream_t s) {
  using C = ColCfg<N>;
  int rc = func_smem((const void *)k_col_pass<N, DIR>, C::smem());
  if (rc) return rc;
  const dim3 grd((unsigned)((a.nlines + kColLines - 1) / kColLines), (unsigned)ngrids);
  k_col_pass<N, DIR><<<grd, C::NTH, C::smem(), s>>>(a);
  CRAVA_LAUNCH_CHECK();
  return CRAVA_GPU_OK;
}

// The z pass that completes the y transform of planes split in two (plane.cu).
int z_parts_launch(const ColPassArgs &a, int n, int ngrids, int dir, cudaStream_t s);

// The compiled lengths (fft_len.cu).
using ColLaunch = int (*)(const ColPassArgs &, int ngrids, int dir, cudaStream_t);
using RowLaunch = int (*)(const RowPassArgs &, int ngrids, int dir, cudaStream_t);
ColLaunch col_launch(int n);  // null: not compiled
RowLaunch row_launch(int nx);
template <int N>
int run_cols(const ColPassArgs &a, int ngrids, int dir, cudaStream_t s) {
  return dir < 0 ? launch_cols<N, -1>(a, ngrids, s) : launch_cols<N, 1>(a, ngrids, s);
}
template <int NX>
int run_rows(const RowPassArgs &a, int ngrids, int dir, cudaStream_t s) {
  return dir < 0 ? launch_rows<NX, -1>(a, ngrids, s) : launch_rows<NX, 1>(a, ngrids, s);
}
// Rows: the even ones 32 .. 512 and the odd ones 25 .. 255.
template <int NX>
RowLaunch row_of() {
  if constexpr (NX % 2 == 0 ? NX >= 32 : NX <= 255) return run_rows<NX>;
  else return nullptr;
}
// Synthetic seismic: the lengths of two or three stages of its radices.
template <int N>
SyntLaunch synt_of() {
  if constexpr (synt_list(N).n >= 2) return run_synt_pass<N>;
  else return nullptr;
}

}  // namespace crava
