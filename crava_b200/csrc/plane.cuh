// plane.cuh -- the x and y passes of a 3-D transform in one kernel, for small
// planes with power-of-two sides: a z-plane lives in a CTA's shared memory
// between the two passes, three CTAs per SM.
//
// The split of the packed x line into the half spectrum pairs column k with
// nh - k; the first y stage (forward) or the last one (inverse) takes the two
// columns of a pair together and does it in registers, so the plane makes three
// trips through shared memory where the separate passes make three and a trip
// through L2.  128x128x256, a grid at a time: 12.8 / 12.4 us forward / inverse
// against 16.8 / 16.7 us for the separate row and column passes.
//
// Larger planes were tried and are not built: 256x256 split over two CTAs of 150
// KB (the last radix-2 step of y in the z pass) took 92 + 71 us per transform,
// over four CTAs of 74 KB 75 + 83 us, and both passes in one cluster kernel with
// the exchange through L2 104 + 53 us, against 43 + 44 + 52 us for the three
// separate passes over a batch of grids: those run at the HBM rate, and a CTA
// that fills the SM has nothing to run while its loads are on the way.
#pragma once

#include "fft_pass.cuh"

namespace crava {

template <int NX, int NY>
struct PlaneCfg {
  static constexpr int NH = NX / 2, CX = NH + 1, NP = NH / 2;
  static constexpr RowBanks kBanks = row_banks(NH);
  using XF = LineOf<NH, kBanks.sf, false>;
  using XI = LineOf<NH, kBanks.si, true>;
  // the y line: the stage that holds a column pair has radix 8
  using YF = CtLine<0, 8, NY / 8>;
  using YI = CtLine<0, NY / 8, 8>;
  // a row holds its padded line and a spare slot (the Nyquist column); the
  // pitch keeps the residue that its bank layout wants
  static constexpr int pitch(int line, int want) { return want > line ? want : line + 1 + (want - line - 1 + 1600) % 16; }
  static constexpr int PF = pitch(XF::R(0) * XF::S(0), kBanks.pf), PI = pitch(XI::R(0) * XI::S(0), kBanks.pi);
  static constexpr size_t smem(int dir) { return sizeof(float2) * (size_t)NY * (dir < 0 ? PF : PI); }
  static constexpr int NTH = 256;
};

struct PlaneArgs {
  PassGrids g;
  const float2 *twx, *twy, *wx;  // stage tables, W_nxp^k
};

template <int NX, int NY>
__global__ void __launch_bounds__(PlaneCfg<NX, NY>::NTH, 4) k_plane_fwd(const __grid_constant__ PlaneArgs a) {
  using C = PlaneCfg<NX, NY>;
  using LX = typename C::XF;
  using LY = typename C::YF;
  constexpr LX lx{};
  constexpr LY ly{};
  constexpr int NTH = C::NTH, NQ = NY, NH = C::NH, CX = C::CX, NP = C::NP, P = C::PF, SPARE = LX::R(0) * LX::S(0);
  static_assert(LX::nst() == 2 && LY::nst() == 2, "two-stage lines");
  extern __shared__ float4 sm4[];
  float2 *A = reinterpret_cast<float2 *>(sm4);
  const int tid = threadIdx.x;
  const int g = blockIdx.y;
  const long long off = (long long)blockIdx.x * CX * NY;
  const float2 *src = reinterpret_cast<const float2 *>(a.g.src[g]) + off;
  float2 *dst = reinterpret_cast<float2 *>(a.g.dst[g]) + off;
  const float scale = a.g.scale[g], h = 0.5f * scale;

  // 1. x, first stage: HBM -> registers -> shared memory
  {
    constexpr int R = LX::R(0), M = LX::M(0), S = LX::S(0), G = rounds_group(R, 16, ceil_div(NQ * M, NTH));
    float2 v[G][R];
    rounds<NQ * M, NTH, G>(
        tid,
        [&](int u, int t) {
          const float2 *row = src + (t / M) * CX + t % M;
#pragma unroll
          for (int i = 0; i < R; ++i) v[u][i] = row[i * M];
        },
        [&](int u, int t) {
          Dft<R, -1>::run(v[u]);
          float2 *o = A + (t / M) * P + t % M;
#pragma unroll
          for (int i = 0; i < R; ++i) o[i * S] = v[u][i];
        });
  }
  __syncthreads();
  // 2. x, last stage, in place
  row_stage<LX, 1, -1, NQ, P, NTH>(A, a.twx, tid);
  __syncthreads();

  // 3. the split and the first y stage, column pairs k, nh - k
  {
    constexpr int R = LY::R(0), M = LY::M(0);
#pragma unroll 1
    for (int t = tid; t < NP * M; t += NTH) {
      const int j = t / NP, k = t % NP;
      float2 *ok = A + j * P + line_out(lx, k);
      float2 *om = A + j * P + (k == 0 ? SPARE : line_out(lx, NH - k));
      float2 x[R], y[R];
      if (k > 0) {
        // e = z_k + conj z_m, T = -i W^k (z_k - conj z_m):
        // X_k = (e + T) / 2, X_m = conj(e - T) / 2
        float2 w = __ldg(a.wx + k);
        w = make_float2(h * w.y, -(h * w.x));
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float2 zk = ok[i * M * P], zm = om[i * M * P];
          const float2 e = make_float2(zk.x + zm.x, zk.y - zm.y);
          const float2 T = cmul(make_float2(zk.x - zm.x, zk.y + zm.y), w);
          x[i] = make_float2(h * e.x + T.x, h * e.y + T.y);
          y[i] = make_float2(h * e.x - T.x, T.y - h * e.y);
        }
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i) {  // DC and Nyquist from z_0
          const float2 z = ok[i * M * P];
          x[i] = make_float2(scale * (z.x + z.y), 0.f);
          y[i] = make_float2(scale * (z.x - z.y), 0.f);
        }
      }
      Dft<R, -1>::run(x);
      Dft<R, -1>::run(y);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        ok[i * M * P] = x[i];
        om[i * M * P] = y[i];
      }
      if (k == 0) {
        float2 *oc = A + j * P + line_out(lx, NH / 2);  // its own partner: conj z
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float2 z = oc[i * M * P];
          x[i] = make_float2(scale * z.x, -(scale * z.y));
        }
        Dft<R, -1>::run(x);
#pragma unroll
        for (int i = 0; i < R; ++i) oc[i * M * P] = x[i];
      }
    }
  }
  __syncthreads();

  // 4. y, last stage: shared memory -> registers -> HBM
  {
    constexpr int R = LY::R(1), M = LY::M(1), S = LY::S(1);
#pragma unroll 1
    for (int t = tid; t < CX * M; t += NTH) {
      const int j = t / CX, k = t % CX;
      const float2 *o = A + line_slot(ly, 1, j) * P + (k == NH ? SPARE : line_out(lx, k));
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = o[i * S * P];
      line_twiddle<R, -1>(ly, 1, j, v, a.twy);
      Dft<R, -1>::run(v);
      float2 *d = dst + j * CX + k;
#pragma unroll
      for (int i = 0; i < R; ++i) d[i * M * CX] = v[i];
    }
  }
}

template <int NX, int NY>
__global__ void __launch_bounds__(PlaneCfg<NX, NY>::NTH, 4) k_plane_inv(const __grid_constant__ PlaneArgs a) {
  using C = PlaneCfg<NX, NY>;
  using LX = typename C::XI;
  using LY = typename C::YI;
  constexpr LX lx{};
  constexpr LY ly{};
  constexpr int NTH = C::NTH, NQ = NY, NH = C::NH, CX = C::CX, NP = C::NP, P = C::PI, SPARE = LX::R(0) * LX::S(0);
  extern __shared__ float4 sm4[];
  float2 *A = reinterpret_cast<float2 *>(sm4);
  const int tid = threadIdx.x;
  const int g = blockIdx.y;
  const long long off = (long long)blockIdx.x * CX * NY;
  const float2 *src = reinterpret_cast<const float2 *>(a.g.src[g]) + off;
  float2 *dst = reinterpret_cast<float2 *>(a.g.dst[g]) + off;
  const float2 *add = a.g.add[g] ? reinterpret_cast<const float2 *>(a.g.add[g]) + off : nullptr;
  const float scale = a.g.scale[g];

  // 1. y, first stage: HBM -> registers -> shared memory
  {
    constexpr int R = LY::R(0), M = LY::M(0);
#pragma unroll 1
    for (int t = tid; t < CX * M; t += NTH) {
      const int j = t / CX, k = t % CX;
      const float2 *o = src + j * CX + k;
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = o[i * M * CX];
      Dft<R, 1>::run(v);
      float2 *d = A + j * P + (k == NH ? SPARE : line_in(lx, k));
#pragma unroll
      for (int i = 0; i < R; ++i) d[i * M * P] = v[i];
    }
  }
  __syncthreads();

  // 2. y, last stage, and the pre-split of the column pairs, in place
  {
    constexpr int R = LY::R(1), M = LY::M(1), S = LY::S(1);
#pragma unroll 1
    for (int t = tid; t < NP * M; t += NTH) {
      const int j = t / NP, k = t % NP;
      float2 *row = A + line_slot(ly, 1, j) * P;
      float2 *ok = row + line_in(lx, k), *om = row + (k == 0 ? SPARE : line_in(lx, NH - k));
      float2 x[R], y[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        x[i] = ok[i * S * P];
        y[i] = om[i * S * P];
      }
      line_twiddle<R, 1>(ly, 1, j, x, a.twy);
      line_twiddle<R, 1>(ly, 1, j, y, a.twy);
      Dft<R, 1>::run(x);
      Dft<R, 1>::run(y);
      if (k > 0) {
        // e = X_k + conj X_m, T = i conj(W^k) (X_k - conj X_m):
        // Z_k = e + T, Z_m = conj(e - T)
        float2 w = __ldg(a.wx + k);
        w = make_float2(w.y, w.x);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float2 e = make_float2(x[i].x + y[i].x, x[i].y - y[i].y);
          const float2 T = cmul(make_float2(x[i].x - y[i].x, x[i].y + y[i].y), w);
          ok[i * S * P] = cadd(e, T);
          om[i * S * P] = make_float2(e.x - T.x, T.y - e.y);
        }
      } else {
        // DC and Nyquist: their imaginary parts are ignored
#pragma unroll
        for (int i = 0; i < R; ++i) ok[i * S * P] = make_float2(x[i].x + y[i].x, x[i].x - y[i].x);
        float2 *oc = row + line_in(lx, NH / 2);
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = oc[i * S * P];
        line_twiddle<R, 1>(ly, 1, j, x, a.twy);
        Dft<R, 1>::run(x);
#pragma unroll
        for (int i = 0; i < R; ++i) oc[i * S * P] = make_float2(2.f * x[i].x, -2.f * x[i].y);
      }
    }
  }
  __syncthreads();
  // 3. x, first stage, in place
  row_stage<LX, 0, 1, NQ, P, NTH>(A, a.twx, tid);
  __syncthreads();

  // 4. x, last stage: shared memory -> registers -> HBM (scale, addend, zero pad)
  {
    constexpr int R = LX::R(1), M = LX::M(1), ST = LX::S(1);
#pragma unroll 1
    for (int t = tid; t < NQ * M; t += NTH) {
      const int q = t / M, j = t % M;
      const float2 *o = A + line_out(ly, q) * P + line_slot(lx, 1, j);  // y output q sits in its line's slot
      float2 v[R], w[R];
      if (add) {  // its loads run under the butterfly
        const float2 *e = add + q * CX + j;
#pragma unroll
        for (int i = 0; i < R; ++i) w[i] = e[i * M];
      }
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = o[i * ST];
      line_twiddle<R, 1>(lx, 1, j, v, a.twx);
      Dft<R, 1>::run(v);
      float2 *d = dst + q * CX + j;
      if (add) {
#pragma unroll
        for (int i = 0; i < R; ++i) d[i * M] = cadd(cscale(v[i], scale), w[i]);
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i) d[i * M] = cscale(v[i], scale);
      }
      if (j == 0) d[NH] = make_float2(0.f, 0.f);
    }
  }
}

}  // namespace crava
