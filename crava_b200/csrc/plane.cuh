// plane.cuh -- the x and y passes of a 3-D transform in one kernel, for planes
// with power-of-two sides: a z-plane, or half of its rows, lives in a CTA's
// shared memory between the two passes, so a transform moves 4 grids of HBM
// traffic (this pass and the z pass) where separate x, y and z passes move 6.
//
// Planes up to 128x128, and 256x64, are one CTA's (CS = 1): 23 to 45 KB and 256
// threads up to 64x128 and 128x64, 88 and 78 KB, 512 threads and two CTAs per SM at
// 128x128 and 256x64.  Of a 256x256 plane CTA r of CS = 2 holds the rows y = CS q + r, q < NQ = nyp / CS
// (149 KB, 1024 threads).  With ky = k1 + NQ k2,
//   Y[k1 + NQ k2] = sum_r W_CS^{r k2} [ W_nyp^{r k1} sum_q x[CS q + r] W_NQ^{q k1} ]:
// the kernel does the brackets, leaves bracket (k1, r) in row k1 + NQ r, and the
// radix-CS step over r, which needs rows from both CTAs, is the z pass's first
// butterfly (k_col_parts, 8 adjacent columns of both parts): the rows meet in its
// registers and cost no extra traffic and no exchange between CTAs.  The inverse
// runs the same steps backwards.  In place a CTA's output rows are the other
// CTA's input rows: the two form a cluster, each arrives at its barrier when its
// loads are done and waits there before its first store.
//
// Where no such z pass follows (the x and y passes of a slab, or another z pass
// by the tuning) the kernel does the radix-2 step itself (WHOLE), with the same
// values.  Forward each CTA takes the rows of half of the k1 and pushes its
// brackets of the other half into the partner's shared memory, in the order of
// the columns (66 KB more, 215 in all); inverse each CTA reads both rows k1 and
// k1 + NQ of the pair and forms its own part's, the second reading coming from
// L2 as the two run at once.  One slab of 256x256x512: 116 / 97 us forward /
// inverse, of 64 planes 20.6 / 17.5 (the earlier cluster of four CTAs 121 / 110 and
// 24.7 / 20.6; the parts kernel and a radix-2 pass after it 141 / 140 and 24.1 /
// 22.9).  Forward, the partner's brackets pulled from the slots they lie in,
// scattered over the banks, took 131 us, handed over through L2 123.
//
// The split of the packed x line into the half spectrum pairs column k with
// nh - k; the first y stage (forward) or the last one (inverse) takes the two
// columns of a pair together and does it in registers.
//
// Measured, 128x128x256 one grid at a time: 12.8 / 12.4 us forward / inverse
// (separate row and column passes 16.8 / 16.7 us; the earlier two-CTA cluster
// kernel 19.0 / 16.7 us).  256x256x512 in a unit of 15 grids, one launch: 81 / 85
// us and the z pass with the radix-2 step 53 / 50 us (41 us at the copy rate);
// one CTA per SM runs its loads, barriers and stores one after the other, with
// the next CTA's input on its way into L2 meanwhile (fetch_l2).  Against it, per
// grid and before that fetch (88 / 93, z 66 / 61): an earlier form over a cluster
// of four CTAs with the last step through distributed shared memory 108 / 100 us
// (z 54 / 50); four parts of 74 KB 75 / 74 us, but 86 / 80 us in the z pass, whose
// runs shrink to 32 bytes; both passes in one cluster kernel with the exchange
// through L2 105 / 103 us; separate row and column passes 43 + 44 / 46 + 51 us at
// the start of a series, but they draw enough power through the HBM that the
// clock falls and a unit takes 5.08 ms instead of 4.90 (4.47 with the fetch).
#pragma once

#include "fft_pass.cuh"

namespace crava {

template <int NX, int NY, int CS>
struct PlaneCfg {
  using R = RowCfg<NX>;
  static constexpr int NH = NX / 2, CX = NH + 1, NQ = NY / CS, NP = NH / 2;
  static constexpr RowBanks kBanks = row_banks(NH);
  using XF = LineOf<NH, kBanks.sf, false>;
  using XI = LineOf<NH, kBanks.si, true>;
  // the y line: the stage that holds a column pair has the smaller radix
  using YF = CtLine<0, NQ == 64 ? 8 : NQ == 128 ? 8 : 16, NQ == 64 ? 8 : 16>;
  using YI = CtLine<0, NQ == 64 ? 8 : 16, NQ == 64 ? 8 : NQ == 128 ? 8 : 16>;
  // a row holds its padded line and a spare slot (the Nyquist column); the
  // pitch keeps the residue that its bank layout wants (a unit of 128x128x256, five
  // angles: 530 us with pitch 88 and two CTAs of 512 threads per SM, 575 with the
  // least pitch, 73, and three of 256)
  static constexpr int pitch(int line, int want) { return want > line ? want : line + 1 + (want - line - 1 + 1600) % 16; }
  static constexpr int PF = pitch(XF::R(0) * XF::S(0), kBanks.pf), PI = pitch(XI::R(0) * XI::S(0), kBanks.pi);
  static constexpr size_t smem(int dir) {
    return sizeof(float2) * ((size_t)NQ * (dir < 0 ? PF : PI) + (CS > 1 ? NQ : 0));
  }
  // the forward kernel that completes y receives half of the partner's rows
  static constexpr size_t smem_whole(int dir) { return smem(dir) + (dir < 0 ? sizeof(float2) * (size_t)(NQ / 2) * CX : 0); }
  static constexpr int kCtas = 224 * 1024 / (int)(smem(PF > PI ? -1 : 1) + 1024) >= 3 ? 3
                               : 224 * 1024 / (int)(smem(PF > PI ? -1 : 1) + 1024) >= 2 ? 2 : 1;
  static constexpr int NTH = kCtas == 3 ? 256 : kCtas == 2 ? 512 : 1024;
  static constexpr int kMinB = NTH == 256 ? 4 : NTH == 512 ? 2 : 1;
};

// a s, kept out of the butterflies that follow: contracted into their sums, the
// product would be rounded in one operand only, and equal rows (the transform
// of a constant mean) would no longer cancel exactly.
__device__ __forceinline__ float2 scaled(float2 a, float s) { return make_float2(__fmul_rn(a.x, s), __fmul_rn(a.y, s)); }

struct PlaneArgs {
  PassGrids g;
  const float2 *twx, *twy, *wx, *wy;  // stage tables, W_nxp^k, W_nyp^k
  int ahead;                          // CTAs ahead whose input is fetched into L2 (CS > 1)
};

// With one CTA per SM nothing runs under a CTA's loads, so it asks for the data
// of the CTA that will take its place, one wave on, as soon as its own loads are
// done: HBM then works under its butterflies and stores, and the next loads find
// their lines in L2 (a wave's reads are 20 MB).  256x256x512, a unit of 15 grids
// in one launch, per grid: 88 / 93 -> 81 / 85 us forward / inverse, and the z
// pass of the parts (k_col_parts) 66 / 61 -> 53 / 50.  Half the wave ahead or the
// wave: the same in the plane passes; 1.75 CTAs per SM ahead of 3 resident are
// best in the z pass (2 and 1.5 per SM 54 / 50 and 54 / 52, 3 per SM 57 / 53, 1
// per SM 58 / 58, 6 per SM 70 / 68).  In
// the row and column passes of smaller grids (several CTAs per SM, inputs mostly
// in L2) nothing is gained: within 1 % at 1 to 4 per SM.
__device__ __forceinline__ void fetch_l2(const float2 *p, int n, int tid, int nth) {
  for (int k = 16 * tid; k < n; k += 16 * nth) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p + k));
}
// The CTA `ahead` places on in the order of the launch: its PART values, which
// the plane's other CTAs complete (all of the plane's rows are read by one of
// them).  Nothing past the launch's last CTA.
template <int PART>
__device__ __forceinline__ void fetch_next(const PlaneArgs &a, int tid, int nth) {
  unsigned b = blockIdx.x + (unsigned)a.ahead, g = blockIdx.y;
  while (b >= gridDim.x) {
    b -= gridDim.x;
    ++g;
  }
  if (g < gridDim.y)
    fetch_l2(reinterpret_cast<const float2 *>(a.g.src[g]) + (long long)b * PART, PART, tid, nth);
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }

__device__ __forceinline__ uint32_t cluster_addr(const void *smem, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(smem)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}

template <int NX, int NY, int CS, bool WHOLE>
__global__ void __launch_bounds__(PlaneCfg<NX, NY, CS>::NTH, PlaneCfg<NX, NY, CS>::kMinB)
    k_plane_fwd(const __grid_constant__ PlaneArgs a) {
  using C = PlaneCfg<NX, NY, CS>;
  using LX = typename C::XF;
  using LY = typename C::YF;
  constexpr LX lx{};
  constexpr LY ly{};
  constexpr int NTH = C::NTH, NQ = C::NQ, NH = C::NH, CX = C::CX, NP = C::NP, P = C::PF, SPARE = LX::R(0) * LX::S(0);
  static_assert(LX::nst() == 2 && LY::nst() == 2, "two-stage lines");
  static_assert(!WHOLE || CS == 2, "the radix-2 step over two parts");
  extern __shared__ float4 sm4[];
  float2 *A = reinterpret_cast<float2 *>(sm4), *twr = A + NQ * P;
  const int tid = threadIdx.x;
  const int plane = blockIdx.x / CS, r = blockIdx.x % CS, g = blockIdx.y;
  const float2 *src = reinterpret_cast<const float2 *>(a.g.src[g]) + (long long)plane * CX * NY + r * CX;
  float2 *dst = reinterpret_cast<float2 *>(a.g.dst[g]) + (long long)plane * CX * NY + (long long)r * NQ * CX;
  const float scale = a.g.scale[g];

  // 1. x, first stage: HBM -> registers -> shared memory
  {
    constexpr int R = LX::R(0), M = LX::M(0), S = LX::S(0), G = rounds_group(R, 16, ceil_div(NQ * M, NTH));
    float2 v[G][R];
    rounds<NQ * M, NTH, G>(
        tid,
        [&](int u, int t) {
          const float2 *row = src + (t / M) * (CS * CX) + t % M;
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
  if constexpr (CS > 1) {
    for (int k = tid; k < NQ; k += NTH) twr[k] = a.wy[r * k];
    if (WHOLE || a.g.src[g] == a.g.dst[g]) cluster_arrive();  // this CTA's rows are read
    fetch_next<NQ * CX>(a, tid, NTH);
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
        const float2 w = __ldg(a.wx + k);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          split_pair(ok[i * M * P], om[i * M * P], w, &x[i], &y[i]);
          x[i] = scaled(x[i], scale);
          y[i] = scaled(y[i], scale);
        }
      } else {
#pragma unroll
        for (int i = 0; i < R; ++i) {  // DC and Nyquist from z_0
          const float2 z = ok[i * M * P];
          x[i] = scaled(make_float2(z.x + z.y, 0.f), scale);
          y[i] = scaled(make_float2(z.x - z.y, 0.f), scale);
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
          x[i] = scaled(cconj(z), scale);
        }
        Dft<R, -1>::run(x);
#pragma unroll
        for (int i = 0; i < R; ++i) oc[i * M * P] = x[i];
      }
    }
  }
  __syncthreads();

  // 4. y, last stage: shared memory -> registers -> HBM
  constexpr int R = LY::R(1), M = LY::M(1), S = LY::S(1);
  auto last = [&](int t, float2 *v) {  // the brackets of rows j + i M, column k; their first slot
    const int j = t / CX, k = t % CX;
    float2 *o = A + line_slot(ly, 1, j) * P + (k == NH ? SPARE : line_out(lx, k));
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = o[i * S * P];
    line_twiddle<R, -1>(ly, 1, j, v, a.twy);
    Dft<R, -1>::run(v);
    if constexpr (CS > 1) {
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = cmul(v[i], twr[j + i * M]);
    }
    return o;
  };
  if constexpr (!WHOLE) {
    if constexpr (CS > 1) if (a.g.src[g] == a.g.dst[g]) cluster_wait();  // every CTA of the plane has read its rows
#pragma unroll 1
    for (int t = tid; t < CX * M; t += NTH) {
      float2 v[R];
      last(t, v);
      float2 *d = dst + (t / CX) * CX + t % CX;
#pragma unroll
      for (int i = 0; i < R; ++i) d[i * M * CX] = v[i];
    }
  } else {
    // and the radix-2 step: this CTA takes the rows of half of the i.  A
    // butterfly keeps that half (in registers; those of the columns past a whole
    // round, a few, in their slots) and pushes the other into the partner's
    // shared memory, in the order of the columns
    constexpr int H = R / 2;
    static_assert(NTH < CX * M && CX * M <= 2 * NTH, "one butterfly per thread and a remainder");
    const int i0 = r * H;  // first i of this CTA's rows
    float2 *B = twr + NQ;  // [H][CX M]: the partner's brackets of this CTA's rows
    const uint32_t to = cluster_addr(B, r ^ 1);
    float2 *out = reinterpret_cast<float2 *>(a.g.dst[g]) + (long long)plane * CX * NY;
    const int t1 = tid + NTH;
    const bool rest = t1 < CX * M;
    cluster_wait();  // the partner runs, and has read its rows
    auto push = [&](int t, const float2 *v) {
#pragma unroll
      for (int i = 0; i < H; ++i) cluster_store(to + (uint32_t)sizeof(float2) * (i * CX * M + t), r == 0 ? v[i + H] : v[i]);
    };
    float2 keep[H];
    float2 *slot = nullptr;
    if (rest) {
      float2 v[R];
      slot = last(t1, v) + i0 * S * P;
      push(t1, v);
#pragma unroll
      for (int i = 0; i < H; ++i) slot[i * S * P] = r == 0 ? v[i] : v[i + H];
    }
    {
      float2 v[R];
      last(tid, v);
      push(tid, v);
#pragma unroll
      for (int i = 0; i < H; ++i) keep[i] = r == 0 ? v[i] : v[i + H];
    }
    cluster_arrive();  // this CTA's pushes are done
    cluster_wait();
    auto finish = [&](int t) {
      float2 *d = out + (t / CX + i0 * M) * CX + t % CX;
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const float2 his = B[i * CX * M + t];
        float2 v[2] = {r == 0 ? keep[i] : his, r == 0 ? his : keep[i]};
        Dft<2, -1>::run(v);
        d[i * M * CX] = v[0];
        d[(i * M + NQ) * CX] = v[1];
      }
    };
    finish(tid);
    if (rest) {
#pragma unroll
      for (int i = 0; i < H; ++i) keep[i] = slot[i * S * P];
      finish(t1);
    }
  }
}

template <int NX, int NY, int CS, bool WHOLE>
__global__ void __launch_bounds__(PlaneCfg<NX, NY, CS>::NTH, PlaneCfg<NX, NY, CS>::kMinB)
    k_plane_inv(const __grid_constant__ PlaneArgs a) {
  using C = PlaneCfg<NX, NY, CS>;
  using LX = typename C::XI;
  using LY = typename C::YI;
  constexpr LX lx{};
  constexpr LY ly{};
  constexpr int NTH = C::NTH, NQ = C::NQ, NH = C::NH, CX = C::CX, NP = C::NP, P = C::PI, SPARE = LX::R(0) * LX::S(0);
  extern __shared__ float4 sm4[];
  float2 *A = reinterpret_cast<float2 *>(sm4), *twr = A + NQ * P;
  const int tid = threadIdx.x;
  const int plane = blockIdx.x / CS, r = blockIdx.x % CS, g = blockIdx.y;
  static_assert(!WHOLE || CS == 2, "the radix-2 step over two parts");
  const float2 *src = reinterpret_cast<const float2 *>(a.g.src[g]) + (long long)plane * CX * NY +
                      (WHOLE ? 0 : (long long)r * NQ * CX);
  const long long off = (long long)plane * CX * NY + r * CX;
  float2 *dst = reinterpret_cast<float2 *>(a.g.dst[g]) + off;
  const float2 *add = a.g.add[g] ? reinterpret_cast<const float2 *>(a.g.add[g]) + off : nullptr;
  const float scale = a.g.scale[g];
  if constexpr (CS > 1) {
    for (int k = tid; k < NQ; k += NTH) twr[k] = cconj(a.wy[r * k]);
    __syncthreads();
  }

  // 1. y, first stage: HBM -> registers -> shared memory
  {
    constexpr int R = LY::R(0), M = LY::M(0);
#pragma unroll 1
    for (int t = tid; t < CX * M; t += NTH) {
      const int j = t / CX, k = t % CX;
      const float2 *o = src + j * CX + k;
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        v[i] = o[i * M * CX];
        if constexpr (WHOLE) {  // the radix-2 step over the two parts: this part's output
          const float2 w = o[(i * M + NQ) * CX];
          v[i] = r == 0 ? cadd(v[i], w) : csub(v[i], w);
        }
      }
      if constexpr (CS > 1) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = cmul(v[i], twr[j + i * M]);
      }
      Dft<R, 1>::run(v);
      float2 *d = A + j * P + (k == NH ? SPARE : line_in(lx, k));
#pragma unroll
      for (int i = 0; i < R; ++i) d[i * M * P] = v[i];
    }
  }
  if constexpr (CS > 1) {
    cluster_arrive();
    fetch_next<NQ * CX>(a, tid, NTH);
    if (a.g.add[g])  // the plane's addend, read in the last step
      fetch_l2(reinterpret_cast<const float2 *>(a.g.add[g]) + (long long)blockIdx.x * (NQ * CX), NQ * CX, tid, NTH);
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
        const float2 w = __ldg(a.wx + k);
#pragma unroll
        for (int i = 0; i < R; ++i) merge_pair(x[i], y[i], w, ok + i * S * P, om + i * S * P);
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
  if constexpr (CS > 1) cluster_wait();
  {
    constexpr int R = LX::R(1), M = LX::M(1), ST = LX::S(1);
#pragma unroll 1
    for (int t = tid; t < NQ * M; t += NTH) {
      const int q = t / M, j = t % M;
      const float2 *o = A + line_out(ly, q) * P + line_slot(lx, 1, j);  // y output q sits in its line's slot
      float2 v[R], w[R];
      if (add) {  // its loads run under the butterfly
        const float2 *e = add + q * (CS * CX) + j;
#pragma unroll
        for (int i = 0; i < R; ++i) w[i] = e[i * M];
      }
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = o[i * ST];
      line_twiddle<R, 1>(lx, 1, j, v, a.twx);
      Dft<R, 1>::run(v);
      float2 *d = dst + q * (CS * CX) + j;
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

// ------------------------------------------------------------------ z pass of a split plane
// 16 / CS adjacent columns of all CS parts, rows k1 + NQ r: the radix-CS
// butterfly over r on registers with the first stage's inputs (forward) or the
// last stage's outputs (inverse).
template <int CS>
__device__ __forceinline__ int swz(int e, int p) { return e * kColLines + ((p + kColLines / CS * e) & (kColLines - 1)); }
template <int N, int DIR, int CS>
__global__ void __launch_bounds__(256, 3) k_col_parts(const __grid_constant__ ColPassArgs a) {
  using L = LineOf<N, 0, true>;
  constexpr L l{};
  constexpr int TXC = kColLines / CS, NTH = 256, TPB = NTH / kColLines;
  extern __shared__ float4 sm4[];
  float2 *B = reinterpret_cast<float2 *>(sm4);  // [N][kColLines]
  const int tid = threadIdx.x, g = blockIdx.y;
  const uint32_t part = (uint32_t)a.nlines, es = a.es;  // lines per part; lines per plane
  const uint32_t f0 = blockIdx.x * TXC;
  float2 *data = a.dst[g];
  const int p = tid % kColLines, t0 = tid / kColLines;
  const int pc = tid % TXC, tc = tid / TXC;
  constexpr int TPC = NTH / TXC;
  const uint32_t line = f0 + p % TXC + (p / TXC) * part;  // of column p of the tile
  const bool ok = f0 + p % TXC < part, okc = f0 + pc < part;
  if constexpr (DIR < 0) {
    constexpr int R = L::R(0), M = L::M(0);
#pragma unroll 1
    for (int j = tc; j < M; j += TPC) {
      if (!okc) break;
      const uint32_t o = f0 + pc + j * es;
      float2 v[CS][R];
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int r = 0; r < CS; ++r) v[r][i] = data[o + i * M * es + r * part];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float2 u[CS];
#pragma unroll
        for (int r = 0; r < CS; ++r) u[r] = v[r][i];
        Dft<CS, -1>::run(u);
#pragma unroll
        for (int r = 0; r < CS; ++r) v[r][i] = u[r];
      }
#pragma unroll
      for (int r = 0; r < CS; ++r) {
        Dft<R, -1>::run(v[r]);
#pragma unroll
        for (int i = 0; i < R; ++i) B[swz<CS>(j + i * L::S(0), r * TXC + pc)] = v[r][i];
      }
    }
  } else {
    constexpr int R = L::R(0), M = L::M(0);
#pragma unroll 2
    for (int j = t0; j < M; j += TPB) {
      if (!ok) break;
      const uint32_t o = line + j * es;
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = data[o + i * M * es];
      Dft<R, 1>::run(v);
#pragma unroll
      for (int i = 0; i < R; ++i) B[swz<CS>(j + i * L::S(0), p)] = v[i];
    }
  }
  {  // a later tile's runs into L2 (see fetch_l2)
    uint32_t nb = blockIdx.x + a.ahead, ng = g;
    while (nb >= gridDim.x) {
      nb -= gridDim.x;
      ++ng;
    }
    if (ng < gridDim.y) {
      const float2 *next = a.dst[ng] + nb * TXC;
      for (int k = tid; k < N * CS; k += NTH)
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(next + (k / CS) * es + (k % CS) * part));
    }
  }
  __syncthreads();
  if constexpr (L::nst() > 2) {
    constexpr int R = L::R(1), M = L::M(1), ST = L::S(1);
#pragma unroll 1
    for (int j = t0; j < M; j += TPB) {
      const int o = line_slot(l, 1, j);
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = B[swz<CS>(o + i * ST, p)];
      line_twiddle<R, DIR>(l, 1, j, v, a.tw);
      Dft<R, DIR>::run(v);
#pragma unroll
      for (int i = 0; i < R; ++i) B[swz<CS>(o + i * ST, p)] = v[i];
    }
    __syncthreads();
  }
  constexpr int S = L::nst() - 1, R = L::R(S), M = L::M(S), ST = L::S(S);
  if constexpr (DIR < 0) {
    ZPrior zp;
    zp.mode = a.mode[g];
    zp.v = a.v[g];
    zp.nf_bits = a.nf_bits;
    zp.nf_any = a.nf_any;
#pragma unroll 1
    for (int j = t0; j < M; j += TPB) {
      if (!ok) break;
      unsigned gated = 0u;
      if (zp.mode) {
#pragma unroll
        for (int i = 0; i < R; ++i) gated |= __ldg(a.inv + j + i * M) == 0 ? 1u << i : 0u;
      }
      const int o = line_slot(l, S, j);
      float2 v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = B[swz<CS>(o + i * ST, p)];
      line_twiddle<R, -1>(l, S, j, v, a.tw);
      Dft<R, -1>::run(v);
      if (gated) {
#pragma unroll
        for (int i = 0; i < R; ++i)
          if ((gated >> i) & 1u) v[i] = zprior_apply(zp, v[i], line + (j + i * M) * es);
      }
      const uint32_t d = line + j * es;
#pragma unroll
      for (int i = 0; i < R; ++i) data[d + i * M * es] = v[i];
    }
  } else {
#pragma unroll 1
    for (int j = tc; j < M; j += TPC) {
      if (!okc) break;
      const int b = line_slot(l, S, j);
      float2 v[CS][R];
#pragma unroll
      for (int r = 0; r < CS; ++r) {
#pragma unroll
        for (int i = 0; i < R; ++i) v[r][i] = B[swz<CS>(b + i * ST, r * TXC + pc)];
        line_twiddle<R, 1>(l, S, j, v[r], a.tw);
        Dft<R, 1>::run(v[r]);
      }
      const uint32_t d = f0 + pc + j * es;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float2 u[CS];
#pragma unroll
        for (int r = 0; r < CS; ++r) u[r] = v[r][i];
        Dft<CS, 1>::run(u);
#pragma unroll
        for (int r = 0; r < CS; ++r) data[d + i * M * es + r * part] = u[r];
      }
    }
  }
}

}  // namespace crava
