// fft_line.cuh -- in-place line transforms in shared memory, the engine of
// the built-in x, y and z passes (fft_pass.cuh).
//
// A line of n = R_0 R_1 .. R_{s-1} points is transformed by s radix stages
// of the Stockham arithmetic of fft_core.cuh (twiddle on the inputs, then
// the butterfly), but every butterfly writes its outputs to the very slots
// its inputs came from.  So a stage needs one barrier after it, not two,
// and no second buffer; the first stage takes its inputs from HBM and the
// last leaves for HBM, which makes a line cost s - 1 trips through shared
// memory.  What the in-place order moves around is the digits of the index:
// after stage t, logical element
//   l = d_0 + d_1 R_0 + .. + d_t (R_0 .. R_{t-1}) + rest (R_0 .. R_t)
// sits in slot d_0 S_0 + d_1 S_1 + .. + d_t S_t + rest with
// S_t = n / (R_0 .. R_t), so a stage's inputs are equally spaced and the
// last stage's outputs leave in natural order.  S_0 may be padded (one spare
// element): lanes that walk d_0 then fall into different banks.
//
// Radices go up to 20 (composite ones in registers), so that of the 89
// 2, 3, 5, 7-smooth lengths 24 .. 512 61 take two stages and the others
// three.  Every such length is compiled with its radices, strides and
// twiddle offsets as constants: a first form with the radices in a struct
// and a switch spent 76 instead of about 40 warp instructions per point and
// warp on a 300-point line (index arithmetic, spills, instruction misses).
#pragma once

#include <utility>

#include "fft_core.cuh"

namespace crava {

// Composite radices.  A B with A, B coprime (6, 10, 12, 14, 15, 18, 20): the
// Good-Thomas map needs no twiddles between the two parts.  9 = 3 x 3.
template <int A, int B, int DIR>
struct DftCoprime {
  static constexpr int N = A * B;
  static __host__ __device__ constexpr int inv(int a, int m) {  // a^-1 mod m
    for (int x = 1; x < m; ++x)
      if (a * x % m == 1) return x;
    return 1;
  }
  static __device__ __forceinline__ void run(float2 *v) {
    constexpr int EA = B * inv(B % A, A) % N, EB = A * inv(A % B, B) % N;  // CRT basis
    float2 y[A][B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      float2 t[A];
#pragma unroll
      for (int a = 0; a < A; ++a) t[a] = v[(B * a + A * b) % N];
      Dft<A, DIR>::run(t);
#pragma unroll
      for (int a = 0; a < A; ++a) y[a][b] = t[a];
    }
#pragma unroll
    for (int a = 0; a < A; ++a) {
      Dft<B, DIR>::run(y[a]);
#pragma unroll
      for (int b = 0; b < B; ++b) v[(EA * a + EB * b) % N] = y[a][b];
    }
  }
};
template <int DIR> struct Dft<6, DIR> : DftCoprime<2, 3, DIR> {};
template <int DIR> struct Dft<10, DIR> : DftCoprime<2, 5, DIR> {};
template <int DIR> struct Dft<12, DIR> : DftCoprime<4, 3, DIR> {};
template <int DIR> struct Dft<14, DIR> : DftCoprime<2, 7, DIR> {};
template <int DIR> struct Dft<15, DIR> : DftCoprime<3, 5, DIR> {};
template <int DIR> struct Dft<20, DIR> : DftCoprime<4, 5, DIR> {};

template <int DIR>
struct Dft<9, DIR> {
  static __device__ __forceinline__ float2 tw(float2 a, int m) {  // a e^{DIR 2 pi i m / 9}
    const float c = m == 1 ? 0.76604444311897803520f : m == 2 ? 0.17364817766693034885f : -0.93969262078590838405f;
    const float s = DIR * (m == 1 ? 0.64278760968653932632f : m == 2 ? 0.98480775301220805937f : 0.34202014332566873304f);
    return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
  }
  static __device__ __forceinline__ void run(float2 *v) {
    float2 y[3][3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      float2 t[3] = {v[b], v[3 + b], v[6 + b]};
      Dft<3, DIR>::run(t);
      y[b][0] = t[0];
      y[b][1] = b ? tw(t[1], b) : t[1];
      y[b][2] = b ? tw(t[2], 2 * b) : t[2];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float2 t[3] = {y[0][k], y[1][k], y[2][k]};
      Dft<3, DIR>::run(t);
#pragma unroll
      for (int q = 0; q < 3; ++q) v[k + 3 * q] = t[q];
    }
  }
};

template <int DIR> struct Dft<18, DIR> : DftCoprime<2, 9, DIR> {};

// Radices of a length, ascending: as few stages as radices up to 20 allow,
// the largest radix as small as possible; 32, 64, 128, 256 and 512 take the
// list of the other passes (CtRadix).  n = 0: none.
struct LineList {
  int n = 0;
  int r[4] = {};
};
__host__ __device__ constexpr bool line_radix_ok(int r) {
  return (r >= 2 && r <= 10) || r == 12 || (r >= 14 && r <= 16) || r == 18 || r == 20;
}
__host__ __device__ constexpr LineList line_list(int n) {
  LineList l{};
  if (n == 32 || n == 64 || n == 128 || n == 256 || n == 512) {
    l.n = CtRadix::count(n);
    for (int s = 0; s < l.n; ++s) l.r[s] = CtRadix::at(n, s);
    return l;
  }
  for (int b = 2; b <= 20; ++b)
    if (line_radix_ok(b) && n % b == 0 && n / b <= b && line_radix_ok(n / b)) {
      l.n = 2;
      l.r[0] = n / b;
      l.r[1] = b;
      return l;
    }
  for (int c = 2; c <= 20; ++c)
    for (int b = c; b >= 2; --b)
      if (line_radix_ok(c) && n % c == 0 && line_radix_ok(b) && (n / c) % b == 0 && n / c / b <= b &&
          line_radix_ok(n / c / b)) {
        l.n = 3;
        l.r[0] = n / c / b;
        l.r[1] = b;
        l.r[2] = c;
        return l;
      }
  return l;
}

// A line with compile-time radices; S0: the padded step of its first digit (0:
// none).
template <int S0, int... RS>
struct CtLine {
  static constexpr int kStages = sizeof...(RS);
  __host__ __device__ static constexpr int R(int s) {
    const int r[] = {RS...};
    return r[s];
  }
  __host__ __device__ static constexpr int prod(int s) {  // R_0 .. R_{s-1}
    int p = 1;
    for (int i = 0; i < s; ++i) p *= R(i);
    return p;
  }
  __host__ __device__ static constexpr int n() { return prod(kStages); }
  __host__ __device__ static constexpr int nst() { return kStages; }
  __host__ __device__ static constexpr int NS(int s) { return prod(s); }
  __host__ __device__ static constexpr int M(int s) { return n() / R(s); }
  __host__ __device__ static constexpr int S(int s) { return s == 0 && S0 > 0 ? S0 : n() / prod(s + 1); }
  __host__ __device__ static constexpr int T(int s) {
    int o = 0;
    for (int i = 1; i < s; ++i) o += prod(i + 1);
    return o;
  }
  __host__ __device__ static constexpr int entries() { return T(kStages); }
  __device__ static __forceinline__ int divR(int x, int s) { return (int)((unsigned)x / (unsigned)R(s)); }
  __device__ static __forceinline__ int divM(int x, int s) { return (int)((unsigned)x / (unsigned)M(s)); }
};

// The line of a length: radices ascending or descending (as listed at 32, whose
// x pass so keeps the values of the other x passes, and at 64, 128, 256 and 512
// points without padding, the y and z passes).
template <int N, int S0, bool DESC, class I>
struct LineOfImpl;
template <int N, int S0, bool DESC, size_t... I>
struct LineOfImpl<N, S0, DESC, std::index_sequence<I...>> {
  static constexpr LineList kL = line_list(N);
  static constexpr bool kAsListed = N == 32 || (S0 == 0 && (N == 64 || N == 128 || N == 256 || N == 512));
  static constexpr bool kFlip = !kAsListed && (kL.r[0] > kL.r[kL.n - 1]) != DESC && kL.r[0] != kL.r[kL.n - 1];
  using type = CtLine<S0, kL.r[kFlip ? kL.n - 1 - I : I]...>;
};
template <int N, int S0, bool DESC>
using LineOf = typename LineOfImpl<N, S0, DESC, std::make_index_sequence<line_list(N).n>>::type;

// Slot of input 0 of stage s's butterfly j; its other inputs are S(s) apart.
template <class L>
__device__ __forceinline__ int line_slot(const L &l, int s, int j) {
  if (s == 0) return j;
  int t = l.divR(j, 0);
  int a = (j - t * l.R(0)) * l.S(0);
  if (s > 1) {
    const int u = l.divR(t, 1);
    a += (t - u * l.R(1)) * l.S(1);
    t = u;
  }
  if (s > 2) {
    const int u = l.divR(t, 2);
    a += (t - u * l.R(2)) * l.S(2);
    t = u;
  }
  return a + t;
}
// Slot of input element e (before the first stage) and of output element k
// (after the last).
template <class L>
__device__ __forceinline__ int line_in(const L &l, int e) {
  const int q = l.divM(e, 0);
  return q * l.S(0) + (e - q * l.M(0));
}
template <class L>
__device__ __forceinline__ int line_out(const L &l, int k) {
  return line_slot(l, l.nst() - 1, k % l.M(l.nst() - 1)) + (k / l.M(l.nst() - 1)) * l.S(l.nst() - 1);
}

// j mod NS(s), s >= 1 (the last stage has M = NS: j itself).
template <class L>
__device__ __forceinline__ int line_base(const L &l, int s, int j) {
  if (s + 1 == l.nst()) return j;
  int t = l.divR(j, 0);
  if (s > 1) t = l.divR(t, 1);
  return j - t * l.NS(s);
}

// Twiddles of stage s, butterfly j on its R inputs (tw: the stage tables in
// device memory, entry q NS + (j mod NS) of stage s; they stay in L1).
template <int R, int DIR, class L>
__device__ __forceinline__ void line_twiddle(const L &l, int s, int j, float2 *v, const float2 *__restrict__ tw) {
  const float2 *t = tw + l.T(s) + line_base(l, s, j);
#pragma unroll
  for (int q = 1; q < R; ++q) {
    float2 w = __ldg(t + q * l.NS(s));
    if (DIR > 0) w.y = -w.y;
    v[q] = cmul(v[q], w);
  }
}

}  // namespace crava
