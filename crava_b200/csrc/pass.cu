// pass.cu -- host side of the built-in passes (fft_pass.cuh): which lengths
// are compiled, the stage tables, and the launches.
#include <math.h>

#include <vector>

#include "fft_lengths.cuh"
#include "fft_pass.cuh"

namespace crava {

#define CRAVA_DECL(N)        \
  ColLaunch col_launch_##N(); \
  RowLaunch row_launch_##N(); \
  SyntLaunch synt_launch_##N();
CRAVA_LINE_LENGTHS(CRAVA_DECL)
#undef CRAVA_DECL

#define CRAVA_FIND(N) case N: return CRAVA_WHICH(N)();
#define CRAVA_WHICH(N) col_launch_##N
ColLaunch col_launch(int n) {
  switch (n) { CRAVA_LINE_LENGTHS(CRAVA_FIND) default: return nullptr; }
}
#undef CRAVA_WHICH
#define CRAVA_WHICH(N) row_launch_##N
RowLaunch row_launch(int nx) {
  switch (nx) { CRAVA_LINE_LENGTHS(CRAVA_FIND) default: return nullptr; }
}
#undef CRAVA_WHICH
#define CRAVA_WHICH(N) synt_launch_##N
SyntLaunch synt_launch(int n) {
  switch (n) { CRAVA_LINE_LENGTHS(CRAVA_FIND) default: return nullptr; }
}
#undef CRAVA_WHICH
#undef CRAVA_FIND

namespace {

// Tables of one geometry, gathered on the host and uploaded in one copy: the
// pointers are set when the device buffer exists.
struct Tables {
  std::vector<float2> host;
  std::vector<std::pair<float2 **, size_t>> at;
  void add(const std::vector<float2> &v, float2 **out) {
    at.emplace_back(out, host.size());
    host.insert(host.end(), v.begin(), v.end());
  }
};

float2 root(long long k, int n) {  // e^{-2 pi i k / n}
  const double ang = -2.0 * M_PI * (double)(k % n) / (double)n;
  return make_float2((float)cos(ang), (float)sin(ang));
}

// The stage tables of a line: stage s >= 1, entry q NS + b holds
// W_n^{q b n / (NS R)}.
void stage_tables(const LineList &l, int n, Tables *to, float2 **out) {
  std::vector<float2> t;
  int ns = l.r[0];
  for (int s = 1; s < l.n; ++s) {
    for (int q = 0; q < l.r[s]; ++q)
      for (int b = 0; b < ns; ++b) t.push_back(root((long long)q * b * (n / (ns * l.r[s])), n));
    ns *= l.r[s];
  }
  to->add(t, out);
}

// The radices of LineOf<n, pad, desc>.
LineList line_order(int n, bool pad, bool desc) {
  LineList l = line_list(n);
  const bool listed = n == 32 || (!pad && (n == 64 || n == 128 || n == 256 || n == 512));
  if (!listed && l.r[0] != l.r[l.n - 1] && (l.r[0] > l.r[l.n - 1]) != desc)
    for (int i = 0; i < l.n / 2; ++i) {
      const int t = l.r[i];
      l.r[i] = l.r[l.n - 1 - i];
      l.r[l.n - 1 - i] = t;
    }
  return l;
}

}  // namespace

int pass_plan_create(const Geom &g, PassPlan *p) {
  Tables t;
  auto roots = [&](int n, int count, float2 **out) {
    std::vector<float2> w(count);
    for (int k = 0; k < count; ++k) w[k] = root(k, n);
    t.add(w, out);
  };
  if (row_launch(g.nxp)) {
    const int n = g.nxp % 2 ? g.nxp : g.nxp / 2;
    stage_tables(line_order(n, true, false), n, &t, &p->xf);
    stage_tables(line_order(n, true, true), n, &t, &p->xi);
    roots(g.nxp, g.nxp / 2 + 1, &p->wx);
  }
  // 32-bit line numbers and offsets in the column passes
  const bool fits = (long long)g.cnxp * g.nyp < (1LL << 31) && (long long)g.cnxp * g.nzp < (1LL << 31) &&
                    g.csize < (1LL << 32);
  if (fits && col_launch(g.nyp)) stage_tables(line_order(g.nyp, false, true), g.nyp, &t, &p->y);
  if (fits && col_launch(g.nzp)) stage_tables(line_order(g.nzp, false, true), g.nzp, &t, &p->z);
  if (fits && synt_launch(g.nzp)) stage_tables(synt_list(g.nzp), g.nzp, &t, &p->synt);
  p->parts = plane_parts(g);
  if (p->parts) {
    // the y line of a part: the stage that holds a column pair (radix 8) first
    // (forward) or last
    const int nq = g.nyp / p->parts;
    LineList f{}, i{};
    f.n = i.n = 2;
    f.r[0] = i.r[1] = 8;
    f.r[1] = i.r[0] = nq / 8;
    stage_tables(f, nq, &t, &p->pyf);
    stage_tables(i, nq, &t, &p->pyi);
    roots(g.nyp, g.nyp, &p->wy);
  }
  if (t.host.empty()) return CRAVA_GPU_OK;
  const size_t bytes = sizeof(float2) * t.host.size();
  CRAVA_CUDA_TRY(cudaMalloc(&p->tables, bytes));
  CRAVA_CUDA_TRY(cudaMemcpy(p->tables, t.host.data(), bytes, cudaMemcpyHostToDevice));
  for (auto &e : t.at) *e.first = p->tables + e.second;
  return CRAVA_GPU_OK;
}

void pass_plan_destroy(PassPlan *p) {
  cudaFree(p->tables);
  *p = PassPlan{};
}

int rows_batch(const FftPlans &p, const GridBatch &b, int dir, cudaStream_t s) {
  RowPassArgs a;
  for (int i = 0; i < b.n; ++i) {
    a.g.src[i] = dir < 0 && b.src[i] ? b.src[i] : b.dst[i];
    a.g.dst[i] = b.dst[i];
    a.g.add[i] = b.add[i];
    a.g.scale[i] = b.scale[i];
  }
  const int pairs = (p.g.nyp + 1) / 2;
  a.nlines = (uint32_t)(p.g.nxp % 2 ? pairs : p.g.nyp) * (uint32_t)p.g.nzp;  // sides up to 4096
  a.odd = (uint32_t)(p.g.nyp % 2);
  a.fpairs = make_fastdiv((uint32_t)pairs);
  a.tw = dir < 0 ? p.pass.xf : p.pass.xi;
  a.post = p.pass.wx;
  return row_launch(p.g.nxp)(a, b.n, dir, s);
}

static ColPassArgs col_args(const GridBatch &b, int dir, const ZPrior *zp) {
  ColPassArgs a;
  a.inv = nullptr;
  a.nf_bits = a.nf_any = nullptr;
  for (int i = 0; i < b.n; ++i) {
    a.dst[i] = reinterpret_cast<float2 *>(b.dst[i]);
    a.mode[i] = 0;
    a.v[i] = 0.0;
    if (zp && dir < 0 && zp[i].inv) {
      a.mode[i] = zp[i].mode;
      a.v[i] = zp[i].v;
      a.inv = zp[i].inv;
      a.nf_bits = zp[i].nf_bits;
      a.nf_any = zp[i].nf_any;
    }
  }
  return a;
}

int y_batch(const FftPlans &p, const GridBatch &b, int dir, cudaStream_t s) {
  const Geom &g = p.g;
  ColPassArgs a = col_args(b, dir, nullptr);
  a.nlines = (long long)g.cnxp * g.nzp;
  a.inner = (uint32_t)g.cnxp;
  a.finner = make_fastdiv(a.inner);
  a.outer = (uint32_t)(g.cnxp * g.nyp);
  a.es = (uint32_t)g.cnxp;
  a.tw = p.pass.y;
  return col_launch(g.nyp)(a, b.n, dir, s);
}

int z_batch(const FftPlans &p, const GridBatch &b, int dir, bool parts, const ZPrior *zp, cudaStream_t s) {
  const Geom &g = p.g;
  ColPassArgs a = col_args(b, dir, zp);
  const int plane = g.cnxp * g.nyp;
  a.nlines = parts ? plane / p.pass.parts : plane;
  a.inner = (uint32_t)plane;
  a.finner = make_fastdiv(a.inner);
  a.outer = 0;
  a.es = (uint32_t)plane;
  a.tw = p.pass.z;
  return parts ? z_parts_launch(a, g.nzp, b.n, dir, s) : col_launch(g.nzp)(a, b.n, dir, s);
}

}  // namespace crava
