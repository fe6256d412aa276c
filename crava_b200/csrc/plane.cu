// plane.cu -- host side of the fused x + y pass (plane.cuh).
#include "plane.cuh"

namespace crava {

namespace {

template <int NX, int NY>
int launch_plane(const PlaneArgs &a, int dir, int nplanes, int ngrids, cudaStream_t s) {
  using C = PlaneCfg<NX, NY>;
  const void *fn = dir < 0 ? (const void *)k_plane_fwd<NX, NY> : (const void *)k_plane_inv<NX, NY>;
  const size_t smem = C::smem(dir);
  int rc = func_smem(fn, smem);
  if (rc) return rc;
  const dim3 grd((unsigned)nplanes, (unsigned)ngrids);
  if (dir < 0) k_plane_fwd<NX, NY><<<grd, C::NTH, smem, s>>>(a);
  else k_plane_inv<NX, NY><<<grd, C::NTH, smem, s>>>(a);
  CRAVA_LAUNCH_CHECK();
  return CRAVA_GPU_OK;
}

}  // namespace

bool plane_xy_supported(const Geom &g) {
  // three CTAs per SM: the rows of a plane in 75 KB
  const bool px = g.nxp == 64 || g.nxp == 128, py = g.nyp == 64 || g.nyp == 128;
  return (px && py) || (g.nxp == 256 && g.nyp == 64);
}

int plane_batch(const FftPlans &p, const GridBatch &b, int dir, cudaStream_t s) {
  const Geom &g = p.g;
  PlaneArgs a;
  for (int i = 0; i < b.n; ++i) {
    a.g.src[i] = dir < 0 && b.src[i] ? b.src[i] : b.dst[i];
    a.g.dst[i] = b.dst[i];
    a.g.add[i] = b.add[i];
    a.g.scale[i] = b.scale[i];
  }
  a.twx = dir < 0 ? p.pass.xf : p.pass.xi;
  a.twy = dir < 0 ? p.pass.pyf : p.pass.pyi;
  a.wx = p.pass.wx;
#define CRAVA_PLANE(NX, NY) \
  if (g.nxp == NX && g.nyp == NY) return launch_plane<NX, NY>(a, dir, g.nzp, b.n, s);
  CRAVA_PLANE(64, 64) CRAVA_PLANE(64, 128) CRAVA_PLANE(128, 64) CRAVA_PLANE(128, 128) CRAVA_PLANE(256, 64)
#undef CRAVA_PLANE
  return CRAVA_GPU_ERR_ARG;
}

}  // namespace crava
