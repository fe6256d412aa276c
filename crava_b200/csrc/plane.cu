// plane.cu -- host side of the fused x + y pass (plane.cuh).
#include "plane.cuh"

namespace crava {

namespace {

int sm_count(int *n) {
  int dev = 0;
  CRAVA_CUDA_TRY(cudaGetDevice(&dev));
  CRAVA_CUDA_TRY(cudaDeviceGetAttribute(n, cudaDevAttrMultiProcessorCount, dev));
  return CRAVA_GPU_OK;
}

template <int NX, int NY, int CS, bool WHOLE = false>
int launch_plane(PlaneArgs a, int dir, int nplanes, int ngrids, cudaStream_t s) {
  using C = PlaneCfg<NX, NY, CS>;
  const void *fn = dir < 0 ? (const void *)k_plane_fwd<NX, NY, CS, WHOLE> : (const void *)k_plane_inv<NX, NY, CS, WHOLE>;
  const size_t smem = WHOLE ? C::smem_whole(dir) : C::smem(dir);
  int rc = func_smem(fn, smem);
  if (rc) return rc;
  a.ahead = 0;
  if (CS > 1 && (rc = sm_count(&a.ahead))) return rc;  // one CTA per SM
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nplanes * CS), (unsigned)ngrids);
  cfg.blockDim = dim3(C::NTH);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  if (dir < 0) CRAVA_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_plane_fwd<NX, NY, CS, WHOLE>, a));
  else CRAVA_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_plane_inv<NX, NY, CS, WHOLE>, a));
  note_launch();
  return CRAVA_GPU_OK;
}

template <int N, int CS>
int launch_parts(ColPassArgs a, int ngrids, int dir, cudaStream_t s) {
  const size_t smem = sizeof(float2) * (size_t)N * kColLines;
  const void *fn = dir < 0 ? (const void *)k_col_parts<N, -1, CS> : (const void *)k_col_parts<N, 1, CS>;
  int sms = 0, rc = func_smem(fn, smem);
  if (rc || (rc = sm_count(&sms))) return rc;
  a.ahead = (uint32_t)(7 * sms / 4);  // of 3 resident per SM; see fetch_l2
  constexpr int TXC = kColLines / CS;
  const dim3 grd((unsigned)((a.nlines + TXC - 1) / TXC), (unsigned)ngrids);
  if (dir < 0) k_col_parts<N, -1, CS><<<grd, 256, smem, s>>>(a);
  else k_col_parts<N, 1, CS><<<grd, 256, smem, s>>>(a);
  CRAVA_LAUNCH_CHECK();
  return CRAVA_GPU_OK;
}

}  // namespace

// CTAs per plane; 0: the plane has the separate passes alone.  One where a plane
// fits a CTA with others on the SM, two at 256x256.
int plane_parts(const Geom &g) {
  const bool px = g.nxp == 64 || g.nxp == 128, py = g.nyp == 64 || g.nyp == 128;
  if ((px && py) || (g.nxp == 256 && g.nyp == 64)) return 1;
  return g.nxp == 256 && g.nyp == 256 ? 2 : 0;
}

bool plane_xy_supported(const Geom &g) { return plane_parts(g) > 0; }

int plane_batch(const FftPlans &p, const GridBatch &b, int dir, bool whole, cudaStream_t s) {
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
  a.wy = p.pass.wy;
#define CRAVA_PLANE(NX, NY, CS) \
  if (g.nxp == NX && g.nyp == NY) return launch_plane<NX, NY, CS>(a, dir, g.nzp, b.n, s);
  CRAVA_PLANE(64, 64, 1) CRAVA_PLANE(64, 128, 1)
  CRAVA_PLANE(128, 64, 1) CRAVA_PLANE(128, 128, 1)
  CRAVA_PLANE(256, 64, 1)
#undef CRAVA_PLANE
  if (g.nxp == 256 && g.nyp == 256)
    return whole ? launch_plane<256, 256, 2, true>(a, dir, g.nzp, b.n, s) : launch_plane<256, 256, 2>(a, dir, g.nzp, b.n, s);
  return CRAVA_GPU_ERR_ARG;
}

int z_parts_launch(const ColPassArgs &a, int n, int ngrids, int dir, cudaStream_t s) {
  switch (n) {  // z_parts_length
    case 64: return launch_parts<64, 2>(a, ngrids, dir, s);
    case 128: return launch_parts<128, 2>(a, ngrids, dir, s);
    case 256: return launch_parts<256, 2>(a, ngrids, dir, s);
    case 512: return launch_parts<512, 2>(a, ngrids, dir, s);
    default: return CRAVA_GPU_ERR_ARG;
  }
}

}  // namespace crava
