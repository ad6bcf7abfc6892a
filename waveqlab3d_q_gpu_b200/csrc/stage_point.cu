// Launcher of the two-role point kernels (full stages of separable Cartesian
// and curvilinear blocks), compiled once per precision.
#include "wql3d_point.cuh"
#include "wql3d_stage.cuh"

namespace wql3d {

template <typename T, int MESH, int RESP, bool PML>
static void launch_point(Blk<T> &b, const StageCtx &c, const StageArgs &a) {
  // Elastic blocks and FP32 take the flattened points with 6 resident CTAs
  // (the roles' taps are short enough for 80 registers): FP64 ms per step
  // 0.69 flattened / 0.71 by the warp map on Cartesian 101^3.  Memory variables in FP64 want the
  // registers of 4 CTAs and no boundary columns among a warp's central ones:
  // 1.57 by the map / 1.77 flattened on Q4 with PML of 93 x 118 x 75 points.
  constexpr bool FLAT = sizeof(T) == 4 || RESP == RESP_EL;
  const WarpMap m = warp_map(b);
  const long long n = FLAT ? ((long long)b.nx * b.ny * b.nz + 127) / 128 : (map_warps(b, m) + 3) / 4;
  k_point<T, MESH, RESP, PML, FLAT, FLAT ? 6 : 4><<<(unsigned)(2 * n), 128, 0, c.stream>>>(b, a, m);
  ++*c.launches;
}

template <typename T, int MESH, bool PML>
static void launch_resp(Blk<T> &b, const StageCtx &c, const StageArgs &a) {
  switch (c.response) {
    case RESP_EL: launch_point<T, MESH, RESP_EL, PML>(b, c, a); break;
    case RESP_Q4: launch_point<T, MESH, RESP_Q4, PML>(b, c, a); break;
    case RESP_Q8: launch_point<T, MESH, RESP_Q8, PML>(b, c, a); break;
    default: launch_point<T, MESH, RESP_FQ8, PML>(b, c, a); break;
  }
}

template <typename T>
void launch_point_stage(Blk<T> &b, int mesh, const StageCtx &c, const StageArgs &a) {
  StageArgs la = a;
  la.pf = sizeof(T) == 4 ? 1 : 0;   // L2 prefetch of the memory variables (FP32 only: see k_curv_fused)
  bool pml = false;
  for (int f = 0; f < 6; ++f) pml = pml || b.pml_on[f];
  if (pml) launch_resp<T, MESH_CART, true>(b, c, la);
  else launch_resp<T, MESH_CART, false>(b, c, la);
}

// The point kernels keep one PML slab per axis: blocks whose two slabs on an
// axis overlap (2 npml > n) take the generic passes.  Cartesian blocks need a
// separable metric.
template <typename T>
bool point_stage_ok(const Blk<T> &b, int mesh) {
  const int nax[3] = {b.nx, b.ny, b.nz};
  for (int ax = 0; ax < 3; ++ax)
    if (b.pml_on[2 * ax] && b.pml_on[2 * ax + 1] && 2 * b.npml > nax[ax]) return false;
  return mesh == MESH_CART && tuning().point && b.sep;
}

template void launch_point_stage<WQL3D_REAL>(Blk<WQL3D_REAL> &, int, const StageCtx &, const StageArgs &);
template bool point_stage_ok<WQL3D_REAL>(const Blk<WQL3D_REAL> &, int);
int WQL3D_CAT(upload_tables_point_, WQL3D_TAG)(const ConstTables &t) { return upload_tables_here(t); }

}  // namespace wql3d
