// Launcher of the two-role point kernels (full stages of separable Cartesian
// and curvilinear blocks), compiled once per precision.
#include "wql3d_point.cuh"
#include "wql3d_stage.cuh"

namespace wql3d {

template <typename T, int MESH, int RESP, bool PML, bool UP>
static void launch_point(Blk<T> &b, const StageCtx &c, const StageArgs &a) {
  // Elastic blocks and FP32 take the flattened points with 6 resident CTAs
  // (the roles' taps are short enough for 80 registers): FP64 ms per step
  // 0.56 flattened / 0.68 by the warp map on 83 x 121 x 67 curvilinear points,
  // 0.69 / 0.71 on Cartesian 101^3 (8 CTAs flattened: 0.61 and 0.76).  FP32 with at
  // most 4 mechanisms has room for 8 CTAs: 0.546 against 0.603 on Cartesian
  // 101^3, 1.21 against 1.24 on Q4 with PML of 93 x 118 x 75 (fQ8: 7.06 against
  // 6.29 on 96 x 160 x 128 twice, so 6 there).  Memory variables in FP64 want
  // the registers of 4 CTAs and no boundary columns among a warp's central
  // ones: 22.8 by the map / 23.4 flattened on the two-block Q8 hill of 201^3
  // points (27.7 with 6 CTAs), 1.57 / 1.77 on Q4 with PML of 93 x 118 x 75.
  constexpr bool FLAT = sizeof(T) == 4 || RESP == RESP_EL;
  const WarpMap m = warp_map(b);
  const long long n = FLAT ? ((long long)b.nx * b.ny * b.nz + 127) / 128 : (map_warps(b, m) + 3) / 4;
  constexpr int MINB = !FLAT ? 4 : sizeof(T) == 4 && (RESP == RESP_EL || RESP == RESP_Q4) ? 8 : 6;
  k_point<T, MESH, RESP, PML, FLAT, MINB, UP><<<(unsigned)(2 * n), 128, 0, c.stream>>>(b, a, m);
  ++*c.launches;
}

template <typename T, int MESH, bool PML, bool UP = false>
static void launch_resp(Blk<T> &b, const StageCtx &c, const StageArgs &a) {
  switch (c.response) {
    case RESP_EL: launch_point<T, MESH, RESP_EL, PML, UP>(b, c, a); break;
    case RESP_Q4: launch_point<T, MESH, RESP_Q4, PML, UP>(b, c, a); break;
    case RESP_Q8: launch_point<T, MESH, RESP_Q8, PML, UP>(b, c, a); break;
    default: launch_point<T, MESH, RESP_FQ8, PML, UP>(b, c, a); break;
  }
}

template <typename T>
void launch_point_stage(Blk<T> &b, int mesh, const StageCtx &c, const StageArgs &a) {
  StageArgs la = a;
  la.pf = sizeof(T) == 4 ? 1 : 0;   // L2 prefetch of the memory variables (FP32 only: see k_curv_fused)
  bool pml = false;
  for (int f = 0; f < 6; ++f) pml = pml || b.pml_on[f];
  if (b.fd != 0) {
    if (mesh == MESH_CART) {
      launch_resp<T, MESH_CART, false, true>(b, c, la);
      return;
    }
    if (b.foff[6] > 0) {
      k_curv_face_sat<T><<<(b.foff[6] + 127) / 128, 128, 0, c.stream>>>(b, a.cur);
      ++*c.launches;
    }
    launch_resp<T, MESH_CURV, false, true>(b, c, la);
    return;
  }
  if (mesh == MESH_CART) {
    if (pml) launch_resp<T, MESH_CART, true>(b, c, la);
    else launch_resp<T, MESH_CART, false>(b, c, la);
  } else {
    if (b.foff[6] > 0) {
      k_curv_face_sat<T><<<(b.foff[6] + 127) / 128, 128, 0, c.stream>>>(b, a.cur);
      ++*c.launches;
    }
    if (pml) {
      launch_resp<T, MESH_CURV, true>(b, c, la);
      SlabCtas m;
      m.first[0] = 0;
      for (int f = 0; f < 6; ++f)
        m.first[f + 1] = m.first[f] + (b.pml_on[f] ? (int)((b.pvol[f] + 127) / 128) : 0);
      k_pml_velocity<T><<<m.first[6], 128, 0, c.stream>>>(b, a, m);
      ++*c.launches;
    } else launch_resp<T, MESH_CURV, false>(b, c, la);
  }
}

// The point kernels keep one PML slab per axis: blocks whose two slabs on an
// axis overlap (2 npml > n) take the generic passes.  Cartesian blocks need a
// separable metric.  FP32 curvilinear blocks with memory variables stay with
// k_curv_fused: 6.27 against 6.55 ms per step on the hill of 145^3 points
// (both roles' code beside the 96 memory-variable streams outgrows the
// instruction cache there).
template <typename T>
bool point_stage_ok(const Blk<T> &b, int mesh) {
  const int nax[3] = {b.nx, b.ny, b.nz};
  for (int ax = 0; ax < 3; ++ax)
    if (b.pml_on[2 * ax] && b.pml_on[2 * ax + 1] && 2 * b.npml > nax[ax]) return false;
  if (b.fd != 0) {
    for (int f = 0; f < 6; ++f)
      if (b.pml_on[f]) return false;   // upwind blocks with PML: the generic kernel
  }
  if (mesh == MESH_CART) return tuning().point && b.sep;
  return tuning().curv_fused && tuning().lean && !(sizeof(T) == 4 && b.nmech > 0 && b.fd == 0);
}

template <typename T>
void launch_fluxes(const Blk<T> &b, const StageCtx &c, int cur, int z0, int z1) {
  const long long n = (long long)b.nx * b.ny * (z1 - z0 + 1);
  k_fluxes<T><<<(unsigned)((n + 127) / 128), 128, 0, c.stream>>>(b, cur, z0, z1);
  ++*c.launches;
}

template void launch_fluxes<WQL3D_REAL>(const Blk<WQL3D_REAL> &, const StageCtx &, int, int, int);
template void launch_point_stage<WQL3D_REAL>(Blk<WQL3D_REAL> &, int, const StageCtx &, const StageArgs &);
template bool point_stage_ok<WQL3D_REAL>(const Blk<WQL3D_REAL> &, int);
int WQL3D_CAT(upload_tables_point_, WQL3D_TAG)(const ConstTables &t) { return upload_tables_here(t); }

}  // namespace wql3d
