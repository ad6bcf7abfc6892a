// Launcher of the two-role point kernels (full stages of separable Cartesian
// and curvilinear blocks), compiled once per precision.
#include "wql3d_point.cuh"
#include "wql3d_stage.cuh"

namespace wql3d {

template <typename T, int MESH, int RESP, bool PML, bool UP, bool FLAT, int MINB>
static void launch_as(Blk<T> &b, const StageCtx &c, const StageArgs &a) {
  const WarpMap m = warp_map(b);
  const long long n = FLAT ? ((long long)b.nx * b.ny * b.nz + 127) / 128 : (map_warps(b, m) + 3) / 4;
  k_point<T, MESH, RESP, PML, FLAT, MINB, UP><<<(unsigned)(2 * n), 128, 0, c.stream>>>(b, a, m);
  ++*c.launches;
}

template <typename T, int MESH, int RESP, bool PML, bool UP>
static void launch_point(Blk<T> &b, const StageCtx &c, const StageArgs &a) {
  if constexpr (RESP == RESP_EL && MESH == MESH_CART && !UP) {
    // Elastic Cartesian blocks: the flattened points while rows are short, the
    // warp map (its warps start on their rows' lines) from 125 points a row, 96
    // with PML.  FP64 with 5 and 6 resident CTAs, FP32 with 8; ms per step,
    // flattened / mapped:
    //              81^3         101^3        137^3        160^3        200 x 90 x 200  90 x 200 x 200
    //   FP64       0.39 / 0.47  0.69 / 0.73  1.72 / 1.53  2.50 / 2.34  2.46 / 1.96     2.27 / 2.48
    //   FP64, PML  0.77 / 0.77  1.48 / 1.39               4.99 / 3.49
    //   FP32       0.31 / 0.36  0.56 / 0.58  1.41 / 1.29  2.12 / 1.94  1.89 / 1.66     2.00 / 2.10
    //   FP32, PML  0.55 / 0.57  1.04 / 1.00               3.63 / 2.69
    // FP64 flattened with 6 CTAs spills 136 bytes (272 with PML; 5 CTAs: none, 32):
    // 0.70 at 101^3, 0.088 against 0.082 at 41^3.  A block that shares the GPU with
    // the domain's other one gains from the sixth: two of 121 x 101 x 111 points
    // 2.05 against 2.10, with PML two of 81 x 83 x 85 1.52 against 1.56.
    if (b.nx >= (PML ? 96 : 125)) launch_as<T, MESH, RESP, PML, UP, false, sizeof(T) == 4 ? 8 : 6>(b, c, a);
    else if (c.alone) launch_as<T, MESH, RESP, PML, UP, true, sizeof(T) == 4 ? 8 : 5>(b, c, a);
    else launch_as<T, MESH, RESP, PML, UP, true, sizeof(T) == 4 ? 8 : 6>(b, c, a);
  } else if constexpr (RESP == RESP_EL && MESH == MESH_CURV && PML) {
    // Elastic curvilinear blocks with PML: the same line at 96 points a row, FP64
    // with 5 resident CTAs (6 spill 32 to 40 bytes), FP32 with 8; ms per step,
    // k_curv_fused / flattened / mapped (FP64 flattened with 6 CTAs):
    //          61^3                       101^3                      160^3                      160 x 31 x 160
    //   FP64   0.47 / 0.45 / 0.50 (0.49)  1.69 / 1.69 / 1.68 (1.78)  5.62 / 5.39 / 4.41 (5.55)  1.28 / 1.34 / 1.24 (1.42)
    //   FP32   0.35 / 0.34 / 0.36         1.20 / 1.27 / 1.30         4.24 / 3.98 / 3.37         1.02 / 1.01 / 0.94
    constexpr int MINB = sizeof(T) == 4 ? 8 : 5;
    if (b.nx >= 96) launch_as<T, MESH, RESP, PML, UP, false, MINB>(b, c, a);
    else launch_as<T, MESH, RESP, PML, UP, true, MINB>(b, c, a);
  } else if constexpr (MESH == MESH_CART || UP || (sizeof(T) == 4 ? RESP == RESP_EL : RESP != RESP_FQ8 || !PML)) {
    // (the curvilinear blocks this leaves out run k_curv_fused: point_stage_ok)
    // The other elastic blocks and FP32 take the flattened points with 6 resident
    // CTAs (FP64 ms per step 0.56 flattened / 0.68 by the warp map on
    // 83 x 121 x 67 curvilinear points).  FP32 with at most 4 mechanisms runs
    // with 8 CTAs, which spills 8 to 104 bytes and still gains: 1.21 against 1.24
    // on Q4 with PML of 93 x 118 x 75 (fQ8: 7.06 against 6.29 on 96 x 160 x 128
    // twice, so 6 there).  Memory variables in FP64
    // want the registers of 4 CTAs and no boundary columns among a warp's central
    // ones: 22.8 by the map / 23.4 flattened on the two-block Q8 hill of 201^3
    // points (27.7 with 6 CTAs), 1.57 / 1.77 on Q4 with PML of 93 x 118 x 75.
    // fQ8 on a curvilinear block spills 236 bytes at 4 CTAs, none at 3: 2.79 ms
    // per step against 3.13 on 101^3 (k_curv_fused 2.95).
    constexpr bool FLAT = sizeof(T) == 4 || RESP == RESP_EL;
    constexpr int MINB = !FLAT ? (RESP == RESP_FQ8 && MESH == MESH_CURV && !UP ? 3 : 4)
                               : sizeof(T) == 4 && (RESP == RESP_EL || RESP == RESP_Q4) ? 8 : 6;
    launch_as<T, MESH, RESP, PML, UP, FLAT, MINB>(b, c, a);
  }
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

// The elastic Cartesian blocks that the tile kernel beside the shell is the
// faster one for (ms per step, tiles / point kernel).
//  * FP64 without PML, shortest axis 139 points or more: 137^3 1.55 / 1.53,
//    145 x 141 x 139 1.75 / 1.82, 160^3 2.29 / 2.34, 201^3 4.14 / 4.22; a short
//    axis makes the shell large: 200 x 200 x 90 1.97 / 1.86, 160 x 160 x 31 0.66 /
//    0.50.
//  * FP64 with PML, little of it and little shell: the point kernel's PML form
//    costs every point, the tiles' only the slabs.  Slabs of `layer` points on
//    `faces` faces, shell (its share of the points) and slab share beside it:
//      101^3          1 face of 5    .32  .05   0.94 / 1.04
//      101^3          2 faces of 10  .38  .19   1.14 / 1.22
//      101^3          3 faces of 10  .40  .27   1.24 / 1.25
//      145^3          2 faces of 5   .23  .07   2.36 / 2.69
//      145^3          3 faces of 10  .30  .19   2.84 / 2.80
//      160^3          5 faces of 8   .26  .23   3.61 / 3.49
//       81 x 79 x 83  1 face of 5    .38  .06   0.66 / 0.59
//      short rows, flattened, lose at any slab share:
//       70 x 160 x 160  3 faces of 10  .38  .25   1.90 / 2.19
//  * FP32 with PML: 145^3 1 face of 5 (.23, .03) 2.00 / 2.08, 2 faces of 10
//    (.27, .13) 2.33 / 2.16.
template <typename T>
static bool tiles_faster(const Blk<T> &b) {
  if (b.nmech > 0) return false;
  const int n[3] = {b.nx, b.ny, b.nz};
  double inner = 1.0, clear = 1.0;
  for (int ax = 0; ax < 3; ++ax) {
    inner *= (double)(b.hi[ax] - b.lo[ax] + 1) / n[ax];
    clear *= 1.0 - (double)b.npml * (b.pml_on[2 * ax] + b.pml_on[2 * ax + 1]) / n[ax];
  }
  const double shell = 1.0 - inner, slab = 1.0 - clear;
  if (slab == 0.0) return sizeof(T) == 8 && b.nx >= 139 && b.ny >= 139 && b.nz >= 139;
  if (sizeof(T) == 4) return shell < 0.24 && slab < 0.1;
  return shell < 0.38 && (b.nx < 96 || slab < 0.2);
}

// The curvilinear blocks that k_curv_fused is the faster kernel for (ms per
// step, fused / point kernels).
//  * FP32 with memory variables: 6.27 / 6.55 on the hill of 145^3 (likely both
//    roles' code, beside 96 memory-variable streams, in the instruction cache).
//    With an upwind pair the other path is the generic kernel: 3.61 / 1.17 on
//    97 x 89 x 83 points, Q8, upwind-4.
//  * FP64 fQ8 with PML: 1.84 / 1.94 on 81^3, 5.26 / 5.30 on 121^3, with the
//    registers of 3 CTAs (4 spill: 2.10, 5.73).
//  * Small blocks with PML, whose third launch (k_pml_velocity) shows.  FP64
//    elastic up to 2^16 points: 0.130 / 0.150 on 17^3, 0.140 / 0.147 on 33^3,
//    0.208 / 0.179 on 41^3.  FP64 Q4 and Q8 from 2^14 to 2^16: 0.161 / 0.147 and
//    0.171 / 0.161 on 25^3, 0.164 / 0.207 and 0.217 / 0.252 on 36^3, 0.278 /
//    0.253 and 0.370 / 0.333 on 41^3.  FP32 elastic up to 1.2 million points:
//    0.144 / 0.161 on 41^3, 1.20 / 1.27 on 101^3, 1.98 / 1.83 on 121^3.
//    Not where a second block's kernels fill the gaps: two FP64 elastic blocks
//    of 41 x 63 x 57 points 0.76 / 0.63, FP32 0.61 / 0.51.
template <typename T>
static bool fused_faster(const Blk<T> &b, int response, bool alone) {
  bool pml = false;
  for (int f = 0; f < 6; ++f) pml = pml || b.pml_on[f];
  const long long n = (long long)b.nx * b.ny * b.nz;
  if (sizeof(T) == 4) return b.nmech > 0 || (pml && alone && n < 1200000);
  if (!pml) return false;
  if (response == RESP_FQ8) return true;
  return alone && n < (1 << 16) && (b.nmech == 0 || n >= (1 << 14));
}

// The point kernels keep one PML slab per axis: blocks whose two slabs on an
// axis overlap (2 npml > n) take the generic passes.  Cartesian blocks need a
// separable metric.  alone: the domain's only block.
template <typename T>
bool point_stage_ok(const Blk<T> &b, int mesh, int response, bool alone) {
  const int nax[3] = {b.nx, b.ny, b.nz};
  for (int ax = 0; ax < 3; ++ax)
    if (b.pml_on[2 * ax] && b.pml_on[2 * ax + 1] && 2 * b.npml > nax[ax]) return false;
  if (b.fd != 0) {
    for (int f = 0; f < 6; ++f)
      if (b.pml_on[f]) return false;   // upwind blocks with PML: the generic kernel
  }
  if (mesh == MESH_CART) return tuning().point && b.sep && (b.fd != 0 || !tiles_faster(b));
  return tuning().curv_fused && tuning().lean && (b.fd != 0 || !fused_faster(b, response, alone));
}

template <typename T>
void launch_fluxes(const Blk<T> &b, const StageCtx &c, int cur, int z0, int z1) {
  const long long n = (long long)b.nx * b.ny * (z1 - z0 + 1);
  k_fluxes<T><<<(unsigned)((n + 127) / 128), 128, 0, c.stream>>>(b, cur, z0, z1);
  ++*c.launches;
}

template void launch_fluxes<WQL3D_REAL>(const Blk<WQL3D_REAL> &, const StageCtx &, int, int, int);
template void launch_point_stage<WQL3D_REAL>(Blk<WQL3D_REAL> &, int, const StageCtx &, const StageArgs &);
template bool point_stage_ok<WQL3D_REAL>(const Blk<WQL3D_REAL> &, int, int, bool);
int WQL3D_CAT(upload_tables_point_, WQL3D_TAG)(const ConstTables &t) { return upload_tables_here(t); }

}  // namespace wql3d
