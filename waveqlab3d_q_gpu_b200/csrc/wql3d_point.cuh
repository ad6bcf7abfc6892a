// Two-role point kernels of the full RK stage.
//
// A stage of one block is a gather: every point reads its stencil
// neighbourhood from the current field buffer and writes its own nine fields
// to the other buffer, its rates, memory variables and PML fields.  The work
// of a point splits in two halves that share nothing but inputs:
//   role V: velocity rates from the stress fluxes, fields and rates 0-2;
//   role S: stress rates from the velocity gradients, fields and rates 3-8,
//           memory variables, sources.
// Either half takes nine derivatives of three fields per axis.  One CTA runs
// one role over a tile of points, the two roles of a tile being neighbours in
// the launch, so that what both read comes from HBM once.
//
// What bounds the kernel is the latency of the gathers: a warp's taps are
// independent of one another, so they are issued together (one straight-line
// batch per point where all three rows are central, one batch per axis at
// the boundaries) with the registers to hold them, instead of axis by axis
// behind branches.
#pragma once

#include "wql3d_device.cuh"

namespace wql3d {

constexpr int ROLE_V = 0, ROLE_S = 1;
constexpr int EDGE = 6;   // closure rows at either end of an axis

template <int ROLE>
struct RoleComps {
  static constexpr int C0 = ROLE == ROLE_V ? 0 : 3;
  static constexpr int N = ROLE == ROLE_V ? 3 : 6;
};

template <int AX, typename T>
__device__ __forceinline__ int axis_len(const Blk<T> &b) {
  return AX == 0 ? b.nx : AX == 1 ? b.ny : b.nz;
}
template <int AX, typename T>
__device__ __forceinline__ T axis_metric(const Blk<T> &b, int i) {
  return AX == 0 ? ld(b.mq + i) : AX == 1 ? ld(b.mr + i) : ld(b.ms + i);
}

// stress components of tensor row r
template <int R>
struct Sym {
  static constexpr int c0 = R == 0 ? 3 : R == 1 ? 6 : 7;
  static constexpr int c1 = R == 0 ? 6 : R == 1 ? 4 : 8;
  static constexpr int c2 = R == 0 ? 7 : R == 1 ? 8 : 5;
};

// an element of a component array at a 32-bit element offset
template <typename T>
__device__ __forceinline__ T at(const T *__restrict__ base, unsigned o) {
  return __ldg(base + o);
}

// the nine arrays a role differentiates: component c along axis a.  Role S:
// the velocities; role V: the stresses of tensor row a (Cartesian) or the
// contravariant fluxes J sum_r X_r,a sigma_rc (curvilinear)
template <typename T, int MESH, int ROLE, int AX, int C>
__device__ __forceinline__ const T *tap_array(const T *__restrict__ F, long long V) {
  if constexpr (ROLE == ROLE_S) return F + C * V;
  else if constexpr (MESH == MESH_CURV) return F + (3 * AX + C) * V;
  else return F + (C == 0 ? Sym<AX>::c0 : C == 1 ? Sym<AX>::c1 : Sym<AX>::c2) * V;
}

template <typename T>
__device__ __forceinline__ T central(const T t[6]) {
  const T c1 = (T)0.75, c2 = (T)-0.15, c3 = (T)(1.0 / 60.0);
  return c3 * (t[5] - t[0]) + (c2 * (t[4] - t[1]) + c1 * (t[3] - t[2]));
}

// six central taps of one array
template <typename T>
__device__ __forceinline__ void load6(const T *__restrict__ f, unsigned o, int st, T t[6]) {
  t[0] = at(f, o - (unsigned)(3 * st));
  t[1] = at(f, o - (unsigned)(2 * st));
  t[2] = at(f, o - (unsigned)st);
  t[3] = at(f, o + (unsigned)st);
  t[4] = at(f, o + (unsigned)(2 * st));
  t[5] = at(f, o + (unsigned)(3 * st));
}

template <typename T, int MESH, int ROLE, int AX>
__device__ __forceinline__ void axis_central(const T *__restrict__ F, long long V, unsigned o, int st, T d[3]) {
  T t0[6], t1[6], t2[6];
  load6(tap_array<T, MESH, ROLE, AX, 0>(F, V), o, st, t0);
  load6(tap_array<T, MESH, ROLE, AX, 1>(F, V), o, st, t1);
  load6(tap_array<T, MESH, ROLE, AX, 2>(F, V), o, st, t2);
  d[0] = central(t0);
  d[1] = central(t1);
  d[2] = central(t2);
}

// closure rows (i <= 6 or i >= n - 5) of one axis, eight tap slots each
template <typename T, int MESH, int ROLE, int AX>
__device__ __forceinline__ void axis_closure(const Blk<T> &b, int i, const T *__restrict__ F, long long V, unsigned o,
                                             int st, T d[3]) {
  const int n = axis_len<AX>(b);
  const bool left = i <= 6;
  const int row = left ? i - 1 : n - i;
  const T *__restrict__ f0 = tap_array<T, MESH, ROLE, AX, 0>(F, V), *__restrict__ f1 = tap_array<T, MESH, ROLE, AX, 1>(F, V),
                       *__restrict__ f2 = tap_array<T, MESH, ROLE, AX, 2>(F, V);
  const double *rc = b.rowc + (left ? row : 6 + row) * 8;
  const int *ro = b.rowo + (left ? row : 6 + row) * 8;
  T c[8], t0[8], t1[8], t2[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    // y and z rows are the same for a whole warp of a central tile: constant
    // memory; x rows differ by lane: the global table
    int off;
    if constexpr (AX == 0) {
      c[k] = (T)__ldg(rc + k);
      off = __ldg(ro + k);
    } else {
      c[k] = (T)c_sbp_c[b.lit][row][k];
      off = c[k] != (T)0 ? c_sbp_idx[row][k] - (row + 1) : 0;
      if (!left) { c[k] = -c[k]; off = -off; }
    }
    const unsigned q = o + (unsigned)(off * st);
    t0[k] = at(f0, q);
    t1[k] = at(f1, q);
    t2[k] = at(f2, q);
  }
  d[0] = d[1] = d[2] = (T)0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (c[k] != (T)0) {
      d[0] = d[0] + c[k] * t0[k];
      d[1] = d[1] + c[k] * t1[k];
      d[2] = d[2] + c[k] * t2[k];
    }
  }
}

template <typename T, int MESH, int ROLE, int AX>
__device__ __forceinline__ void axis_any(const Blk<T> &b, int i, const T *__restrict__ F, long long V, unsigned o,
                                         int st, T d[3]) {
  if (central_row(b, AX, i, axis_len<AX>(b))) axis_central<T, MESH, ROLE, AX>(F, V, o, st, d);
  else axis_closure<T, MESH, ROLE, AX>(b, i, F, V, o, st, d);
}

// upwind pairs: the forward rows on the velocities, the backward rows on the
// stresses (or fluxes), from the block's row table (Blk::urowc), four taps'
// loads at a time (Q8, upwind-4, 61^3 points in FP64: 0.63 ms per step, 1.48
// through the generic kernel's 255 registers and 8 warps per SM)
template <typename T, int MESH, int ROLE, int AX>
__device__ __forceinline__ void axis_upwind(const Blk<T> &b, int i, const T *__restrict__ F, long long V, unsigned o,
                                            int st, T d[3]) {
  const int row = up_row(b, ROLE == ROLE_S, i, axis_len<AX>(b));
  const int cnt = __ldg(b.urown + row);
  const double *__restrict__ rc = b.urowc + row * 16;
  const int *__restrict__ ro = b.urowo + row * 16;
  const T *__restrict__ f0 = tap_array<T, MESH, ROLE, AX, 0>(F, V), *__restrict__ f1 = tap_array<T, MESH, ROLE, AX, 1>(F, V),
                       *__restrict__ f2 = tap_array<T, MESH, ROLE, AX, 2>(F, V);
  d[0] = d[1] = d[2] = (T)0;
#pragma unroll 4
  for (int k = 0; k < cnt; ++k) {
    const T c = (T)__ldg(rc + k);
    const unsigned q = o + (unsigned)(__ldg(ro + k) * st);
    d[0] = d[0] + c * at(f0, q);
    d[1] = d[1] + c * at(f1, q);
    d[2] = d[2] + c * at(f2, q);
  }
}

// the nine derivatives of a role at one point, g[a][c] with the axis metric
// (Cartesian) and 1/h applied.  inner: every lane of the warp has central
// rows on all three axes.  UP: the block's upwind pair
template <typename T, int MESH, int ROLE, bool UP>
__device__ __forceinline__ void derivatives(const Blk<T> &b, const T *__restrict__ F, bool inner, int x, int y, int z,
                                            unsigned o, T g[3][3]) {
  const long long V = b.vol;
  const int sy = (int)b.sy, sz = (int)b.sz;
  if constexpr (UP) {
    axis_upwind<T, MESH, ROLE, 0>(b, x, F, V, o, 1, g[0]);
    axis_upwind<T, MESH, ROLE, 1>(b, y, F, V, o, sy, g[1]);
    axis_upwind<T, MESH, ROLE, 2>(b, z, F, V, o, sz, g[2]);
  } else if (inner) {
    axis_central<T, MESH, ROLE, 0>(F, V, o, 1, g[0]);
    axis_central<T, MESH, ROLE, 1>(F, V, o, sy, g[1]);
    axis_central<T, MESH, ROLE, 2>(F, V, o, sz, g[2]);
  } else {
    axis_any<T, MESH, ROLE, 0>(b, x, F, V, o, 1, g[0]);
    axis_any<T, MESH, ROLE, 1>(b, y, F, V, o, sy, g[1]);
    axis_any<T, MESH, ROLE, 2>(b, z, F, V, o, sz, g[2]);
  }
  T hx = b.ihq, hy = b.ihr, hz = b.ihs;
  if constexpr (MESH == MESH_CART) { hx *= ld(b.mq + x); hy *= ld(b.mr + y); hz *= ld(b.ms + z); }
#pragma unroll
  for (int c = 0; c < 3; ++c) { g[0][c] *= hx; g[1][c] *= hy; g[2][c] *= hz; }
}

// PML slab of a point on axis AX: its face, or -1 (the host sends blocks whose
// two slabs on an axis overlap to the generic update)
template <int AX, typename T>
__device__ __forceinline__ int axis_slab_face(const Blk<T> &b, int x, int y, int z) {
  if (slab_has<T, 2 * AX + 1>(b, x, y, z)) return 2 * AX + 1;
  if (slab_has<T, 2 * AX>(b, x, y, z)) return 2 * AX;
  return -1;
}
template <typename T>
__device__ __forceinline__ long long slab_at(const Blk<T> &b, int f, int x, int y, int z) {
  const int *B = b.pb[f];
  return (long long)(x - B[0]) +
         (long long)(B[1] - B[0] + 1) * ((long long)(y - B[2]) + (long long)(B[3] - B[2] + 1) * (long long)(z - B[4]));
}
template <int AX, typename T>
__device__ __forceinline__ T slab_damp(const Blk<T> &b, int f, int i) {
  const int n = axis_len<AX>(b);
  const T v = (f == 4) ? (T)(i - b.npml) : ((f & 1) ? (T)(i - (n - b.npml)) : (T)(i - (1 + b.npml)));
  return b.d0 * fabs(v / (T)b.npml);
}

// Physical-boundary term of the face of axis AX this point lies on (face f):
// rates d -= dsat, and dq, what the face's PML slab subtracts from DQ
// (impose_boundary_condition, src/RHS_Interior.f90:1584-1768).  Curvilinear:
// from the k_curv_face_sat buffers.  Cartesian: the face basis is the axes,
// so the characteristic terms of BC_* (src/BoundaryConditions.f90:50-924) are
// scalar per component: impedance Zp along the axis, Zs across it.
template <int AX, typename T, int MESH, int ROLE>
__device__ __forceinline__ void face_term(const Blk<T> &b, const T *__restrict__ F, int f, int x, int y, int z,
                                          long long p, T dsat[RoleComps<ROLE>::N], T dq[RoleComps<ROLE>::N]) {
  constexpr int C0 = RoleComps<ROLE>::C0, NC = RoleComps<ROLE>::N;
  if constexpr (MESH == MESH_CURV) {
    const int fn = b.foff[f + 1] - b.foff[f];
    const int k = AX == 0 ? (y - 1) + b.ny * (z - 1) : AX == 1 ? (x - 1) + b.nx * (z - 1) : (x - 1) + b.nx * (y - 1);
    const T *o = b.fsat[f] + k;
#pragma unroll
    for (int c = 0; c < NC; ++c) dsat[c] = o[(C0 + c) * fn];
    const T *q = b.fdq[f];
#pragma unroll
    for (int c = 0; c < NC; ++c) dq[c] = q ? q[(C0 + c) * fn + k] : (T)0;
  } else {
    using C = Sym<AX>;
    const long long V = b.vol;
    const int type = b.bc[f];
    const T r = type == 1 ? (T)0 : type == 2 ? (T)1 : (T)-1;
    const T sg = (f & 1) ? (T)1 : (T)-1;
    const T lam = b.M[p], mu = b.M[V + p], rho = b.M[2 * V + p];
    const T l2m = (T)2 * mu + lam;
    const T Zp = rho * sqrt(l2m / rho), Zs = rho * sqrt(mu / rho);
    const T v[3] = {F[p], F[V + p], F[2 * V + p]};
    const T t[3] = {F[C::c0 * V + p], F[C::c1 * V + p], F[C::c2 * V + p]};
    const T pen = b.tau0 / (AX == 0 ? b.hq : AX == 1 ? b.hr : b.hs);
    const T pn = pen * axis_metric<AX>(b, AX == 0 ? x : AX == 1 ? y : z);
    const T half = (T)0.5, one = (T)1;
    if constexpr (ROLE == ROLE_V) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        dq[c] = pn * (half * ((one - r) * (c == AX ? Zp : Zs) * v[c] + sg * ((one + r) * t[c])));
        dsat[c] = dq[c] / rho;
      }
    } else {
      T g[3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
        g[c] = sg * (pn * (half * ((one - r) * v[c] + sg * ((one + r) / (c == AX ? Zp : Zs) * t[c]))));
#pragma unroll
      for (int c = 0; c < 6; ++c) { dq[c] = 0; dsat[c] = 0; }
#pragma unroll
      for (int c = 0; c < 3; ++c) dsat[c] = (c == AX ? l2m : lam) * g[AX];
      dq[C::c0 - 3] = g[0]; dq[C::c1 - 3] = g[1]; dq[C::c2 - 3] = g[2];
      if (AX != 0) dsat[C::c0 - 3] = mu * g[0];
      if (AX != 1) dsat[C::c1 - 3] = mu * g[1];
      if (AX != 2) dsat[C::c2 - 3] = mu * g[2];
    }
  }
}

// PML slab and physical boundary of axis AX for this role's components: G
// holds the axis' three source terms (fluxes over J, or velocity gradients)
template <int AX, typename T, int MESH, int ROLE, bool PML>
__device__ __forceinline__ void axis_finish(const Blk<T> &b, const StageArgs &a, const T *__restrict__ F, int x, int y,
                                            int z, long long p, const T G[3], T irho, T l2m, T lam, T mu,
                                            T df[RoleComps<ROLE>::N], T e[6]) {
  constexpr int C0 = RoleComps<ROLE>::C0, NC = RoleComps<ROLE>::N;
  using C = Sym<AX>;
  const int i = AX == 0 ? x : AX == 1 ? y : z;
  const int n = axis_len<AX>(b);
  T dq[NC];
  const int f = i == 1 ? 2 * AX : i == n ? 2 * AX + 1 : -1;
  const bool sat = f >= 0 && b.bc[f] > 0;
  if (sat) {
    T ds[NC];
    face_term<AX, T, MESH, ROLE>(b, F, f, x, y, z, p, ds, dq);
#pragma unroll
    for (int c = 0; c < NC; ++c) df[c] = df[c] - ds[c];
  }
  if constexpr (PML) {
    const int s = axis_slab_face<AX>(b, x, y, z);
    if (s >= 0) {
      const long long PV = b.pvol[s];
      const long long q = slab_at(b, s, x, y, z) + C0 * PV;
      T *__restrict__ Qp = b.Q[s] + q;
      T *__restrict__ DQp = b.DQ[s] + q;
      const T d = slab_damp<AX>(b, s, i);
      const T A = (T)a.A, Bdt = (T)a.Bdt;
      if constexpr (ROLE == ROLE_V && MESH == MESH_CURV) {
        // the auxiliary velocities themselves: k_pml_velocity
#pragma unroll
        for (int c = 0; c < 3; ++c) df[c] = df[c] - d * Qp[c * PV] * irho;
      } else {
        T Q[NC], DQ[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          Q[c] = Qp[c * PV];
          DQ[c] = A * DQp[c * PV];
        }
        if constexpr (ROLE == ROLE_V) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            df[c] = df[c] - d * Q[c] * irho;
            DQ[c] = DQ[c] + G[c] - (d + (T)1) * Q[c];
          }
        } else {
          df[0] = df[0] - d * (l2m * Q[0] + lam * Q[1] + lam * Q[2]);
          df[1] = df[1] - d * (lam * Q[0] + l2m * Q[1] + lam * Q[2]);
          df[2] = df[2] - d * (lam * Q[0] + lam * Q[1] + l2m * Q[2]);
#pragma unroll
          for (int c = 3; c < 6; ++c) df[c] = df[c] - mu * d * Q[c];
          // strain rates of the memory variables (src/RHS_Interior.f90:2351-2451)
          e[C::c0 - 3] = e[C::c0 - 3] - d * Q[C::c0 - 3];
          e[C::c1 - 3] = e[C::c1 - 3] - d * Q[C::c1 - 3];
          e[C::c2 - 3] = e[C::c2 - 3] - d * Q[C::c2 - 3];
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            const T src = c == C::c0 - 3 ? G[0] : c == C::c1 - 3 ? G[1] : c == C::c2 - 3 ? G[2] : (T)0;
            DQ[c] = DQ[c] + src - (d + (T)1) * Q[c];
          }
        }
        if (sat && s == f) {
#pragma unroll
          for (int c = 0; c < NC; ++c) DQ[c] = DQ[c] - dq[c];
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          DQp[c * PV] = DQ[c];
          Qp[c * PV] = Q[c] + Bdt * DQ[c];
        }
      }
    }
  }
}

// rates to memory and F <- F + B dt DF (Kahan-compensated in FP32); f holds
// the old fields on entry, the new ones on return
template <typename T, int ROLE>
__device__ __forceinline__ void role_store(const Blk<T> &b, const StageArgs &a, unsigned o,
                                           const T df[RoleComps<ROLE>::N], T f[RoleComps<ROLE>::N]) {
  constexpr int C0 = RoleComps<ROLE>::C0, NC = RoleComps<ROLE>::N;
  const long long V = b.vol;
  T *__restrict__ Fn = a.cur ? b.F0 : b.F1;
  const T Bdt = (T)a.Bdt;
  if constexpr (sizeof(T) == 4) {
    T fc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) fc[c] = (b.FC + (C0 + c) * V)[o];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const T yv = Bdt * df[c] - fc[c];
      const T tv = f[c] + yv;
      (b.FC + (C0 + c) * V)[o] = (tv - f[c]) - yv;
      f[c] = tv;
    }
  } else {
#pragma unroll
    for (int c = 0; c < NC; ++c) f[c] = f[c] + Bdt * df[c];
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    (Fn + (C0 + c) * V)[o] = f[c];
    (b.DF + (C0 + c) * V)[o] = df[c];
  }
}

template <typename T, int ROLE>
__device__ __forceinline__ void iface_term(const Blk<T> &b, int x, int y, int z, T df[RoleComps<ROLE>::N]) {
  // interface SAT, src/RHS_Interior.f90:1813-1837: DF(face) -= tau0/hx * (F_x | G_x)
  constexpr int C0 = RoleComps<ROLE>::C0, NC = RoleComps<ROLE>::N;
  const int side = x == 1 ? 0 : (x == b.nx ? 1 : -1);
  if (side >= 0 && b.isat[side]) {
    const T pen = b.tau0 / b.hq;
    const long long fn = (long long)b.ny * b.nz;
    const T *o = b.isat[side] + C0 * fn + (long long)(y - 1) + (long long)b.ny * (z - 1);
#pragma unroll
    for (int c = 0; c < NC; ++c) df[c] = df[c] - pen * o[c * fn];
  }
}

// Memory variables of stress component c (0-5): the stress rate df loses the
// sum of the old values.  The loads of a component go out together; the
// barrier keeps the next component's from being hoisted above these stores,
// so that one component's pairs are live (all six at once spilled, four
// mechanisms at a time left too few loads in flight: 14.7 against 11.8 ms per
// step on the fQ8 blocks of 112 x 176 x 112 points in FP64).
template <typename T, int RESP>
__device__ __forceinline__ void memory_component(const Blk<T> &b, const StageArgs &a, int c, int active, unsigned o,
                                                 T ge, T gt, T l2t, T m2t, T &df) {
  constexpr int N = RESP == RESP_Q4 ? 4 : 8;
  const long long V = b.vol;
  const T A = (T)a.A, Bdt = (T)a.Bdt;
  T *__restrict__ ep = b.eta + (long long)(c * N) * V;
  T *__restrict__ dp = b.deta + (long long)(c * N) * V;
  T ev[N], dv[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    ev[i] = (ep + i * V)[o];
    dv[i] = (dp + i * V)[o];
  }
  T sum = ev[0];
#pragma unroll
  for (int i = 1; i < N; ++i) sum = sum + ev[i];
  df = df - sum;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T d = A * dv[i];
    if constexpr (RESP == RESP_FQ8) {
      if (!b.coarse || (i + 1) == active) {
        if (c < 3) d = d + ((b.ss[i] * ge + (b.ps[i] * l2t - b.ss[i] * m2t)) - ev[i]) * b.itau[i];
        else d = d + (b.ss[i] * ge - ev[i]) * b.itau[i];
      }
    } else {
      if (c < 3) d = d + ((b.w[i] * ge + b.w[i] * gt) - ev[i]) * b.itau[i];
      else d = d + (b.w[i] * ge - ev[i]) * b.itau[i];
    }
    (dp + i * V)[o] = d;
    (ep + i * V)[o] = ev[i] + Bdt * d;
  }
  asm volatile("" ::: "memory");
}

// contravariant stress fluxes G[3 a + c] = J sum_r X_r,a sigma_rc of one
// point (f: stresses xx yy zz xy xz yz)
template <typename T>
__device__ __forceinline__ void store_fluxes(const Blk<T> &b, T *__restrict__ G, unsigned o, const T f[6]) {
  const long long V = b.vol;
  const T J = at(b.J, o);
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const T x0 = J * at(b.met + ax * V, o), x1 = J * at(b.met + (3 + ax) * V, o), x2 = J * at(b.met + (6 + ax) * V, o);
    (G + (3 * ax) * V)[o] = x0 * f[0] + x1 * f[3] + x2 * f[4];
    (G + (3 * ax + 1) * V)[o] = x0 * f[3] + x1 * f[1] + x2 * f[5];
    (G + (3 * ax + 2) * V)[o] = x0 * f[4] + x1 * f[5] + x2 * f[2];
  }
}

// one point of a full stage (flags F_ALL), velocity half
template <typename T, int MESH, bool PML, bool UP>
__device__ __forceinline__ void point_v(const Blk<T> &b, const StageArgs &a, bool inner, int x, int y, int z) {
  const long long V = b.vol;
  const unsigned o = (unsigned)pidx(b, x, y, z);
  const T *__restrict__ F = a.cur ? b.F1 : b.F0;
  if (sizeof(T) == 4) {
#pragma unroll
    for (int c = 0; c < 3; ++c) prefetch_l2(b.FC + c * V + o);
  }
  T df[3], f[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) df[c] = (b.DF + c * V)[o];
  const T rho = at(b.M + 2 * V, o);
  const T J = MESH == MESH_CURV ? at(b.J, o) : (T)1;
#pragma unroll
  for (int c = 0; c < 3; ++c) f[c] = at(F + c * V, o);
  T g[3][3];
  derivatives<T, MESH, ROLE_V, UP>(b, MESH == MESH_CURV ? b.G + (a.cur ? 9 * V : 0) : F, inner, x, y, z, o, g);
  if (MESH == MESH_CURV && a.rec) {
    T *E = reinterpret_cast<T *>(a.rec);
#pragma unroll
    for (int c = 0; c < 3; ++c) (E + (6 + c) * V)[o] = g[0][c] + g[1][c] + g[2][c];
  }
  const T irho = (T)1 / rho;
  const T a1 = MESH == MESH_CURV ? (T)1 / (rho * J) : irho;
#pragma unroll
  for (int c = 0; c < 3; ++c) df[c] = (T)a.A * df[c] + (g[0][c] + g[1][c] + g[2][c]) * a1;
  axis_finish<0, T, MESH, ROLE_V, PML>(b, a, F, x, y, z, o, g[0], irho, (T)0, (T)0, (T)0, df, nullptr);
  axis_finish<1, T, MESH, ROLE_V, PML>(b, a, F, x, y, z, o, g[1], irho, (T)0, (T)0, (T)0, df, nullptr);
  axis_finish<2, T, MESH, ROLE_V, PML>(b, a, F, x, y, z, o, g[2], irho, (T)0, (T)0, (T)0, df, nullptr);
  iface_term<T, ROLE_V>(b, x, y, z, df);
  role_store<T, ROLE_V>(b, a, o, df, f);
}

// one point of a full stage (flags F_ALL), stress half
template <typename T, int MESH, int RESP, bool PML, bool UP>
__device__ __forceinline__ void point_s(const Blk<T> &b, const StageArgs &a, bool inner, int x, int y, int z) {
  const long long V = b.vol;
  const unsigned o = (unsigned)pidx(b, x, y, z);
  const T *__restrict__ F = a.cur ? b.F1 : b.F0;
#pragma unroll
  for (int c = 3; c < 9; ++c) {
    prefetch_l2(F + c * V + o);
    if (sizeof(T) == 4) prefetch_l2(b.FC + c * V + o);
  }
  if (RESP != RESP_EL && a.pf) {
    constexpr int NM = RESP == RESP_Q4 ? 4 : 8;
#pragma unroll 8
    for (int c = 0; c < 6 * NM; ++c) {
      prefetch_l2(b.eta + (long long)c * V + o);
      prefetch_l2(b.deta + (long long)c * V + o);
    }
  }
  T df[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) df[c] = (b.DF + (3 + c) * V)[o];
  const T lam = at(b.M, o), mu = at(b.M + V, o);
  T g[3][3];
  derivatives<T, MESH, ROLE_S, UP>(b, F, inner, x, y, z, o, g);
  if constexpr (MESH == MESH_CURV) {
    T u[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const T x0 = at(b.met + (3 * r) * V, o), x1 = at(b.met + (3 * r + 1) * V, o), x2 = at(b.met + (3 * r + 2) * V, o);
#pragma unroll
      for (int c = 0; c < 3; ++c) u[r][c] = x0 * g[0][c] + x1 * g[1][c] + x2 * g[2][c];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) g[r][c] = u[r][c];
  }
  // g[r][c] = d v_c / d x_r
  T e[6] = {g[0][0], g[1][1], g[2][2], g[1][0] + g[0][1], g[2][0] + g[0][2], g[2][1] + g[1][2]};
  if (MESH == MESH_CURV && a.rec) {
    T *E = reinterpret_cast<T *>(a.rec);
#pragma unroll
    for (int c = 0; c < 6; ++c) (E + c * V)[o] = e[c];
  }
  const T l2m = lam + (T)2 * mu;
#pragma unroll
  for (int c = 0; c < 6; ++c) df[c] = (T)a.A * df[c];
  df[0] = df[0] + (l2m * e[0] + lam * (e[1] + e[2]));
  df[1] = df[1] + (l2m * e[1] + lam * (e[0] + e[2]));
  df[2] = df[2] + (l2m * e[2] + lam * (e[0] + e[1]));
  df[3] = df[3] + mu * e[3];
  df[4] = df[4] + mu * e[4];
  df[5] = df[5] + mu * e[5];
  axis_finish<0, T, MESH, ROLE_S, PML>(b, a, F, x, y, z, o, g[0], (T)0, l2m, lam, mu, df, e);
  axis_finish<1, T, MESH, ROLE_S, PML>(b, a, F, x, y, z, o, g[1], (T)0, l2m, lam, mu, df, e);
  axis_finish<2, T, MESH, ROLE_S, PML>(b, a, F, x, y, z, o, g[2], (T)0, l2m, lam, mu, df, e);
  if (b.nsrc > 0 && x >= b.sbox[0] && x <= b.sbox[1] && y >= b.sbox[2] && y <= b.sbox[3] && z >= b.sbox[4] &&
      z <= b.sbox[5]) {
    const double t0 = a.time ? a.time->t : 0.0;
    const double tst = a.stage <= 1 ? t0 : t0 + c_rkC[a.stage - 1] * a.dt;
    T d9[9] = {0, 0, 0, df[0], df[1], df[2], df[3], df[4], df[5]};
    add_sources<T, MESH>(b, tst, x, y, z, o, d9);
#pragma unroll
    for (int c = 0; c < 6; ++c) df[c] = d9[3 + c];
  }
  iface_term<T, ROLE_S>(b, x, y, z, df);
  if constexpr (RESP != RESP_EL) {
    const int active = 1 + ((x - 1) & 1) + 2 * ((y - 1) & 1) + 4 * ((z - 1) & 1);
    const T tr = e[0] + e[1] + e[2];
    T fn, ft, fs, l2, two_mu;
    mv_factors<T, RESP>(b, o, lam, mu, fn, ft, fs, l2, two_mu);
#pragma unroll
    for (int c = 0; c < 6; ++c)
      memory_component<T, RESP>(b, a, c, active, o, (c < 3 ? fn : fs) * e[c], ft * tr, l2 * tr, two_mu * tr, df[c]);
  }
  T f[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) f[c] = at(F + (3 + c) * V, o);
  role_store<T, ROLE_S>(b, a, o, df, f);
  if constexpr (MESH == MESH_CURV) store_fluxes<T>(b, b.G + (a.cur ? 0 : 9 * V), o, f);
}

// Work map of a block, in warps: rows are taken two at a time (a row pair).
// Each row has m whole warps of central columns (x = 7 .. 6 + 32 m); the
// other ec columns of a row, the two closures' and the remainder, go to the
// pair's last e warps (e = 1: both rows in one warp, ec <= 16).  Consecutive
// warps stay close in memory, which the many streams of a point need: with
// the boundary columns in CTAs of their own, far from their rows in time,
// every line they share with the rows was read twice.
struct WarpMap {
  int m, ec, e;
  int per;      // warps of a row pair
  int pairs;    // row pairs of a plane
};

template <typename T>
inline WarpMap warp_map(const Blk<T> &b) {
  WarpMap w;
  w.m = (b.nx - 2 * EDGE) / 32;
  w.ec = b.nx - 32 * w.m;
  if (w.ec > 32) { w.m += 1; w.ec = 2 * EDGE; }
  w.e = w.ec <= 16 ? 1 : 2;
  w.per = 2 * w.m + w.e;
  w.pairs = (b.ny + 1) / 2;
  return w;
}
template <typename T>
inline long long map_warps(const Blk<T> &b, const WarpMap &w) {
  return (long long)w.per * w.pairs * b.nz;
}

// point of a lane of warp `warp` of the map; false outside the block
template <typename T>
__device__ __forceinline__ bool warp_point(const Blk<T> &b, const WarpMap &w, int warp, int lane, int &x, int &y,
                                           int &z) {
  const int g = warp / w.per, k = warp - g * w.per;
  const int zi = g / w.pairs;
  z = zi + 1;
  y = 2 * (g - zi * w.pairs) + 1;
  if (k < 2 * w.m) {
    const int row = k >= w.m ? 1 : 0;
    y += row;
    x = EDGE + 1 + 32 * (k - row * w.m) + lane;
    return z <= b.nz && y <= b.ny && x <= b.nx - EDGE;
  }
  int c = lane;
  if (w.e == 1) {
    const int row = lane >= w.ec ? 1 : 0;
    c = lane - row * w.ec;
    y += row;
  } else {
    y += k - 2 * w.m;
  }
  x = c < EDGE ? c + 1 : b.nx - w.ec + 1 + c;
  return c < w.ec && z <= b.nz && y <= b.ny;
}

// point of 0-based index j of the flattened block (x fastest); false past its end
template <typename T>
__device__ __forceinline__ bool flat_index(const Blk<T> &b, int j, int &x, int &y, int &z) {
  if (j >= b.nx * b.ny * b.nz) return false;
  const int r = j / b.nx;
  x = j - r * b.nx + 1;
  z = r / b.ny;
  y = r - z * b.ny + 1;
  z = z + 1;
  return true;
}

// one role at one point, the warp's lanes agreeing on the straight-line taps
template <typename T, int MESH, int RESP, bool PML, bool UP = false>
__device__ __forceinline__ void run_role(const Blk<T> &b, const StageArgs &a, int role, int x, int y, int z) {
  const bool c = central_row(b, 0, x, b.nx) && central_row(b, 1, y, b.ny) && central_row(b, 2, z, b.nz);
  const bool inner = __all_sync(__activemask(), c);
  if (role == ROLE_S) point_s<T, MESH, RESP, PML, UP>(b, a, inner, x, y, z);
  else point_v<T, MESH, PML, UP>(b, a, inner, x, y, z);
}

// CTA pair (2 k, 2 k + 1): the two roles of 128 points.  FLAT: consecutive
// points of the flattened block (every lane busy; warps straddle row ends),
// else four warps of the work map m (no warp mixes boundary columns with
// central ones).
template <typename T, int MESH, int RESP, bool PML, bool FLAT, int MINB, bool UP>
__global__ void __launch_bounds__(128, MINB) k_point(const __grid_constant__ Blk<T> b,
                                                     const __grid_constant__ StageArgs a, WarpMap m) {
  int x, y, z;
  const int t = (blockIdx.x >> 1) * 128 + threadIdx.x;
  if (FLAT ? !flat_index(b, t, x, y, z) : !warp_point(b, m, t >> 5, t & 31, x, y, z)) return;
  run_role<T, MESH, RESP, PML, UP>(b, a, blockIdx.x & 1 ? ROLE_S : ROLE_V, x, y, z);
}

// The contravariant fluxes of the fields F on planes z0 .. z1 (ghost planes
// of open faces included), where no stage has left them: fields set by the
// caller, restored or updated in place
template <typename T>
__global__ void __launch_bounds__(128) k_fluxes(Blk<T> b, int cur, int z0, int z1) {
  const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long plane = (long long)b.nx * b.ny;
  if (j >= plane * (z1 - z0 + 1)) return;
  const int z = z0 + (int)(j / plane);
  const int r = (int)(j % plane), y = r / b.nx + 1, x = r % b.nx + 1;
  const unsigned o = (unsigned)pidx(b, x, y, z);
  const T *F = cur ? b.F1 : b.F0;
  T f[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) f[c] = (F + (3 + c) * b.vol)[o];
  store_fluxes<T>(b, b.G + (cur ? 9 * b.vol : 0), o, f);
}

// Auxiliary velocities (Q, DQ 0-2) of every PML slab of a curvilinear block,
// src/RHS_Interior.f90:1913-2265: the source on the slab of axis A is the
// flux divergence of metric row A alone, D_a(J X_A,a sigma_Ac) / J, which the
// summed fluxes of the velocity half do not hold, so it is gathered here, for
// slab points only.  Runs after the velocity half, which damps with the old Q.
// One thread per slab point, `first` the CTA offsets of the six faces.
struct SlabCtas {
  int first[7];
};
template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 4 : 8) k_pml_velocity(const __grid_constant__ Blk<T> b,
                                                                            const __grid_constant__ StageArgs a,
                                                                            SlabCtas m) {
  int f = 0;
#pragma unroll
  for (int g = 1; g < 6; ++g)
    if ((int)blockIdx.x >= m.first[g]) f = g;
  const long long k = (long long)(blockIdx.x - m.first[f]) * 128 + threadIdx.x;
  const long long PV = b.pvol[f];
  if (k >= PV) return;
  const int *B = b.pb[f];
  const int wx = B[1] - B[0] + 1, wy = B[3] - B[2] + 1;
  const int r = (int)(k / wx), x = B[0] + (int)(k - (long long)r * wx), z = B[4] + r / wy, y = B[2] + r % wy;
  const unsigned o = (unsigned)pidx(b, x, y, z);
  const long long V = b.vol;
  const T *__restrict__ F = a.cur ? b.F1 : b.F0;
  T *__restrict__ Qp = b.Q[f] + k;
  T *__restrict__ DQp = b.DQ[f] + k;
  const int AX = f >> 1;
  const T *__restrict__ s0 = F + (AX == 0 ? 3 : 5 + AX) * V;   // sigma_A0
  const T *__restrict__ s1 = F + (AX == 1 ? 4 : 6 + AX) * V;   // sigma_A1
  const T *__restrict__ s2 = F + (AX == 2 ? 5 : 7 + AX) * V;   // sigma_A2
  T Q[3], DQ[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    Q[c] = Qp[c * PV];
    DQ[c] = DQp[c * PV];
  }
  const int pos[3] = {x, y, z}, nn[3] = {b.nx, b.ny, b.nz}, st[3] = {1, (int)b.sy, (int)b.sz};
  const T ih[3] = {b.ihq, b.ihr, b.ihs};
  T S[3] = {0, 0, 0};
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const T *__restrict__ X = b.met + (long long)(3 * AX + ax) * V;
    const int i = pos[ax], n = nn[ax];
    T d[3] = {0, 0, 0};
    if (central_row(b, ax, i, n)) {
      T w[6], t0[6], t1[6], t2[6];
      load6(b.J, o, st[ax], w);
      load6(X, o, st[ax], t0);
#pragma unroll
      for (int q = 0; q < 6; ++q) w[q] *= t0[q];
      load6(s0, o, st[ax], t0);
      load6(s1, o, st[ax], t1);
      load6(s2, o, st[ax], t2);
#pragma unroll
      for (int q = 0; q < 6; ++q) { t0[q] *= w[q]; t1[q] *= w[q]; t2[q] *= w[q]; }
      d[0] = central(t0); d[1] = central(t1); d[2] = central(t2);
    } else {
      const int row = i <= 6 ? i - 1 : 6 + (n - i);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const T c = (T)__ldg(b.rowc + row * 8 + q);
        if (c != (T)0) {
          const unsigned p = o + (unsigned)(__ldg(b.rowo + row * 8 + q) * st[ax]);
          const T w = c * (at(b.J, p) * at(X, p));
          d[0] = d[0] + w * at(s0, p);
          d[1] = d[1] + w * at(s1, p);
          d[2] = d[2] + w * at(s2, p);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) S[c] = S[c] + ih[ax] * d[c];
  }
  const T iJ = (T)1 / at(b.J, o);
  const T d = AX == 0 ? slab_damp<0>(b, f, x) : AX == 1 ? slab_damp<1>(b, f, y) : slab_damp<2>(b, f, z);
  const bool face = (f & 1) ? pos[AX] == nn[AX] : pos[AX] == 1;
  const T *__restrict__ fq = b.fdq[f];
  const int fn = b.foff[f + 1] - b.foff[f];
  const int fk = AX == 0 ? (y - 1) + b.ny * (z - 1) : AX == 1 ? (x - 1) + b.nx * (z - 1) : (x - 1) + b.nx * (y - 1);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    T q = (T)a.A * DQ[c] + S[c] * iJ - (d + (T)1) * Q[c];
    if (face && fq) q = q - fq[c * fn + fk];
    DQp[c * PV] = q;
    Qp[c * PV] = Q[c] + (T)a.Bdt * q;
  }
}

}  // namespace wql3d
