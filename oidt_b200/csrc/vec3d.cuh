// vec3d.cuh -- 3D Yee E and H half-steps, vector form.
//
// One launch per half-step, in two roles over one x-plane per grid row:
//
// * vector role: the z-clean cells, k in [kz0, kz1) = [kb + P, ke - P)
//   rounded inward to multiples of 4, where no cell is in a z slab or on the
//   rim.  A thread owns a group of four (float64: two) consecutive cells along
//   z (the guide axis, contiguous in memory) of one (i, j) row.  Rows are padded to nzp (a
//   multiple of 4 cells) and every sub-buffer starts on a 256-byte boundary,
//   so each field, dt/eps grid, z kappa array and x/y-slab psi row moves in
//   16-byte accesses (float4, or double2 in float64).  The x-slab terms
//   are uniform over a block and the y-slab terms over a row, and so are the
//   component update ranges (only i = ib and j = jb leave a component out):
//   no per-cell test runs in this role.  A plane is a flat list of (row,
//   group) pairs, so no lane idles whatever nz is.
// * edge role: every other group (the z slabs, the rim and the row
//   padding: 9 % of the cells of a 256-cell guide with a 10-cell CPML), with
//   each component's update range tested per cell and the z-slab psi moved
//   per group in rows padded to whole groups.
//
// Per cell the arithmetic is the sequence of kernels.cuh's y3_e_compute /
// y3_h_compute (the reference's fdtd_funcs.py:43-266 in its launch order):
// curl update, soft source, then the CPML terms of the x, y and z slabs.  With
// EXACT arithmetic every operation is the reference's IEEE operation, so
// float64 runs equal the reference and the oracle bit for bit.
//
// With the 'TM' source (Hy) the reference subtracts J from Hy between the E
// curl and the E CPML kernels, so the x-slab term of Ez and the z-slab term of
// Ex read Hy - J (src_diffs).
#pragma once
#include "kernels.cuh"

namespace oidt {

constexpr int kVecThreads = 128;
// Six resident blocks per SM in FP32 (at most 80 registers a thread): the
// vector role's loads in flight come from occupancy, and the edge role's
// longer code would otherwise raise the whole kernel's register count
// (measured: with six blocks C2 73.9 us and a 384 x 384 x 256 grid 0.612 ms
// per step, against 83.6 and 0.694 with the compiler's own 96-107 registers).
// The E half-step runs seven blocks (72
// registers, a few spills to L1): C2 71.6 against 72.8 us per step; eight
// blocks (64 registers) spill more and lose (76.1).
// FP64 with two cells a thread: 97 x 114 x 187 fast 63.9 us per step with
// seven / six blocks, 64.9 with six / six, 66.7 with six / five; EXACT 107.3,
// 103.8, 101.7 (79.5 now, with the source terms in SRC instances only and the
// kappa tables' padding in the quotients' range).
template <typename T, bool EXACT> constexpr int kVecBlocksPerSM = sizeof(T) == 8 && EXACT ? 5 : 6;   // H half-step
template <typename T, bool EXACT> constexpr int kVecBlocksPerSME = sizeof(T) == 8 && EXACT ? 6 : 7;  // E half-step

// Cells of a thread's group along z: 16 bytes of them in k_v3_e / k_v3_h, four
// in float32 and two in float64 (four float64 cells took 168 registers, three
// blocks an SM: the same grid 75.0 us per step fast, 120 EXACT; with two the
// loads in flight come from twice the warps).  The ordered form keeps four.
template <typename T> constexpr int kVecW = 16 / (int)sizeof(T);

template <typename T, int W> struct VW { T v[W]; };

// read-only data of this launch (non-coherent path)
__device__ __forceinline__ void ldg16(float *a, const float *p) {
  const float4 x = __ldg(reinterpret_cast<const float4 *>(p));
  a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
}
__device__ __forceinline__ void ldg16(double *a, const double *p) {
  const double2 x = __ldg(reinterpret_cast<const double2 *>(p));
  a[0] = x.x; a[1] = x.y;
}
__device__ __forceinline__ void ldcg16(float *a, const float *p) {
  const float4 x = __ldcg(reinterpret_cast<const float4 *>(p));
  a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
}
__device__ __forceinline__ void ldcg16(double *a, const double *p) {
  const double2 x = __ldcg(reinterpret_cast<const double2 *>(p));
  a[0] = x.x; a[1] = x.y;
}
__device__ __forceinline__ void ld16(float *a, const float *p) {
  const float4 x = *reinterpret_cast<const float4 *>(p);
  a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
}
__device__ __forceinline__ void ld16(double *a, const double *p) {
  const double2 x = *reinterpret_cast<const double2 *>(p);
  a[0] = x.x; a[1] = x.y;
}
__device__ __forceinline__ void st16(float *p, const float *v) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void st16(double *p, const double *v) { *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]); }
template <typename T, int W> __device__ __forceinline__ void ld4(VW<T, W> &a, const T *p) {
#pragma unroll
  for (int m = 0; m < W; m += kVecW<T>) ldg16(a.v + m, p + m);
}
// E in an H update: L2 only (CG) where the same launch may have written E on
// another SM, whose writes an SM's L1 does not see; the read-only path otherwise
template <bool CG, typename T, int W> __device__ __forceinline__ void ld4e(VW<T, W> &a, const T *p) {
#pragma unroll
  for (int m = 0; m < W; m += kVecW<T>)
    if (CG) ldcg16(a.v + m, p + m);
    else ldg16(a.v + m, p + m);
}
// data this launch also writes (each element only by the thread reading it)
template <typename T, int W> __device__ __forceinline__ void ldw4(VW<T, W> &a, const T *p) {
#pragma unroll
  for (int m = 0; m < W; m += kVecW<T>) ld16(a.v + m, p + m);
}
template <typename T, int W> __device__ __forceinline__ void st4(T *p, const T (&v)[W]) {
#pragma unroll
  for (int m = 0; m < W; m += kVecW<T>) st16(p + m, v + m);
}

// dt/eps of a group: from the material index and its table (one byte per
// cell, the table entries read through L1) or from the three grids.
__device__ __forceinline__ void tab_entry(const float *t, unsigned q, float &a, float &b, float &c) {
  const float4 e = __ldg(reinterpret_cast<const float4 *>(t) + q);
  a = e.x; b = e.y; c = e.z;
}
__device__ __forceinline__ void tab_entry(const double *t, unsigned q, double &a, double &b, double &c) {
  const double2 e = __ldg(reinterpret_cast<const double2 *>(t) + 2 * q), f = __ldg(reinterpret_cast<const double2 *>(t) + 2 * q + 1);
  a = e.x; b = e.y; c = f.x;
}
template <typename T, int W>
__device__ __forceinline__ void load_cb(const Params<T> &p, long long bi, int o, VW<T, W> &C0, VW<T, W> &C1, VW<T, W> &C2) {
  if (p.mat) {
    if constexpr (W == 4) {
      const uchar4 m = __ldg(reinterpret_cast<const uchar4 *>(p.mat + bi + o));
      tab_entry(p.mtab, m.x, C0.v[0], C1.v[0], C2.v[0]);
      tab_entry(p.mtab, m.y, C0.v[1], C1.v[1], C2.v[1]);
      tab_entry(p.mtab, m.z, C0.v[2], C1.v[2], C2.v[2]);
      tab_entry(p.mtab, m.w, C0.v[3], C1.v[3], C2.v[3]);
    } else {
      const uchar2 m = __ldg(reinterpret_cast<const uchar2 *>(p.mat + bi + o));
      tab_entry(p.mtab, m.x, C0.v[0], C1.v[0], C2.v[0]);
      tab_entry(p.mtab, m.y, C0.v[1], C1.v[1], C2.v[1]);
    }
  } else {
    ld4(C0, p.cb[0] + bi + o);
    ld4(C1, p.cb[1] + bi + o);
    ld4(C2, p.cb[2] + bi + o);
  }
}

// Prefetch (into L2) of the CPML psi lines a group reads after its curl (its
// x- and y-slab rows and, in the edge role, its z-slab row), issued before the
// field loads so that the late loads find the lines on chip.  A prefetch holds
// no register; the addresses are those the group loads later.  Used by both
// roles of the H half-step and by the E half-step's edge role: in the E
// vector role it measured slower on large grids (the 384 x 384 x 256 E
// half-step 301 against 286 us), elsewhere faster (C2 step 68.1 against
// 69.8 us).
__device__ __forceinline__ void prefetch_line(const void *a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); }
template <typename T, bool HALF_H, int W>
__device__ __forceinline__ void psi_prefetch(const Params<T> &p, int i, int j, int k0, bool zslab) {
  constexpr int FX0 = HALF_H ? HY : EY, FX1 = HALF_H ? HZ : EZ, FY0 = HALF_H ? HX : EX, FY1 = HALF_H ? HZ : EZ;
  constexpr int FZ0 = HALF_H ? HX : EX, FZ1 = HALF_H ? HY : EY;
  const int P = p.P;
  int d, side;
  if ((HALF_H ? h_slab(i, p.ib, p.ie, P, d, side) : e_slab(i, p.ib, p.ie, P, d, side)) >= 0) {
    const long long oa = ((long long)d * p.ny + j) * p.psx + k0;
    prefetch_line(p.psi[FX0][AX][side] + oa);
    prefetch_line(p.psi[FX1][AX][side] + oa);
  }
  if ((HALF_H ? h_slab(j, p.jb, p.je, P, d, side) : e_slab(j, p.jb, p.je, P, d, side)) >= 0) {
    const long long oa = ((long long)i * P + d) * p.psy + k0;
    prefetch_line(p.psi[FY0][AY][side] + oa);
    prefetch_line(p.psi[FY1][AY][side] + oa);
  }
  if (zslab) {  // the side whose slab cells the group holds (the low one if both)
    const bool lo = k0 <= p.kb + P - 1 && k0 + (W - 1) >= p.kb, hi = k0 + (W - 1) >= p.ke - P && k0 <= p.ke - 1;
    if (lo || hi) {
      const int sd = lo ? LO : HI;
      const long long oz = ((long long)i * p.ny + j) * p.psz + (k0 - (sd ? p.ke - P : p.kb));
      prefetch_line(p.psi[FZ0][AZ][sd] + oz);
      prefetch_line(p.psi[FZ1][AZ][sd] + oz);
    }
  }
}

// EXACT quotients of a group: one range test (numerators `in`, reciprocals
// `yin`) and one branch for all of them, so that their chains overlap.
// Measured on a B200, 97 x 114 x 187 float64 EXACT: 144 us per step with a
// test and a branch a quotient, 117 with one a cell, 120 with one a group of
// four cells, 102 with one a group of two (and six / five blocks an SM; 79.5 now,
// see kVecBlocksPerSM and kappa.h); float32 EXACT 88, 84 and 64.
template <typename T, bool EXACT> __device__ __forceinline__ bool yin3(T y) {
  if constexpr (EXACT) return Ar<T, EXACT>::yin(y);
  else return true;
}
template <typename T, bool EXACT, int W> __device__ __forceinline__ bool yin4(const T (&y)[W]) {
  bool ok = true;
#pragma unroll
  for (int m = 0; m < W; ++m) ok &= yin3<T, EXACT>(y[m]);
  return ok;
}
template <typename T, bool EXACT, int N> __device__ __forceinline__ bool in3(const T (&d)[N]) {
  bool ok = true;
  if constexpr (EXACT)
#pragma unroll
    for (int m = 0; m < N; ++m) ok &= Ar<T, EXACT>::in(d[m]);
  return ok;
}
// EXACT: next psi of a group, b psi + c d / dx (dok: 1 / dx is in range).
template <typename T, bool EXACT, int W>
__device__ __forceinline__ void psi4(T (&v)[W], const T (&b)[W], const T (&psi)[W], const T (&c)[W], const T (&d)[W], T dx,
                                     T rdx, bool dok) {
  using A = Ar<T, EXACT>;
  T n[W];
#pragma unroll
  for (int m = 0; m < W; ++m) n[m] = A::mul(c[m], d[m]);
  const bool ok = in3<T, EXACT>(n) & dok;
  if (ok) {
#pragma unroll
    for (int m = 0; m < W; ++m) v[m] = A::add(A::mul(b[m], psi[m]), A::quo(n[m], dx, rdx));
  } else {
#pragma unroll
    for (int m = 0; m < W; ++m) v[m] = A::add(A::mul(b[m], psi[m]), A::ieee(n[m], dx));
  }
}
template <typename T, bool EXACT, int W>
__device__ __forceinline__ void psi4(T (&v)[W], T b, const T (&psi)[W], T c, const T (&d)[W], T dx, T rdx, bool dok) {
  T b4[W], c4[W];
#pragma unroll
  for (int m = 0; m < W; ++m) b4[m] = b, c4[m] = c;
  psi4<T, EXACT, W>(v, b4, psi, c4, d, dx, rdx, dok);
}
// One cell's next psi (EXACT: v, as psi4 gave it).
template <typename T, bool EXACT> __device__ __forceinline__ T psi_of(T v, T b, T psi, T c, T d, T dx, T rdx) {
  using A = Ar<T, EXACT>;
  if constexpr (EXACT) return v;
  else return A::add(A::mul(b, psi), A::div(A::mul(c, d), dx, rdx));
}

// Split of a row between the roles (computed on the host per job).
struct VecGeom {
  int kz0, kz1;  // vector role: k in [kz0, kz1), multiples of 4
  int nvc;       // groups per row in the vector role
  int nedge;     // edge-role cells per row: [0, kz0) and [kz1, nzp)
  int nb_vec;    // blocks of the vector role per plane (the edge role follows)
};

// 'TM' source (Hy): Ez's x-slab term reads Hy - J at i and i + 1, Ex's z-slab
// term at k and k + 1.  Only the E half-steps of jobs whose source meets a slab
// so (SRC; engine.cu, src_meets_cpml) hold anything for it: in every job's it
// takes registers (float32 128 x 128 x 256 64.5 us per step without, 65.4 with).
//
// src_diffs forms the differences of a group's x- and z-slab terms again, with
// Hy - J at the cells of the source box.  Measured on a B200, float32, 'TM'
// source in, at or 2 cells past the z slab, against the group's cells one after
// another inline / out of line: 48 x 40 x 96 10.2 against 20.4 / 21.3 us per
// step, 64 x 64 x 128 14.8 against 20.8-23.0 / 23.3-24.8, 128 x 128 x 256 65.4
// against 67.3 / 68.1.
template <typename T, bool EXACT, int W>
__device__ __forceinline__ void src_diffs(const Params<T> &p, int i, int j, int k0, int s, const T (&hy)[W], T hyk,
                                          const T (&hyx)[W], T (&dyz)[W], T (&dyx)[W]) {
  using A = Ar<T, EXACT>;
  if (p.src_field != HY || i < p.slo[0] - 1 || i >= p.shi[0] || j < p.slo[1] || j >= p.shi[1] || k0 + W < p.slo[2] ||
      k0 >= p.shi[2])
    return;
  const T Jn = p.jsrc[p.state[0] + s];
  const bool in0 = i >= p.slo[0], in1 = i + 1 < p.shi[0];  // the box holds cells of plane i, of plane i + 1
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const int k = k0 + m;
    const bool at = k >= p.slo[2] && k < p.shi[2], next = k + 1 >= p.slo[2] && k + 1 < p.shi[2];
    const T h1 = m < W - 1 ? hy[m < W - 1 ? m + 1 : 0] : hyk;
    const T c = in0 && at ? A::sub(hy[m], Jn) : hy[m];
    dyz[m] = A::sub(in0 && next ? A::sub(h1, Jn) : h1, c);
    dyx[m] = A::sub(in1 && at ? A::sub(hyx[m], Jn) : hyx[m], c);
  }
}
// float32 EXACT: such groups run cell after cell, out of line (v3_src_e), and
// every job's kernel holds the call: without it, or with src_diffs, the code
// the compiler makes of the EXACT branches is slower (128 x 128 x 256 195 -> 226
// us per step while most of the grid is still below the fast quotient's range,
// 99 -> 101 over a whole run; 72 x 80 x 192 74 -> 87).
template <typename T, bool EXACT> constexpr bool kSrcCells = sizeof(T) == 4 && EXACT;
// A cell of the group has a term that reads the source (zs: z slabs too).
template <typename T> __device__ __forceinline__ bool src_in_cpml(const Params<T> &p, int i, int j, int k0, int nk, bool zs) {
  if (p.src_field != HY || i < p.slo[0] - 1 || i >= p.shi[0] || j < p.slo[1] || j >= p.shi[1] || k0 + nk < p.slo[2] ||
      k0 >= p.shi[2])
    return false;
  int d, side;
  if (k0 + nk > p.slo[2] && e_slab(i, p.ib, p.ie, p.P, d, side) >= 0) return true;
  if (zs && i >= p.slo[0])
    for (int k = max(k0, p.slo[2] - 1); k < min(k0 + nk, p.shi[2]); ++k)
      if (e_slab(k, p.kb, p.ke, p.P, d, side) >= 0) return true;
  return false;
}
template <typename T, bool EXACT>
__device__ __noinline__ void v3_src_e(const Params<T> &p, int i, int j, int k0, int k1, int s) {
  for (int k = k0; k < k1; ++k) y3_e_cell<T, EXACT, true>(p, i, j, k, p.state[0] + s, s);
}

// The source box holds cells of the group (field fld).
template <typename T> __device__ __forceinline__ bool src_group(const Params<T> &p, int fld, int i, int j, int k0, int nk) {
  return p.src_field == fld && i >= p.slo[0] && i < p.shi[0] && j >= p.slo[1] && j < p.shi[1] && k0 + nk > p.slo[2] &&
         k0 < p.shi[2];
}

// Edge role: groups k0 in [0, kz0) and [kz1, nzp) -- the z slabs,
// the rim and the row padding -- with the update range of every component
// tested per cell.  A group's z-slab psi values are one 16-byte vector of the
// padded z-slab rows, unless the group holds cells of both z slabs (then cell
// by cell); all old values of a group are read before the first write.
template <int W, typename T>
__device__ __forceinline__ bool edge_group(const Params<T> &p, const VecGeom &g, int bx, int &j, int &k0) {
  const int nge = g.nedge >> (W == 4 ? 2 : 1);
  const int t = (bx - g.nb_vec) * kVecThreads + threadIdx.x;
  if (t >= (p.je - p.jb) * nge) return false;
  const int r = t / nge, e4 = W * (t - r * nge);
  j = p.jb + r;
  k0 = e4 < g.kz0 ? e4 : g.kz1 + (e4 - g.kz0);
  return true;
}

template <typename T, bool EXACT, int W, bool SRC>
__device__ __forceinline__ void v3_edge_e(const Params<T> &p, const VecGeom &g, int i, int bx, int s) {
  int j, k0;
  if (!edge_group<W>(p, g, bx, j, k0)) return;
  if constexpr (SRC && kSrcCells<T, EXACT>)
    if (src_in_cpml(p, i, j, k0, W, true)) {
      v3_src_e<T, EXACT>(p, i, j, k0, min(k0 + W, p.nz), s);
      return;
    }
  using A = Ar<T, EXACT>;
  const int P = p.P;
  const bool iex = i > p.ib, jey = j > p.jb;
  bool mex[W], mey[W], mez[W];
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const int k = k0 + m;
    const bool kc = k >= p.kb && k < p.ke;
    mex[m] = iex && kc;
    mey[m] = jey && kc;
    mez[m] = k > p.kb && k < p.ke;
  }
  const int sy = p.nzp;
  const long long sx = (long long)p.ny * p.nzp, bi = (long long)i * sx;
  const int o = j * sy + k0;
  psi_prefetch<T, false, W>(p, i, j, k0, true);
  const T *const hx = p.f[HX] + bi, *const hy = p.f[HY] + bi, *const hz = p.f[HZ] + bi;
  VW<T, W> Hx, Hy, Hz, Hzy, Hxy, Hzx, Hyx, C0, C1, C2, Ex, Ey, Ez, Rz, Kz;
  ld4(Hx, hx + o);
  ld4(Hy, hy + o);
  ld4(Hz, hz + o);
  ld4(Hzy, hz + (o + sy));
  ld4(Hxy, hx + (o + sy));
  ld4(Hzx, hz + sx + o);
  ld4(Hyx, hy + sx + o);
  const bool kn = k0 + W < p.nzp;  // the k + 1 neighbour of the last cell
  const T hyk = kn ? __ldg(hy + (o + W)) : T(0), hxk = kn ? __ldg(hx + (o + W)) : T(0);
  load_cb(p, bi, o, C0, C1, C2);
  T *const ex = p.f[EX] + bi, *const ey = p.f[EY] + bi, *const ez = p.f[EZ] + bi;
  ldw4(Ex, ex + o);
  ldw4(Ey, ey + o);
  ldw4(Ez, ez + o);
  ld4(Rz, p.rkd[2] + k0);
  if (EXACT) ld4(Kz, p.kd[2] + k0);
  const T rkx = p.rkd[0][i], rky = p.rkd[1][j];
  const T kx = EXACT ? p.kd[0][i] : T(0), ky = EXACT ? p.kd[1][j] : T(0);
  const bool dok = yin3<T, EXACT>(p.rdx), yok = yin3<T, EXACT>(rkx) & yin3<T, EXACT>(rky) & yin4<T, EXACT>(Rz.v);
  T e0[W], e1[W], e2[W], dzy[W], dyz[W], dxz[W], dzx[W], dyx[W], dxy[W];
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const T hy1 = m < W - 1 ? Hy.v[m + 1] : hyk, hx1 = m < W - 1 ? Hx.v[m + 1] : hxk;
    dzy[m] = A::sub(Hzy.v[m], Hz.v[m]);
    dyz[m] = A::sub(hy1, Hy.v[m]);
    dxz[m] = A::sub(hx1, Hx.v[m]);
    dzx[m] = A::sub(Hzx.v[m], Hz.v[m]);
    dyx[m] = A::sub(Hyx.v[m], Hy.v[m]);
    dxy[m] = A::sub(Hxy.v[m], Hx.v[m]);
    if constexpr (!EXACT) {
      e0[m] = A::add(Ex.v[m], A::mul(C0.v[m], A::sub(A::div(dzy[m], ky, rky), A::div(dyz[m], T(0), Rz.v[m]))));
      e1[m] = A::add(Ey.v[m], A::mul(C1.v[m], A::sub(A::div(dxz[m], T(0), Rz.v[m]), A::div(dzx[m], kx, rkx))));
      e2[m] = A::add(Ez.v[m], A::mul(C2.v[m], A::sub(A::div(dyx[m], kx, rkx), A::div(dxy[m], ky, rky))));
    }
  }
  if constexpr (EXACT) {  // one test and one branch for the group's quotients
    auto curl = [&](auto quo) {
#pragma unroll
      for (int m = 0; m < W; ++m) {
        const T kz = Kz.v[m];
        e0[m] = A::add(Ex.v[m], A::mul(C0.v[m], A::sub(quo(dzy[m], ky, rky), quo(dyz[m], kz, Rz.v[m]))));
        e1[m] = A::add(Ey.v[m], A::mul(C1.v[m], A::sub(quo(dxz[m], kz, Rz.v[m]), quo(dzx[m], kx, rkx))));
        e2[m] = A::add(Ez.v[m], A::mul(C2.v[m], A::sub(quo(dyx[m], kx, rkx), quo(dxy[m], ky, rky))));
      }
    };
    const bool ok = yok & in3<T, EXACT>(dzy) & in3<T, EXACT>(dyz) & in3<T, EXACT>(dxz) & in3<T, EXACT>(dzx) & in3<T, EXACT>(dyx) &
                    in3<T, EXACT>(dxy);
    if (ok) curl([](T a, T b, T y) { return A::quo(a, b, y); });
    else curl([](T a, T b, T) { return A::ieee(a, b); });
  }
  if (src_group(p, EY, i, j, k0, W)) {  // soft source on Ey ('TE'): after the curl, before the CPML terms
    const T Jn = p.jsrc[p.state[0] + s];
#pragma unroll
    for (int m = 0; m < W; ++m)
      if (mey[m] && k0 + m >= p.slo[2] && k0 + m < p.shi[2]) e1[m] = A::sub(e1[m], Jn);
  }
  if constexpr (SRC && !kSrcCells<T, EXACT>) src_diffs<T, EXACT, W>(p, i, j, k0, s, Hy.v, hyk, Hyx.v, dyz, dyx);
  int d, side, q;
  if ((q = e_slab(i, p.ib, p.ie, P, d, side)) >= 0) {  // update_pml_ey_xinc, update_pml_ez_xinc
    const long long oa = ((long long)d * p.ny + j) * p.psx + k0;
    const T be = p.be[q], ce = p.ce[q];
    T *const py = p.psi[EY][AX][side] + oa, *const pz = p.psi[EZ][AX][side] + oa;
    VW<T, W> Py, Pz;
    ldw4(Py, py);
    ldw4(Pz, pz);
    T v0[W], v1[W];  // EXACT: before the masks
    if constexpr (EXACT) {
      psi4<T, EXACT, W>(v0, be, Py.v, ce, dzx, p.dx, p.rdx, dok);
      psi4<T, EXACT, W>(v1, be, Pz.v, ce, dyx, p.dx, p.rdx, dok);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (mey[m]) {
        Py.v[m] = psi_of<T, EXACT>(v0[m], be, Py.v[m], ce, dzx[m], p.dx, p.rdx);
        e1[m] = A::sub(e1[m], A::mul(C1.v[m], Py.v[m]));
      }
      if (mez[m]) {
        Pz.v[m] = psi_of<T, EXACT>(v1[m], be, Pz.v[m], ce, dyx[m], p.dx, p.rdx);
        e2[m] = A::add(e2[m], A::mul(C2.v[m], Pz.v[m]));
      }
    }
    st4(py, Py.v);
    st4(pz, Pz.v);
  }
  if ((q = e_slab(j, p.jb, p.je, P, d, side)) >= 0) {  // update_pml_ex_yinc, update_pml_ez_yinc
    const long long oa = ((long long)i * P + d) * p.psy + k0;
    const T be = p.be[q], ce = p.ce[q];
    T *const px = p.psi[EX][AY][side] + oa, *const pz = p.psi[EZ][AY][side] + oa;
    VW<T, W> Px, Pz;
    ldw4(Px, px);
    ldw4(Pz, pz);
    T v0[W], v1[W];  // EXACT: before the masks
    if constexpr (EXACT) {
      psi4<T, EXACT, W>(v0, be, Px.v, ce, dzy, p.dx, p.rdx, dok);
      psi4<T, EXACT, W>(v1, be, Pz.v, ce, dxy, p.dx, p.rdx, dok);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (mex[m]) {
        Px.v[m] = psi_of<T, EXACT>(v0[m], be, Px.v[m], ce, dzy[m], p.dx, p.rdx);
        e0[m] = A::add(e0[m], A::mul(C0.v[m], Px.v[m]));
      }
      if (mez[m]) {
        Pz.v[m] = psi_of<T, EXACT>(v1[m], be, Pz.v[m], ce, dxy[m], p.dx, p.rdx);
        e2[m] = A::sub(e2[m], A::mul(C2.v[m], Pz.v[m]));
      }
    }
    st4(px, Px.v);
    st4(pz, Pz.v);
  }
  // update_pml_ex_zinc, update_pml_ey_zinc.  The z-slab psi rows are padded to whole four-cell
  // groups: when the group's slab cells lie on one side (always unless
  // ke - kb < 2P + 3), its values are one 16-byte aligned vector of the
  // row (the rim cells' elements are padding, written back as read);
  // otherwise cell by cell.
  int qz[W], dz[W], zside = -1;
  bool zmix = false;
#pragma unroll
  for (int m = 0; m < W; ++m) {
    int sd = 0;
    dz[m] = 0;
    qz[m] = mex[m] || mey[m] ? e_slab(k0 + m, p.kb, p.ke, P, dz[m], sd) : -1;
    if (qz[m] >= 0) {
      zmix |= zside >= 0 && zside != sd;
      zside = sd;
    }
  }
  const long long ob = ((long long)i * p.ny + j) * p.psz;  // z-slab psi row (i, j)
  if (zside >= 0 && !zmix) {
    const int off = k0 - (zside ? p.ke - P : p.kb);  // slab index d of the group's first cell
    T *const qx = p.psi[EX][AZ][zside] + (ob + off), *const qy = p.psi[EY][AZ][zside] + (ob + off);
    VW<T, W> Zx, Zy;
    ldw4(Zx, qx);
    ldw4(Zy, qy);
    T v0[W], v1[W];
    if constexpr (EXACT) {
      T b4[W], c4[W];
#pragma unroll
      for (int m = 0; m < W; ++m) {
        b4[m] = p.be[max(qz[m], 0)];
        c4[m] = p.ce[max(qz[m], 0)];
      }
      psi4<T, EXACT, W>(v0, b4, Zx.v, c4, dyz, p.dx, p.rdx, dok);
      psi4<T, EXACT, W>(v1, b4, Zy.v, c4, dxz, p.dx, p.rdx, dok);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (qz[m] < 0) continue;
      const T be = p.be[qz[m]], ce = p.ce[qz[m]];
      if (mex[m]) {
        Zx.v[m] = psi_of<T, EXACT>(v0[m], be, Zx.v[m], ce, dyz[m], p.dx, p.rdx);
        e0[m] = A::sub(e0[m], A::mul(C0.v[m], Zx.v[m]));
      }
      if (mey[m]) {
        Zy.v[m] = psi_of<T, EXACT>(v1[m], be, Zy.v[m], ce, dxz[m], p.dx, p.rdx);
        e1[m] = A::add(e1[m], A::mul(C1.v[m], Zy.v[m]));
      }
    }
    st4(qx, Zx.v);
    st4(qy, Zy.v);
  } else if (zmix) {
    T zx[W], zy[W];
    int sz[W];
#pragma unroll
    for (int m = 0; m < W; ++m) {
      int dd = 0;
      sz[m] = 0;
      if (qz[m] >= 0) {e_slab(k0 + m, p.kb, p.ke, P, dd, sz[m]);}
      zx[m] = qz[m] >= 0 && mex[m] ? p.psi[EX][AZ][sz[m]][ob + dz[m]] : T(0);
      zy[m] = qz[m] >= 0 && mey[m] ? p.psi[EY][AZ][sz[m]][ob + dz[m]] : T(0);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (qz[m] < 0) continue;
      const T be = p.be[qz[m]], ce = p.ce[qz[m]];
      if (mex[m]) {
        zx[m] = A::add(A::mul(be, zx[m]), A::div(A::mul(ce, dyz[m]), p.dx, p.rdx));
        p.psi[EX][AZ][sz[m]][ob + dz[m]] = zx[m];
        e0[m] = A::sub(e0[m], A::mul(C0.v[m], zx[m]));
      }
      if (mey[m]) {
        zy[m] = A::add(A::mul(be, zy[m]), A::div(A::mul(ce, dxz[m]), p.dx, p.rdx));
        p.psi[EY][AZ][sz[m]][ob + dz[m]] = zy[m];
        e1[m] = A::add(e1[m], A::mul(C1.v[m], zy[m]));
      }
    }
  }
#pragma unroll
  for (int m = 0; m < W; ++m) {  // cells outside a component's range keep their value
    e0[m] = mex[m] ? e0[m] : Ex.v[m];
    e1[m] = mey[m] ? e1[m] : Ey.v[m];
    e2[m] = mez[m] ? e2[m] : Ez.v[m];
  }
  st4(ex + o, e0);
  st4(ey + o, e1);
  st4(ez + o, e2);
#pragma unroll
  for (int pq = 0; pq < 2; ++pq) {
    const int dm = p.port_pos[pq] - k0;
    if ((unsigned)dm < (unsigned)W) {
      const long long pc = (long long)i * p.ny + j;
#pragma unroll
      for (int m = 0; m < W; ++m)
        if (m == dm) {
          if (mex[m]) capture(p, s, pq, 0, pc, e0[m]);
          if (mey[m]) capture(p, s, pq, 1, pc, e1[m]);
        }
    }
  }
}

template <typename T, bool EXACT, bool CG, int W>
__device__ __forceinline__ void v3_edge_h(const Params<T> &p, const VecGeom &g, int i, int bx, int s) {
  int j, k0;
  if (!edge_group<W>(p, g, bx, j, k0)) return;
  using A = Ar<T, EXACT>;
  const int P = p.P;
  const bool ihy = i > p.ib, jhx = j > p.jb;
  bool mhx[W], mhy[W], mhz[W];
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const int k = k0 + m;
    const bool kc = k >= p.kb && k < p.ke, ko = k > p.kb && k < p.ke;
    mhx[m] = jhx && ko;
    mhy[m] = ihy && ko;
    mhz[m] = ihy && jhx && kc;
  }
  const int sy = p.nzp;
  const long long sx = (long long)p.ny * p.nzp, bi = (long long)i * sx;
  const int o = j * sy + k0;
  psi_prefetch<T, true, W>(p, i, j, k0, true);
  const T *const ex = p.f[EX] + bi, *const ey = p.f[EY] + bi, *const ez = p.f[EZ] + bi;
  VW<T, W> Ex, Ey, Ez, Ezy, Exy, Ezx, Eyx, Hx, Hy, Hz, Rz, Kz;
  ld4e<CG>(Ex, ex + o);
  ld4e<CG>(Ey, ey + o);
  ld4e<CG>(Ez, ez + o);
  ld4e<CG>(Ezy, ez + (o - sy));
  ld4e<CG>(Exy, ex + (o - sy));
  ld4e<CG>(Ezx, ez - sx + o);
  ld4e<CG>(Eyx, ey - sx + o);
  const bool kp = k0 > 0;  // the k - 1 neighbour of the first cell
  const T eyk = kp ? ld_e<CG>(ey + (o - 1)) : T(0), exk = kp ? ld_e<CG>(ex + (o - 1)) : T(0);
  T *const hx = p.f[HX] + bi, *const hy = p.f[HY] + bi, *const hz = p.f[HZ] + bi;
  ldw4(Hx, hx + o);
  ldw4(Hy, hy + o);
  ldw4(Hz, hz + o);
  if (src_group(p, HY, i, j, k0, W)) {  // soft source on Hy ('TM'): subtracted before the Hy update
    const T Jn = p.jsrc[p.state[0] + s];
#pragma unroll
    for (int m = 0; m < W; ++m)
      if (mhy[m] && k0 + m >= p.slo[2] && k0 + m < p.shi[2]) Hy.v[m] = A::sub(Hy.v[m], Jn);
  }
  ld4(Rz, p.rkd[5] + k0);
  if (EXACT) ld4(Kz, p.kd[5] + k0);
  const T rkx = p.rkd[3][i], rky = p.rkd[4][j];
  const T kx = EXACT ? p.kd[3][i] : T(0), ky = EXACT ? p.kd[4][j] : T(0);
  const bool dok = yin3<T, EXACT>(p.rdx), yok = yin3<T, EXACT>(rkx) & yin3<T, EXACT>(rky) & yin4<T, EXACT>(Rz.v);
  const T db = p.db;
  T h0[W], h1[W], h2[W], dyz[W], dzy[W], dzx[W], dxz[W], dxy[W], dyx[W];
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const T ey1 = m > 0 ? Ey.v[m - 1] : eyk, ex1 = m > 0 ? Ex.v[m - 1] : exk;
    dyz[m] = A::sub(Ey.v[m], ey1);
    dzy[m] = A::sub(Ez.v[m], Ezy.v[m]);
    dzx[m] = A::sub(Ez.v[m], Ezx.v[m]);
    dxz[m] = A::sub(Ex.v[m], ex1);
    dxy[m] = A::sub(Ex.v[m], Exy.v[m]);
    dyx[m] = A::sub(Ey.v[m], Eyx.v[m]);
    if constexpr (!EXACT) {
      h0[m] = A::add(Hx.v[m], A::mul(db, A::sub(A::div(dyz[m], T(0), Rz.v[m]), A::div(dzy[m], ky, rky))));
      h1[m] = A::add(Hy.v[m], A::mul(db, A::sub(A::div(dzx[m], kx, rkx), A::div(dxz[m], T(0), Rz.v[m]))));
      h2[m] = A::add(Hz.v[m], A::mul(db, A::sub(A::div(dxy[m], ky, rky), A::div(dyx[m], kx, rkx))));
    }
  }
  if constexpr (EXACT) {  // one test and one branch for the group's quotients
    auto curl = [&](auto quo) {
#pragma unroll
      for (int m = 0; m < W; ++m) {
        const T kz = Kz.v[m];
        h0[m] = A::add(Hx.v[m], A::mul(db, A::sub(quo(dyz[m], kz, Rz.v[m]), quo(dzy[m], ky, rky))));
        h1[m] = A::add(Hy.v[m], A::mul(db, A::sub(quo(dzx[m], kx, rkx), quo(dxz[m], kz, Rz.v[m]))));
        h2[m] = A::add(Hz.v[m], A::mul(db, A::sub(quo(dxy[m], ky, rky), quo(dyx[m], kx, rkx))));
      }
    };
    const bool ok = yok & in3<T, EXACT>(dzy) & in3<T, EXACT>(dyz) & in3<T, EXACT>(dxz) & in3<T, EXACT>(dzx) & in3<T, EXACT>(dyx) &
                    in3<T, EXACT>(dxy);
    if (ok) curl([](T a, T b, T y) { return A::quo(a, b, y); });
    else curl([](T a, T b, T) { return A::ieee(a, b); });
  }
  int d, side, q;
  if ((q = h_slab(i, p.ib, p.ie, P, d, side)) >= 0) {  // update_pml_hy_xinc, update_pml_hz_xinc
    const long long oa = ((long long)d * p.ny + j) * p.psx + k0;
    const T bh = p.bh[q], ch = p.ch[q];
    T *const py = p.psi[HY][AX][side] + oa, *const pz = p.psi[HZ][AX][side] + oa;
    VW<T, W> Py, Pz;
    ldw4(Py, py);
    ldw4(Pz, pz);
    T v0[W], v1[W];  // EXACT: before the masks
    if constexpr (EXACT) {
      psi4<T, EXACT, W>(v0, bh, Py.v, ch, dzx, p.dx, p.rdx, dok);
      psi4<T, EXACT, W>(v1, bh, Pz.v, ch, dyx, p.dx, p.rdx, dok);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (mhy[m]) {
        Py.v[m] = psi_of<T, EXACT>(v0[m], bh, Py.v[m], ch, dzx[m], p.dx, p.rdx);
        h1[m] = A::add(h1[m], A::mul(db, Py.v[m]));
      }
      if (mhz[m]) {
        Pz.v[m] = psi_of<T, EXACT>(v1[m], bh, Pz.v[m], ch, dyx[m], p.dx, p.rdx);
        h2[m] = A::sub(h2[m], A::mul(db, Pz.v[m]));
      }
    }
    st4(py, Py.v);
    st4(pz, Pz.v);
  }
  if ((q = h_slab(j, p.jb, p.je, P, d, side)) >= 0) {  // update_pml_hx_yinc, update_pml_hz_yinc
    const long long oa = ((long long)i * P + d) * p.psy + k0;
    const T bh = p.bh[q], ch = p.ch[q];
    T *const px = p.psi[HX][AY][side] + oa, *const pz = p.psi[HZ][AY][side] + oa;
    VW<T, W> Px, Pz;
    ldw4(Px, px);
    ldw4(Pz, pz);
    T v0[W], v1[W];  // EXACT: before the masks
    if constexpr (EXACT) {
      psi4<T, EXACT, W>(v0, bh, Px.v, ch, dzy, p.dx, p.rdx, dok);
      psi4<T, EXACT, W>(v1, bh, Pz.v, ch, dxy, p.dx, p.rdx, dok);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (mhx[m]) {
        Px.v[m] = psi_of<T, EXACT>(v0[m], bh, Px.v[m], ch, dzy[m], p.dx, p.rdx);
        h0[m] = A::sub(h0[m], A::mul(db, Px.v[m]));
      }
      if (mhz[m]) {
        Pz.v[m] = psi_of<T, EXACT>(v1[m], bh, Pz.v[m], ch, dxy[m], p.dx, p.rdx);
        h2[m] = A::add(h2[m], A::mul(db, Pz.v[m]));
      }
    }
    st4(px, Px.v);
    st4(pz, Pz.v);
  }
  // update_pml_hx_zinc, update_pml_hy_zinc.  The z-slab psi rows are padded to whole four-cell
  // groups: when the group's slab cells lie on one side (always unless
  // ke - kb < 2P + 3), its values are one 16-byte aligned vector of the
  // row (the rim cells' elements are padding, written back as read);
  // otherwise cell by cell.
  int qz[W], dz[W], zside = -1;
  bool zmix = false;
#pragma unroll
  for (int m = 0; m < W; ++m) {
    int sd = 0;
    dz[m] = 0;
    qz[m] = mhx[m] || mhy[m] ? h_slab(k0 + m, p.kb, p.ke, P, dz[m], sd) : -1;
    if (qz[m] >= 0) {
      zmix |= zside >= 0 && zside != sd;
      zside = sd;
    }
  }
  const long long ob = ((long long)i * p.ny + j) * p.psz;  // z-slab psi row (i, j)
  if (zside >= 0 && !zmix) {
    const int off = k0 - (zside ? p.ke - P : p.kb);  // slab index d of the group's first cell
    T *const qx = p.psi[HX][AZ][zside] + (ob + off), *const qy = p.psi[HY][AZ][zside] + (ob + off);
    VW<T, W> Zx, Zy;
    ldw4(Zx, qx);
    ldw4(Zy, qy);
    T v0[W], v1[W];
    if constexpr (EXACT) {
      T b4[W], c4[W];
#pragma unroll
      for (int m = 0; m < W; ++m) {
        b4[m] = p.bh[max(qz[m], 0)];
        c4[m] = p.ch[max(qz[m], 0)];
      }
      psi4<T, EXACT, W>(v0, b4, Zx.v, c4, dyz, p.dx, p.rdx, dok);
      psi4<T, EXACT, W>(v1, b4, Zy.v, c4, dxz, p.dx, p.rdx, dok);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (qz[m] < 0) continue;
      const T bh = p.bh[qz[m]], ch = p.ch[qz[m]];
      if (mhx[m]) {
        Zx.v[m] = psi_of<T, EXACT>(v0[m], bh, Zx.v[m], ch, dyz[m], p.dx, p.rdx);
        h0[m] = A::add(h0[m], A::mul(db, Zx.v[m]));
      }
      if (mhy[m]) {
        Zy.v[m] = psi_of<T, EXACT>(v1[m], bh, Zy.v[m], ch, dxz[m], p.dx, p.rdx);
        h1[m] = A::sub(h1[m], A::mul(db, Zy.v[m]));
      }
    }
    st4(qx, Zx.v);
    st4(qy, Zy.v);
  } else if (zmix) {
    T zx[W], zy[W];
    int sz[W];
#pragma unroll
    for (int m = 0; m < W; ++m) {
      int dd = 0;
      sz[m] = 0;
      if (qz[m] >= 0) {h_slab(k0 + m, p.kb, p.ke, P, dd, sz[m]);}
      zx[m] = qz[m] >= 0 && mhx[m] ? p.psi[HX][AZ][sz[m]][ob + dz[m]] : T(0);
      zy[m] = qz[m] >= 0 && mhy[m] ? p.psi[HY][AZ][sz[m]][ob + dz[m]] : T(0);
    }
#pragma unroll
    for (int m = 0; m < W; ++m) {
      if (qz[m] < 0) continue;
      const T bh = p.bh[qz[m]], ch = p.ch[qz[m]];
      if (mhx[m]) {
        zx[m] = A::add(A::mul(bh, zx[m]), A::div(A::mul(ch, dyz[m]), p.dx, p.rdx));
        p.psi[HX][AZ][sz[m]][ob + dz[m]] = zx[m];
        h0[m] = A::add(h0[m], A::mul(db, zx[m]));
      }
      if (mhy[m]) {
        zy[m] = A::add(A::mul(bh, zy[m]), A::div(A::mul(ch, dxz[m]), p.dx, p.rdx));
        p.psi[HY][AZ][sz[m]][ob + dz[m]] = zy[m];
        h1[m] = A::sub(h1[m], A::mul(db, zy[m]));
      }
    }
  }
#pragma unroll
  for (int m = 0; m < W; ++m) {
    h0[m] = mhx[m] ? h0[m] : Hx.v[m];
    h1[m] = mhy[m] ? h1[m] : Hy.v[m];
    h2[m] = mhz[m] ? h2[m] : Hz.v[m];
  }
  st4(hx + o, h0);
  st4(hy + o, h1);
  st4(hz + o, h2);
#pragma unroll
  for (int pq = 0; pq < 2; ++pq) {
    const int dm = p.port_pos[pq] - k0;
    if ((unsigned)(dm + 1) < W + 1u) {
      const long long pc = (long long)i * p.ny + j;
#pragma unroll
      for (int m = 0; m < W; ++m) {
        if (m == dm) {
          if (mhx[m]) capture(p, s, pq, 2, pc, h0[m]);
          if (mhy[m]) capture(p, s, pq, 4, pc, h1[m]);
        }
        if (m == dm + 1) {
          if (mhx[m]) capture(p, s, pq, 3, pc, h0[m]);
          if (mhy[m]) capture(p, s, pq, 5, pc, h1[m]);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// E half-step.  Updated: Ex i (ib,ie) j [jb,je) k [kb,ke); Ey i [ib,ie)
// j (jb,je) k [kb,ke); Ez i [ib,ie) j [jb,je) k (kb,ke).  Grid: (vector-role
// then edge-role blocks, x-planes ib..ie-1).
// ---------------------------------------------------------------------------
// One block of x-plane i: bx < nb_vec a vector-role block, the edge role above.
template <typename T, bool EXACT, int W, bool SRC>
__device__ __forceinline__ void v3_e_block(const Params<T> &p, const VecGeom &g, int i, int bx, int s) {
  if (bx >= g.nb_vec) {
    v3_edge_e<T, EXACT, W, SRC>(p, g, i, bx, s);
    return;
  }
  const int t = bx * kVecThreads + threadIdx.x;
  if (t >= (p.je - p.jb) * g.nvc) return;
  const int r = t / g.nvc;
  const int j = p.jb + r, k0 = g.kz0 + W * (t - r * g.nvc);
  if constexpr (SRC && kSrcCells<T, EXACT>)
    if (src_in_cpml(p, i, j, k0, W, false)) {
      v3_src_e<T, EXACT>(p, i, j, k0, k0 + W, s);
      return;
    }
  using A = Ar<T, EXACT>;
  const int sy = p.nzp;
  const long long sx = (long long)p.ny * p.nzp, bi = (long long)i * sx;
  const int o = j * sy + k0;
  const T *const hx = p.f[HX] + bi, *const hy = p.f[HY] + bi, *const hz = p.f[HZ] + bi;
  VW<T, W> Hx, Hy, Hz, Hzy, Hxy, Hzx, Hyx, C0, C1, C2, Ex, Ey, Ez, Rz, Kz;
  ld4(Hx, hx + o);
  ld4(Hy, hy + o);
  ld4(Hz, hz + o);
  ld4(Hzy, hz + (o + sy));
  ld4(Hxy, hx + (o + sy));
  ld4(Hzx, hz + sx + o);
  ld4(Hyx, hy + sx + o);
  const T hyk = __ldg(hy + (o + W)), hxk = __ldg(hx + (o + W));  // k0 + W <= kz1 <= nz - 2
  load_cb(p, bi, o, C0, C1, C2);
  T *const ex = p.f[EX] + bi, *const ey = p.f[EY] + bi, *const ez = p.f[EZ] + bi;
  ldw4(Ex, ex + o);
  ldw4(Ey, ey + o);
  ldw4(Ez, ez + o);
  ld4(Rz, p.rkd[2] + k0);
  if (EXACT) ld4(Kz, p.kd[2] + k0);
  const T rkx = p.rkd[0][i], rky = p.rkd[1][j];
  const T kx = EXACT ? p.kd[0][i] : T(0), ky = EXACT ? p.kd[1][j] : T(0);
  const bool dok = yin3<T, EXACT>(p.rdx), yok = yin3<T, EXACT>(rkx) & yin3<T, EXACT>(rky) & yin4<T, EXACT>(Rz.v);
  // update ranges: all cells of the group are inside (kb, ke); Ex leaves out i = ib,
  // Ey j = jb
  const bool mex = i > p.ib, mey = j > p.jb;
  T e0[W], e1[W], e2[W], dzy[W], dyz[W], dxz[W], dzx[W], dyx[W], dxy[W];
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const T hy1 = m < W - 1 ? Hy.v[m + 1] : hyk, hx1 = m < W - 1 ? Hx.v[m + 1] : hxk;
    dzy[m] = A::sub(Hzy.v[m], Hz.v[m]);
    dyz[m] = A::sub(hy1, Hy.v[m]);
    dxz[m] = A::sub(hx1, Hx.v[m]);
    dzx[m] = A::sub(Hzx.v[m], Hz.v[m]);
    dyx[m] = A::sub(Hyx.v[m], Hy.v[m]);
    dxy[m] = A::sub(Hxy.v[m], Hx.v[m]);
    if constexpr (!EXACT) {
      e0[m] = A::add(Ex.v[m], A::mul(C0.v[m], A::sub(A::div(dzy[m], ky, rky), A::div(dyz[m], T(0), Rz.v[m]))));
      e1[m] = A::add(Ey.v[m], A::mul(C1.v[m], A::sub(A::div(dxz[m], T(0), Rz.v[m]), A::div(dzx[m], kx, rkx))));
      e2[m] = A::add(Ez.v[m], A::mul(C2.v[m], A::sub(A::div(dyx[m], kx, rkx), A::div(dxy[m], ky, rky))));
    }
  }
  if constexpr (EXACT) {  // one test and one branch for the group's quotients
    auto curl = [&](auto quo) {
#pragma unroll
      for (int m = 0; m < W; ++m) {
        const T kz = Kz.v[m];
        e0[m] = A::add(Ex.v[m], A::mul(C0.v[m], A::sub(quo(dzy[m], ky, rky), quo(dyz[m], kz, Rz.v[m]))));
        e1[m] = A::add(Ey.v[m], A::mul(C1.v[m], A::sub(quo(dxz[m], kz, Rz.v[m]), quo(dzx[m], kx, rkx))));
        e2[m] = A::add(Ez.v[m], A::mul(C2.v[m], A::sub(quo(dyx[m], kx, rkx), quo(dxy[m], ky, rky))));
      }
    };
    const bool ok = yok & in3<T, EXACT>(dzy) & in3<T, EXACT>(dyz) & in3<T, EXACT>(dxz) & in3<T, EXACT>(dzx) & in3<T, EXACT>(dyx) &
                    in3<T, EXACT>(dxy);
    if (ok) curl([](T a, T b, T y) { return A::quo(a, b, y); });
    else curl([](T a, T b, T) { return A::ieee(a, b); });
  }
  // soft source on Ey ('TE'): after the curl, before the CPML terms
  if (mey && src_group(p, EY, i, j, k0, W)) {
    const T Jn = p.jsrc[p.state[0] + s];
#pragma unroll
    for (int m = 0; m < W; ++m)
      if (k0 + m >= p.slo[2] && k0 + m < p.shi[2]) e1[m] = A::sub(e1[m], Jn);
  }
  if constexpr (SRC && !kSrcCells<T, EXACT>) src_diffs<T, EXACT, W>(p, i, j, k0, s, Hy.v, hyk, Hyx.v, dyz, dyx);
  const int P = p.P;
  int d, side, q;
  if ((q = e_slab(i, p.ib, p.ie, P, d, side)) >= 0) {  // update_pml_ey_xinc, update_pml_ez_xinc
    const long long oa = ((long long)d * p.ny + j) * p.psx + k0;
    const T be = p.be[q], ce = p.ce[q];
    if (mey) {
      T *const py = p.psi[EY][AX][side] + oa;
      VW<T, W> Py;
      ldw4(Py, py);
      T v[W];
      if constexpr (EXACT) psi4<T, EXACT, W>(v, be, Py.v, ce, dzx, p.dx, p.rdx, dok);
#pragma unroll
      for (int m = 0; m < W; ++m) {
        Py.v[m] = psi_of<T, EXACT>(v[m], be, Py.v[m], ce, dzx[m], p.dx, p.rdx);
        e1[m] = A::sub(e1[m], A::mul(C1.v[m], Py.v[m]));
      }
      st4(py, Py.v);
    }
    T *const pz = p.psi[EZ][AX][side] + oa;
    VW<T, W> Pz;
    ldw4(Pz, pz);
    T v[W];
    if constexpr (EXACT) psi4<T, EXACT, W>(v, be, Pz.v, ce, dyx, p.dx, p.rdx, dok);
#pragma unroll
    for (int m = 0; m < W; ++m) {
      Pz.v[m] = psi_of<T, EXACT>(v[m], be, Pz.v[m], ce, dyx[m], p.dx, p.rdx);
      e2[m] = A::add(e2[m], A::mul(C2.v[m], Pz.v[m]));
    }
    st4(pz, Pz.v);
  }
  if ((q = e_slab(j, p.jb, p.je, P, d, side)) >= 0) {  // update_pml_ex_yinc, update_pml_ez_yinc
    const long long oa = ((long long)i * P + d) * p.psy + k0;
    const T be = p.be[q], ce = p.ce[q];
    if (mex) {
      T *const px = p.psi[EX][AY][side] + oa;
      VW<T, W> Px;
      ldw4(Px, px);
      T v[W];
      if constexpr (EXACT) psi4<T, EXACT, W>(v, be, Px.v, ce, dzy, p.dx, p.rdx, dok);
#pragma unroll
      for (int m = 0; m < W; ++m) {
        Px.v[m] = psi_of<T, EXACT>(v[m], be, Px.v[m], ce, dzy[m], p.dx, p.rdx);
        e0[m] = A::add(e0[m], A::mul(C0.v[m], Px.v[m]));
      }
      st4(px, Px.v);
    }
    T *const pz = p.psi[EZ][AY][side] + oa;
    VW<T, W> Pz;
    ldw4(Pz, pz);
    T v[W];
    if constexpr (EXACT) psi4<T, EXACT, W>(v, be, Pz.v, ce, dxy, p.dx, p.rdx, dok);
#pragma unroll
    for (int m = 0; m < W; ++m) {
      Pz.v[m] = psi_of<T, EXACT>(v[m], be, Pz.v[m], ce, dxy[m], p.dx, p.rdx);
      e2[m] = A::sub(e2[m], A::mul(C2.v[m], Pz.v[m]));
    }
    st4(pz, Pz.v);
  }
  if (mex) st4(ex + o, e0);
  if (mey) st4(ey + o, e1);
  st4(ez + o, e2);
  // port planes: raw Ex, Ey samples for the DFT fold
#pragma unroll
  for (int pq = 0; pq < 2; ++pq) {
    const int dm = p.port_pos[pq] - k0;
    if ((unsigned)dm < (unsigned)W) {
      const long long pc = (long long)i * p.ny + j;
#pragma unroll
      for (int m = 0; m < W; ++m)
        if (m == dm) {
          if (mex) capture(p, s, pq, 0, pc, e0[m]);
          if (mey) capture(p, s, pq, 1, pc, e1[m]);
        }
    }
  }
}

// ---------------------------------------------------------------------------
// H half-step.  Updated: Hx i [ib,ie) j (jb,je) k (kb,ke); Hy i (ib,ie)
// j [jb,je) k (kb,ke); Hz i (ib,ie) j (jb,je) k [kb,ke).  Planes run in
// decreasing i: the launch starts on the E planes the E half-step wrote last
// (still in L2) and ends on the planes the next E half-step reads first.
// ---------------------------------------------------------------------------
template <typename T, bool EXACT, bool CG, int W>
__device__ __forceinline__ void v3_h_block(const Params<T> &p, const VecGeom &g, int i, int bx, int s) {
  if (bx >= g.nb_vec) {
    v3_edge_h<T, EXACT, CG, W>(p, g, i, bx, s);
    return;
  }
  const int t = bx * kVecThreads + threadIdx.x;
  if (t >= (p.je - p.jb) * g.nvc) return;
  const int r = t / g.nvc;
  const int j = p.jb + r, k0 = g.kz0 + W * (t - r * g.nvc);
  using A = Ar<T, EXACT>;
  const int sy = p.nzp;
  const long long sx = (long long)p.ny * p.nzp, bi = (long long)i * sx;
  const int o = j * sy + k0;
  psi_prefetch<T, true, W>(p, i, j, k0, false);
  const T *const ex = p.f[EX] + bi, *const ey = p.f[EY] + bi, *const ez = p.f[EZ] + bi;
  VW<T, W> Ex, Ey, Ez, Ezy, Exy, Ezx, Eyx, Hx, Hy, Hz, Rz, Kz;
  ld4e<CG>(Ex, ex + o);
  ld4e<CG>(Ey, ey + o);
  ld4e<CG>(Ez, ez + o);
  ld4e<CG>(Ezy, ez + (o - sy));
  ld4e<CG>(Exy, ex + (o - sy));
  ld4e<CG>(Ezx, ez - sx + o);
  ld4e<CG>(Eyx, ey - sx + o);
  const T eyk = ld_e<CG>(ey + (o - 1)), exk = ld_e<CG>(ex + (o - 1));  // k0 - 1 >= kz0 - 1 >= kb + P - 1
  T *const hx = p.f[HX] + bi, *const hy = p.f[HY] + bi, *const hz = p.f[HZ] + bi;
  ldw4(Hx, hx + o);
  ldw4(Hy, hy + o);
  ldw4(Hz, hz + o);
  ld4(Rz, p.rkd[5] + k0);
  if (EXACT) ld4(Kz, p.kd[5] + k0);
  const T rkx = p.rkd[3][i], rky = p.rkd[4][j];
  const T kx = EXACT ? p.kd[3][i] : T(0), ky = EXACT ? p.kd[4][j] : T(0);
  const bool dok = yin3<T, EXACT>(p.rdx), yok = yin3<T, EXACT>(rkx) & yin3<T, EXACT>(rky) & yin4<T, EXACT>(Rz.v);
  const T db = p.db;
  // update ranges: all cells of the group are inside (kb, ke); Hx leaves out j = jb,
  // Hy i = ib, Hz both
  const bool mhx = j > p.jb, mhy = i > p.ib, mhz = mhx && mhy;
  // soft source on Hy ('TM'): subtracted before the Hy update
  const bool src = mhy && src_group(p, HY, i, j, k0, W);
  const T Jn = src ? p.jsrc[p.state[0] + s] : T(0);
  T h0[W], h1[W], h2[W], dyz[W], dzy[W], dzx[W], dxz[W], dxy[W], dyx[W];
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const T ey1 = m > 0 ? Ey.v[m - 1] : eyk, ex1 = m > 0 ? Ex.v[m - 1] : exk;
    dyz[m] = A::sub(Ey.v[m], ey1);
    dzy[m] = A::sub(Ez.v[m], Ezy.v[m]);
    dzx[m] = A::sub(Ez.v[m], Ezx.v[m]);
    dxz[m] = A::sub(Ex.v[m], ex1);
    dxy[m] = A::sub(Ex.v[m], Exy.v[m]);
    dyx[m] = A::sub(Ey.v[m], Eyx.v[m]);
    if (src && k0 + m >= p.slo[2] && k0 + m < p.shi[2]) Hy.v[m] = A::sub(Hy.v[m], Jn);
    if constexpr (!EXACT) {
      h0[m] = A::add(Hx.v[m], A::mul(db, A::sub(A::div(dyz[m], T(0), Rz.v[m]), A::div(dzy[m], ky, rky))));
      h1[m] = A::add(Hy.v[m], A::mul(db, A::sub(A::div(dzx[m], kx, rkx), A::div(dxz[m], T(0), Rz.v[m]))));
      h2[m] = A::add(Hz.v[m], A::mul(db, A::sub(A::div(dxy[m], ky, rky), A::div(dyx[m], kx, rkx))));
    }
  }
  if constexpr (EXACT) {  // one test and one branch for the group's quotients
    auto curl = [&](auto quo) {
#pragma unroll
      for (int m = 0; m < W; ++m) {
        const T kz = Kz.v[m];
        h0[m] = A::add(Hx.v[m], A::mul(db, A::sub(quo(dyz[m], kz, Rz.v[m]), quo(dzy[m], ky, rky))));
        h1[m] = A::add(Hy.v[m], A::mul(db, A::sub(quo(dzx[m], kx, rkx), quo(dxz[m], kz, Rz.v[m]))));
        h2[m] = A::add(Hz.v[m], A::mul(db, A::sub(quo(dxy[m], ky, rky), quo(dyx[m], kx, rkx))));
      }
    };
    const bool ok = yok & in3<T, EXACT>(dzy) & in3<T, EXACT>(dyz) & in3<T, EXACT>(dxz) & in3<T, EXACT>(dzx) & in3<T, EXACT>(dyx) &
                    in3<T, EXACT>(dxy);
    if (ok) curl([](T a, T b, T y) { return A::quo(a, b, y); });
    else curl([](T a, T b, T) { return A::ieee(a, b); });
  }
  const int P = p.P;
  int d, side, q;
  if (mhy && (q = h_slab(i, p.ib, p.ie, P, d, side)) >= 0) {  // update_pml_hy_xinc, update_pml_hz_xinc
    const long long oa = ((long long)d * p.ny + j) * p.psx + k0;
    const T bh = p.bh[q], ch = p.ch[q];
    T *const py = p.psi[HY][AX][side] + oa;
    VW<T, W> Py;
    ldw4(Py, py);
    T v[W];
    if constexpr (EXACT) psi4<T, EXACT, W>(v, bh, Py.v, ch, dzx, p.dx, p.rdx, dok);
#pragma unroll
    for (int m = 0; m < W; ++m) {
      Py.v[m] = psi_of<T, EXACT>(v[m], bh, Py.v[m], ch, dzx[m], p.dx, p.rdx);
      h1[m] = A::add(h1[m], A::mul(db, Py.v[m]));
    }
    st4(py, Py.v);
    if (mhz) {
      T *const pz = p.psi[HZ][AX][side] + oa;
      VW<T, W> Pz;
      ldw4(Pz, pz);
      T v[W];
      if constexpr (EXACT) psi4<T, EXACT, W>(v, bh, Pz.v, ch, dyx, p.dx, p.rdx, dok);
#pragma unroll
      for (int m = 0; m < W; ++m) {
        Pz.v[m] = psi_of<T, EXACT>(v[m], bh, Pz.v[m], ch, dyx[m], p.dx, p.rdx);
        h2[m] = A::sub(h2[m], A::mul(db, Pz.v[m]));
      }
      st4(pz, Pz.v);
    }
  }
  if (mhx && (q = h_slab(j, p.jb, p.je, P, d, side)) >= 0) {  // update_pml_hx_yinc, update_pml_hz_yinc
    const long long oa = ((long long)i * P + d) * p.psy + k0;
    const T bh = p.bh[q], ch = p.ch[q];
    T *const px = p.psi[HX][AY][side] + oa;
    VW<T, W> Px;
    ldw4(Px, px);
    T v[W];
    if constexpr (EXACT) psi4<T, EXACT, W>(v, bh, Px.v, ch, dzy, p.dx, p.rdx, dok);
#pragma unroll
    for (int m = 0; m < W; ++m) {
      Px.v[m] = psi_of<T, EXACT>(v[m], bh, Px.v[m], ch, dzy[m], p.dx, p.rdx);
      h0[m] = A::sub(h0[m], A::mul(db, Px.v[m]));
    }
    st4(px, Px.v);
    if (mhz) {
      T *const pz = p.psi[HZ][AY][side] + oa;
      VW<T, W> Pz;
      ldw4(Pz, pz);
      T v[W];
      if constexpr (EXACT) psi4<T, EXACT, W>(v, bh, Pz.v, ch, dxy, p.dx, p.rdx, dok);
#pragma unroll
      for (int m = 0; m < W; ++m) {
        Pz.v[m] = psi_of<T, EXACT>(v[m], bh, Pz.v[m], ch, dxy[m], p.dx, p.rdx);
        h2[m] = A::add(h2[m], A::mul(db, Pz.v[m]));
      }
      st4(pz, Pz.v);
    }
  }
  if (mhx) st4(hx + o, h0);
  if (mhy) st4(hy + o, h1);
  if (mhz) st4(hz + o, h2);
  // port planes: raw Hx, Hy at k = port and port + 1
#pragma unroll
  for (int pq = 0; pq < 2; ++pq) {
    const int dm = p.port_pos[pq] - k0;
    if ((unsigned)(dm + 1) < W + 1u) {  // k = port or port + 1 among the group's cells
      const long long pc = (long long)i * p.ny + j;
#pragma unroll
      for (int m = 0; m < W; ++m) {
        if (m == dm) {
          if (mhx) capture(p, s, pq, 2, pc, h0[m]);
          if (mhy) capture(p, s, pq, 4, pc, h1[m]);
        }
        if (m == dm + 1) {
          if (mhx) capture(p, s, pq, 3, pc, h0[m]);
          if (mhy) capture(p, s, pq, 5, pc, h1[m]);
        }
      }
    }
  }
}

template <typename T, bool EXACT, bool SRC>
__global__ void __launch_bounds__(kVecThreads, kVecBlocksPerSME<T, EXACT>) k_v3_e(const __grid_constant__ Params<T> p, VecGeom g, int s) {
  pdl_wait();
  v3_e_block<T, EXACT, kVecW<T>, SRC>(p, g, p.ib + blockIdx.y, blockIdx.x, s);
}

template <typename T, bool EXACT>
__global__ void __launch_bounds__(kVecThreads, kVecBlocksPerSM<T, EXACT>) k_v3_h(Params<T> p, VecGeom g, int s) {
  pdl_wait();
  v3_h_block<T, EXACT, false, kVecW<T>>(p, g, p.ie - 1 - blockIdx.y, blockIdx.x, s);
}

// ---------------------------------------------------------------------------
// Ordered form: one launch per time step runs both half-steps, plane by
// plane: E(0) .. E(D-1), then for q = 0 .. n-1 the pair E(q+D) (while q+D <
// n), H(q) -- a unit of nb blocks each, n = ie - ib updated planes, q = i -
// ib, D the lag (wave.lag).  H(q) reads new E of planes q and q-1 and
// overwrites the H of plane q that E(q) and E(q-1) read, so its blocks wait
// until every block of E(q) and E(q-1) has finished; no other dependence
// exists inside a step.  A block's place in the order is its block index; the
// hardware dispatches a 1D grid in increasing block index, so the E blocks an
// H block waits for were dispatched D units or more earlier, and those never
// wait: the waits end, and with the lag they are rarely needed at all.  Each
// wait is bounded (kWaitCycles); on expiry the block records state[1] = 2
// and returns without updating, and oidt_job_sync reports the job as timed
// out -- should a dependence ever not be resident, the launch ends with that
// error instead of hanging.  H blocks read E through L2 (another SM's L1 may
// hold lines written in this launch).  The new E of planes q and q-1 and the
// H of plane q were touched D units earlier, and D is chosen so that D planes
// of the step's arrays fit in L2: H reads them from L2 and DRAM carries each
// field word about once per step.
// ---------------------------------------------------------------------------
struct WaveArgs {
  int *done;  // [n]: E blocks finished per plane, summed over the steps run
  int nb;     // blocks per plane and half-step (vector + edge role)
  int lag;    // D, 1 <= D <= n
};

// __grid_constant__, as in k_v3_e: v3_src_e takes the parameters by reference,
// and of a plain by-value parameter each thread would keep a copy of 1 KB in
// local memory (128 x 128 x 256 float32 393 us per step with it, 82 without).
template <typename T, bool EXACT, bool SRC>
__global__ void __launch_bounds__(kVecThreads, sizeof(T) == 4 ? kVecBlocksPerSM<T, EXACT> : 3)
    k_v3_wave(const __grid_constant__ Params<T> p, VecGeom g, WaveArgs w, int s) {
  pdl_wait();
  __shared__ int s_ok;
  const int n = p.ie - p.ib, D = w.lag;
  const int u = (int)(blockIdx.x / w.nb), bx = (int)(blockIdx.x - (unsigned)u * w.nb);
  bool is_h;
  int q;
  if (u < D) {
    is_h = false;
    q = u;
  } else if (u < D + 2 * (n - D)) {
    const int r = u - D;
    is_h = r & 1;
    q = is_h ? r >> 1 : (r >> 1) + D;
  } else {
    is_h = true;
    q = n - D + (u - D - 2 * (n - D));
  }
  if (!is_h) {
    v3_e_block<T, EXACT, 4, SRC>(p, g, p.ib + q, bx, s);
    __threadfence();  // this thread's stores visible to the whole GPU ...
    __syncthreads();  // ... for every thread of the block, before the count
    if (threadIdx.x == 0) atomicAdd(w.done + q, 1);
    return;
  }
  if (threadIdx.x == 0) {
    s_ok = 1;
    const int want = (int)(((long long)p.state[0] + s + 1) * w.nb);  // counts after this step's E
    const long long t0 = clock64();
    for (int d = 0; d < 2 && q - d >= 0 && s_ok; ++d)
      while (ld_acquire(w.done + (q - d)) < want)
        if (clock64() - t0 > kWaitCycles) {
          atomicExch(p.state + 1, 2);  // reported to the host by oidt_job_sync
          s_ok = 0;
          break;
        }
  }
  __syncthreads();
  if (s_ok) v3_h_block<T, EXACT, true, 4>(p, g, p.ib + q, bx, s);
}

}  // namespace oidt
