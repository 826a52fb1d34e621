// strip2d.cuh -- 2D TM / TE time steps in tiles, float32 fast arithmetic.
//
// The tile form of tile2d.cuh with strips of cells per thread and a lighter
// exchange between tiles; the grid advances in sub-blocks of up to `halo`
// steps, a launch covering one sub-block or a whole ring block of them.
//
// * The grid is cut into tiles, one block each.  Block (bi, bj) owns the
//   cells [oi0, oi1) x [oj0, oj1) and also computes `halo` cells on every side
//   of them ([wi0, wi1) x [wj0, wj1), clipped to the grid).  A step's E half
//   reads H at (i + 1, j) and (i, j + 1), its H half E at (i - 1, j) and
//   (i, j - 1), so after s steps the cells a block holds are exact s cells
//   inside the held tile's edges (and up to the grid's edges, where there is
//   nothing to read): after cnt <= halo steps the owned cells are exact.
// * A thread holds a strip of C cells of one column (C consecutive rows; lanes
//   run along the rows' contiguous axis), fields and CPML psi in registers
//   through the whole launch.  A strip's neighbours along x are its own
//   registers except at its ends, so it publishes in shared memory all rows of
//   the fields read along y and one row of the field read along x.  The cells'
//   updates of a half-step are one straight run (their chains overlap); what
//   few cells need -- source, slabs, captures, values kept where a component
//   is not updated -- is behind one branch a half-step.  A block of 512
//   threads holds up to 2048 cells, twice the one-cell form's 1024.
// * A launch of one sub-block (cnt <= halo) reads one field / psi buffer and
//   writes its owned cells to the other, so no block sees cells another has
//   advanced; a grid with more tiles than the GPU holds runs in waves.
// * A launch of several sub-blocks is cooperative (all tiles resident at
//   once).  Between sub-blocks a tile needs its halo cells from its (up to 8)
//   neighbours, which own them.  They cross through an exchange buffer whose
//   64-bit words carry a value beside the number of the sub-block that wrote
//   it: the reader polls the data word itself until the number is the one it
//   waits for.  A 64-bit access is single-copy atomic, so no fence, flag or
//   barrier orders data against a flag.  The loads of a poll are predicated,
//   not branched around, so all are in flight together.  Two buffers
//   alternate: a tile writes sub-block b + 1's words over those of b - 1 only
//   after it has read its neighbours' b, which they publish after reading its
//   b - 1.  Each wait is bounded (p.wait_cycles); on expiry the block records
//   state[1] = 3 and goes on without waiting again.
//
// What bounds it: latency -- two block barriers and a dependent chain a step,
// an L2 store and load a crossing.  Strips of four hold twice the cells of a
// block and hide the chain; strips of one have the shorter half-step, for
// grids of which 148 tiles hold a thread's worth a cell (engine.cu,
// strip_plan).  Measured on a B200 (advances of 2560 steps, folds included)
// against the one-cell form with its state exchanged through global memory
// behind counters: 613 x 227 1.57 against 3.46 us per step (that form ran in
// waves there), 675 x 141 1.46 / 2.99, TE 1.71 / 3.14, 400 x 200 1.13 / 1.81,
// 603 x 1601 10.9 / 21.7.
//
// float64 and EXACT runs stay in tile2d.cuh's one-cell form: with strips their
// registers spill (400 x 200, us per step: float64 fast 2.20, EXACT 3.57; the
// one-cell form 2.05 and 2.87 then, 1.64 and 2.30 now).
//
// Per cell the arithmetic is that of kernels.cuh's tm2_e_cell / tm2_h_cell /
// te2_e_cell / te2_h_cell (the reference's fdtd_funcs.py of FDTD_2D_TM and
// FDTD_2D_TE, lines 43-124, in its launch order), operation for operation, so
// a run equals the per-cell launches' bit for bit; halo cells are computed
// with the same operations and never written back.
#pragma once

#include "tile2d.cuh"

namespace oidt {

constexpr int kStripThreads = 512;  // threads of a block at most (128 registers each; one-cell strips: twice)
constexpr int kStripCells = 4;      // cells of a thread's strip at most
constexpr int kStripHaloMax = 8;    // steps per sub-block at most

struct StripArgs {
  int s0;      // ring slot of the launch's first step
  int cnt;     // steps of this launch (more than halo: a cooperative launch of several sub-blocks)
  int ti, tj;  // owned tile extent: rows (x), columns (y)
  int gj;      // tiles along y
  int halo;    // cells computed on each side of the owned tile; steps per sub-block
  int cells;   // cells of a thread's strip: 1 or 4
  int threads; // of a block
  int *epoch;  // per tile: sub-blocks completed (cooperative launches)
  unsigned long long *xch;  // exchange words, two buffers ...
  long long xbuf;           // ... of xbuf words
};

// Shared memory of a block: three fields of rows x cols held cells (rows
// rounded up to whole strips), row and column tables [6] each and the source
// samples of the launch's steps.
inline size_t strip2d_smem(int rows, int cols, int C, int steps) {
  const size_t r = (size_t)(rows + C - 1) / C * C;
  return (3 * r * cols + 6 * r + 6 * (size_t)cols + steps) * sizeof(float);
}
// Exchange words of a job (64-bit), two buffers of: f0, f1 [nx ny][2], x-slab
// psi of E, H [side][P][ny][2], y-slab psi [side][nx][P][2], f2 [nx ny].
inline size_t strip2d_xch_buf(long long nx, long long ny, long long P) { return (size_t)((3 * nx * ny + 4 * P * (nx + ny) + 1) / 2 * 2); }

// Cell flags.  TM: E1 = Ez update, H1 = Hx, H2 = Hy; TE: E1 = Ex, E2 = Ey,
// H1 = Hz.  XE / YE / XH / YH: the cell's component is in the E / H x- /
// y-slab of the CPML (and updated).  CE, CH, CN: the cell's E (ring slot 0)
// and H (slot 1) on a port's line x = port, its H (slot 2) on x = port + 1,
// are captured.  kOwn: owned; kBand: owned and held by a neighbour tile;
// kHeld: held; kRim: some component is not updated.
enum : unsigned {
  kS_E1 = 1u, kS_E2 = 2u, kS_H1 = 4u, kS_H2 = 8u, kS_Src = 16u, kS_XE = 32u, kS_YE = 64u, kS_XH = 128u, kS_YH = 256u,
  kS_CE = 512u, kS_CH = 1024u, kS_CN = 2048u, kS_Own = 4096u, kS_Band = 8192u, kS_Held = 16384u, kS_Rim = 32768u
};

template <int MODE, int C>
__global__ void __launch_bounds__(C == 1 ? 2 * kStripThreads : kStripThreads, 1)
    k_2d_strip(const __grid_constant__ Params<float> p, StripArgs a) {
  using A = Ar<float, false>;
  constexpr bool TM = MODE == OIDT_MODE_TM2;
  // fields f0, f1 (E in TE, H in TM), f2 (H); the fields carrying each psi array
  constexpr int FA = TM ? EZ : EX, FB = TM ? HX : EY, FC = TM ? HY : HZ;
  constexpr int EXS = TM ? EZ : EY, EYS = TM ? EZ : EX, HXS = TM ? HY : HZ, HYS = TM ? HX : HZ;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int nx = p.nx, ny = p.ny, P = p.P, H = a.halo;
  const int bi = (int)blockIdx.x / a.gj, bj = (int)blockIdx.x - bi * a.gj;
  const int oi0 = bi * a.ti, oi1 = min(nx, oi0 + a.ti), oj0 = bj * a.tj, oj1 = min(ny, oj0 + a.tj);
  const int wi0 = max(0, oi0 - H), wi1 = min(nx, oi1 + H), wj0 = max(0, oj0 - H), wj1 = min(ny, oj1 + H);
  const int nrow = wi1 - wi0, ncol = wj1 - wj0, nst = (nrow + C - 1) / C, M = nst * ncol, nh = C * M;
  float *const F0 = reinterpret_cast<float *>(smem_raw), *const F1 = F0 + nh, *const F2 = F1 + nh;
  float *const RT = F2 + nh;           // [rows][6]: 1 / (kappa dx) of E and H along x, CPML be ce bh ch
  float *const CT = RT + 6 * nst * C;  // [6][columns], the same along y
  float *const JS = CT + 6 * ncol;     // source samples of the launch's steps
  const int t = threadIdx.x;
  const bool act = t < M;
  const int tr = act ? t / ncol : 0, tc = act ? t - tr * ncol : 0;
  const int l0 = tr * C, i0 = wi0 + l0, j = wj0 + tc;  // the strip's first row (held, grid) and its column
  // in the shared fields cell q of thread t is at q M + t: a warp's accesses are 32 consecutive words
  const int sc = act ? t : 0;
  int g0 = i0 * ny + j;                                // ... and in the [nx][ny] arrays (2^31 cells at most)
  auto table = [&](float *r, int stride, int k, int axis, int b, int e) {
    int d, side;
    const int qe = e_slab(k, b, e, P, d, side), qh = h_slab(k, b, e, P, d, side);
    r[0] = __ldg(p.rkd[axis] + k);
    r[stride] = __ldg(p.rkd[axis + 3] + k);
    r[2 * stride] = qe >= 0 ? __ldg(p.be + qe) : 0.0f;
    r[3 * stride] = qe >= 0 ? __ldg(p.ce + qe) : 0.0f;
    r[4 * stride] = qh >= 0 ? __ldg(p.bh + qh) : 0.0f;
    r[5 * stride] = qh >= 0 ? __ldg(p.ch + qh) : 0.0f;
  };
  for (int u = t; u < nst * C; u += blockDim.x) table(RT + 6 * u, 1, min(wi0 + u, nx - 1), 0, p.ib, p.ie);
  for (int u = t; u < ncol; u += blockDim.x) table(CT + u, ncol, wj0 + u, 1, p.jb, p.je);
  int dy = 0, sy = 0, qye = -1, qyh = -1;  // the column's y slab: layer, side, E and H coefficient
  if (act) {
    qye = e_slab(j, p.jb, p.je, P, dy, sy);
    qyh = h_slab(j, p.jb, p.je, P, dy, sy);  // an E-slab column: same layer and side
  }
  // ---- the cells' constants ---------------------------------------------------------------
  unsigned fl[C], any = 0;
  float cbA[C], cbB[TM ? 1 : C];  // dt/eps of the cells' E components
  int cport = 0;                  // the port whose lines the strip's rows meet
#pragma unroll
  for (int q = 0; q < C; ++q) {
    const int i = i0 + q;
    unsigned f = 0;
    cbA[q] = 0.0f;
    if (!TM) cbB[TM ? 0 : q] = 0.0f;
    if (act && l0 + q < nrow) {
      int d, side;
      f |= kS_Held;
      const bool own = i >= oi0 && i < oi1 && j >= oj0 && j < oj1;
      if (own) f |= kS_Own;
      if (own && (i - oi0 < H || oi1 - i <= H || j - oj0 < H || oj1 - j <= H)) f |= kS_Band;
      // (a halo cell on the tile's edge updates from whatever the neighbour's place holds: it is
      // no more off than a cell left alone, and neither reaches an owned cell within `halo` steps)
      const bool ic = i >= p.ib && i < p.ie, io = i > p.ib && i < p.ie;
      const bool jc = j >= p.jb && j < p.je, jo = j > p.jb && j < p.je;
      if (TM) {
        if (ic && jc) f |= kS_E1;  // update_ez :44-49
        if (ic && jo) f |= kS_H1;  // update_hx :53-58
        if (io && jc) f |= kS_H2;  // update_hy :62-67
        if (in_src(p, EZ, i, j, 0)) f |= kS_Src;
        cbA[q] = __ldg(p.cb[2] + g0 + q * ny);
      } else {
        if (io && jc) f |= kS_E1;  // update_ex :43-49
        if (ic && jo) f |= kS_E2;  // update_ey :52-58
        if (io && jo) f |= kS_H1;  // update_hz :61-67
        if (in_src(p, HZ, i, j, 0)) f |= kS_Src;
        cbA[q] = __ldg(p.cb[0] + g0 + q * ny);
        cbB[TM ? 0 : q] = __ldg(p.cb[1] + g0 + q * ny);
      }
      constexpr unsigned kAll = TM ? kS_E1 | kS_H1 | kS_H2 : kS_E1 | kS_E2 | kS_H1, kEx = TM ? kS_E1 : kS_E2,
                         kHx = TM ? kS_H2 : kS_H1;  // the components with x slabs
      if ((f & kAll) != kAll) f |= kS_Rim;
      if ((f & kEx) && e_slab(i, p.ib, p.ie, P, d, side) >= 0) f |= kS_XE;
      if ((f & kHx) && h_slab(i, p.ib, p.ie, P, d, side) >= 0) f |= kS_XH;
      if ((f & kS_E1) && qye >= 0) f |= kS_YE;
      if ((f & kS_H1) && qyh >= 0) f |= kS_YH;
      if (!(f & (TM ? kS_E1 : kS_H1))) f &= ~kS_Src;
      for (int port = 0; port < 2 && own; ++port) {
        const int x = p.port_pos[port];
        if (i == x || i == x + 1) cport = port;
        if (i == x && (f & kEx)) f |= kS_CE;
        if (i == x && (f & kHx)) f |= kS_CH;
        if (i == x + 1 && (f & kHx)) f |= kS_CN;
      }
    }
    fl[q] = f;
    any |= f;
  }
  const float db = p.db, dx = p.dx, rdx = p.rdx;
  const int nsub = (a.cnt + H - 1) / H;
  // a cell's place in the x-slab [side][P][ny] and y-slab [side][nx][P] psi arrays
  auto xoff = [&](int i, int &side) {
    side = i < p.ib + P ? 0 : 1;
    return (side ? i - p.ie + P : i - p.ib) * ny + j;
  };
  __syncthreads();
  pdl_wait();  // the previous launch's state is complete (and visible) from here on
  if (p.src_field >= 0) {
    const int n0 = p.state[0] + a.s0;
    for (int u = t; u < a.cnt; u += blockDim.x) JS[u] = __ldg(p.jsrc + n0 + u);
  }
  const unsigned e0 = nsub > 1 ? (unsigned)a.epoch[blockIdx.x] : 0u;  // equal for every tile at launch
  float f0[C], f1[C], f2[C], xe[C], ye[C], xh[C], yh[C];  // the cells' values
#pragma unroll
  for (int q = 0; q < C; ++q) {
    f0[q] = f1[q] = f2[q] = xe[q] = ye[q] = xh[q] = yh[q] = 0.0f;
    if (fl[q] & kS_Held) {
      const int g = g0 + q * ny;
      f0[q] = __ldcg(p.f[FA] + g);
      f1[q] = __ldcg(p.f[FB] + g);
      f2[q] = __ldcg(p.f[FC] + g);
      int side = 0;
      const int ox = xoff(i0 + q, side), oy = (i0 + q) * P + dy;
      if (fl[q] & kS_XE) xe[q] = __ldcg(p.psi[EXS][AX][side] + ox);
      if (fl[q] & kS_XH) xh[q] = __ldcg(p.psi[HXS][AX][side] + ox);
      if (fl[q] & kS_YE) ye[q] = __ldcg(p.psi[EYS][AY][sy] + oy);
      if (fl[q] & kS_YH) yh[q] = __ldcg(p.psi[HYS][AY][sy] + oy);
    }
    if (act) {
      F0[sc + q * M] = f0[q];
      F1[sc + q * M] = f1[q];
      F2[sc + q * M] = f2[q];
    }
  }
  __syncthreads();
  // The step's ring slots of the strip's port.  Ports no more than C rows apart may both meet a strip: then
  // every captured row is tested against both.
  const int pslot = p.nslot * (int)p.plane, plane = (int)p.plane;
  const bool near = abs(p.port_pos[0] - p.port_pos[1]) <= C;
  float *ring = p.ring + (long long)a.s0 * 2 * pslot + (near ? 0 : cport * pslot) + j;
  auto capture_near = [&](int q, bool h, float v) {
    for (int port = 0; port < 2; ++port) {
      const int dm = i0 + q - p.port_pos[port];
      if (!h && dm == 0) ring[port * pslot] = v;
      if (h && (unsigned)dm < 2u) ring[port * pslot + (1 + dm) * plane] = v;
    }
  };
  // the cells below and above the strip (outside the tile: not an exact cell's)
  const int sc_dn = min(sc + ncol, M - 1), sc_up = max(sc - ncol, 0) + (C - 1) * M;
  const float *const rt = RT + 6 * l0, *const ct = CT + tc;
  const float rkye = ct[0], rkyh = ct[ncol];
  bool waits = true;
  for (int sb = 0; sb < nsub; ++sb) {
    const int s1 = min(a.cnt, (sb + 1) * H);
    for (int s = sb * H; s < s1; ++s) {
      float e[C], e2[C], dA[C], dB[C];  // new values; the differences along x and along y
      // ---- E half-step ------------------------------------------------------------------
      if (TM) {
        const float hyn = F2[sc_dn];
#pragma unroll
        for (int q = 0; q < C; ++q) {  // update_ez :44-49
          dA[q] = A::sub(q < C - 1 ? f2[q + 1 < C ? q + 1 : 0] : hyn, f2[q]);
          dB[q] = A::sub(F1[sc + q * M + 1], f1[q]);
          e[q] = A::curl(f0[q], cbA[q], dA[q], 0.0f, rt[6 * q], dB[q], 0.0f, rkye);
        }
      } else {
        const float hzn = F2[sc_dn];
#pragma unroll
        for (int q = 0; q < C; ++q) {  // update_ex :43-49, update_ey :52-58
          dA[q] = A::sub(f2[q], q < C - 1 ? f2[q + 1 < C ? q + 1 : 0] : hzn);
          dB[q] = A::sub(F2[sc + q * M + 1], f2[q]);
          e[q] = A::step(f0[q], cbA[q], dB[q], 0.0f, rkye);
          e2[q] = A::step(f1[q], cbB[TM ? 0 : q], dA[q], 0.0f, rt[6 * q]);
        }
      }
      if (any & (kS_Src | kS_XE | kS_YE | kS_Rim)) {
        if (TM && (any & kS_Src))
#pragma unroll
          for (int q = 0; q < C; ++q)
            if (fl[q] & kS_Src) e[q] = A::sub(e[q], JS[s]);  // update_source :71-76
        if (any & kS_XE)
#pragma unroll
          for (int q = 0; q < C; ++q)
            if (fl[q] & kS_XE) {  // update_pml_ez_xinc :80-88, update_pml_ey_xinc :91-99
              xe[q] = A::psi(rt[6 * q + 2], xe[q], rt[6 * q + 3], TM ? dA[q] : -dA[q], dx, rdx);
              if (TM) e[q] = A::inc(e[q], cbA[q], xe[q]);
              else e2[q] = A::dec(e2[q], cbB[TM ? 0 : q], xe[q]);
            }
        if (any & kS_YE)
#pragma unroll
          for (int q = 0; q < C; ++q)
            if (fl[q] & kS_YE) {  // update_pml_ez_yinc :92-100, update_pml_ex_yinc :79-87
              ye[q] = A::psi(ct[2 * ncol], ye[q], ct[3 * ncol], dB[q], dx, rdx);
              e[q] = TM ? A::dec(e[q], cbA[q], ye[q]) : A::inc(e[q], cbA[q], ye[q]);
            }
        if (any & kS_Rim)
#pragma unroll
          for (int q = 0; q < C; ++q) {
            e[q] = (fl[q] & kS_E1) ? e[q] : f0[q];
            if (!TM) e2[q] = (fl[q] & kS_E2) ? e2[q] : f1[q];
          }
      }
#pragma unroll
      for (int q = 0; q < C; ++q) {
        f0[q] = e[q];
        if (!TM) f1[q] = e2[q];
        if (act) F0[sc + q * M] = f0[q];
      }
      if (!TM && act) F1[sc + (C - 1) * M] = f1[C - 1];
      if (any & kS_CE)
#pragma unroll
        for (int q = 0; q < C; ++q)
          if (fl[q] & kS_CE) {
            if (near) capture_near(q, false, TM ? f0[q] : f1[q]);
            else *ring = TM ? f0[q] : f1[q];
          }
      __syncthreads();
      // ---- H half-step ------------------------------------------------------------------
      if (TM) {
        const float ezu = F0[sc_up];
#pragma unroll
        for (int q = 0; q < C; ++q) {  // update_hx :53-58, update_hy :62-67
          dB[q] = A::sub(F0[max(sc + q * M - 1, 0)], f0[q]);
          dA[q] = A::sub(f0[q], q > 0 ? f0[q > 0 ? q - 1 : 0] : ezu);
          e[q] = A::step(f1[q], db, dB[q], 0.0f, rkyh);
          e2[q] = A::step(f2[q], db, dA[q], 0.0f, rt[6 * q + 1]);
        }
      } else {
        const float eyu = F1[sc_up];
#pragma unroll
        for (int q = 0; q < C; ++q) {  // update_hz :61-67
          dB[q] = A::sub(f0[q], F0[max(sc + q * M - 1, 0)]);
          dA[q] = A::sub(f1[q], q > 0 ? f1[q > 0 ? q - 1 : 0] : eyu);
          e2[q] = A::curl(f2[q], db, dB[q], 0.0f, rkyh, dA[q], 0.0f, rt[6 * q + 1]);
        }
      }
      if (any & (kS_Src | kS_XH | kS_YH | kS_Rim)) {
        if (!TM && (any & kS_Src))
#pragma unroll
          for (int q = 0; q < C; ++q)
            if (fl[q] & kS_Src) e2[q] = A::sub(e2[q], JS[s]);  // source after update_hz
        if (any & kS_XH)
#pragma unroll
          for (int q = 0; q < C; ++q)
            if (fl[q] & kS_XH) {  // update_pml_hy_xinc :116-124, update_pml_hz_xinc :103-111
              xh[q] = A::psi(rt[6 * q + 4], xh[q], rt[6 * q + 5], dA[q], dx, rdx);
              e2[q] = TM ? A::inc(e2[q], db, xh[q]) : A::dec(e2[q], db, xh[q]);
            }
        if (any & kS_YH)
#pragma unroll
          for (int q = 0; q < C; ++q)
            if (fl[q] & kS_YH) {  // update_pml_hx_yinc :104-112, update_pml_hz_yinc :115-123
              yh[q] = A::psi(ct[4 * ncol], yh[q], ct[5 * ncol], TM ? -dB[q] : dB[q], dx, rdx);
              if (TM) e[q] = A::dec(e[q], db, yh[q]);
              else e2[q] = A::inc(e2[q], db, yh[q]);
            }
        if (any & kS_Rim)
#pragma unroll
          for (int q = 0; q < C; ++q) {
            if (TM) e[q] = (fl[q] & kS_H1) ? e[q] : f1[q];
            e2[q] = (fl[q] & (TM ? kS_H2 : kS_H1)) ? e2[q] : f2[q];
          }
      }
#pragma unroll
      for (int q = 0; q < C; ++q) {
        if (TM) f1[q] = e[q];
        f2[q] = e2[q];
        if (act) (TM ? F1 : F2)[sc + q * M] = TM ? f1[q] : f2[q];
      }
      if (TM && act) F2[sc] = f2[0];
      if (any & (kS_CH | kS_CN))
#pragma unroll
        for (int q = 0; q < C; ++q) {
          if (near) {
            if (fl[q] & (kS_CH | kS_CN)) capture_near(q, true, f2[q]);
          } else {
            if (fl[q] & kS_CH) ring[plane] = f2[q];
            if (fl[q] & kS_CN) ring[2 * plane] = f2[q];
          }
        }
      ring += 2 * pslot;
      __syncthreads();
    }
    if (sb == nsub - 1) break;
    // ---- between sub-blocks: publish the owned cells other tiles hold, fetch the halo cells ----
    const unsigned n = e0 + sb + 1;
    asm volatile("" : "+r"(g0), "+r"(dy));  // the exchange addresses are formed here, not held through the steps
    const int N = nx * ny, SX = 2 * P * ny, SY = 2 * nx * P;
    unsigned long long *const xb = a.xch + ((n & 1) ? a.xbuf : 0);
    unsigned long long *const x01 = xb + 2 * (long long)g0, *const x2 = xb + 2 * (long long)(N + SX + SY) + g0;
    auto psi_x = [&](int q) {  // the cell's x-slab and y-slab words
      int side = 0;
      const int o = xoff(i0 + q, side);
      return xb + 2 * (long long)(N + o + side * P * ny);
    };
    auto psi_y = [&](int q) { return xb + 2 * (long long)(N + SX + (i0 + q) * P + dy + sy * nx * P); };
#pragma unroll
    for (int q = 0; q < C; ++q)
      if (fl[q] & kS_Band) {
        xch_put(x01 + 2 * q * ny, f0[q], f1[q], n);
        xch_put(x2 + q * ny, f2[q], n);
        if (fl[q] & (kS_XE | kS_XH)) xch_put(psi_x(q), xe[q], xh[q], n);
        if (fl[q] & (kS_YE | kS_YH)) xch_put(psi_y(q), ye[q], yh[q], n);
      }
    bool need = false, psi = false;
#pragma unroll
    for (int q = 0; q < C; ++q)
      if ((fl[q] & (kS_Held | kS_Own)) == kS_Held) {
        need = true;
        psi |= (fl[q] & (kS_XE | kS_YE | kS_XH | kS_YH)) != 0;
      }
    if (need) {
      const long long t0 = clock64();
      unsigned round = 0;
      for (;;) {
        bool ok = true;
        unsigned long long w[C][4] = {};
#pragma unroll
        for (int q = 0; q < C; ++q) {
          const bool on = (fl[q] & (kS_Held | kS_Own)) == kS_Held;
          xch_load2(w[q], x01 + 2 * q * ny, on);
          xch_load(w[q][2], x2 + q * ny, on);
        }
#pragma unroll
        for (int q = 0; q < C; ++q) {
          const bool on = (fl[q] & (kS_Held | kS_Own)) == kS_Held;
          ok &= xch_take(w[q][0], f0[q], n, on);
          ok &= xch_take(w[q][1], f1[q], n, on);
          ok &= xch_take(w[q][2], f2[q], n, on);
        }
        if (psi) {
#pragma unroll
          for (int q = 0; q < C; ++q) {
            const bool on = (fl[q] & (kS_Held | kS_Own)) == kS_Held;
            xch_load2(w[q], psi_x(q), on && (fl[q] & (kS_XE | kS_XH)));
            xch_load2(w[q] + 2, psi_y(q), on && (fl[q] & (kS_YE | kS_YH)));
          }
#pragma unroll
          for (int q = 0; q < C; ++q) {
            const bool on = (fl[q] & (kS_Held | kS_Own)) == kS_Held;
            const bool ox = on && (fl[q] & (kS_XE | kS_XH)), oy = on && (fl[q] & (kS_YE | kS_YH));
            ok &= xch_take(w[q][0], xe[q], n, ox);
            ok &= xch_take(w[q][1], xh[q], n, ox);
            ok &= xch_take(w[q][2], ye[q], n, oy);
            ok &= xch_take(w[q][3], yh[q], n, oy);
          }
        }
        if (ok || !waits) break;
        if (clock64() - t0 > p.wait_cycles) {
          atomicExch(p.state + 1, 3);  // reported to the host by oidt_job_sync
          waits = false;
        } else if (++round % 64 == 0 && ld_acquire(p.state + 1) != 0) {  // an earlier wait expired: stop waiting
          waits = false;
        }
      }
#pragma unroll
      for (int q = 0; q < C; ++q)
        if ((fl[q] & (kS_Held | kS_Own)) == kS_Held) {
          F0[sc + q * M] = f0[q];
          F1[sc + q * M] = f1[q];
          F2[sc + q * M] = f2[q];
        }
    }
    __syncthreads();
  }
  // ---- owned cells to the other buffer ------------------------------------------------------
#pragma unroll
  for (int q = 0; q < C; ++q)
    if (fl[q] & kS_Own) {
      const int g = g0 + q * ny;
      p.fn[FA][g] = f0[q];
      p.fn[FB][g] = f1[q];
      p.fn[FC][g] = f2[q];
      int side = 0;
      const int ox = xoff(i0 + q, side), oy = (i0 + q) * P + dy;
      if (fl[q] & kS_XE) p.psin[EXS][AX][side][ox] = xe[q];
      if (fl[q] & kS_YE) p.psin[EYS][AY][sy][oy] = ye[q];
      if (fl[q] & kS_XH) p.psin[HXS][AX][side][ox] = xh[q];
      if (fl[q] & kS_YH) p.psin[HYS][AY][sy][oy] = yh[q];
    }
  if (nsub > 1 && t == 0) a.epoch[blockIdx.x] = (int)(e0 + nsub);
}

}  // namespace oidt
