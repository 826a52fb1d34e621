// tile2d.cuh -- 2D TM / TE time steps, temporally blocked in tiles: float64 and
// EXACT runs (float32 fast runs: strip2d.cuh).
//
// A 2D job of the served sizes (a few hundred x a few hundred cells) is too
// small to fill the GPU, so with one launch per half-step its step time is
// launch latency.  Here the grid advances in sub-blocks of up to `halo` steps,
// a launch covering one sub-block or a whole ring block of them:
//
// * The grid is cut into tiles, one block each.  Block (bi, bj) owns the
//   cells [oi0, oi1) x [oj0, oj1) and also computes `halo` cells on every side
//   of them ([wi0, wi1) x [wj0, wj1), clipped to the grid).  A step's E half
//   reads H at (i + 1, j) and (i, j + 1), its H half E at (i - 1, j) and
//   (i, j - 1), so after s steps the cells a block holds are exact s cells
//   inside the held tile's edges (and up to the grid's edges, where there is
//   nothing to read): after cnt <= halo steps the owned cells are exact.
// * A held tile has at most kTileThreads cells, one per thread.  A thread
//   works out its cell's update conditions, CPML slab coefficients and dt/eps
//   values once per launch and keeps them in registers, and so its cell's
//   three field values and CPML psi values through a sub-block of up to
//   `halo` steps.  Shared memory holds the tile's fields only for the
//   neighbours' reads (each value written once per half-step by its cell's
//   thread), the CPML coefficient tables, and the kappa dx divisors with
//   their reciprocals for the tile's rows and columns; __syncthreads
//   separates the half-steps.
// * A launch of one sub-block (cnt <= halo) reads one field / psi buffer and
//   writes its owned cells to the other, so no block sees cells another has
//   advanced; a grid with more tiles than SMs simply runs in waves.
// * A launch of several sub-blocks is cooperative (all tiles resident at
//   once).  Between sub-blocks only what other tiles read moves: a tile puts
//   its owned cells within `halo` of its edges (fields and psi) into the
//   exchange words and polls its halo cells' words, which their tiles (up to
//   8, as halo width <= tile extent) put there; everything else stays in
//   registers, and the owned cells are stored once, after the last sub-block.
//   Two buffers of words alternate: a tile writes sub-block b + 1's words over
//   those of b - 1 only after it has read its neighbours' b, which they put
//   after reading its b - 1.  Each wait is bounded (p.wait_cycles); on expiry
//   the block records state[1] = 3 and goes on without waiting again.
//
// What bounds it: latency -- two block barriers and a dependent chain a step,
// an L2 store and load a crossing.  A crossing through the field buffers
// behind per-tile counters (fence, release, acquire, then the loads) took 3.5 us
// where the words take 2.1.  Measured on a B200, 400 x 200 float64 in sub-blocks
// of 4: EXACT 2.95 -> 2.62 us per step with the words, -> 2.45 with the range
// test on the integer pipe (kernels.cuh, Ar), -> 2.30 without spills in the
// steps; fast 2.09 -> 1.64 with the words and without spills.
//
// Per cell the arithmetic is that of kernels.cuh's tm2_e_cell / tm2_h_cell /
// te2_e_cell / te2_h_cell (the reference's fdtd_funcs.py of FDTD_2D_TM and
// FDTD_2D_TE, lines 43-124, in its launch order), operation for operation, so
// EXACT runs equal the reference and the oracle bit for bit; halo cells are
// computed with the same operations and never written back.
#pragma once

#include "kernels.cuh"

namespace oidt {

constexpr int kTileThreads = 1024;  // also the most cells a held tile has
constexpr int kTileHaloMax = 8;     // steps per sub-block at most

struct TileArgs {
  int s0;      // ring slot of the launch's first step
  int cnt;     // steps of this launch (more than halo: a cooperative launch of several sub-blocks)
  int ti, tj;  // owned tile extent: rows (x), columns (y)
  int gj;      // tiles along y
  int halo;    // cells computed on each side of the owned tile; steps per sub-block
  int *epoch;  // per tile: sub-blocks completed (cooperative launches)
  unsigned long long *xch;  // exchange words, two buffers ...
  long long xbuf;           // ... of xbuf words
};

// Exchange words (64 bits: 32 bits of a value beside the 32-bit number of the
// sub-block that wrote it).  A 64-bit access is single-copy atomic, so the
// reader polls the data word itself until the number is the one it waits for;
// no fence, flag or barrier orders data against a flag.  A float32 value is one
// word, a float64 value two.
__device__ __forceinline__ void xch_put(unsigned long long *q, float v0, float v1, unsigned n) {  // two values to q[0..1]
  const unsigned long long h = (unsigned long long)n << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(q), "l"(h | __float_as_uint(v0)),
               "l"(h | __float_as_uint(v1))
               : "memory");
}
__device__ __forceinline__ void xch_put(unsigned long long *q, float v, unsigned n) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(q), "l"((unsigned long long)n << 32 | __float_as_uint(v))
               : "memory");
}
__device__ __forceinline__ void xch_put(unsigned long long *q, double v, unsigned n) {  // to q[0..1]
  const unsigned long long h = (unsigned long long)n << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(q), "l"(h | (unsigned)__double2loint(v)),
               "l"(h | (unsigned)__double2hiint(v))
               : "memory");
}
// Predicated (all loads of a poll are in flight together): q[0..1], or q[0],
// is loaded where `on`, else w is left.
__device__ __forceinline__ void xch_load(unsigned long long &w, const unsigned long long *q, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p ld.relaxed.gpu.global.b64 %0, [%1];\n}\n"
               : "+l"(w)
               : "l"(q), "r"((unsigned)on)
               : "memory");
}
__device__ __forceinline__ void xch_load2(unsigned long long *w, const unsigned long long *q, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n}\n"
               : "+l"(w[0]), "+l"(w[1])
               : "l"(q), "r"((unsigned)on)
               : "memory");
}
__device__ __forceinline__ bool xch_take(unsigned long long w, float &v, unsigned n, bool on) {
  v = on ? __uint_as_float((unsigned)w) : v;
  return !on || (unsigned)(w >> 32) == n;
}
// A value's words in tile2d's exchange.
__device__ __forceinline__ void xch_load(unsigned long long *w, const unsigned long long *q, bool on, float) { xch_load(w[0], q, on); }
__device__ __forceinline__ void xch_load(unsigned long long *w, const unsigned long long *q, bool on, double) { xch_load2(w, q, on); }
__device__ __forceinline__ bool xch_take(const unsigned long long *w, float &v, unsigned n, bool on) { return xch_take(w[0], v, n, on); }
__device__ __forceinline__ bool xch_take(const unsigned long long *w, double &v, unsigned n, bool on) {
  v = on ? __hiloint2double((int)(unsigned)w[1], (int)(unsigned)w[0]) : v;
  return !on || ((unsigned)(w[0] >> 32) == n && (unsigned)(w[1] >> 32) == n);
}
// Words of one buffer: the three fields [nx ny], x-slab psi of E and H
// [2 sides][P][ny], y-slab psi of E and H [2 sides][nx][P].
inline size_t tile2d_xch_buf(int esz, long long nx, long long ny, long long P) {
  return (size_t)(esz / 4) * (3 * nx * ny + 4 * P * (nx + ny) + (nx * ny & 1));
}

// Shared memory of a block: the tile's three fields (kTileThreads cells each),
// the CPML coefficient tables be, ce, bh, ch (P each), and per held row (at
// most rows) kd0, 1/kd0, kd3, 1/kd3, per held column (at most cols) kd1,
// 1/kd1, kd4, 1/kd4 (the kappa dx arrays: E x, H x, E y, H y).
inline size_t tile2d_smem(int esz, int P, int rows, int cols) {
  return (3 * (size_t)kTileThreads + 4 * (size_t)P + 4 * (size_t)rows + 4 * (size_t)cols) * esz;
}

// Cell flags.  TM: E1 = Ez update, H1 = Hx, H2 = Hy; TE: E1 = Ex, E2 = Ey,
// H1 = Hz.  XE / YE / XH / YH: the cell is in the E / H x- / y-slab of the
// CPML.  CE0 / CE1, CH0 / CH1: the cell's E / H value is captured into the
// ring for port 0 / 1 (E slot 0 and H slot 1 at x = port, H slot 2 at
// x = port + 1).
enum : unsigned {
  kE1 = 1u, kE2 = 2u, kH1 = 4u, kH2 = 8u, kSrc = 16u, kXE = 32u, kYE = 64u, kXH = 128u, kYH = 256u,
  kCE0 = 512u, kCE1 = 1024u, kCH0 = 2048u, kCH1 = 4096u, kOwn = 8192u, kBand = 16384u
};

template <typename T, bool EXACT, int MODE>
__global__ void __launch_bounds__(kTileThreads, 1) k_2d_tile(const __grid_constant__ Params<T> p, TileArgs a) {
  using A = Ar<T, EXACT>;
  constexpr bool TM = MODE == OIDT_MODE_TM2;
  // fields f0, f1 (E in TE, H in TM), f2 (H); the fields carrying each psi array
  constexpr int FA = TM ? EZ : EX, FB = TM ? HX : EY, FC = TM ? HY : HZ;
  constexpr int EXS = TM ? EZ : EY, EYS = TM ? EZ : EX, HXS = TM ? HY : HZ, HYS = TM ? HX : HZ;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T *const F0 = reinterpret_cast<T *>(smem_raw), *const F1 = F0 + kTileThreads, *const F2 = F1 + kTileThreads;
  T *const BE = F2 + kTileThreads, *const CE = BE + p.P, *const BH = CE + p.P, *const CH = BH + p.P;
  // kd, 1/kd tables (one array each, consecutive columns in consecutive banks): rows kd0 1/kd0 kd3 1/kd3,
  // columns kd1 1/kd1 kd4 1/kd4
  const int RM = a.ti + 2 * a.halo, CM = a.tj + 2 * a.halo;
  T *const KR = CH + p.P, *const KC = KR + 4 * RM;
  const int nx = p.nx, ny = p.ny, P = p.P, H = a.halo;
  const int bi = (int)blockIdx.x / a.gj, bj = (int)blockIdx.x - bi * a.gj;
  const int oi0 = bi * a.ti, oi1 = min(nx, oi0 + a.ti), oj0 = bj * a.tj, oj1 = min(ny, oj0 + a.tj);
  const int wi0 = max(0, oi0 - H), wi1 = min(nx, oi1 + H), wj0 = max(0, oj0 - H), wj1 = min(ny, oj1 + H);
  const int nrow = wi1 - wi0, ncol = wj1 - wj0;
  const int t = threadIdx.x;
  const bool act = t < nrow * ncol;
  const int li = act ? t / ncol : 0, lj = act ? t - li * ncol : 0;
  int i = wi0 + li, j = wj0 + lj;
  auto cell = [&] { return i * ny + j; };  // the cell in the [nx][ny] arrays (2^31 cells at most)
  // its place in the x-slab [side][P][ny] and y-slab [side][nx][P] psi arrays (an H-slab cell is an E-slab cell
  // of the same layer and side).  These, the captures' and the exchange words' places are formed where they are
  // used: held through the steps they took some twenty of a thread's 64 registers, and the float64 kernels
  // spilled in the steps (64 to 72 bytes a thread; 8 to 16 now).  400 x 200 float64 fast 1.96 -> 1.64 us per
  // step, EXACT 2.45 -> 2.30; 603 x 1601 (waves) 25.8 -> 22.5 and 30.0 -> 26.8.
  auto xslab = [&](int &side) {
    side = i < p.ib + P ? LO : HI;
    return (side ? i - p.ie + P : i - p.ib) * ny + j;
  };
  auto yslab = [&](int &side) {
    side = j < p.jb + P ? LO : HI;
    return i * P + (side ? j - p.je + P : j - p.jb);
  };
  // ---- the cell's constants ------------------------------------------------------------
  unsigned fl = 0;
  int qE = 0, qH = 0;  // slab coefficient indices + 1: x slab in bits 0-15, y slab in bits 16-31
  T cbA = T(0), cbB = T(0);  // dt/eps of the cell's E components
  // this thread's entries of the coefficient and kappa dx tables, loaded first so that
  // their latency overlaps the cell's own loads (leftovers past kTileThreads below)
  const int nk = 4 * (nrow + ncol);
  auto co_src = [&](int u) { return __ldg((u < P ? p.be : u < 2 * P ? p.ce : u < 3 * P ? p.bh : p.ch) + u % P); };
  auto k_src = [&](int u, int &dst) {  // rows kd0 1/kd0 kd3 1/kd3, then columns kd1 1/kd1 kd4 1/kd4
    const bool row = u < 4 * nrow;
    const int v = row ? u : u - 4 * nrow, n = row ? nrow : ncol, c = v / n, r = v - c * n;
    const int a_ = row ? (c < 2 ? 0 : 3) : (c < 2 ? 1 : 4);
    dst = row ? c * RM + r : 4 * RM + c * CM + r;
    return __ldg((c & 1 ? p.rkd[a_] : p.kd[a_]) + (row ? wi0 : wj0) + r);
  };
  int kdst = 0;
  const T vco = t < 4 * P ? co_src(t) : T(0);
  const T vk = t < nk ? k_src(t, kdst) : T(0);
  if (act) {
    int d, side, q;
    if ((q = e_slab(i, p.ib, p.ie, P, d, side)) >= 0) {
      fl |= kXE;
      qE |= q + 1;
    }
    if ((q = e_slab(j, p.jb, p.je, P, d, side)) >= 0) {
      fl |= kYE;
      qE |= (q + 1) << 16;
    }
    if ((q = h_slab(i, p.ib, p.ie, P, d, side)) >= 0) {
      fl |= kXH;
      qH |= q + 1;
    }
    if ((q = h_slab(j, p.jb, p.je, P, d, side)) >= 0) {
      fl |= kYH;
      qH |= (q + 1) << 16;
    }
    // neighbours at (i + 1, j), (i, j + 1) [E] and (i - 1, j), (i, j - 1) [H] exist in
    // the tile except on its edges, whose cells are halo cells when not on the grid's edge
    const bool up = li + 1 < nrow, right = lj + 1 < ncol, down = li > 0, left = lj > 0;
    const bool own = i >= oi0 && i < oi1 && j >= oj0 && j < oj1;
    if (own) fl |= kOwn;
    if (own && (i - oi0 < H || oi1 - i <= H || j - oj0 < H || oj1 - j <= H)) fl |= kBand;  // read by neighbour tiles
    if (TM) {
      if (i >= p.ib && i < p.ie && j >= p.jb && j < p.je && up && right) fl |= kE1;   // update_ez :44-49
      if (i >= p.ib && i < p.ie && j > p.jb && j < p.je && left) fl |= kH1;          // update_hx :53-58
      if (i > p.ib && i < p.ie && j >= p.jb && j < p.je && down) fl |= kH2;          // update_hy :62-67
      if (in_src(p, EZ, i, j, 0)) fl |= kSrc;
      cbA = __ldg(p.cb[2] + cell());
    } else {
      if (i > p.ib && i < p.ie && j >= p.jb && j < p.je && right) fl |= kE1;         // update_ex :43-49
      if (i >= p.ib && i < p.ie && j > p.jb && j < p.je && up) fl |= kE2;            // update_ey :52-58
      if (i > p.ib && i < p.ie && j > p.jb && j < p.je && down && left) fl |= kH1;   // update_hz :61-67
      if (in_src(p, HZ, i, j, 0)) fl |= kSrc;
      cbA = __ldg(p.cb[0] + cell());
      cbB = __ldg(p.cb[1] + cell());
    }
    // ring captures of an owned cell on a port plane (where the update of the captured component runs)
    for (int port = 0; port < 2 && own; ++port) {
      const int x = p.port_pos[port];
      if (i == x && (fl & (TM ? kE1 : kE2))) fl |= kCE0 << port;
      if ((i == x || i == x + 1) && (fl & (TM ? kH2 : kH1))) fl |= kCH0 << port;
    }
  }
  if (t < 4 * P) BE[t] = vco;  // the CPML coefficients be ce bh ch, and the kappa dx tables
  if (t < nk) KR[kdst] = vk;
  for (int u = t + kTileThreads; u < 4 * P; u += kTileThreads) BE[u] = co_src(u);
  for (int u = t + kTileThreads; u < nk; u += kTileThreads) {
    int dst;
    const T x = k_src(u, dst);
    KR[dst] = x;
  }
  const T *const kr = KR + li, *const kc = KC + lj;  // kr[0, RM, 2 RM, 3 RM]: kd0 1/kd0 kd3 1/kd3; kc likewise
  const T db = p.db;
  const long long cstride = 2LL * p.nslot * p.plane;  // ring slot pitch
  const int nsub = (a.cnt + H - 1) / H;
  pdl_wait();  // the previous launch's state is complete (and visible) from here on
  const int n0 = p.state[0] + a.s0;
  const int e0 = nsub > 1 ? a.epoch[blockIdx.x] : 0;  // equal for every tile at launch
  T f0 = T(0), f1 = T(0), f2 = T(0), xe = T(0), ye = T(0), xh = T(0), yh = T(0);  // the cell's values
  if (act) {  // the held tile
    const int g = cell();
    f0 = __ldcg(p.f[FA] + g);
    f1 = __ldcg(p.f[FB] + g);
    f2 = __ldcg(p.f[FC] + g);
    F0[t] = f0;
    F1[t] = f1;
    F2[t] = f2;
    int sx, sy;
    const int ox = xslab(sx), oy = yslab(sy);
    if (fl & kXE) xe = __ldcg(p.psi[EXS][AX][sx] + ox);
    if (fl & kYE) ye = __ldcg(p.psi[EYS][AY][sy] + oy);
    if (fl & kXH) xh = __ldcg(p.psi[HXS][AX][sx] + ox);
    if (fl & kYH) yh = __ldcg(p.psi[HYS][AY][sy] + oy);
  }
  __syncthreads();
  // captures of an owned cell into the step's ring slot: E to slot 0, H to slot 1 (x = port) or 2 (x = port + 1)
  auto capture_e = [&](T *ring, T v) {
    if (fl & kCE0) ring[j] = v;
    if (fl & kCE1) ring[p.nslot * (int)p.plane + j] = v;
  };
  auto capture_h = [&](T *ring, T v) {
    if (fl & kCH0) ring[(i == p.port_pos[0] ? 1 : 2) * (int)p.plane + j] = v;
    if (fl & kCH1) ring[(p.nslot + (i == p.port_pos[1] ? 1 : 2)) * (int)p.plane + j] = v;
  };
  bool waits = true;
  for (int sb = 0; sb < nsub; ++sb) {
    const int s1 = min(a.cnt, (sb + 1) * H);
    for (int s = sb * H; s < s1; ++s) {
      T *const ring = p.ring + (a.s0 + s) * cstride;  // the step's ring slot
      // ---- E half-step ------------------------------------------------------------------
      if (TM) {
        if (fl & kE1) {  // update_ez :44-49
          const T dhy = A::sub(F2[t + ncol], f2);
          const T dhx = A::sub(F1[t + 1], f1);
          T e = A::curl(f0, cbA, dhy, kr[0], kr[RM], dhx, kc[0], kc[CM]);
          if (fl & kSrc) e = A::sub(e, __ldg(p.jsrc + n0 + s));  // update_source :71-76
          if (fl & kXE) {                                        // update_pml_ez_xinc :80-88
            const int q = (qE & 0xffff) - 1;
            xe = A::psi(BE[q], xe, CE[q], dhy, p.dx, p.rdx);
            e = A::inc(e, cbA, xe);
          }
          if (fl & kYE) {                                        // update_pml_ez_yinc :92-100
            const int q = (qE >> 16) - 1;
            ye = A::psi(BE[q], ye, CE[q], dhx, p.dx, p.rdx);
            e = A::dec(e, cbA, ye);
          }
          f0 = e;
          F0[t] = e;
          if (fl & (kCE0 | kCE1)) capture_e(ring, e);
        }
      } else {
        if (fl & kE1) {  // update_ex :43-49
          const T dhz = A::sub(F2[t + 1], f2);
          T e = A::step(f0, cbA, dhz, kc[0], kc[CM]);
          if (fl & kYE) {                                        // update_pml_ex_yinc :79-87
            const int q = (qE >> 16) - 1;
            ye = A::psi(BE[q], ye, CE[q], dhz, p.dx, p.rdx);
            e = A::inc(e, cbA, ye);
          }
          f0 = e;
          F0[t] = e;
        }
        if (fl & kE2) {  // update_ey :52-58
          const T hz1 = F2[t + ncol];
          T e = A::step(f1, cbB, A::sub(f2, hz1), kr[0], kr[RM]);
          if (fl & kXE) {                                        // update_pml_ey_xinc :91-99
            const int q = (qE & 0xffff) - 1;
            xe = A::psi(BE[q], xe, CE[q], A::sub(hz1, f2), p.dx, p.rdx);
            e = A::dec(e, cbB, xe);
          }
          f1 = e;
          F1[t] = e;
          if (fl & (kCE0 | kCE1)) capture_e(ring, e);
        }
      }
      __syncthreads();
      // ---- H half-step ------------------------------------------------------------------
      if (TM) {
        if (fl & kH1) {  // update_hx :53-58
          const T ezm = F0[t - 1];
          T h = A::step(f1, db, A::sub(ezm, f0), kc[2 * CM], kc[3 * CM]);
          if (fl & kYH) {                                        // update_pml_hx_yinc :104-112
            const int q = (qH >> 16) - 1;
            yh = A::psi(BH[q], yh, CH[q], A::sub(f0, ezm), p.dx, p.rdx);
            h = A::dec(h, db, yh);
          }
          f1 = h;
          F1[t] = h;
        }
        if (fl & kH2) {  // update_hy :62-67
          const T dez = A::sub(f0, F0[t - ncol]);
          T h = A::step(f2, db, dez, kr[2 * RM], kr[3 * RM]);
          if (fl & kXH) {                                        // update_pml_hy_xinc :116-124
            const int q = (qH & 0xffff) - 1;
            xh = A::psi(BH[q], xh, CH[q], dez, p.dx, p.rdx);
            h = A::inc(h, db, xh);
          }
          f2 = h;
          F2[t] = h;
          if (fl & (kCH0 | kCH1)) capture_h(ring, h);
        }
      } else {
        if (fl & kH1) {  // update_hz :61-67
          const T dex = A::sub(f0, F0[t - 1]);
          const T dey = A::sub(f1, F1[t - ncol]);
          T h = A::curl(f2, db, dex, kc[2 * CM], kc[3 * CM], dey, kr[2 * RM], kr[3 * RM]);
          if (fl & kSrc) h = A::sub(h, __ldg(p.jsrc + n0 + s));  // source after update_hz
          if (fl & kXH) {                                        // update_pml_hz_xinc :103-111
            const int q = (qH & 0xffff) - 1;
            xh = A::psi(BH[q], xh, CH[q], dey, p.dx, p.rdx);
            h = A::dec(h, db, xh);
          }
          if (fl & kYH) {                                        // update_pml_hz_yinc :115-123
            const int q = (qH >> 16) - 1;
            yh = A::psi(BH[q], yh, CH[q], dex, p.dx, p.rdx);
            h = A::inc(h, db, yh);
          }
          f2 = h;
          F2[t] = h;
          if (fl & (kCH0 | kCH1)) capture_h(ring, h);
        }
      }
      __syncthreads();
    }
    if (sb == nsub - 1) break;
    // ---- between sub-blocks: put the owned cells other tiles hold, fetch the halo cells ----
    const unsigned n = (unsigned)(e0 + sb + 1);
    constexpr int XW = (int)sizeof(T) / 4;
    const int N = nx * ny, SX = 2 * P * ny, SY = 2 * nx * P;
    unsigned long long *const xb = a.xch + ((n & 1) ? a.xbuf : 0);
    auto word = [&](int v) { return xb + (long long)XW * v; };
    auto places = [&](int &gx, int &pxe, int &pye) {  // of the cell's fields, x-slab and y-slab psi of E (H: + SX, + SY)
      asm volatile("" : "+r"(i), "+r"(j));  // formed anew at each use
      int sx, sy;
      const int ox = xslab(sx), oy = yslab(sy);
      gx = cell();
      pxe = 3 * N + sx * P * ny + ox;
      pye = 3 * N + 2 * SX + sy * nx * P + oy;
    };
    int gx, pxe, pye;
    if (fl & kBand) {
      places(gx, pxe, pye);
      xch_put(word(gx), f0, n);
      xch_put(word(N + gx), f1, n);
      xch_put(word(2 * N + gx), f2, n);
      if (fl & kXE) xch_put(word(pxe), xe, n);
      if (fl & kYE) xch_put(word(pye), ye, n);
      if (fl & kXH) xch_put(word(pxe + SX), xh, n);
      if (fl & kYH) xch_put(word(pye + SY), yh, n);
    }
    if (act && !(fl & kOwn)) {
      const long long t0 = clock64();
      unsigned round = 0;
      for (;;) {
        unsigned long long w[4][XW] = {};
        places(gx, pxe, pye);
        xch_load(w[0], word(gx), true, T(0));
        xch_load(w[1], word(N + gx), true, T(0));
        xch_load(w[2], word(2 * N + gx), true, T(0));
        bool ok = xch_take(w[0], f0, n, true);
        ok &= xch_take(w[1], f1, n, true);
        ok &= xch_take(w[2], f2, n, true);
        if (fl & (kXE | kYE | kXH | kYH)) {
          xch_load(w[0], word(pxe), fl & kXE, T(0));
          xch_load(w[1], word(pye), fl & kYE, T(0));
          xch_load(w[2], word(pxe + SX), fl & kXH, T(0));
          xch_load(w[3], word(pye + SY), fl & kYH, T(0));
          ok &= xch_take(w[0], xe, n, fl & kXE);
          ok &= xch_take(w[1], ye, n, fl & kYE);
          ok &= xch_take(w[2], xh, n, fl & kXH);
          ok &= xch_take(w[3], yh, n, fl & kYH);
        }
        if (ok || !waits) break;
        if (clock64() - t0 > p.wait_cycles) {
          atomicExch(p.state + 1, 3);  // reported to the host by oidt_job_sync
          waits = false;
        } else if (++round % 64 == 0 && ld_acquire(p.state + 1) != 0) {  // an earlier wait expired: stop waiting
          waits = false;
        }
      }
      F0[t] = f0;
      F1[t] = f1;
      F2[t] = f2;
    }
    __syncthreads();
  }
  // ---- owned cells to the other buffer ----------------------------------------------------
  if (fl & kOwn) {
    const int g = cell();
    p.fn[FA][g] = f0;
    p.fn[FB][g] = f1;
    p.fn[FC][g] = f2;
    int sx, sy;
    const int ox = xslab(sx), oy = yslab(sy);
    if (fl & kXE) p.psin[EXS][AX][sx][ox] = xe;
    if (fl & kYE) p.psin[EYS][AY][sy][oy] = ye;
    if (fl & kXH) p.psin[HXS][AX][sx][ox] = xh;
    if (fl & kYH) p.psin[HYS][AY][sy][oy] = yh;
  }
  if (nsub > 1 && t == 0) a.epoch[blockIdx.x] = e0 + nsub;
}

}  // namespace oidt
