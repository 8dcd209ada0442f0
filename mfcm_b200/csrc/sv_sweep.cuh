// sv_sweep.cuh -- column-sweep stage kernels.
//
// One warp owns a strip of 32 columns (28 output columns plus a 2-column halo on each side) and
// marches down its output rows. Each lane holds its column's last three rows of (h, u, v, z,
// dz/dx, dz/dy) in registers; x neighbours come from warp shuffles, y neighbours from the
// rolling window. Every face flux and every difference quotient is computed once and reused by
// both cells / both slopes that need it, and there is no block-level barrier.
//
// A strip is of one of three classes (strip_class_kernel):
//   kStripInterior  its whole window lies inside the mesh: sweep_rows without edge tests
//   kStripEdge      the window meets the mesh edge: sweep_rows with warp-uniform branches for
//                   one-sided slopes, wall faces and edge boundaries
//   kStripGeneral   the window holds a coded-out (NaN) bed or one outside the range below:
//                   sweep_rows_general, which follows the reference's functions literally
// The edge form costs an interior strip 15 % (FP32: 474 against 403 us a stage at 4096 x 4096;
// FP64: 1028 against 923). The persistent batch kernel runs every strip in the edge form all the
// same: its warps mix strips of all members at all times, and the two codes evicted each other
// from the instruction cache (3.3 cycles of no_instruction stall per issue; 149 ms against 122
// for 16 catchments). So do single sweeps whose strips are all resident at once (splits_forms).
//
// sweep_rows computes the same values as sweep_rows_general with far fewer instructions. In
// FP64 the results are bit-identical (up to the sign of zeros) as long as every h, u, v of the
// window is zero or has a magnitude in [2^-200, 2^200): then no intermediate value is non-finite,
// and no difference or product that is divided by the cell size leaves the range in which
// Markstein's division is exact. Each row is tested as it enters the window (a vote per row);
// the first row that fails sends the rest of the strip to sweep_rows_general. Under that
// condition:
//  * the two-sided Minmod3 slope is sign * min(2 min(|qL|, |qR|), |qC| / 2) when qL and qR agree
//    in sign and zero otherwise: qC has their sign then, since rounding is monotone. Half of it,
//    min(min(|qL|, |qR|), |qC| / 4), is kept: scalings by powers of two commute with rounding,
//    so d * (slope / 2) is the reference's 0.5 d * slope.
//  * a face side that is not above the face bed contributes nothing: its h and velocities set
//    to zero turn the two-sided flux into the reference's one-sided branches (adding an exact
//    zero), and both sides dead into the dry branch but for its normal momentum.
//  * fluxes are kept doubled (Sh - a Dh for 0.5 Sh - 0.5 a Dh) and divided by 2 d.
//  * with dx and dy powers of two the quotients are differences scaled by a power of two, so
//    slopes stay undivided and a cell's rate is scaled once at its end.
//  * the friction increment never has the velocity's sign, so its cap is a magnitude test.
// In FP32 the same formulas are used, with fused multiply-adds where the cell sizes are powers of
// two and with quotients and separate products elsewhere (MeshOps); a non-finite state stays non-finite in
// its own cells, which is what the controller tests.
#pragma once
#include <cstddef>
#include <type_traits>

namespace svk {

// A value that is the same in every lane, in a form the compiler knows to be so (a warp reduction
// ends in a uniform register): what follows from it -- loop counters, row addresses, branches --
// leaves the lanes' registers and needs no reconvergence.
__device__ __forceinline__ int uniform(int x) { return __reduce_max_sync(kFull, x); }

template <typename T> __device__ __forceinline__ T up1(T v) { return __shfl_up_sync(kFull, v, 1); }
template <typename T> __device__ __forceinline__ T dn1(T v) { return __shfl_down_sync(kFull, v, 1); }

template <typename T> struct RowV { T h, u, v, z, zx, zy; };
template <typename T> struct SlopeV { T hx, ux, vx, hy, uy, vy; };

template <typename T>
__device__ __forceinline__ CellV<T> mkcell(const RowV<T>& r, const SlopeV<T>& s) {
  CellV<T> c;
  c.h = r.h; c.u = r.u; c.v = r.v; c.z = r.z;
  c.dhdx = s.hx; c.dudx = s.ux; c.dvdx = s.vx; c.dzdx = r.zx;
  c.dhdy = s.hy; c.dudy = s.uy; c.dvdy = s.vy; c.dzdy = r.zy;
  return c;
}
template <typename T> __device__ __forceinline__ CellV<T> shfl_cell_up(const CellV<T>& a) {
  CellV<T> c;
  c.h = up1(a.h); c.u = up1(a.u); c.v = up1(a.v); c.z = up1(a.z);
  c.dhdx = up1(a.dhdx); c.dudx = up1(a.dudx); c.dvdx = up1(a.dvdx); c.dzdx = up1(a.dzdx);
  c.dhdy = up1(a.dhdy); c.dudy = up1(a.dudy); c.dvdy = up1(a.dvdy); c.dzdy = up1(a.dzdy);
  return c;
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = nmax(v, __shfl_down_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
  for (int o = 16; o > 0; o >>= 1) v = nmin(v, __shfl_down_sync(kFull, v, o));
  return v;
}

constexpr int kSweepOut = 28;  // output columns per warp

// Row ring of a sweeping warp. The next row of every field a stage reads -- the window fields
// (stage input, bed, bed slopes) of row k+1, the per-cell fields of output row k-1 -- is copied
// to shared memory by 16-byte asynchronous copies while row k is worked on, so no load waits for
// L2 or DRAM and no register holds a row ahead (prefetches into L1 left a third of the warps'
// cycles waiting on loads). A field row is 32 columns starting anywhere, so kCpr aligned chunks
// of 16 bytes cover it; the chunks of all fields are numbered and dealt to the lanes, kWSlots
// chunks per lane for the window and kCSlots for the per-cell fields, five (FP32) or nine (FP64)
// copy instructions per row instead of fourteen loads with their address arithmetic. Fields have
// at least kFieldPad bytes behind them (a row of chunks reaches past the last cell); in rows whose length is
// not a multiple of the chunk the first column's place in its chunk changes from row to row.
template <typename T> struct RowRing {
  static constexpr int kChunk = 16 / int(sizeof(T));               // values per chunk
  static constexpr int kCpr = (32 + 2 * (kChunk - 1)) / kChunk;    // chunks per field row: 9, 17
  static constexpr int kWSlots = (6 * kCpr + 31) / 32;             // 2, 4
  static constexpr int kCSlots = sizeof(T) == 4 ? 3 : 5;
  static constexpr int kCellFields = kCSlots * 32 / kCpr;          // 10, 9 fit
  static constexpr int kStage = (kWSlots + kCSlots) * 512;         // bytes per row
  static constexpr int kStages = 2;
  static constexpr int kBytes = kStages * kStage;                  // per warp
  static constexpr int kFieldBytes = kCpr * 16;
};
constexpr int kFieldPad = 288;
static_assert(kFieldPad >= RowRing<float>::kFieldBytes && kFieldPad >= RowRing<double>::kFieldBytes, "row of chunks");
__device__ __forceinline__ void copy16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Per-lane sums of a strip: tallies and volume in FP64, the CFL extremes in T (exact).
template <typename T> struct SweepAcc {
  double rain = 0.0, removed = 0.0, walls = 0.0, vol = 0.0;
  T xmax = T(0), xmin = T(1.0 / 0.0);
};

// Constants of a stage at the solver's present timestep.
template <typename T> struct StepConst {
  double dt_d, tsub_d, L, rL;
  T dt, rdt, cA, cB, rq0, rq1, rain_w, rain_q;
  T ck[4];  // general tableaux: the coefficients of k_0 .. k_st
  __device__ __forceinline__ void set(const StageParams<T>& P, int st) volatile {
    const double d = P.ctl->dt, tsub = P.ctl->t_local + P.c[st] * d, w = (tsub + 0.5 * d) / P.L;
    dt_d = d; tsub_d = tsub; L = P.L; rL = 1.0 / P.L;
    dt = T(d); rdt = T(1.0 / d);
    cA = T(P.a[st][st] * d); cB = T(P.b[st] * d);
    for (int j = 0; j <= st; ++j) ck[j] = T((st == P.nstages - 1 ? P.b[j] : P.a[st][j]) * d);
    const double q0 = P.fc->rq0, q1 = P.fc->rq1;
    rq0 = T(q0); rq1 = T(q1);
    // FP32 rain: the mean of the step's linear rain over the stage's timestep, as a weight of its
    // two ends formed in FP64
    rain_w = T(w); rain_q = T(q0 + (q1 - q0) * w);
  }
};

// What a sweeping warp keeps in shared memory besides its row ring: addresses and constants that
// every row uses once or twice. In registers they would cost the sweep a third of its resident
// warps (FP32: 50 registers of 128) or be spilled.
template <typename T> struct alignas(16) SweepShared {  // rings of 16-byte copies: aligned in an array of them
  using RR = RowRing<T>;
  unsigned char ring[RR::kBytes];
  const T* src[RR::kWSlots + RR::kCSlots][32];  // each lane's chunks: address in row 0
  double vol[32];                               // last stage: per-lane volume and CFL extremes
  T xmax[32], xmin[32];
  StepConst<T> step;
};
static_assert(sizeof(SweepShared<float>) % 16 == 0 && sizeof(SweepShared<double>) % 16 == 0 &&
                  offsetof(SweepShared<float>, ring) == 0 && offsetof(SweepShared<double>, ring) == 0,
              "16-byte copies need aligned rings");

// ---------------------------------------------------------------------------------------
// Output rows y0 .. y1-1 of the strip of column `tile_x`, any bed and any state: the
// reference's functions, with masks at every face. Strips with coded-out beds, and the rest
// of a strip whose state leaves the range of sweep_rows. Out of line: one copy per kernel.
// ---------------------------------------------------------------------------------------
template <typename T, bool EDDY, bool COH>
__device__ __noinline__ void sweep_rows_general(const StageParams<T>& P, int st, int tile_x, int y0, int y1, SweepAcc<T>& acc) {
  using DX = Div<T>;
  const Ctl* ctl = P.ctl;
  const int nx = P.nx, ny = P.ny;
  const int lane = threadIdx.x;
  const int gx = tile_x * kSweepOut - 2 + lane;
  const int gxc = min(max(gx, 0), nx - 1);
  const bool out_lane = lane >= 2 && lane < 2 + kSweepOut && gx < nx;
  const bool wface_lane = lane >= 2 && lane <= 2 + kSweepOut && gx <= nx;
  const bool hasW = gx > 0, hasE = gx < nx - 1;

  const int cur = ctl->cur;
  const double dt_d = ctl->dt;
  const double tsub = ctl->t_local + P.c[st] * dt_d;
  const T *Yh = P.in(st, cur, 0), *Yu = P.in(st, cur, 1), *Yv = P.in(st, cur, 2);
  const DX divx = MkDivX<DX>::make(P.dx), divy = MkDivX<DX>::make(P.dy);
  const T hdx = T(0.5) * T(P.dx), hdy = T(0.5) * T(P.dy);
  CellCtx<T, DX> c;
  c.divx = divx; c.divy = divy;
  c.divdt = mkdiv<T>(dt_d);
  c.divL = mkdiv<T>(P.L);
  c.dt = T(dt_d); c.dt_d = dt_d; c.tsub_d = tsub;
  c.manning = P.manning; c.rain_mode = P.rain_mode; c.head_first = P.head_first;
  const DevForcing fc = *P.fc;

  // FP32 with tile datums: the window keeps each cell's raw bed offset; a face whose two
  // cells lie in different datum tiles is evaluated in its lower cell's frame (face_frame),
  // the same whichever strip computes it, so the flux out of one cell is the flux into the
  // other and the volume is conserved across strip boundaries
  auto load_row = [&](int gy) {
    const int r = min(max(gy, 0), ny - 1);
    const long long g = (long long)r * nx + gxc;
    RowV<T> v;
    v.h = ldst<COH>(Yh, g); v.u = ldst<COH>(Yu, g); v.v = ldst<COH>(Yv, g);
    v.z = ld(P.z, g);
    v.zx = ld(P.zx, g); v.zy = ld(P.zy, g);
    return v;
  };

  RowV<T> Rm{}, R0{}, Rp{};   // rows k-2, k-1, k
  SlopeV<T> Sm{}, S0{};       // slopes of rows k-2, k-1
  T Smm_uy = T(0), Smm_vy = T(0);  // y slopes of u, v of row k-3 (eddy viscosity)
  T fyA[3] = {}, fyB[3] = {};  // (U[k-1]-U[k-2])/dy, (U[k]-U[k-1])/dy
  FaceF<T> FS{}, FN{};

#pragma unroll 1
  for (int k = y0 - 2; k <= y1 + 1; ++k) {
    Rm = R0; R0 = Rp; Rp = load_row(k);
    if constexpr (EDDY) { Smm_uy = Sm.uy; Smm_vy = Sm.vy; }
    Sm = S0;
    fyA[0] = fyB[0]; fyA[1] = fyB[1]; fyA[2] = fyB[2];
    // forward y quotients between rows k-1 and k
    if (k >= y0 - 1) {
      fyB[0] = divy(Rp.h - R0.h);
      fyB[1] = divy(Rp.u - R0.u);
      fyB[2] = divy(Rp.v - R0.v);
    }
    // slopes of row k-1 (State.cpp:187-192): Y axis uses north (row k) as the left neighbour
    if (k >= y0) {
      const int r = k - 1;
      const bool hasN = r < ny - 1, hasS = r > 0;
      S0.hy = minmod3q<T>(-fyB[0], hasN, -fyA[0], hasS, divy(Rm.h - Rp.h));
      S0.uy = minmod3q<T>(-fyB[1], hasN, -fyA[1], hasS, divy(Rm.u - Rp.u));
      S0.vy = minmod3q<T>(-fyB[2], hasN, -fyA[2], hasS, divy(Rm.v - Rp.v));
      {
        T r_ = dn1(R0.h), l_ = up1(R0.h);
        T fq = divx(r_ - R0.h);
        S0.hx = minmod3q<T>(up1(fq), hasW, fq, hasE, divx(r_ - l_));
      }
      {
        T r_ = dn1(R0.u), l_ = up1(R0.u);
        T fq = divx(r_ - R0.u);
        S0.ux = minmod3q<T>(up1(fq), hasW, fq, hasE, divx(r_ - l_));
      }
      {
        T r_ = dn1(R0.v), l_ = up1(R0.v);
        T fq = divx(r_ - R0.v);
        S0.vx = minmod3q<T>(up1(fq), hasW, fq, hasE, divx(r_ - l_));
      }
    }
    // horizontal face between rows k-2 and k-1 (face row fy = k-1), Fluxes.cpp:55-64
    if (k >= y0 + 1 && out_lane) {
      const int fy = k - 1;
      if (fy <= ny) {
        const int edge = fy == 0 ? -1 : (fy == ny ? 1 : 0);
        const CellV<T> lo = mkcell(Rm, Sm), hi = mkcell(R0, S0);
        if (P.zdat && edge == 0) {
          CellV<T> lo2 = lo, hi2 = hi;
          face_frame<T>(P, lo2, hi2, gx, fy - 1, gx, fy);
          face_flux<T, 1>(lo2, hi2, edge, hdy, divy, FN);
        } else {
          face_flux<T, 1>(edge == -1 ? hi : lo, edge == 1 ? lo : hi, edge, hdy, divy, FN);
        }
      }
    }
    // output row k-2
    if (k >= y0 + 2) {
      const int r = k - 2;
      const CellV<T> me = mkcell(Rm, Sm);
      const CellV<T> lf = shfl_cell_up(me);
      EddyIn<T> ed{};
      if constexpr (EDDY) {
        if (P.eddy) {  // second derivatives of row r: x by shuffles, y from rows r+1, r, r-1
          ed.ux = Sm.ux; ed.uy = Sm.uy; ed.vx = Sm.vx; ed.vy = Sm.vy;
          {
            T r_ = dn1(Sm.ux), l_ = up1(Sm.ux);
            T fq = divx(r_ - Sm.ux);
            ed.uxx = minmod3q<T>(up1(fq), hasW, fq, hasE, divx(r_ - l_));
          }
          {
            T r_ = dn1(Sm.vx), l_ = up1(Sm.vx);
            T fq = divx(r_ - Sm.vx);
            ed.vxx = minmod3q<T>(up1(fq), hasW, fq, hasE, divx(r_ - l_));
          }
          const bool hasN = r < ny - 1, hasS = r > 0;  // Y axis: north is the left neighbour
          ed.uyy = minmod3q<T>(divy(Sm.uy - S0.uy), hasN, divy(Smm_uy - Sm.uy), hasS, divy(Smm_uy - S0.uy));
          ed.vyy = minmod3q<T>(divy(Sm.vy - S0.vy), hasN, divy(Smm_vy - Sm.vy), hasS, divy(Smm_vy - S0.vy));
        }
      }
      FaceF<T> FW{T(0), T(0), T(0), T(0)};
      if (wface_lane && r < ny) {
        const int edge = gx == 0 ? -1 : (gx == nx ? 1 : 0);
        if (P.zdat && edge == 0) {
          CellV<T> lf2 = lf, me2 = me;
          face_frame<T>(P, lf2, me2, gx - 1, r, gx, r);
          face_flux<T, 0>(lf2, me2, edge, hdx, divx, FW);
        } else {
          face_flux<T, 0>(edge == -1 ? me : lf, edge == 1 ? lf : me, edge, hdx, divx, FW);
        }
      }
      const FaceF<T> FE{dn1(FW.h), dn1(FW.u), dn1(FW.v), dn1(FW.z)};
      if (out_lane && r < ny) {
        const long long g = (long long)r * nx + gx;
        finish_cell<T, CellCtx<T, DX>, EDDY, COH>(P, st, fc, c, g, gx, r, me.h, me.u, me.v, me.dhdx, me.dhdy,
                                                        me.dzdx, me.dzdy, FW, FE, FS, FN, cur, dt_d,
                                                        acc.rain, acc.removed, acc.walls, acc.xmax, acc.xmin, acc.vol,
                                                        &ed);
      }
    }
    FS = FN;
  }
}

// ---------------------------------------------------------------------------------------
// Strip classes.
// ---------------------------------------------------------------------------------------
constexpr unsigned kStripGeneral = 0, kStripInterior = 1, kStripEdge = 2;

// x is zero or 2^-200 <= |x| < 2^200 (false for NaN and infinities)
__device__ __forceinline__ bool in_range(double x) {
  const int hi = __double2hiint(x);
  const unsigned e = (unsigned(hi) >> 20) & 0x7ffu;
  return e - (1023u - 200u) < 400u || ((hi & 0x7fffffff) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool in_range(float x) { return x == x; }

// Whether the whole window (32 columns x the output rows and two more on each side) of strip
// `gw` of strips of `rows` output rows lies inside the mesh, with a column to spare.
__host__ __device__ inline bool strip_inside(long long gw, int nx, int ny, int rows) {
  const int tiles_x = (nx + kSweepOut - 1) / kSweepOut;
  const int x0 = int(gw % tiles_x) * kSweepOut, y0 = int(gw / tiles_x) * rows;
  return x0 >= 2 && x0 + 30 <= nx && y0 >= 2 && y0 + rows + 2 <= ny;
}

// Class of each strip; `exact`: the cell sizes allow sweep_rows (FP64: within 2^-30 .. 2^40 m,
// so that its quotients stay in the range of the exact division). One warp per strip.
template <typename T>
__global__ void strip_class_kernel(const T* __restrict__ z, int nx, int ny, int rows, long long nstrips, bool exact,
                                   unsigned char* __restrict__ cls) {
  const long long gw = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (gw >= nstrips) return;  // whole warp
  const int lane = threadIdx.x & 31;
  const int tiles_x = (nx + kSweepOut - 1) / kSweepOut;
  const int gx = min(max(int(gw % tiles_x) * kSweepOut - 2 + lane, 0), nx - 1), y0 = int(gw / tiles_x) * rows;
  bool ok = exact;
  for (int r = max(y0 - 2, 0); r <= min(y0 + rows + 1, ny - 1); ++r)
    if (!in_range(z[(long long)r * nx + gx])) ok = false;
  ok = __all_sync(kFull, ok);
  if (lane == 0) cls[gw] = ok ? (strip_inside(gw, nx, ny, rows) ? kStripInterior : kStripEdge) : kStripGeneral;
}

// ---------------------------------------------------------------------------------------
// Arithmetic of sweep_rows (see the top of this file).
// ---------------------------------------------------------------------------------------
// x / d without the range tests of DivD (the caller's values are in the range)
__device__ __forceinline__ double div_exact(double x, double d, double rd) {
  const double q0 = x * rd;
  return fma(fma(-q0, d, x), rd, q0);
}
__device__ __forceinline__ float div_exact(float x, float, float rd) { return x * rd; }

// half the two-sided Minmod3 slope of the quotients (or differences) qL, qR, qC
__device__ __forceinline__ float half_slope(float a, float b, float c) {
  float m;  // min(|a|, |b|), negative when a and b differ in sign
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
  m = fminf(fmaxf(m, 0.0f), 0.25f * fabsf(c));
  return __int_as_float(__float_as_int(m) | (__float_as_int(a) & 0x80000000));
}
__device__ __forceinline__ double half_slope(double a, double b, double c) {
  const double c4 = 0.25 * c;
  double m = fabs(a) < fabs(b) ? a : b;
  m = fabs(m) < fabs(c4) ? m : c4;
  return (__double2hiint(a) ^ __double2hiint(b)) < 0 ? 0.0 : m;
}
__device__ __forceinline__ float pick_max(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double pick_max(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ float clip0(float x) { return fmaxf(x, 0.0f); }
__device__ __forceinline__ double clip0(double x) { return __double2hiint(x) < 0 ? 0.0 : x; }
// the divider of a launch constant and its reciprocal
template <typename T> __device__ __forceinline__ Div<T> div_by(T d, T rd);
template <> __device__ __forceinline__ DivD div_by<double>(double d, double rd) { return DivD{d, rd}; }
template <> __device__ __forceinline__ DivF div_by<float>(float, float rd) { return DivF{rd}; }
// a * b + c, rounded once
__device__ __forceinline__ float sfma_(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double sfma_(double a, double b, double c) { return fma(a, b, c); }
// a * b + c: the product rounded by itself in FP64 (the reference's arithmetic), fused in FP32.
// Written out, since FP32 too is compiled without contraction: every instantiation of a formula
// then rounds alike, and a cell's FP32 result does not depend on the strip height, the strip's
// class or the kernel that computed it.
__device__ __forceinline__ float mad_(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double mad_(double a, double b, double c) { return a * b + c; }
// x with its sign flipped when s is negative
__device__ __forceinline__ float flip_sign(float x, float s) {
  return __int_as_float(__float_as_int(x) ^ (__float_as_int(s) & 0x80000000));
}
__device__ __forceinline__ double flip_sign(double x, double s) {
  return __hiloint2double(__double2hiint(x) ^ (__double2hiint(s) & 0x80000000), __double2loint(x));
}

// Quotients by the mesh spacing. With dx and dy powers of two, differences are kept undivided
// (diff_x, diff_y) and scaled where they are used; else they are divided (FP64: exactly; FP32: by
// the rounded reciprocal). FP32 could stay undivided with any spacing, and would be a little
// faster, but a velocity reconstructed across a full one-sided slope is then an exact zero where
// the quotients leave a rounding error, and a face whose velocity is an exact zero has no
// upwinding at all: results would move by 1e-4 of the velocity at a dam break's first timesteps.
// For the same reason FP32 rounds the products of face_pair and friction by themselves there. With
// power-of-two cells (StageParams::p2) the quotient form fuses them like the undivided one and, its
// scalings being exact, gives the same bits: a batch of both kinds runs the quotient form for all,
// and every member keeps its solo run's bits (both forms compiled into one kernel evicted each
// other from the instruction cache: 62 against 51 ms for 16 catchments in the persistent kernel).
template <typename T, bool P2> struct MeshOps {
  static constexpr bool SCALED = P2;
  const MeshConst<T>& mc;
  __device__ __forceinline__ T diff_x(T x) const { if constexpr (SCALED) return x; else return div_exact(x, mc.dx, mc.rdx); }
  __device__ __forceinline__ T diff_y(T x) const { if constexpr (SCALED) return x; else return div_exact(x, mc.dy, mc.rdy); }
  __device__ __forceinline__ T over_2dx(T x) const {
    if constexpr (SCALED) return x * mc.kx; else return div_exact(x, mc.dx2, mc.kx);
  }
  __device__ __forceinline__ T over_2dy(T x) const {
    if constexpr (SCALED) return x * mc.ky; else return div_exact(x, mc.dy2, mc.ky);
  }
  __device__ __forceinline__ T over_dx(T x) const { if constexpr (SCALED) return x * mc.rdx; else return diff_x(x); }
  __device__ __forceinline__ T over_dy(T x) const { if constexpr (SCALED) return x * mc.rdy; else return diff_y(x); }
  // bed at a face side: z + 0.5 d * slope, the product rounded by itself unless it is exact
  __device__ __forceinline__ static T zside(T hd, T s, T z) { if constexpr (SCALED || sizeof(T) == 4) return sfma_(hd, s, z); else return z + hd * s; }
  // what is kept of half a slope for the faces: the half jump 0.5 d * slope, but in FP32 with
  // quotients half the slope itself (side_x and side_y then add d times it, fused)
  __device__ __forceinline__ T jump_x(T hs) const { if constexpr (SCALED || sizeof(T) == 4) return hs; else return mc.dx * hs; }
  __device__ __forceinline__ T jump_y(T hs) const { if constexpr (SCALED || sizeof(T) == 4) return hs; else return mc.dy * hs; }
  // a cell's value plus a half jump
  __device__ __forceinline__ T side_x(T v, T j) const { if constexpr (!SCALED && sizeof(T) == 4) return sfma_(mc.dx, j, v); else return v + j; }
  __device__ __forceinline__ T side_y(T v, T j) const { if constexpr (!SCALED && sizeof(T) == 4) return sfma_(mc.dy, j, v); else return v + j; }
};

// Doubled fluxes of a face: depth, normal and tangential momentum, bed step.
template <typename T> struct FaceG { T h, n, t, z; };

// The doubled fluxes of a face from its two sides (FluxKernel.cpp:189-291); dv(x) is x / (2 d).
// strict: products rounded by themselves (the same thing in FP64).
template <typename T, typename DV>
__device__ __forceinline__ FaceG<T> face_pair(const Side<T>& m, const Side<T>& p, const DV& dv, bool strict) {
  const T g = T(kG);
  const bool rise = p.zb > m.zb;
  const T zf = rise ? p.zb : m.zb;
  const bool am = m.zb + m.h > zf, ap = p.zb + p.h > zf;
  T hm = m.h, um = m.un, tm = m.ut, hp = p.h, up = p.un, tp = p.ut;
  FaceG<T> G;
  G.z = (m.zb - p.zb) * (T(2) * g);
  T dry_n = T(0);
  bool dry = false;
  if (!(am && ap)) {
    dry = !am && !ap;
    const T t = clip0((dry ? rise : ap) ? hm : hp);
    const T gt = g * t;
    dry_n = rise ? gt : -gt;
    G.z = dry ? -dry_n : T(4) * dv(t);
    if (!am) hm = um = tm = T(0);
    if (!ap) hp = up = tp = T(0);
  }
  const T gm = g * hm, gp = g * hp;
  const T cm = ssqrt(gm), cp = ssqrt(gp);
  // |u + sign(u) c|: 0 when u is an exact zero
  const T a_m = um == T(0) ? T(0) : sfabs(um) + cm;
  const T a_p = up == T(0) ? T(0) : sfabs(up) + cp;
  const T a = pick_max(a_p, a_m);
  const T nm = mad_(um, T(0.5) * um, gm);
  const T np = mad_(up, T(0.5) * up, am ? -gp : gp);
  if (sizeof(T) == 4 && strict) {
    G.h = (hp * up + hm * um) - a * (hp - hm);
    G.n = (np + nm) - a * (up - um);
    G.t = (tp * up + tm * um) - a * (tp - tm);
  } else {
    G.h = mad_(-a, hp - hm, mad_(hp, up, hm * um));
    G.n = mad_(-a, up - um, np + nm);
    G.t = mad_(-a, tp - tm, mad_(tp, up, tm * um));
  }
  if (dry) G.n = dry_n;
  return G;
}

// Friction of a cell (ManningRoughnessSourceTerm.cpp:53-87), added to du, dv: FP64 in the
// reference's order; FP32 as one rate, min(g Sf, 1 / dt) (the cap of both components).
template <typename T> __device__ __forceinline__ T manning_n(T h, T ns, T nd, T ds, T dd) {
  if (ns == nd) return ns;  // mix(n, n, t) = n + 0*t = n: t = smoothstep(...) is always finite
  const T t = sfmin(sfmax((h - ds) / (dd - ds), T(0)), T(1));
  const T ss = t * t * (T(3) - T(2) * t);
  return ns + (nd - ns) * ss;
}
__device__ __forceinline__ void friction(double h, double u, double v, double n, double dt, double, double& du,
                                         double& dv, bool) {
  const double sf = n * n * ssqrt(u * u + v * v) * pow43_(manning_inv_h(h));
  double fu = -kG * sf * u, fv = -kG * sf * v;
  if (fabs(fu * dt) > fabs(u)) fu = -div_slow(u, dt);
  if (fabs(fv * dt) > fabs(v)) fv = -div_slow(v, dt);
  du = du + fu;
  dv = dv + fv;
}
__device__ __forceinline__ void friction(float h, float u, float v, float n, float dt, float rdt, float& du, float& dv,
                                         bool strict) {
  if (strict) {
    const float sf = n * n * ssqrt(mad_(u, u, v * v)) * pow43_(manning_inv_h(h));
    float fu = -float(kG) * sf * u, fv = -float(kG) * sf * v;
    if (fabsf(fu * dt) > fabsf(u)) fu = -u * rdt;
    if (fabsf(fv * dt) > fabsf(v)) fv = -v * rdt;
    du = du + fu;
    dv = dv + fv;
    return;
  }
  const float rate = fminf(float(kG) * (n * n * ssqrt(mad_(u, u, v * v)) * pow43_(manning_inv_h(h))), rdt);
  du = mad_(-rate, u, du);
  dv = mad_(-rate, v, dv);
}

// One cell of a stage after its four face fluxes are known (W, E: faces along x; GS, GN: along y;
// doubled): its rates, then the Runge-Kutta combination (RungeKutta.hpp:377-388) and, on the last
// stage, the CFL quantity and depth passed to totals(). jhx, jhy: half jumps of h (y: towards
// row + 1); shx, shy: its slopes where they are not kept undivided. medge: the cell may lie on the
// mesh edge. cells: the cell's values of U_[0], the running sum and the per-cell fields.
template <typename T, bool P2, bool EXTRA, bool COH, typename Cells, typename Totals>
__device__ __forceinline__ void lean_cell(const StageParams<T>& P, int st, int cur, const volatile StepConst<T>& k, int rk,
                                          bool rain_any, long long g, int gx, int r, const RowV<T>& R, T jhx, T jhy,
                                          T shx, T shy, const FaceG<T>& W, const FaceG<T>& E, const FaceG<T>& GS,
                                          const FaceG<T>& GN, bool medge, const EddyIn<T>& ed, const Cells& cells,
                                          SweepAcc<T>& acc, const Totals& totals) {
  constexpr bool F32 = sizeof(T) == 4;
  constexpr bool SCALED = P2;
  const int nx = P.nx, ny = P.ny;
  const bool first = st == 0, last = st == P.nstages - 1;
  const auto& mc = P.mc;
  const MeshOps<T, P2> mo{mc};
  const T h = R.h, u = R.u, v = R.v;
  // flux divergence, depth slope, bed step (TemporalDerivativeKernel.cpp:53-98)
  T dh, du, dv;
  if constexpr (F32) {
    // each difference is scaled before the next is added: beside a wall the momentum and
    // bed-step fluxes of one face are large and cancel, and the order decides what is left
    // of their rounding
    dh = mad_(GS.h - GN.h, mc.ky, (W.h - E.h) * mc.kx);
    du = mad_(GS.t - GN.t, mc.ky, (W.n - E.n) * mc.kx);
    dv = mad_(GS.n - GN.n, mc.ky, (W.t - E.t) * mc.kx);
    if constexpr (SCALED) {
      du = mad_(-mc.gx, jhx, du);
      dv = mad_(mc.gy, jhy, dv);
    } else {
      du = mad_(T(-kG), shx, du);
      dv = mad_(T(-kG), shy, dv);
    }
    du = mad_(W.z - E.z, mc.kx, du);
    dv = mad_(GS.z - GN.z, mc.ky, dv);
  } else if constexpr (SCALED) {
    const T g4 = T(4) * T(kG);
    const T ry = mc.ry;
    dh = sfma_(GS.h - GN.h, ry, W.h - E.h) * mc.kx;
    du = sfma_(GS.t - GN.t, ry, W.n - E.n);
    dv = sfma_(GS.n - GN.n, ry, W.t - E.t);
    du = mad_(-g4, jhx, du);
    dv = sfma_(g4 * jhy, ry, dv);
    du = (du + (W.z - E.z)) * mc.kx;
    dv = sfma_(GS.z - GN.z, ry, dv) * mc.kx;
  } else {
    dh = mo.over_2dx(W.h - E.h) + mo.over_2dy(GS.h - GN.h);
    du = mo.over_2dx(W.n - E.n) + mo.over_2dy(GS.t - GN.t);
    dv = mo.over_2dx(W.t - E.t) + mo.over_2dy(GS.n - GN.n);
    du = du + shx * T(-kG);
    dv = dv + shy * T(-kG);
    du = du + mo.over_2dx(W.z - E.z);
    dv = dv + mo.over_2dy(GS.z - GN.z);
  }
  // limited bed slope
  {
    const T lx = mo.over_dx(h), ly = mo.over_dy(h);
    const T zx = R.zx, zy = R.zy;
    du = mad_(T(-kG), (sfabs(zx) > lx && zx != T(0)) ? flip_sign(lx, zx) : zx, du);
    dv = mad_(T(-kG), (sfabs(zy) > ly && zy != T(0)) ? flip_sign(ly, zy) : zy, dv);
  }
  auto roughness = [&]() {
    if (!(P.manning && h > T(1e-6))) return;
    const T ns = P.man_p[0] ? cells.ns(g) : P.man_s[0];
    const T nd = P.man_p[1] ? (P.man_p[1] == P.man_p[0] ? ns : cells.nd(g)) : P.man_s[1];
    T n = ns;
    if (ns != nd)
      n = manning_n<T>(h, ns, nd, P.man_p[2] ? ld(P.man_p[2], g) : P.man_s[2],
                       P.man_p[3] ? ld(P.man_p[3], g) : P.man_s[3]);
    friction(h, u, v, n, k.dt, k.rdt, du, dv, !P2 && !P.p2);
  };
  if constexpr (!EXTRA) {
    roughness();
  } else {  // the momentum terms in configuration order, then infiltration
    CellCtx<T> c;
    c.dt = k.dt;
    c.divdt = div_by<T>(k.dt, k.rdt);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int term = (P.term_order >> (2 * i)) & 3;
      if (term == 1) roughness();
      if (term == 2 && P.efx)
        energy_loss_apply<T>(h, u, v, cells.ex(g), cells.ey(g), c, du, dv);
      if (term == 3 && P.eddy) {
        const T mu = P.eddy == 2 ? smagorinsky_mu<T>(P.eddy_c, P.eddy_s, T(P.cell_area), ed)
                                 : (P.eddy_mup ? ld(P.eddy_mup, g) : P.eddy_mu);
        T fu = T(0), fv = T(0);
        if (eddy_term<T>(h, u, v, mu, ed, c, fu, fv)) { du = du + fu; dv = dv + fv; }
      }
    }
    if (P.irate) {  // infiltration (InfiltrationSourceTerm.cpp:43-62), capacity consumed in place
      const T cap = cells.ic(g);
      const T d = infiltration_depth<T>(h, cells.ir(g), cap, c);
      dh = dh - c.divdt(d);
      P.icap[g] = cap - d;
    }
  }
  if (medge) {
    double w = 0.0;
    if (gx == 0) w += double(mo.over_2dx(W.h));
    if (gx == nx - 1) w -= double(mo.over_2dx(E.h));
    if (r == 0) w += double(mo.over_2dy(GS.h));
    if (r == ny - 1) w -= double(mo.over_2dy(GN.h));
    acc.walls += w;
  }
  auto do_rain = [&]() {
    if (rk == 0) return;
    T rate;
    bool applied;
    const T dt = k.dt;
    if constexpr (F32) {
      if (rk == 2) {
        const T q0 = cells.r0(P.q0p, g), q1 = cells.r1(P.q1p, g);
        applied = q0 != T(0) || q1 != T(0);
        rate = mad_(q1 - q0, k.rain_w, q0);
      } else {
        const T pp = rk == 3 ? cells.r0(P.pat, g) : T(1);
        applied = rain_any && pp != T(0);
        rate = pp * k.rain_q;
      }
      const T dhr = rate * dt;
      if (P.rain_mode == 0 ? (h - dhr <= T(0)) : (h + dhr <= T(0))) rate = -h * k.rdt;
    } else {
      T q0 = k.rq0, q1 = k.rq1;
      if (rk == 2) { q0 = cells.r0(P.q0p, g); q1 = cells.r1(P.q1p, g); }
      else if (rk == 3) { const T pp = cells.r0(P.pat, g); q0 = pp * q0; q1 = pp * q1; }
      applied = q0 != T(0) || q1 != T(0);
      const T dq = DivD{k.L, k.rL}(q1 - q0);
      const T qn = q0 + T(k.tsub_d) * dq;
      rate = T(0.5) * (qn + (qn + dt * dq));
      const T dhr = rate * dt;
      if (P.rain_mode == 0 ? (h - dhr <= T(0)) : (h + dhr <= T(0))) rate = -div_slow(h, dt);
    }
    if (applied) { dh = dh + rate; acc.rain += double(rate); }
  };
  auto do_head = [&]() {
    if (!EXTRA && !medge) return;
    const DevForcing& f = *P.fc;
    const int hk = f.head_kind;
    T h0, h1;
    if (medge && (hk == 1 || hk == 3)) {
      const bool sel = ((f.head_edges & 1u) && gx == 0) || ((f.head_edges & 2u) && gx == nx - 1) ||
                       ((f.head_edges & 4u) && r == 0) || ((f.head_edges & 8u) && r == ny - 1);
      if (!sel) return;
      h0 = T(f.hh0); h1 = T(f.hh1);
    } else if (EXTRA && (hk == 2 || hk == 4)) {
      h0 = ld(P.hb0p, g); h1 = ld(P.hb1p, g);
    } else {
      return;
    }
    if (hk >= 3) {  // water levels: less the bed, in FP64 with tile datums
      if (P.zdat) {
        const double zb = P.zdat[datum_tile(gx, r, P.dtiles_x)] + double(R.z);
        h0 = T(double(h0) - zb); h1 = T(double(h1) - zb);
      } else {
        h0 = h0 - R.z; h1 = h1 - R.z;
      }
    }
    if (!(h0 == h0 && h1 == h1)) return;  // NaN = not selected
    CellCtx<T> c;
    c.divL = mkdiv<T>(P.L);
    c.dt = k.dt; c.tsub_d = k.tsub_d;
    const T before = dh;
    const T d = head_target<T>(h0, h1, c) - h;
    if constexpr (F32) dh = d * k.rdt;
    else dh = div_slow(d, k.dt);
    acc.removed += double(before) - double(dh);
  };
  if (P.head_first) { do_head(); do_rain(); }
  else { do_rain(); do_head(); }
  // Runge-Kutta combination (RungeKutta.hpp:377-388), running accumulator; see finish_cell
  const T kk[3] = {dh, du, dv}, U[3] = {h, u, v};
  const T cA = k.cA, cB = k.cB;
  T out[3];
  bool running_sum = true;
  if constexpr (EXTRA) {
  if (!(P.mode & M_ACC)) {  // general tableau: U0 + k_0 c_0 + k_1 c_1 + ..., stored k's
    running_sum = false;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      T y = first ? U[f] : cells.u0(f);
      for (int j = 0; j < st; ++j) {
        const T kj = cells.k(j, f, g);
        y = mad_(kj, T(k.ck[j]), y);
      }
      y = mad_(kk[f], T(k.ck[st]), y);
      out[f] = y;
      if (last) {
        P.S[cur ^ 1][f][g] = y;
      } else {
        P.K[st][f][g] = kk[f];
        P.out(st, f)[g] = y;
      }
    }
  }
  }
  if (running_sum)
#pragma unroll
  for (int f = 0; f < 3; ++f) {
        const T u0 = first ? U[f] : cells.u0(f);
    const T a0 = first ? T(0) : cells.a0(f);
    T* A = P.S[cur ^ 1][f];
    if constexpr (F32) {  // the accumulator holds the increment
      const T d = mad_(kk[f], cB, a0);
      if (!last) {
        P.out(st, f)[g] = mad_(kk[f], cA, u0);
        A[g] = d;
      } else if (f == 0) {  // U_N.h = U0.h + d with the carried compensation (Neumaier)
        const T y = d + cells.hc(g);
        const T t = u0 + y;
        P.hc[cur ^ 1][g] = (sfabs(u0) >= sfabs(y)) ? (u0 - t) + y : (y - t) + u0;
        out[0] = t;
        A[g] = t;
      } else {
        out[f] = u0 + d;
        A[g] = out[f];
      }
    } else {
      const T a = first ? u0 : a0;
      if (!last) P.out(st, f)[g] = mad_(kk[f], cA, u0);
      out[f] = mad_(kk[f], cB, a);
      A[g] = out[f];
    }
  }
  if (last) {  // CFL quantity and volume of U_[N] (State.cpp:204-228)
    const T cc = ssqrt(T(kG) * sfmax(out[0], T(0)));
    T xx;
    if constexpr (SCALED || F32) xx = mad_(sfabs(out[1]) + cc, mc.rdx, (sfabs(out[2]) + cc) * mc.rdy);
    else xx = DivD{mc.dx, mc.rdx}(sfabs(out[1]) + cc) + DivD{mc.dy, mc.rdy}(sfabs(out[2]) + cc);
    totals(xx, out[0]);
  }
}

// the last stage's sums of a strip's rows from shared memory
template <typename T> __device__ __forceinline__ void sweep_totals(SweepShared<T>& sm, SweepAcc<T>& acc) {
  const int lane = threadIdx.x;
  acc.vol += sm.vol[lane];
  acc.xmax = nmax(acc.xmax, sm.xmax[lane]);
  acc.xmin = nmin(acc.xmin, sm.xmin[lane]);
}

// A cell's values from its row in the ring; o_*: place of a field in the row, or -1 (read directly).
template <typename T, bool COH> struct RingCells {
  const StageParams<T>& P;
  int cur;
  const unsigned char* cell;
  int o_ns, o_nd, o_r0, o_r1, o_hc, o_ex, o_ey, o_ir, o_ic;
  __device__ __forceinline__ T at(int o) const { return *reinterpret_cast<const T*>(cell + o); }
  __device__ __forceinline__ T field(int o, const T* p, long long g) const { return o >= 0 ? at(o) : ld(p, g); }
  __device__ __forceinline__ T u0(int f) const { return at(f * RowRing<T>::kFieldBytes); }
  __device__ __forceinline__ T a0(int f) const { return at((3 + f) * RowRing<T>::kFieldBytes); }
  __device__ __forceinline__ T k(int j, int f, long long g) const {
    const int n = 3 + 3 * j + f;
    return n < RowRing<T>::kCellFields ? at(n * RowRing<T>::kFieldBytes) : ldst<COH>(P.K[j][f], g);
  }
  __device__ __forceinline__ T ns(long long g) const { return field(o_ns, P.man_p[0], g); }
  __device__ __forceinline__ T nd(long long g) const { return field(o_nd, P.man_p[1], g); }
  __device__ __forceinline__ T r0(const T* p, long long g) const { return field(o_r0, p, g); }
  __device__ __forceinline__ T r1(const T* p, long long g) const { return field(o_r1, p, g); }
  __device__ __forceinline__ T hc(long long g) const { return o_hc >= 0 ? at(o_hc) : ldst<COH>(P.hc[cur], g); }
  __device__ __forceinline__ T ex(long long g) const { return field(o_ex, P.efx, g); }
  __device__ __forceinline__ T ey(long long g) const { return field(o_ey, P.efy, g); }
  __device__ __forceinline__ T ir(long long g) const { return field(o_ir, P.irate, g); }
  __device__ __forceinline__ T ic(long long g) const { return o_ic >= 0 ? at(o_ic) : P.icap[g]; }
};

// Output rows y0 .. y1-1 (inside the mesh) of the strip of column `tile_x`. Returns y1, or the
// first row not computed because the state left the range this function is exact for.
// EXTRA: any source term, boundary kind and tableau; without it Manning friction, rain, edge
// heads and a running accumulator.
template <typename T, bool P2, bool EXTRA, bool EDGE, bool COH>
__device__ __forceinline__ int sweep_rows(const StageParams<T>& P, int st, int tile_x, int y0, int y1, SweepShared<T>& sm,
                                          SweepAcc<T>& acc) {
  constexpr bool F32 = sizeof(T) == 4;
  constexpr bool SCALED = P2;  // slopes and fluxes undivided, one scaling per cell
  const Ctl* ctl = P.ctl;
  const int nx = P.nx, ny = P.ny;
  const int lane = threadIdx.x;
  const int gx0 = tile_x * kSweepOut - 2;
  const int gx = gx0 + lane;
  const int gxc = EDGE ? min(max(gx, 0), nx - 1) : gx;
  const bool out_lane = lane >= 2 && lane < 2 + kSweepOut && (!EDGE || gx < nx);
  const bool xedge = EDGE && (gx0 < 0 || gx0 + 31 >= nx - 1);  // the strip holds the mesh's first or last column

  const int cur = uniform(ctl->cur);
  const bool first = st == 0, last = st == P.nstages - 1;
  const T *Yh = P.in(st, cur, 0), *Yu = P.in(st, cur, 1), *Yv = P.in(st, cur, 2);

  const MeshOps<T, P2> mo{P.mc};
  const auto& mc = P.mc;

  // step constants, in shared memory
  volatile SweepShared<T>& vs = sm;
  const int rk = uniform(P.fc->rain_kind);
  const bool rain_any = uniform(P.fc->rq0 != 0.0 || P.fc->rq1 != 0.0);
  __syncwarp();  // a strip swept before this one is done with them and with its rows
  if (lane == 0) vs.step.set(P, st);
  vs.vol[lane] = 0.0;
  vs.xmax[lane] = T(0);
  vs.xmin[lane] = T(1.0 / 0.0);
  // FP32 with tile datums: a vertical face crosses datum tiles where its right cell starts a
  // tile column, a horizontal face where its upper row starts a tile row; there the upper /
  // right cell's bed moves into the other cell's frame (face_frame)
  const bool xcross = F32 && P.zdat != nullptr && (gx % kDatumTX) == 0 && (!EDGE || (gx > 0 && gx < nx));

  // the row ring: this lane's chunks
  using RR = RowRing<T>;
  const int c0 = EDGE ? max(gx0, 0) : gx0;  // first column of the rows copied
  // per-cell fields: place in the ring's row, or -1
  int o_ns = -1, o_nd = -1, o_r0 = -1, o_r1 = -1, o_hc = -1, o_ex = -1, o_ey = -1, o_ir = -1, o_ic = -1;
  int ncell = 0;                                              // per-cell fields in the ring
  {
    auto deal = [&](const T* f, int n, int slot0, int slots) {  // field number n of a class
      for (int s = 0; s < slots; ++s) {
        const int q = lane + 32 * s;
        if (q / RR::kCpr == n) vs.src[slot0 + s][lane] = f + (q % RR::kCpr) * RR::kChunk;
      }
    };
    deal(Yh, 0, 0, RR::kWSlots); deal(Yu, 1, 0, RR::kWSlots); deal(Yv, 2, 0, RR::kWSlots);
    deal(P.z, 3, 0, RR::kWSlots); deal(P.zx, 4, 0, RR::kWSlots); deal(P.zy, 5, 0, RR::kWSlots);
    auto add = [&](const T* f) {
      if (ncell >= RR::kCellFields) return -1;
      deal(f, ncell, RR::kWSlots, RR::kCSlots);
      return ncell++ * RR::kFieldBytes;
    };
    if (!first) {  // U_[0], then the running sum or, of a general tableau, the stored k's
      for (int f = 0; f < 3; ++f) add(P.S[cur][f]);
      if (!EXTRA || (P.mode & M_ACC)) {
        for (int f = 0; f < 3; ++f) add(P.S[cur ^ 1][f]);
      } else {
        for (int j = 0; j < st; ++j)
          for (int f = 0; f < 3; ++f) add(P.K[j][f]);
      }
    }
    if (P.manning) {
      if (P.man_p[0]) o_ns = add(P.man_p[0]);
      if (P.man_p[1] && P.man_p[1] != P.man_p[0]) o_nd = add(P.man_p[1]);
    }
    if (rk == 3) o_r0 = add(P.pat);
    if (rk == 2) { o_r0 = add(P.q0p); o_r1 = add(P.q1p); }
    if (F32 && last && P.hc[0] && (!EXTRA || (P.mode & M_ACC))) o_hc = add(P.hc[cur]);
    if constexpr (EXTRA) {
      if (P.efx) { o_ex = add(P.efx); o_ey = add(P.efy); }
      if (P.irate) { o_ir = add(P.irate); o_ic = add(P.icap); }
    }
  }
  const int ncopies = ncell * RR::kCpr;  // chunks of the per-cell fields
  __syncwarp();
  const unsigned ring0 = unsigned(__cvta_generic_to_shared(sm.ring));
  // copies of window row w (the mesh's nearest one) and per-cell row q into the ring's stage `k & 1`
  auto fetch = [&](int k, int w, int q) {
    const unsigned dst = ring0 + (k & 1) * RR::kStage + lane * 16;
    if (w <= y1 + 1) {
      const long long off = ((long long)(EDGE ? min(max(w, 0), ny - 1) : w) * nx + c0) & ~(long long)(RR::kChunk - 1);
#pragma unroll
      for (int s = 0; s < RR::kWSlots; ++s)
        if (lane + 32 * s < 6 * RR::kCpr) copy16(dst + s * 512, vs.src[s][lane] + off);
    }
    if (q >= y0 && q < y1) {
      const long long off = ((long long)q * nx + c0) & ~(long long)(RR::kChunk - 1);
#pragma unroll
      for (int s = 0; s < RR::kCSlots; ++s)
        if (lane + 32 * s < ncopies) copy16(dst + (RR::kWSlots + s) * 512, vs.src[RR::kWSlots + s][lane] + off);
    }
    copies_commit();
  };
  fetch(y0 - 2, y0 - 2, y0 - 4);

  RowV<T> Rm{}, R0{}, Rp{};     // rows k-2, k-1, k
  SlopeV<T> Jm{}, J0{};         // half jumps (0.5 d * slope) of rows k-2, k-1; y: towards row + 1
  SlopeV<T> Sm{}, S0{};         // EXTRA, or h of a mode that is not scaled: the slopes themselves
  T Smm_uy = T(0), Smm_vy = T(0);
  T fyA[3] = {}, fyB[3] = {};   // forward y quotients of rows k-2, k-1
  FaceG<T> GS{}, GN{};
  T xstep = T(0);  // datum step of the west face in the current tile row (xcross lanes)

#pragma unroll 1
  for (int k = y0 - 2; k <= y1 + 1; ++k) {
    copies_wait();
    __syncwarp();  // row k has arrived for every lane, and every lane is done with row k - 1's stage
    fetch(k + 1, k + 1, k - 1);
    const unsigned char* stage = sm.ring + (k & 1) * RR::kStage;
    Rm = R0; R0 = Rp;
    {
      const int sh = (int(unsigned(EDGE ? min(max(k, 0), ny - 1) : k) * unsigned(nx)) + c0) & (RR::kChunk - 1);
      const T* w = reinterpret_cast<const T*>(stage) + (gxc - c0 + sh);
      constexpr int kF = RR::kFieldBytes / int(sizeof(T));
      Rp.h = w[0]; Rp.u = w[kF]; Rp.v = w[2 * kF];
      Rp.z = w[3 * kF]; Rp.zx = w[4 * kF]; Rp.zy = w[5 * kF];
    }
    if constexpr (!F32) {
      if (__any_sync(kFull, !(in_range(Rp.h) && in_range(Rp.u) && in_range(Rp.v)))) {
        copies_wait();
        sweep_totals(sm, acc);
        return max(k - 2, y0);
      }
    }
    Jm = J0;
    if constexpr (EXTRA || !SCALED) {
      if constexpr (EXTRA) { Smm_uy = Sm.uy; Smm_vy = Sm.vy; }
      Sm = S0;
    }
    if constexpr (!SCALED) {
      fyA[0] = fyB[0]; fyA[1] = fyB[1]; fyA[2] = fyB[2];
      fyB[0] = mo.diff_y(Rp.h - R0.h); fyB[1] = mo.diff_y(Rp.u - R0.u); fyB[2] = mo.diff_y(Rp.v - R0.v);
    } else {
      fyA[0] = R0.h - Rm.h; fyA[1] = R0.u - Rm.u; fyA[2] = R0.v - Rm.v;
      fyB[0] = Rp.h - R0.h; fyB[1] = Rp.u - R0.u; fyB[2] = Rp.v - R0.v;
    }
    // half slopes of row k-1 (State.cpp:187-192). Along y they are formed towards row + 1, the
    // negative of the reference's (its Y axis takes north as the left side).
    if (k >= y0) {
      const int row = k - 1;
      const bool yedge = EDGE && (row <= 0 || row >= ny - 1);
      auto yslope = [&](T a, T b, T lo, T hi, T& j, T& s) {
        T hs = half_slope(a, b, F32 ? a + b : mo.diff_y(hi - lo));
        if (yedge) {  // one-sided: the slope is the present quotient
          if (row >= ny - 1) hs = T(0.5) * a;
          if (row <= 0) hs = ny > 1 ? T(0.5) * b : T(0);
        }
        j = mo.jump_y(hs);
        if constexpr (!SCALED) s = T(-2) * hs;
        else if constexpr (EXTRA) s = T(-2) * hs * mc.rdy;
      };
      yslope(fyA[0], fyB[0], Rm.h, Rp.h, J0.hy, S0.hy);
      yslope(fyA[1], fyB[1], Rm.u, Rp.u, J0.uy, S0.uy);
      yslope(fyA[2], fyB[2], Rm.v, Rp.v, J0.vy, S0.vy);
      auto xslope = [&](T x, T& j, T& s) {
        const T e = dn1(x);
        const T b = mo.diff_x(e - x), a = up1(b);
        T cc;
        if constexpr (F32) cc = a + b;
        else cc = mo.diff_x(e - up1(x));
        T hs = half_slope(a, b, cc);
        if (xedge) {
          if (gx >= nx - 1) hs = T(0.5) * a;
          if (gx <= 0) hs = nx > 1 ? T(0.5) * b : T(0);
        }
        j = mo.jump_x(hs);
        if constexpr (!SCALED) s = T(2) * hs;
        else if constexpr (EXTRA) s = T(2) * hs * mc.rdx;
      };
      xslope(R0.h, J0.hx, S0.hx);
      xslope(R0.u, J0.ux, S0.ux);
      xslope(R0.v, J0.vx, S0.vx);
    }
    // horizontal face between rows k-2 and k-1 (face row fy = k-1), Fluxes.cpp:55-64: the upper
    // side of the lower cell, the lower side of the upper one
    if (k >= y0 + 1) {
      const int fy = k - 1;
      T zhi = R0.z;
      if constexpr (F32) {
        if (P.zdat != nullptr && (fy % kDatumTY) == 0 && (!EDGE || (fy > 0 && fy < ny))) {
          const long long tb = datum_tile(gxc, fy, P.dtiles_x);
          zhi = T(double(zhi) + (P.zdat[tb] - P.zdat[tb - P.dtiles_x]));
        }
      }
      Side<T> m{mo.zside(mc.hdy, Rm.zy, Rm.z), mo.side_y(Rm.h, -Jm.hy), mo.side_y(Rm.v, -Jm.vy), mo.side_y(Rm.u, -Jm.uy)};
      Side<T> p{mo.zside(-mc.hdy, R0.zy, zhi), mo.side_y(R0.h, J0.hy), mo.side_y(R0.v, J0.vy), mo.side_y(R0.u, J0.uy)};
      if (EDGE && (fy <= 0 || fy >= ny)) {  // walls at the mesh edge, FluxKernel.cpp:111-157
        if (fy == 0) m = {R0.z + R0.h * T(2), T(0), T(0), mo.side_y(R0.u, -J0.uy)};
        if (fy == ny) p = {Rm.z + Rm.h * T(2), T(0), T(0), mo.side_y(Rm.u, Jm.uy)};
      }
      GN = face_pair<T>(m, p, [&](T x) { return mo.over_2dy(x); }, !P2 && !P.p2);
    }
    // output row k-2
    if (k >= y0 + 2) {
      const int r = k - 2;
      // west face: the left lane's east side against this lane's west side
      T zw = Rm.z;
      if constexpr (F32) {
        if (xcross) {
          // the datum step across the tile column edge, read once per tile row: datums are
          // multiples of 2^-10 m, so the step is exact in FP32 (below 2^14 m) and z + step
          // rounds as the FP64 sum does; an inexact step (NaN here) takes the FP64 sum
          if (r == y0 || (r % kDatumTY) == 0) {
            const long long tb = datum_tile(gx, r, P.dtiles_x);
            const double s = P.zdat[tb] - P.zdat[tb - 1];
            xstep = double(T(s)) == s ? T(s) : Lim<T>::nan();
          }
          if (xstep == xstep) {
            zw = Rm.z + xstep;
          } else {
            const long long tb = datum_tile(gx, r, P.dtiles_x);
            zw = T(double(Rm.z) + (P.zdat[tb] - P.zdat[tb - 1]));
          }
        }
      }
      Side<T> p{mo.zside(-mc.hdx, Rm.zx, zw), mo.side_x(Rm.h, -Jm.hx), mo.side_x(Rm.u, -Jm.ux), mo.side_x(Rm.v, -Jm.vx)};
      const T eut = mo.side_x(Rm.v, Jm.vx);
      Side<T> m{up1(mo.zside(mc.hdx, Rm.zx, Rm.z)), up1(mo.side_x(Rm.h, Jm.hx)), up1(mo.side_x(Rm.u, Jm.ux)), up1(eut)};
      if (xedge) {
        const T wall = Rm.z + Rm.h * T(2);
        const T wl = up1(wall), utl = up1(p.ut);
        if (gx == 0) m = {wall, T(0), T(0), eut};
        if (gx == nx) p = {wl, T(0), T(0), utl};
      }
      const FaceG<T> W = face_pair<T>(m, p, [&](T x) { return mo.over_2dx(x); }, !P2 && !P.p2);
      const FaceG<T> E{dn1(W.h), dn1(W.n), dn1(W.t), dn1(W.z)};
      EddyIn<T> ed{};
      if constexpr (EXTRA) {
        if (P.eddy) {  // second derivatives of row r: x by shuffles, y from rows r+1, r, r-1
          ed.ux = Sm.ux; ed.uy = Sm.uy; ed.vx = Sm.vx; ed.vy = Sm.vy;
          auto along_x = [&](T x) {
            const T e = dn1(x), b = mo.over_dx(e - x), a = up1(b);
            T hs = half_slope(a, b, mo.over_dx(e - up1(x)));
            if (xedge) {
              if (gx >= nx - 1) hs = T(0.5) * a;
              if (gx <= 0) hs = nx > 1 ? T(0.5) * b : T(0);
            }
            return T(2) * hs;
          };
          auto along_y = [&](T south, T x, T north) {  // the reference's Y axis: north on the left
            const T a = mo.over_dy(x - north), b = mo.over_dy(south - x);
            T hs = half_slope(a, b, mo.over_dy(south - north));
            if (EDGE && r >= ny - 1) hs = T(0.5) * b;
            if (EDGE && r <= 0) hs = ny > 1 ? T(0.5) * a : T(0);
            return T(2) * hs;
          };
          ed.uxx = along_x(Sm.ux);
          ed.vxx = along_x(Sm.vx);
          ed.uyy = along_y(Smm_uy, Sm.uy, S0.uy);
          ed.vyy = along_y(Smm_vy, Sm.vy, S0.vy);
        }
      }
      if (out_lane) {
        const long long g = (long long)r * nx + gx;
        // the per-cell fields of this row in the ring
        RingCells<T, COH> cells{P, cur, stage + RR::kWSlots * 512 +
                                    (gxc - c0 + ((int(unsigned(r) * unsigned(nx)) + c0) & (RR::kChunk - 1))) * int(sizeof(T)),
                                o_ns, o_nd, o_r0, o_r1, o_hc, o_ex, o_ey, o_ir, o_ic};
        lean_cell<T, P2, EXTRA, COH>(P, st, cur, sm.step, rk, rain_any, g, gx, r, Rm, Jm.hx, Jm.hy, Sm.hx, Sm.hy, W, E, GS, GN,
                                     EDGE && (xedge || r == 0 || r == ny - 1), ed, cells, acc,
                                     [&](T xx, T hN) {
                                       vs.xmax[lane] = nmax(T(vs.xmax[lane]), xx);
                                       vs.xmin[lane] = nmin(T(vs.xmin[lane]), xx);
                                       vs.vol[lane] = vs.vol[lane] + double(hN) * P.cell_area;
                                     });
      }
    }
    GS = GN;
  }
  sweep_totals(sm, acc);
  return y1;
}

// A warp's strip sums into the strip's partial slot.
template <typename T>
__device__ __forceinline__ void store_strip_sums(const StageParams<T>& P, int st, long long gw, const SweepAcc<T>& acc) {
  const int lane = threadIdx.x;
  if (st == P.nstages - 1) {
    const double mx = warp_max(double(acc.xmax)), mn = warp_min(double(acc.xmin)), vs = warp_sum(acc.vol);
    if (lane == 0) {
      P.part[gw] = mx;
      P.part[P.nblk + gw] = mn;
      P.part[2 * P.nblk + gw] = vs;
    }
  }
  if (P.mode & M_TALLY) {
    const double rs = warp_sum(acc.rain), os = warp_sum(acc.removed), ws = warp_sum(acc.walls);
    if (lane == 0) store_tallies(P, st, gw, rs, os, ws, P.ctl->dt);
  }
}

// One strip of one solver's stage: its class's sweep, then its partial sums. `entry` is the
// strip's index (row-major over strips of kSweepOut columns x P.rows rows) times 4 plus its
// class. SPLIT: interior strips run the form without edge tests.
template <typename T, bool P2, bool EXTRA, bool SPLIT, bool COH>
__device__ __forceinline__ void sweep_strip(const StageParams<T>& P, int st, unsigned entry, SweepShared<T>& sm) {
  const unsigned e = unsigned(uniform(int(entry)));
  const long long gw = e >> 2;
  const unsigned cls = e & 3u;
  const int tiles_x = (P.nx + kSweepOut - 1) / kSweepOut;
  const int tile_y = int(gw) / tiles_x;
  const int tile_x = int(gw) - tile_y * tiles_x, y0 = tile_y * P.rows, y1 = min(y0 + P.rows, P.ny);
  SweepAcc<T> acc;
  int y = y0;
  if (SPLIT && cls == kStripInterior) y = sweep_rows<T, P2, EXTRA, false, COH>(P, st, tile_x, y0, y1, sm, acc);
  else if (cls != kStripGeneral) y = sweep_rows<T, P2, EXTRA, true, COH>(P, st, tile_x, y0, y1, sm, acc);
  if (y < y1) {
    SweepAcc<T> rest = acc;
    sweep_rows_general<T, EXTRA, COH>(P, st, tile_x, y, y1, rest);
    acc = rest;
  }
  store_strip_sums(P, st, gw, acc);
}

// ---------------------------------------------------------------------------------------
// Row-tile kernel: a strip's rows side by side instead of one after another. One block per strip
// of kTileRows output rows, one warp per row of its window: each warp forms its row's slopes and
// sides, then the face below it, then its cells; neighbours in y come from shared memory. The
// lean sweep's arithmetic, so the same bits. For meshes of few strips, where a marching warp's
// latency is the whole stage's time: an FP64 stage of 100 x 100 cells takes 13 us, 27 in strips of
// 4 rows; 256 x 256 23, against 28 in strips of 4 rows and 117 in strips of 32. Bound by the latency of one row's chain
// of square roots, divisions and barriers. A block whose window holds a value out of sweep_rows' range
// hands its rows to sweep_rows_general.
// ---------------------------------------------------------------------------------------
constexpr int kTileRows = 8, kTileWarps = kTileRows + 4;

// a cell's values loaded ahead into registers (fields the tile kernel does not expect: directly)
template <typename T> struct LoadedCells {
  const StageParams<T>& P;
  int cur;
  T u[3], a[3], n, r;
  __device__ __forceinline__ T u0(int f) const { return u[f]; }
  __device__ __forceinline__ T a0(int f) const { return a[f]; }
  __device__ __forceinline__ T ns(long long) const { return n; }
  __device__ __forceinline__ T nd(long long g) const { return ld(P.man_p[1], g); }
  __device__ __forceinline__ T r0(const T*, long long) const { return r; }
  __device__ __forceinline__ T r1(const T* p, long long g) const { return ld(p, g); }
  __device__ __forceinline__ T hc(long long g) const { return ld(P.hc[cur], g); }
};

template <typename T, bool P2>
__global__ void __launch_bounds__(32 * kTileWarps, sizeof(T) == 8 ? 1 : 2)
    tile_rows_kernel(const __grid_constant__ StageParams<T> P, const int st) {
  constexpr bool F32 = sizeof(T) == 4;
  constexpr bool SCALED = P2;
  __shared__ StepConst<T> step;
  __shared__ T val[3][kTileWarps][32];    // h, u, v
  __shared__ T upper[5][kTileWarps][32];  // a row's upper side: bed, h, normal, tangential; its lower tangential
  __shared__ T face[4][kTileWarps][32];   // the face below a row
  __shared__ double sums[6][kTileRows];
  chain_wait();
  if (P.ctl->done) return;
  const int lane = threadIdx.x, w = uniform(threadIdx.y);
  const int nx = P.nx, ny = P.ny;
  const int tiles_x = (nx + kSweepOut - 1) / kSweepOut;
  const int gw = blockIdx.x, tile_y = gw / tiles_x, tile_x = gw - tile_y * tiles_x;
  const int y0 = tile_y * kTileRows, y1 = min(y0 + kTileRows, ny);
  const int row = y0 - 2 + w;
  const int gx = tile_x * kSweepOut - 2 + lane, gxc = min(max(gx, 0), nx - 1);
  const bool out_row = w >= 2 && row < y1;
  const bool out = out_row && lane >= 2 && lane < 2 + kSweepOut && gx < nx;
  const int cur = uniform(P.ctl->cur);
  const bool first = st == 0, last = st == P.nstages - 1;
  const MeshOps<T, P2> mo{P.mc};
  const auto& mc = P.mc;
  const int rk = uniform(P.fc->rain_kind);
  const bool rain_any = uniform(P.fc->rq0 != 0.0 || P.fc->rq1 != 0.0);

  // every load of the row at once
  const long long gc = (long long)min(max(row, 0), ny - 1) * nx + gxc;
  RowV<T> R;
  R.h = ld(P.in(st, cur, 0), gc); R.u = ld(P.in(st, cur, 1), gc); R.v = ld(P.in(st, cur, 2), gc);
  R.z = ld(P.z, gc); R.zx = ld(P.zx, gc); R.zy = ld(P.zy, gc);
  LoadedCells<T> cells{P, cur};
  if (out_row) {
    if (!first)
#pragma unroll
      for (int f = 0; f < 3; ++f) { cells.u[f] = ld(P.S[cur][f], gc); cells.a[f] = ld(P.S[cur ^ 1][f], gc); }
    if (P.manning && P.man_p[0]) cells.n = ld(P.man_p[0], gc);
    if (rk == 3) cells.r = ld(P.pat, gc);
    if (rk == 2) cells.r = ld(P.q0p, gc);
  }
  if (w == 0 && lane == 0) const_cast<volatile StepConst<T>&>(step).set(P, st);
  val[0][w][lane] = R.h; val[1][w][lane] = R.u; val[2][w][lane] = R.v;
  const bool bad = !(in_range(R.z) && (F32 || (in_range(R.h) && in_range(R.u) && in_range(R.v)))) || !P.exact;
  SweepAcc<T> acc;
  if (__syncthreads_or(bad)) {
    if (w > 0) return;
    sweep_rows_general<T, false, false>(P, st, tile_x, y0, y1, acc);
    store_strip_sums(P, st, gw, acc);
    return;
  }

  // half slopes of the row (State.cpp:187-192), y towards row + 1
  SlopeV<T> J{}, S{};
  if (w > 0 && w < kTileWarps - 1) {
    auto yslope = [&](int f, T x, T& j, T& s) {
      const T lo = val[f][w - 1][lane], hi = val[f][w + 1][lane];
      const T a = mo.diff_y(x - lo), b = mo.diff_y(hi - x);
      T hs = half_slope(a, b, F32 ? a + b : mo.diff_y(hi - lo));
      if (row >= ny - 1) hs = T(0.5) * a;
      if (row <= 0) hs = ny > 1 ? T(0.5) * b : T(0);
      j = mo.jump_y(hs);
      s = T(-2) * hs;
    };
    yslope(0, R.h, J.hy, S.hy);
    yslope(1, R.u, J.uy, S.uy);
    yslope(2, R.v, J.vy, S.vy);
    auto xslope = [&](T x, T& j, T& s) {
      const T e = dn1(x), b = mo.diff_x(e - x), a = up1(b);
      T cc;
      if constexpr (F32) cc = a + b;
      else cc = mo.diff_x(e - up1(x));
      T hs = half_slope(a, b, cc);
      if (gx >= nx - 1) hs = T(0.5) * a;
      if (gx <= 0) hs = nx > 1 ? T(0.5) * b : T(0);
      j = mo.jump_x(hs);
      s = T(2) * hs;
    };
    xslope(R.h, J.hx, S.hx);
    xslope(R.u, J.ux, S.ux);
    xslope(R.v, J.vx, S.vx);
    upper[0][w][lane] = mo.zside(mc.hdy, R.zy, R.z);
    upper[1][w][lane] = mo.side_y(R.h, -J.hy);
    upper[2][w][lane] = mo.side_y(R.v, -J.vy);
    upper[3][w][lane] = mo.side_y(R.u, -J.uy);
    upper[4][w][lane] = mo.side_y(R.u, J.uy);
  }
  __syncthreads();
  // the face below the row (fy = row), Fluxes.cpp:55-64
  FaceG<T> GS{};
  if (w >= 2 && w < kTileWarps - 1) {
    T zhi = R.z;
    if constexpr (F32) {
      if (P.zdat != nullptr && (row % kDatumTY) == 0 && row > 0 && row < ny) {
        const long long tb = datum_tile(gxc, row, P.dtiles_x);
        zhi = T(double(zhi) + (P.zdat[tb] - P.zdat[tb - P.dtiles_x]));
      }
    }
    Side<T> m{upper[0][w - 1][lane], upper[1][w - 1][lane], upper[2][w - 1][lane], upper[3][w - 1][lane]};
    Side<T> p{mo.zside(-mc.hdy, R.zy, zhi), mo.side_y(R.h, J.hy), mo.side_y(R.v, J.vy), mo.side_y(R.u, J.uy)};
    // walls at the mesh edge, FluxKernel.cpp:111-157 (rows past it hold the edge row's values)
    if (row == 0) m = {R.z + R.h * T(2), T(0), T(0), mo.side_y(R.u, -J.uy)};
    if (row == ny) p = {R.z + R.h * T(2), T(0), T(0), upper[4][w - 1][lane]};
    GS = face_pair<T>(m, p, [&](T x) { return mo.over_2dy(x); }, !P2 && !P.p2);
    face[0][w][lane] = GS.h; face[1][w][lane] = GS.n; face[2][w][lane] = GS.t; face[3][w][lane] = GS.z;
  }
  FaceG<T> W{};
  if (out_row) {  // west faces: the left lane's east side against this lane's west side
    T zw = R.z;
    if constexpr (F32) {
      if (P.zdat != nullptr && (gx % kDatumTX) == 0 && gx > 0 && gx < nx) {
        const long long tb = datum_tile(gx, row, P.dtiles_x);
        const double d = P.zdat[tb] - P.zdat[tb - 1];
        zw = double(T(d)) == d ? R.z + T(d) : T(double(R.z) + d);
      }
    }
    Side<T> p{mo.zside(-mc.hdx, R.zx, zw), mo.side_x(R.h, -J.hx), mo.side_x(R.u, -J.ux), mo.side_x(R.v, -J.vx)};
    const T eut = mo.side_x(R.v, J.vx), wall = R.z + R.h * T(2);
    Side<T> m{up1(mo.zside(mc.hdx, R.zx, R.z)), up1(mo.side_x(R.h, J.hx)), up1(mo.side_x(R.u, J.ux)), up1(eut)};
    const T wl = up1(wall), utl = up1(p.ut);
    if (gx == 0) m = {wall, T(0), T(0), eut};
    if (gx == nx) p = {wl, T(0), T(0), utl};
    W = face_pair<T>(m, p, [&](T x) { return mo.over_2dx(x); }, !P2 && !P.p2);
  }
  __syncthreads();
  if (out_row) {
    const FaceG<T> E{dn1(W.h), dn1(W.n), dn1(W.t), dn1(W.z)};
    const FaceG<T> GN{face[0][w + 1][lane], face[1][w + 1][lane], face[2][w + 1][lane], face[3][w + 1][lane]};
    if (out)
      lean_cell<T, P2, false, false>(P, st, cur, step, rk, rain_any, gc, gx, row, R, J.hx, J.hy, S.hx, S.hy, W, E, GS, GN,
                                     gx == 0 || gx == nx - 1 || row == 0 || row == ny - 1, EddyIn<T>{}, cells, acc, [&](T xx, T hN) {
                                       acc.xmax = nmax(acc.xmax, xx);
                                       acc.xmin = nmin(acc.xmin, xx);
                                       acc.vol += double(hN) * P.cell_area;
                                     });
  }
  if (!last && !(P.mode & M_TALLY)) return;
  // the strip's sums: rows by shuffles, then the first warp's lane 0 over the rows in order
  if (out_row) {
    const int i = w - 2;
    if (last) {
      const double mx = warp_max(double(acc.xmax)), mn = warp_min(double(acc.xmin)), vs = warp_sum(acc.vol);
      if (lane == 0) { sums[0][i] = mx; sums[1][i] = mn; sums[2][i] = vs; }
    }
    if (P.mode & M_TALLY) {
      const double rs = warp_sum(acc.rain), os = warp_sum(acc.removed), ws = warp_sum(acc.walls);
      if (lane == 0) { sums[3][i] = rs; sums[4][i] = os; sums[5][i] = ws; }
    }
  }
  __syncthreads();
  if (w != 0 || lane != 0) return;
  const int n = y1 - y0;
  if (last) {
    double mx = sums[0][0], mn = sums[1][0], vs = sums[2][0];
    for (int i = 1; i < n; ++i) { mx = nmax(mx, sums[0][i]); mn = nmin(mn, sums[1][i]); vs += sums[2][i]; }
    P.part[gw] = mx;
    P.part[P.nblk + gw] = mn;
    P.part[2 * P.nblk + gw] = vs;
  }
  if (P.mode & M_TALLY) {
    double rs = 0.0, os = 0.0, ws = 0.0;
    for (int i = 0; i < n; ++i) { rs += sums[3][i]; os += sums[4][i]; ws += sums[5][i]; }
    store_tallies(P, st, gw, rs, os, ws, step.dt_d);
  }
}

constexpr int kSweepWarps = 4;  // warps (strips) per block

// The strips listed in P.strips (general and edge strips first: they take longer, so they do
// not end up as the launch's tail). Four strips a block; a block only shares the launch.
// Per stage at 4096 x 4096: FP32 404 us against 667 before (issue active 77 %, 22 warp instructions
// per cell against 29), FP64 945 against 1966 (38 against 70; 16 warps per SM, issue active
// 57 %: bound by dependent instructions, the FP64 pipe is a third busy). DRAM is at 36 and 32 %
// of the copy bandwidth.
template <typename T, int MINB, bool P2, bool EXTRA, bool SPLIT>
__global__ void __launch_bounds__(32 * kSweepWarps, MINB)
    sweep_kernel(const __grid_constant__ StageParams<T> P, const int st) {
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  chain_wait();
  if (P.ctl->done) return;
  const int w = uniform(threadIdx.y), i = int(blockIdx.x) * kSweepWarps + w;
  if (i >= P.n_strips) return;  // whole warp: no block-level synchronisation below
  sweep_strip<T, P2, EXTRA, SPLIT, false>(P, st, P.strips[i], reinterpret_cast<SweepShared<T>*>(sweep_smem)[w]);
}

// Batched column sweep: the strips of up to kBatchMembers solvers in one launch. Their parameters
// are kernel parameters, so a block reads them as constants, as the single-solver kernel does
// (staged in shared memory instead they took registers from the sweep, which then spilled). A
// block sweeps strips of one solver: first_block[k] is member k's first block.
constexpr int kBatchMembers = 32;
template <typename T> struct BatchParams {
  int n;
  int first_block[kBatchMembers + 1];
  StageParams<T> m[kBatchMembers];
};
static_assert(sizeof(BatchParams<double>) <= 32764 && sizeof(BatchParams<float>) <= 32764, "kernel parameters");

template <typename T, int MINB, bool P2, bool EXTRA>
__global__ void __launch_bounds__(32 * kSweepWarps, MINB)
    sweep_batch_kernel(const __grid_constant__ BatchParams<T> B, const int st) {
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  int k = 0;
  for (int step = kBatchMembers / 2; step > 0; step /= 2)  // the last member that starts at or before this block
    if (k + step < B.n && B.first_block[k + step] <= int(blockIdx.x)) k += step;
  const StageParams<T>& P = B.m[k];
  chain_wait();
  if (P.ctl->done) return;
  const int w = uniform(threadIdx.y), i = (int(blockIdx.x) - B.first_block[k]) * kSweepWarps + w;
  if (i >= P.n_strips) return;
  sweep_strip<T, P2, EXTRA, !EXTRA, false>(P, st, P.strips[i], reinterpret_cast<SweepShared<T>*>(sweep_smem)[w]);
}

}  // namespace svk
