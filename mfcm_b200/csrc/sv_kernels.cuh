// sv_kernels.cuh -- kernels of the Saint-Venant RK time step on sm_100a.
//
//  column sweeps  (sv_sweep.cuh) one launch per RK stage, the form that every caller gets unless
//                 it asks for another variant: warps march strips of 28 columns; slopes and fluxes
//                 stay in registers.
//  stage_kernel   one launch per RK stage. A CTA owns a TX x TY tile of cells, stages the
//                 tile plus a 2-cell halo of (h, u, v, z) in shared memory, computes the
//                 Minmod3 slopes of every cell of the tile plus a 1-cell ring, the fluxes of
//                 every face of the tile, then per cell dU/dt (flux divergence, depth-slope,
//                 limited bed slope, zflux), Manning friction, rainfall and outflow, and the
//                 Runge-Kutta combination. Faces and slopes never leave the SM.
//                 The last stage of either also reduces the CFL quantity and the FP64 volume.
//  finalize_kernel  fixed-order reduction of the partials, the control number, and the dt
//                 controller (accept / repeat / new dt / end-of-step trimming) in FP64, so a
//                 whole step runs without a host round trip.
//  debug kernels  the same per-face / per-cell functions over global arrays, one reference
//                 kernel each, for per-function parity tests.
#pragma once
#include <cooperative_groups.h>

#include "sv_device.cuh"

namespace svk {
using namespace svd;

constexpr unsigned kFull = 0xffffffffu;  // every lane of a warp

// Device-resident controller state of one solver (FP64 times, TT = double).
struct Ctl {
  double t_local;   // time since the start of the step
  double dt;        // current timestep
  double cn;        // control number of the last timestep
  double new_dt;    // dt suggested by the last timestep
  int cur;          // parity of the state buffer that holds U_[0]
  int done;         // 1: the step is complete (auto mode) -- all stage kernels exit
  int repeat;       // last timestep rejected
  int error;        // sticky error code (SV_E_NONFINITE ...)
  unsigned long long accepted, repeated;            // running totals
  unsigned long long step_accepted, step_repeated;  // in the current step
  double rain_in, outflow;      // running tallies over accepted timesteps
  double wall_in;               // running tally of the flow through the mesh-edge faces
  double volume;                // volume of U_[0] after the last accepted timestep
  double pend_rain, pend_out, pend_vol;  // tallies of the last timestep, applied on accept
  double pend_wall;
  long long budget;             // > 0: timesteps left before the loop pauses (done = 2)
};

// Per-step boundary values, kept in device memory so captured graphs stay valid when
// start_new_step changes them (DischargeBoundarySourceTerm.hpp:114-146,
// HeadBoundarySourceTerm.hpp:114-146).
struct DevForcing {
  int rain_kind;        // SV_RAIN_*
  int head_kind;        // SV_HEAD_*
  unsigned head_edges;  // SV_EDGE_* bits
  int pad;
  double rq0, rq1;      // uniform / pattern-scaled rain values at the start / end of the step
  double hh0, hh1;      // head targets at the start / end of the step
};

// Programmatic dependent launch: the kernels of a timestep follow each other without a host round
// trip, so a small mesh's timestep is a chain of launches. Each kernel waits here until the ones
// before it in the stream have completed (their writes are visible then), and lets the next one
// be launched while it runs: the real-time timestep of 64 x 48
// cells (six launches in a stream) 51 -> 37 us, with its begin and result launches merged.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

enum StageMode : int {
  M_ACC = 4,      // diagonal tableau: running accumulator instead of stored k's
  M_STOREK = 8,   // store k_s for later stages (non-diagonal tableaux)
  M_TALLY = 16,   // rain / outflow partials
};

// Constants of the mesh in the solver's value type, formed once on the host.
template <typename T> struct MeshConst {
  T dx, dy, rdx, rdy;    // cell sizes and their reciprocals
  T dx2, dy2, kx, ky;    // 2 d and 1 / (2 d)
  T hdx, hdy;            // d / 2
  T ry;                  // dx / dy
  T gx, gy;              // 2 g / d
  void set(double x, double y) {
    dx = T(x); dy = T(y); rdx = T(1.0 / x); rdy = T(1.0 / y);
    dx2 = T(2.0 * x); dy2 = T(2.0 * y); kx = T(0.5) * rdx; ky = T(0.5) * rdy;
    hdx = T(0.5) * dx; hdy = T(0.5) * dy; ry = T(x / y);
    gx = T(2.0 * 9.81 / x); gy = T(2.0 * 9.81 / y);
  }
};

// One solver's parameters for every stage of a timestep; the stage's index (0-based) goes beside
// them. Stage 0 reads U_[0] and the last one writes U_[N] and the CFL and volume partials.
template <typename T> struct StageParams {
  int nx, ny;
  double dx, dy, L;
  double cell_area;
  MeshConst<T> mc;
  T* S[2][3];            // state parity buffers: S[cur] = U_[0], S[cur^1] = acc / U_[N]
  T* Y[2][3];            // stage s reads Y[(s - 1) & 1] (s > 0) and writes Y[s & 1]
  T* K[3][3];            // stored k_s, all but the last stage's (M_STOREK)
  const T* z;
  const T* zx; const T* zy;   // bed slopes dz/dx, dz/dy (Constants.cpp:39-40), precomputed
  const double* zdat;         // FP32-with-datum mode: per datum tile FP64 datum (z = datum + z_off)
  int dtiles_x;               // datum tiles per row
  const T* man_p[4];     // per-cell n_shallow, n_deep, d_shallow, d_deep, or nullptr
  T man_s[4];            // uniform values where man_p is nullptr
  const DevForcing* fc;  // per-step boundary values
  const T* q0p; const T* q1p; const T* pat;
  const T* hb0p; const T* hb1p;
  const T* irate; T* icap;   // infiltration rate (m/s) and remaining capacity (m), or nullptr
  const T* efx; const T* efy;  // energy-loss coefficients fx/m, fy/m, or nullptr
  T* hc[2];              // FP32: per-cell compensation of the depth update (state parity), or nullptr
  int manning, rain_mode, head_first;
  int eloss_first;       // energy loss applied before roughness (configuration order)
  int nstages, mode;
  double c[4];           // stage s is evaluated at t_local + c[s] * dt
  double a[4][4];        // a[s][j] = a(s+2, j+1), j = 0..s: coefficients of Y_{s+1}
  double b[4];           // b_1..b_N
  Ctl* ctl;
  double* part;          // per-CTA partials (see part_* offsets)
  long long nblk;
  // eddy viscosity (run by the kernels compiled with it): 0 off, 1 constant coefficient
  // (eddy_mup per cell, else eddy_mu), 2 Smagorinsky (eddy_c + eddy_s * area * |strain|)
  int eddy;
  T eddy_mu, eddy_c, eddy_s;
  const T* eddy_mup;
  // the momentum source terms in configuration order, 2 bits per slot: 1 roughness,
  // 2 energy loss, 3 eddy viscosity (each adds to du/dt and dv/dt, so the order sets the
  // rounding); used by the kernels compiled with eddy viscosity
  int term_order;
  // column sweep: strips of kSweepOut columns x `rows` rows, each listed as its index times 4
  // plus its class (strip_class_kernel)
  const unsigned* strips;
  int n_strips, rows;
  int exact;  // the cell sizes allow sweep_rows (exact_mesh)
  int p2;     // dx and dy are powers of two (pow2_mesh): chooses the rounding in FP32 (MeshOps)
  // split schedule: the stage input's slopes dh/dx, du/dx, dv/dx, dh/dy, du/dy, dv/dy as
  // written by slopes_kernel (read by the stage kernel instead of computing them), or null
  T* pslp[6];

  // field f of stage `st`'s input, of its output
  __device__ __forceinline__ const T* in(int st, int cur, int f) const {
    return st == 0 ? S[cur][f] : Y[(st - 1) & 1][f];
  }
  __device__ __forceinline__ T* out(int st, int f) const { return Y[st & 1][f]; }
};

// partial layout: [0, nblk) cn max, [nblk, 2nblk) cn min, [2nblk, 3nblk) volume, then the
// rain, outflow and wall-flow tallies at 3, 4 and 5 nblk. A block's (or warp's) tally slot
// carries the weighted sum over the stages so far, sum_s b_s dt * tally_s, so the finalize
// reads three tally arrays however many stages there are: at 4096 x 4096 and four stages 0.9 MB
// instead of 2.3 MB.
constexpr int kParts = 6;
__host__ __device__ inline long long part_count(long long nblk) { return kParts * nblk; }
// Adds one stage's tallies, weighted by b_s dt in the solver's value type, to slot `i`.
template <typename T>
__device__ __forceinline__ void store_tallies(const StageParams<T>& P, int st, long long i, double rain,
                                              double removed, double wall, double dt) {
  const bool first = st == 0;
  const double w = double(T(P.b[st] * dt));
  double* p = P.part + 3 * P.nblk + i;
  p[0] = first ? w * rain : p[0] + w * rain;
  p[P.nblk] = first ? w * removed : p[P.nblk] + w * removed;
  p[2 * P.nblk] = first ? w * wall : p[2 * P.nblk] + w * wall;
}

template <typename T> __device__ __forceinline__ T ld(const T* p, long long i) { return __ldg(p + i); }
// Loads of the state, stage and accumulator buffers. A launch that writes and later reads them
// itself (the persistent batch kernel, COH) must use coherent loads, ordered by its phase
// fences; every other launch only reads what earlier launches wrote, through the read-only path.
template <bool COH, typename T> __device__ __forceinline__ T ldst(const T* p, long long i) {
  if constexpr (COH) return p[i];
  return __ldg(p + i);
}

// Datum tiles of the FP32-with-datum mode: 32 x 8 cells, each with an FP64 datum; the stored
// bed is the FP32 offset from its tile's datum.
constexpr int kDatumTX = 32, kDatumTY = 8;
__host__ __device__ inline long long datum_tile(int gx, int gy, int dtiles_x) {
  return (long long)(gy / kDatumTY) * dtiles_x + gx / kDatumTX;
}
// FP32 with tile datums: the beds of a face's two cells, (ax, ay) below or left of (bx, by),
// in the frame of the lower cell's datum tile: b's offset moved by the exact FP64 datum
// difference and rounded once, a's unchanged.
template <typename T>
__device__ __forceinline__ void face_frame(const StageParams<T>& P, CellV<T>& a, CellV<T>& b, int ax, int ay, int bx,
                                           int by) {
  const long long ta = datum_tile(ax, ay, P.dtiles_x), tb = datum_tile(bx, by, P.dtiles_x);
  if (ta != tb) b.z = T(double(b.z) + (P.zdat[tb] - P.zdat[ta]));
}

// Bed of cell (gx, gy) in the frame of datum tile `ref`: the stored value itself, or, for a
// cell of another datum tile, its offset moved by the FP64 datum difference and rounded once.
template <typename T>
__device__ __forceinline__ T load_bed(const T* z, const double* zdat, int dtiles_x, long long g, int gx, int gy,
                                      long long ref) {
  const T zo = __ldg(z + g);
  if (!zdat) return zo;
  const long long t = datum_tile(gx, gy, dtiles_x);
  if (t == ref) return zo;
  return T(double(zo) + (__ldg(zdat + t) - __ldg(zdat + ref)));
}

// NaN-propagating max/min for the CFL reduction
__device__ __forceinline__ double nmax(double a, double b) { return (a != a || b != b) ? (a + b) : (a > b ? a : b); }
__device__ __forceinline__ double nmin(double a, double b) { return (a != a || b != b) ? (a + b) : (a < b ? a : b); }
__device__ __forceinline__ float nmax(float a, float b) { return (a != a || b != b) ? (a + b) : (a > b ? a : b); }
__device__ __forceinline__ float nmin(float a, float b) { return (a != a || b != b) ? (a + b) : (a < b ? a : b); }

template <int NT> __device__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NT / 32; ++i) r += red[i];
  }
  return r;
}
template <int NT> __device__ double block_max(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v = nmax(v, __shfl_down_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double r = v;
  if (threadIdx.x == 0) {
    r = red[0];
    for (int i = 1; i < NT / 32; ++i) r = nmax(r, red[i]);
  }
  return r;
}
template <int NT> __device__ double block_min(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v = nmin(v, __shfl_down_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double r = v;
  if (threadIdx.x == 0) {
    r = red[0];
    for (int i = 1; i < NT / 32; ++i) r = nmin(r, red[i]);
  }
  return r;
}

template <typename T> __device__ __forceinline__ Div<T> mkdiv(double d);
template <> __device__ __forceinline__ Div<double> mkdiv<double>(double d) { return make_div(d); }
template <> __device__ __forceinline__ Div<float> mkdiv<float>(double d) { return make_divf(float(d)); }
template <typename DV> struct MkDivX;
template <> struct MkDivX<DivD> { __device__ static DivD make(double d) { return make_div(d); } };
template <> struct MkDivX<DivP2> { __device__ static DivP2 make(double d) { return DivP2{1.0 / d}; } };
template <> struct MkDivX<DivF> { __device__ static DivF make(double d) { return make_divf(float(d)); } };

// Per-cell dU/dt of one stage (TemporalDerivativeKernel.cpp:53-98, then the source terms
// and boundaries in configuration order, Solver.cpp:97-113). fw/fe/fs/fn are the four face
// fluxes; returns the rain rate added, the depth rate removed by the head assignment and the
// depth rate that entered through mesh-edge faces (the reference's walls pass flow through
// their one-sided branches; taken before any boundary assignment).
template <typename T, typename CC, bool EDDY = false>
__device__ __forceinline__ void cell_dudt(const StageParams<T>& P, const DevForcing& fc, const CC& c,
                                          long long g, int gx,
                                          int gy, T h, T u, T v, T dhdx, T dhdy, T dzdx, T dzdy,
                                          const FaceF<T>& fw, const FaceF<T>& fe, const FaceF<T>& fs,
                                          const FaceF<T>& fn, T& kh, T& ku, T& kv, double& rain,
                                          double& removed, double& wall, T* n_out, T* sf_out,
                                          const EddyIn<T>* ed = nullptr) {
  T dhdt = c.divx(fw.h - fe.h) + c.divy(fs.h - fn.h);
  T dudt = c.divx(fw.u - fe.u) + c.divy(fs.u - fn.u);
  T dvdt = c.divx(fw.v - fe.v) + c.divy(fs.v - fn.v);
  dudt = dudt + dhdx * T(-kG);
  dvdt = dvdt + dhdy * T(-kG);
  T hdx = c.divx(h), hdy = c.divy(h);
  if (sfabs(dzdx) > hdx) dzdx = (dzdx > T(0)) ? hdx : ((dzdx < T(0)) ? -hdx : c.divx(ssign(dzdx) * h));
  if (sfabs(dzdy) > hdy) dzdy = (dzdy > T(0)) ? hdy : ((dzdy < T(0)) ? -hdy : c.divy(ssign(dzdy) * h));
  T dudt_bed = T(-kG) * dzdx;
  T dvdt_bed = T(-kG) * dzdy;
  dudt = dudt + c.divx(fw.z - fe.z);
  dvdt = dvdt + c.divy(fs.z - fn.z);
  dudt = dudt + dudt_bed;
  dvdt = dvdt + dvdt_bed;
  // source terms in configuration order (Solver.cpp:98-104): roughness and energy loss both
  // add to du/dt, dv/dt, so only their relative order changes the rounding
  auto do_manning = [&]() {
    if (!P.manning) return;
    T ns = P.man_p[0] ? ld(P.man_p[0], g) : P.man_s[0];
    T nd = P.man_p[1] ? (P.man_p[1] == P.man_p[0] ? ns : ld(P.man_p[1], g)) : P.man_s[1];
    T ds = P.man_p[2] ? ld(P.man_p[2], g) : P.man_s[2];
    T dd = P.man_p[3] ? ld(P.man_p[3], g) : P.man_s[3];
    manning_apply<T>(h, u, v, ns, nd, ds, dd, c, dudt, dvdt, n_out, sf_out);
  };
  auto do_eloss = [&]() {
    if (P.efx) energy_loss_apply<T>(h, u, v, ld(P.efx, g), ld(P.efy, g), c, dudt, dvdt);
  };
  if constexpr (!EDDY) {
    if (P.eloss_first) { do_eloss(); do_manning(); }
    else { do_manning(); do_eloss(); }
  } else {
    // each term's increments depend on the cell's state only; they are added in the
    // configured order
    T fu1 = T(0), fv1 = T(0), fu2 = T(0), fv2 = T(0), fu3 = T(0), fv3 = T(0);
    bool on1 = false, on2 = false, on3 = false;
    if (P.manning) {
      T ns = P.man_p[0] ? ld(P.man_p[0], g) : P.man_s[0];
      T nd = P.man_p[1] ? (P.man_p[1] == P.man_p[0] ? ns : ld(P.man_p[1], g)) : P.man_s[1];
      T ds = P.man_p[2] ? ld(P.man_p[2], g) : P.man_s[2];
      T dd = P.man_p[3] ? ld(P.man_p[3], g) : P.man_s[3];
      on1 = manning_term<T>(h, u, v, ns, nd, ds, dd, c, fu1, fv1, n_out, sf_out);
    }
    if (P.efx) on2 = energy_loss_term<T>(h, u, v, ld(P.efx, g), ld(P.efy, g), c, fu2, fv2);
    if (P.eddy) {
      const T mu = P.eddy == 2 ? smagorinsky_mu<T>(P.eddy_c, P.eddy_s, T(P.cell_area), *ed)
                               : (P.eddy_mup ? ld(P.eddy_mup, g) : P.eddy_mu);
      on3 = eddy_term<T>(h, u, v, mu, *ed, c, fu3, fv3);
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int t = (P.term_order >> (2 * s)) & 3;
      if (t == 1 && on1) { dudt = dudt + fu1; dvdt = dvdt + fv1; }
      else if (t == 2 && on2) { dudt = dudt + fu2; dvdt = dvdt + fv2; }
      else if (t == 3 && on3) { dudt = dudt + fu3; dvdt = dvdt + fv3; }
    }
  }
  if (P.irate) {  // infiltration (InfiltrationSourceTerm.cpp:43-62), capacity consumed in place
    T cap = P.icap[g];
    T dh = infiltration_depth<T>(h, ld(P.irate, g), cap, c);
    dhdt = dhdt - c.divdt(dh);
    P.icap[g] = cap - dh;
  }
  rain = 0.0;
  removed = 0.0;
  wall = 0.0;
  if (gx == 0) wall += double(c.divx(fw.h));
  if (gx == P.nx - 1) wall -= double(c.divx(fe.h));
  if (gy == 0) wall += double(c.divy(fs.h));
  if (gy == P.ny - 1) wall -= double(c.divy(fn.h));
  // head boundary target values for this cell (NaN = not selected); a stage boundary
  // (StageBoundarySourceTerm.cpp:48-52) gives water levels, from which the bed is subtracted
  bool head_sel = false;
  T h0 = T(0), h1 = T(0);
  const int hk = fc.head_kind;
  if (hk == 1 || hk == 3) {
    head_sel = ((fc.head_edges & 1u) && gx == 0) || ((fc.head_edges & 2u) && gx == P.nx - 1) ||
               ((fc.head_edges & 4u) && gy == 0) || ((fc.head_edges & 8u) && gy == P.ny - 1);
    h0 = T(fc.hh0); h1 = T(fc.hh1);
  } else if (hk == 2 || hk == 4) {
    h0 = ld(P.hb0p, g); h1 = ld(P.hb1p, g);
    head_sel = true;
  }
  if (head_sel && hk >= 3) {
    if (P.zdat) {  // absolute bed = FP64 datum + FP32 offset; levels minus bed in FP64
      const double zb = P.zdat[datum_tile(gx, gy, P.dtiles_x)] + double(ld(P.z, g));
      h0 = T(double(h0) - zb); h1 = T(double(h1) - zb);
    } else {
      const T zb = ld(P.z, g);
      h0 = h0 - zb; h1 = h1 - zb;
    }
  }
  if (head_sel && !(h0 == h0 && h1 == h1)) head_sel = false;  // NaN = not selected
  auto do_rain = [&]() {
    if (fc.rain_kind == 0) return;
    T q0, q1;
    if (fc.rain_kind == 1) { q0 = T(fc.rq0); q1 = T(fc.rq1); }
    else if (fc.rain_kind == 2) { q0 = ld(P.q0p, g); q1 = ld(P.q1p, g); }
    else { T pp = ld(P.pat, g); q0 = pp * T(fc.rq0); q1 = pp * T(fc.rq1); }
    bool applied;
    T dh = discharge_rate<T>(q0, q1, h, c, applied);
    if (applied) { dhdt = dhdt + dh; rain = double(dh); }
  };
  auto do_head = [&]() {
    if (!head_sel) return;
    T target = head_target<T>(h0, h1, c);
    T before = dhdt;
    dhdt = c.divdt(target - h);
    removed = double(before) - double(dhdt);
  };
  if (P.head_first) { do_head(); do_rain(); }
  else { do_rain(); do_head(); }
  kh = dhdt; ku = dudt; kv = dvdt;
}

// One cell of one stage after its four face fluxes are known: dU/dt, then the Runge-Kutta
// combination (RungeKutta.hpp:377-388) and, on the last stage, the CFL quantity and volume.
template <typename T, typename CC, bool EDDY = false, bool COH = false>
__device__ __forceinline__ void finish_cell(const StageParams<T>& P, int st, const DevForcing& fc, const CC& c,
                                            long long g, int gx, int gy, T h, T u, T v, T dhdx, T dhdy, T dzdx,
                                            T dzdy, const FaceF<T>& fw, const FaceF<T>& fe, const FaceF<T>& fs,
                                            const FaceF<T>& fn, int cur, double dt_d, double& rain,
                                            double& removed, double& walls, T& xcfl, T& xcfl_min, double& vol, const EddyIn<T>* ed = nullptr) {
  T kh, ku, kv;
  double r_, o_, w_;
  cell_dudt<T, CC, EDDY>(P, fc, c, g, gx, gy, h, u, v, dhdx, dhdy, dzdx, dzdy, fw, fe, fs, fn, kh, ku, kv, r_,
                               o_, w_, (T*)nullptr, (T*)nullptr, ed);
  rain += r_;
  removed += o_;
  walls += w_;
  const bool first = st == 0, last = st == P.nstages - 1;
  if ((P.mode & M_STOREK) && !last) {
    P.K[st][0][g] = kh; P.K[st][1][g] = ku; P.K[st][2][g] = kv;
  }
  T* A[3] = {P.S[cur ^ 1][0], P.S[cur ^ 1][1], P.S[cur ^ 1][2]};
  const T* U0[3] = {P.S[cur][0], P.S[cur][1], P.S[cur][2]};
  T k[3] = {kh, ku, kv};
  T out[3];
  if (P.mode & M_ACC) {
    // diagonal tableau: Y_{s+1} = U0 + k_s*a and acc += k_s*b, in the reference's
    // left-to-right order (RungeKutta.hpp:377-388); the skipped zero-coefficient terms
    // k_j*0 (j < s) can only contribute a NaN, which happens exactly when some earlier
    // k_j is not finite, i.e. when acc is not finite while U0 is.
    const T cB = T(P.b[st] * dt_d);
    // FP32 (hc set): the accumulator holds the increment sum_s k_s cB_s, added to U0 once at
    // the last stage; the depth takes it with a per-cell compensation carried across
    // timesteps. Rounding a small, nearly uniform increment (steady rain) onto the depth at
    // every stage otherwise biases the FP32 volume by ~1e-4 over thousands of timesteps.
    const bool incr = sizeof(T) == 4 && P.hc[0] != nullptr;
    T u0v[3], accv[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      u0v[f] = first ? (f == 0 ? h : (f == 1 ? u : v)) : ldst<COH>(U0[f], g);
      accv[f] = first ? (incr ? T(0) : u0v[f]) : ldst<COH>(A[f], g);
    }
    if (!last) {
      const T cA = T(P.a[st][st] * dt_d);
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        T y = u0v[f] + k[f] * cA;
        // FP32 leaves this out: a non-finite accumulator reaches U_N at the last stage anyway
        if constexpr (sizeof(T) == 8)
          if (!first && finite_(u0v[f]) && !finite_(accv[f])) y = Lim<T>::nan();
        P.out(st, f)[g] = y;
      }
    }
    if (!incr) {
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        out[f] = accv[f] + k[f] * cB;
        A[f][g] = out[f];
      }
    } else {
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const T d = accv[f] + k[f] * cB;  // increment sum so far
        if (!last) {
          A[f][g] = d;
          out[f] = d;
        } else if (f == 0) {  // U_N.h = U0.h + d with the carried compensation (Neumaier)
          const T y = d + ldst<COH>(P.hc[cur], g);
          const T t = u0v[0] + y;
          P.hc[cur ^ 1][g] = (sfabs(u0v[0]) >= sfabs(y)) ? (u0v[0] - t) + y : (y - t) + u0v[0];
          out[0] = t;
          A[0][g] = t;
        } else {
          out[f] = u0v[f] + d;
          A[f][g] = out[f];
        }
      }
    }
  } else {
    // general tableau: Y_{s+1} = ((U0 + k_0 c_0) + k_1 c_1) + ... with stored k_j
    T u0v[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) u0v[f] = first ? (f == 0 ? h : (f == 1 ? u : v)) : ldst<COH>(U0[f], g);
    const double* coef = last ? P.b : P.a[st];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      T y = u0v[f];
      for (int j = 0; j < st; ++j) y = y + ldst<COH>(P.K[j][f], g) * T(coef[j] * dt_d);
      y = y + k[f] * T(coef[st] * dt_d);
      out[f] = y;
      if (last) A[f][g] = y;
      else P.out(st, f)[g] = y;
    }
  }
  if (last) {
    // SaintVenantState::max_control_number (State.cpp:204-228) on U_[N]: per cell
    // x = (|u|+c)/dx + (|v|+c)/dy; cn = max(dt*x) = dt*max(x) (rounding is monotone)
    T hh = sfmax(out[0], T(0));
    T cc = ssqrt(T(kG) * hh);
    T xx = c.divx(sfabs(out[1]) + cc) + c.divy(sfabs(out[2]) + cc);
    xcfl = nmax(xcfl, xx);  // a max or min of T values is exact in T
    xcfl_min = nmin(xcfl_min, xx);
    vol += double(out[0]) * P.cell_area;
  }
}

template <typename T, int TX, int TY>
struct StageSmem {
  static constexpr int RX = TX + 4, RY = TY + 4;  // values with a 2-cell halo
  static constexpr int SX = TX + 2, SY = TY + 2;  // slopes with a 1-cell ring
  T val[4][RY][RX];
  T slp[8][SY][SX];
  T fxf[4][TY][TX + 1];
  T fyf[4][TY + 1][TX];
  double red[TX * TY / 32];
};

// One TX x TY tile of one stage: bx, by = tile coordinates, blk = partial-sum slot.
template <typename T, int TX, int TY, bool P2, bool EDDY, bool PRE = false>
__device__ __forceinline__ void stage_tile(const StageParams<T>& P, int st, int bx, int by, long long blk,
                                           StageSmem<T, TX, TY>& s) {
  using DX = DivX<T, P2>;
  using SM = StageSmem<T, TX, TY>;
  constexpr int NT = TX * TY;

  const Ctl* ctl = P.ctl;
  if (ctl->done) return;
  const int cur = ctl->cur;
  const double dt_d = ctl->dt;
  const double tsub = ctl->t_local + P.c[st] * dt_d;

  const int tid = threadIdx.x;
  const int x0 = bx * TX, y0 = by * TY;
  const int nx = P.nx, ny = P.ny;
  const T *Yh = P.in(st, cur, 0), *Yu = P.in(st, cur, 1), *Yv = P.in(st, cur, 2);

  // phase 1: tile + 2-cell halo of h, u, v, z (clamped at the mesh edge; the clamped
  // copies are never used because edge faces and edge slopes use the cell itself)
  const long long zref = P.zdat ? datum_tile(x0, y0, P.dtiles_x) : 0;
  for (int i = tid; i < SM::RX * SM::RY; i += NT) {
    int lx = i % SM::RX, ly = i / SM::RX;
    int gx = min(max(x0 - 2 + lx, 0), nx - 1);
    int gy = min(max(y0 - 2 + ly, 0), ny - 1);
    long long g = (long long)gy * nx + gx;
    s.val[0][ly][lx] = ld(Yh, g);
    s.val[1][ly][lx] = ld(Yu, g);
    s.val[2][ly][lx] = ld(Yv, g);
    s.val[3][ly][lx] = load_bed(P.z, P.zdat, P.dtiles_x, g, gx, gy, zref);
  }
  __syncthreads();

  const DX divx = MkDivX<DX>::make(P.dx), divy = MkDivX<DX>::make(P.dy);
  // phase 2: Minmod3 slopes of h, u, v (State.cpp:176-193) on the tile + ring; the bed
  // slopes (Constants.cpp:39-40) are precomputed once per bed and loaded
  for (int i = tid; i < SM::SX * SM::SY; i += NT) {
    int sx = i % SM::SX, sy = i / SM::SX;
    if ((sx == 0 || sx == SM::SX - 1) && (sy == 0 || sy == SM::SY - 1)) continue;  // unused corners
    int gx = x0 - 1 + sx, gy = y0 - 1 + sy;
    if (gx < 0 || gx >= nx || gy < 0 || gy >= ny) continue;
    int lx = sx + 1, ly = sy + 1;
    bool hasW = gx > 0, hasE = gx < nx - 1, hasN = gy < ny - 1, hasS = gy > 0;
    long long g = (long long)gy * nx + gx;
    s.slp[3][sy][sx] = ld(P.zx, g);
    s.slp[7][sy][sx] = ld(P.zy, g);
    if constexpr (PRE) {  // split schedule: slopes from the slopes pass
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        s.slp[f][sy][sx] = ld(P.pslp[f], g);
        s.slp[4 + f][sy][sx] = ld(P.pslp[3 + f], g);
      }
    } else {
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        s.slp[f][sy][sx] = minmod3<T>(s.val[f][ly][lx - 1], hasW, s.val[f][ly][lx], hasE, s.val[f][ly][lx + 1], divx);
        // Y axis: north (row + 1) is the left neighbour, south the right
        s.slp[4 + f][sy][sx] =
            minmod3<T>(s.val[f][ly + 1][lx], hasN, s.val[f][ly][lx], hasS, s.val[f][ly - 1][lx], divy);
      }
    }
  }
  __syncthreads();

  auto cellv = [&](int gx, int gy) {
    int sx = gx - (x0 - 1), sy = gy - (y0 - 1);
    int lx = sx + 1, ly = sy + 1;
    CellV<T> c;
    c.h = s.val[0][ly][lx]; c.u = s.val[1][ly][lx]; c.v = s.val[2][ly][lx]; c.z = s.val[3][ly][lx];
    c.dhdx = s.slp[0][sy][sx]; c.dudx = s.slp[1][sy][sx]; c.dvdx = s.slp[2][sy][sx]; c.dzdx = s.slp[3][sy][sx];
    c.dhdy = s.slp[4][sy][sx]; c.dudy = s.slp[5][sy][sx]; c.dvdy = s.slp[6][sy][sx]; c.dzdy = s.slp[7][sy][sx];
    return c;
  };
  // phase 3: face fluxes (Fluxes.cpp:44-65)
  const T hdx = T(0.5) * T(P.dx), hdy = T(0.5) * T(P.dy);
  for (int i = tid; i < (TX + 1) * TY; i += NT) {
    int fx = i % (TX + 1), fy = i / (TX + 1);
    int gfx = x0 + fx, gy = y0 + fy;
    if (gy >= ny || gfx > nx) continue;
    int edge = gfx == 0 ? -1 : (gfx == nx ? 1 : 0);
    int gl = edge == -1 ? 0 : gfx - 1;
    int gr = edge == 1 ? nx - 1 : gfx;
    FaceF<T> F;
    face_flux<T, 0>(cellv(gl, gy), cellv(gr, gy), edge, hdx, divx, F);
    s.fxf[0][fy][fx] = F.h; s.fxf[1][fy][fx] = F.u; s.fxf[2][fy][fx] = F.v; s.fxf[3][fy][fx] = F.z;
  }
  for (int i = tid; i < TX * (TY + 1); i += NT) {
    int fx = i % TX, fy = i / TX;
    int gx = x0 + fx, gfy = y0 + fy;
    if (gx >= nx || gfy > ny) continue;
    int edge = gfy == 0 ? -1 : (gfy == ny ? 1 : 0);
    int gl = edge == -1 ? 0 : gfy - 1;
    int gr = edge == 1 ? ny - 1 : gfy;
    FaceF<T> F;
    face_flux<T, 1>(cellv(gx, gl), cellv(gx, gr), edge, hdy, divy, F);
    s.fyf[0][fy][fx] = F.h; s.fyf[1][fy][fx] = F.u; s.fyf[2][fy][fx] = F.v; s.fyf[3][fy][fx] = F.z;
  }
  __syncthreads();

  // phase 4: per cell
  const int tx = tid % TX, ty = tid / TX;
  const int gx = x0 + tx, gy = y0 + ty;
  const bool valid = gx < nx && gy < ny;
  double rain = 0.0, removed = 0.0, walls = 0.0, vol = 0.0;
  T xcfl = T(0), xcfl_min = T(1.0 / 0.0);
  const bool last = st == P.nstages - 1;
  if (valid) {
    const long long g = (long long)gy * nx + gx;
    CellCtx<T, DX> c;
    c.divx = divx; c.divy = divy;
    c.divdt = mkdiv<T>(dt_d);
    c.divL = mkdiv<T>(P.L);
    c.dt = T(dt_d); c.dt_d = dt_d; c.tsub_d = tsub;
    c.manning = P.manning; c.rain_mode = P.rain_mode; c.head_first = P.head_first;
    const int sx = tx + 1, sy = ty + 1, lx = tx + 2, ly = ty + 2;
    const T h = s.val[0][ly][lx], u = s.val[1][ly][lx], v = s.val[2][ly][lx];
    FaceF<T> fw{s.fxf[0][ty][tx], s.fxf[1][ty][tx], s.fxf[2][ty][tx], s.fxf[3][ty][tx]};
    FaceF<T> fe{s.fxf[0][ty][tx + 1], s.fxf[1][ty][tx + 1], s.fxf[2][ty][tx + 1], s.fxf[3][ty][tx + 1]};
    FaceF<T> fs{s.fyf[0][ty][tx], s.fyf[1][ty][tx], s.fyf[2][ty][tx], s.fyf[3][ty][tx]};
    FaceF<T> fn{s.fyf[0][ty + 1][tx], s.fyf[1][ty + 1][tx], s.fyf[2][ty + 1][tx], s.fyf[3][ty + 1][tx]};
    const DevForcing fc = *P.fc;
    EddyIn<T> ed{};
    if constexpr (EDDY) {
      if (P.eddy) {  // second derivatives from the slopes of the tile + ring
        const bool hasW = gx > 0, hasE = gx < nx - 1, hasN = gy < ny - 1, hasS = gy > 0;
        ed.ux = s.slp[1][sy][sx]; ed.uy = s.slp[5][sy][sx]; ed.vx = s.slp[2][sy][sx]; ed.vy = s.slp[6][sy][sx];
        ed.uxx = minmod3<T>(s.slp[1][sy][sx - 1], hasW, ed.ux, hasE, s.slp[1][sy][sx + 1], divx);
        ed.vxx = minmod3<T>(s.slp[2][sy][sx - 1], hasW, ed.vx, hasE, s.slp[2][sy][sx + 1], divx);
        ed.uyy = minmod3<T>(s.slp[5][sy + 1][sx], hasN, ed.uy, hasS, s.slp[5][sy - 1][sx], divy);
        ed.vyy = minmod3<T>(s.slp[6][sy + 1][sx], hasN, ed.vy, hasS, s.slp[6][sy - 1][sx], divy);
      }
    }
    finish_cell<T, CellCtx<T, DX>, EDDY>(P, st, fc, c, g, gx, gy, h, u, v, s.slp[0][sy][sx], s.slp[4][sy][sx],
                                         s.slp[3][sy][sx], s.slp[7][sy][sx], fw, fe, fs, fn, cur, dt_d,
                                         rain, removed, walls, xcfl, xcfl_min, vol, &ed);
  }
  if (last) {
    double mx = block_max<NT>(double(xcfl), s.red);
    double mn = block_min<NT>(double(xcfl_min), s.red);
    double vs = block_sum<NT>(vol, s.red);
    if (tid == 0) {
      P.part[blk] = mx;
      P.part[P.nblk + blk] = mn;
      P.part[2 * P.nblk + blk] = vs;
    }
  }
  if (P.mode & M_TALLY) {
    double rs = block_sum<NT>(rain, s.red);
    double os = block_sum<NT>(removed, s.red);
    double ws = block_sum<NT>(walls, s.red);
    if (tid == 0) store_tallies(P, st, blk, rs, os, ws, dt_d);
  }
}

template <typename T, int TX, int TY, int MINB, bool P2, bool EDDY, bool PRE = false>
__global__ void __launch_bounds__(TX * TY, MINB) stage_kernel(const __grid_constant__ StageParams<T> P, int st) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& s = *reinterpret_cast<StageSmem<T, TX, TY>*>(smem_raw);
  stage_tile<T, TX, TY, P2, EDDY, PRE>(P, st, blockIdx.x, blockIdx.y, (long long)blockIdx.y * gridDim.x + blockIdx.x, s);
}

// Split schedule, first pass: the Minmod3 slopes of the stage input (State.cpp:176-193), one
// thread per cell, into P.pslp; the stage kernel that follows reads them instead of forming
// them from its tile.
template <typename T, bool P2>
__global__ void __launch_bounds__(256) slopes_kernel(const __grid_constant__ StageParams<T> P, int st) {
  using DX = DivX<T, P2>;
  const Ctl* ctl = P.ctl;
  if (ctl->done) return;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nx = P.nx, ny = P.ny;
  if (i >= (long long)nx * ny) return;
  const int cur = ctl->cur;
  const int gx = int(i % nx), gy = int(i / nx);
  const bool hasW = gx > 0, hasE = gx < nx - 1, hasN = gy < ny - 1, hasS = gy > 0;
  const DX divx = MkDivX<DX>::make(P.dx), divy = MkDivX<DX>::make(P.dy);
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    const T* a = P.in(st, cur, f);
    const T c = ld(a, i);
    const T l = hasW ? ld(a, i - 1) : c, r = hasE ? ld(a, i + 1) : c;
    P.pslp[f][i] = minmod3<T>(l, hasW, c, hasE, r, divx);
    // Y axis: north (row + 1) is the left neighbour, south the right
    const T n = hasN ? ld(a, i + nx) : c, so = hasS ? ld(a, i - nx) : c;
    P.pslp[3 + f][i] = minmod3<T>(n, hasN, c, hasS, so, divy);
  }
}

}  // namespace svk

#include "sv_sweep.cuh"

namespace svk {

// Bed slopes once per bed upload (SaintVenantConstants, Constants.cpp:39-40).
// The slopes are computed in T and stored as TO (FP32 with tile datums: FP64 slopes of the
// FP64 bed, rounded once).
template <typename T, typename TO = T>
__device__ __forceinline__ void bed_slope_cell(const T* z, int nx, int ny, double dx, double dy, TO* zx, TO* zy) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)nx * ny;
  if (i >= n) return;
  int gx = int(i % nx), gy = int(i / nx);
  bool hasW = gx > 0, hasE = gx < nx - 1, hasN = gy < ny - 1, hasS = gy > 0;
  T cz = z[i];
  zx[i] = TO(minmod3<T>(hasW ? z[i - 1] : cz, hasW, cz, hasE, hasE ? z[i + 1] : cz, mkdiv<T>(dx)));
  zy[i] = TO(minmod3<T>(hasN ? z[i + nx] : cz, hasN, cz, hasS, hasS ? z[i - nx] : cz, mkdiv<T>(dy)));
}

template <typename T, typename TO = T>
__global__ void bed_slopes_kernel(const T* z, int nx, int ny, double dx, double dy, TO* zx, TO* zy) {
  bed_slope_cell<T, TO>(z, nx, ny, dx, dy, zx, zy);
}

// Fields arrive and leave in FP64 (the interface's type); a solver of another value type
// converts them here, one rounding per value as a host cast would do.
template <typename TI, typename TO>
__global__ void convert_kernel(const TI* __restrict__ src, TO* __restrict__ dst, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = TO(src[i]);
}

// Whether an FP64 field, once converted to T, differs bit for bit from a stored one: sets *flag.
__device__ __forceinline__ bool same_bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
template <typename T>
__global__ void differs_kernel(const double* __restrict__ src, const T* __restrict__ ref, long long n, int* flag) {
  bool diff = false;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    diff = diff || !same_bits(T(src[i]), ref[i]);
  if (diff) *flag = 1;
}

#ifdef SV_DEFINE_COMMON_KERNELS  // non-template kernels: defined in one unit only
// Datum of each 32 x 8 tile of an FP64 bed: the tile's lowest non-NaN value (among values
// that compare equal, such as -0.0 and 0.0, the first in row-major order), rounded down to a
// multiple of 2^-10 m; 0 for a tile without a valid bed. One warp per tile, a lane per column.
__global__ void datum_tiles_kernel(const double* z, int nx, int ny, int dtiles_x, int dtiles_y, double* zdat) {
  const long long t = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (t >= (long long)dtiles_x * dtiles_y) return;  // whole warp
  const int lane = threadIdx.x & 31;
  const int gx = int(t % dtiles_x) * kDatumTX + lane, ty = int(t / dtiles_x);
  double best = 0.0;
  long long bi = -1;  // row-major index of `best`; -1 = none yet
  if (gx < nx) {
    for (int r = 0; r < kDatumTY; ++r) {
      const int gy = ty * kDatumTY + r;
      if (gy >= ny) break;
      const long long i = (long long)gy * nx + gx;
      const double v = z[i];
      if (v != v) continue;
      if (bi < 0 || v < best) { best = v; bi = i; }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_down_sync(kFull, best, o);
    const long long oi = __shfl_down_sync(kFull, bi, o);
    if (oi >= 0 && (bi < 0 || ob < best || (ob == best && oi < bi))) { best = ob; bi = oi; }
  }
  if (lane == 0) zdat[t] = floor((bi < 0 ? 0.0 : best) * 1024.0) / 1024.0;
}

// FP32 offset of each cell's bed from its tile's datum (FP64 difference, rounded once), or the
// absolute FP64 bed from an offset (`to_abs`).
__global__ void datum_offsets_kernel(const double* z, int nx, int ny, int dtiles_x, const double* zdat, float* off) {
  const long long n = (long long)nx * ny;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    off[i] = float(z[i] - zdat[datum_tile(int(i % nx), int(i / nx), dtiles_x)]);
}
__global__ void datum_absolute_kernel(const float* off, int nx, int ny, int dtiles_x, const double* zdat, double* z) {
  const long long n = (long long)nx * ny;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    z[i] = double(off[i]) + zdat[datum_tile(int(i % nx), int(i / nx), dtiles_x)];
}
#endif

// Steps queued for one batch member by one batched advance. The member runs them back to
// back at its own pace: when a step ends, the controller records it and starts the next one
// on the device (TypedTemporalScheme::solve's loop, TemporalScheme.hpp:244-276, moved onto
// the GPU), so members with large timesteps do not wait for the slowest one at every step.
constexpr int kMaxQueuedSteps = 16;
struct StepQueue {
  int n;           // steps queued (0: the member sits this advance out)
  int k;           // steps completed so far
  int status;      // 0, or -5 (time became NaN) / -7 (step limit reached) in step k
  int keep_first;  // 1: step 0 uses the forcing already in place (f[0] unused)
  int cur;         // the member's state parity when the advance ended (host mirror)
  int pad;
  long long limit; // timesteps allowed per step (0: no limit)
  DevForcing f[kMaxQueuedSteps];                             // forcing of each queued step
  unsigned long long acc[kMaxQueuedSteps], rep[kMaxQueuedSteps];   // per-step counts
  double rain[kMaxQueuedSteps], outflow[kMaxQueuedSteps], volume[kMaxQueuedSteps];  // running, at step end
  double wall[kMaxQueuedSteps];
};

struct FinalizeParams {
  Ctl* ctl;
  StepQueue* q;      // batch members: the step queue (null for a solver on its own)
  DevForcing* fc;    // batch members: the member's forcing slot read by its stage kernels
  const double* part;
  long long nblk;
  double cn_target, max_dt, L;
  double cell_area;
  int auto_mode;   // 1: accept/repeat, advance t_local, trim dt (TemporalScheme.hpp:119-146)
  int tally;
  int is_float;    // control number rounded to T = float
  double* result;  // control number, new dt and the repeat flag for a caller's buffer, or null
};

// Fixed-order sum: thread t adds blocks t, t+NT, ... in order, then a fixed tree.
template <int NT> __device__ double fixed_sum(const double* p, long long n, double* red) {
  double a = 0.0;
  for (long long i = threadIdx.x; i < n; i += NT) a += p[i];
  red[threadIdx.x] = a;
  __syncthreads();
  for (int st = NT / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
    __syncthreads();
  }
  double r = red[0];
  __syncthreads();
  return r;
}

__device__ __forceinline__ void finalize_control(const FinalizeParams& F, double mx, double mn, double vol,
                                                 double rain, double outf, double wall);

// The six reductions of a timestep's finalize over the partial slots.
struct Reduced {
  double mx, mn, vol, rain, outf, wall;
  __device__ __forceinline__ void init() {
    mx = vol = rain = outf = wall = 0.0;
    mn = 1.0 / 0.0;
  }
  __device__ __forceinline__ void add(const Reduced& o) {
    mx = nmax(mx, o.mx);  // CFL max and min: NaN-propagating, order-independent
    mn = nmin(mn, o.mn);
    vol += o.vol;
    rain += o.rain;
    outf += o.outf;
    wall += o.wall;
  }
  __device__ __forceinline__ Reduced down(int o) const {
    return {__shfl_down_sync(kFull, mx, o),   __shfl_down_sync(kFull, mn, o),   __shfl_down_sync(kFull, vol, o),
            __shfl_down_sync(kFull, rain, o), __shfl_down_sync(kFull, outf, o), __shfl_down_sync(kFull, wall, o)};
  }
  // slots t, t + n, t + 2n, ... of the partials, in that order
  __device__ __forceinline__ void slots(const FinalizeParams& F, long long t, long long n) {
    init();
    const double* p = F.part;
    const long long m = F.nblk;
#pragma unroll 4
    for (long long i = t; i < m; i += n) {
      Reduced x{p[i], p[m + i], p[2 * m + i], 0.0, 0.0, 0.0};
      if (F.tally) {
        x.rain = p[3 * m + i];
        x.outf = p[4 * m + i];
        x.wall = p[5 * m + i];
      }
      add(x);
    }
  }
  __device__ __forceinline__ void over_warp() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) add(down(o));
  }
};

// The finalize of one solver by a cluster of CTAS blocks of 1024 threads (CTAS = 1: one block).
// One pass over the partials, all six quantities at once: a fixed order for a given number of
// blocks (strided slots per thread, shuffle tree per warp, warps, then blocks), one block
// barrier and, with several blocks, one cluster barrier. What bounds it is latency: the six
// separate trees of ten barriers each that this replaces took 23.5 us for a mesh of a few
// strips (7.8 now), and one block reading 2.3 MB of partials 67 us at 4096 x 4096 (10 now).
constexpr int kFinalizeThreads = 1024;
// slots above which a cluster of kFinalizeCtas blocks shares the reads: up to two slots per
// thread one block is faster (no cluster launch, no cluster barrier)
constexpr long long kFinalizeClusterSlots = 2 * kFinalizeThreads;
constexpr int kFinalizeCtas = 8;
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
template <int CTAS> __device__ __forceinline__ void finalize_body(const FinalizeParams& F) {
  __shared__ Reduced warp_sum_[kFinalizeThreads / 32];
  __shared__ Reduced block_sum_[CTAS];
  if (F.ctl->done) return;  // the same for every block of the cluster
  const int rank = CTAS > 1 ? int(blockIdx.x % CTAS) : 0;
  if constexpr (CTAS > 1) cluster_arrive();
  Reduced r;
  r.slots(F, (long long)rank * kFinalizeThreads + threadIdx.x, (long long)CTAS * kFinalizeThreads);
  r.over_warp();
  if ((threadIdx.x & 31) == 0) warp_sum_[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x < 32) {
    r = warp_sum_[threadIdx.x];
    r.over_warp();
  }
  if constexpr (CTAS > 1) {
    cluster_wait();  // every block of the cluster runs: block 0's shared memory may be written
    if (threadIdx.x == 0) *cooperative_groups::this_cluster().map_shared_rank(&block_sum_[rank], 0) = r;
    cluster_arrive();
    cluster_wait();
    if (rank != 0 || threadIdx.x != 0) return;
    r = block_sum_[0];
    for (int i = 1; i < CTAS; ++i) r.add(block_sum_[i]);
  }
  if (threadIdx.x != 0) return;
  finalize_control(F, r.mx, r.mn, r.vol, r.rain * F.cell_area, r.outf * F.cell_area, r.wall * F.cell_area);
}

// The rest of a timestep's finalize, one thread, from its reductions (CFL max and min over
// cells of (|u|+c)/dx + (|v|+c)/dy, volume, tallies): the control number, accept / repeat and
// the new dt (RungeKutta.cpp:154-167), the step clock and the end-of-step trimming
// (TemporalScheme.hpp:119-146) and, for a batch member, its step queue.
__device__ __forceinline__ void finalize_control(const FinalizeParams& F, double mx, double mn, double vol,
                                                 double rain, double outf, double wall) {
  Ctl* ctl = F.ctl;
  const double dt = ctl->dt;
  // control number: max over cells of dt * x
  double cn;
  if (mx != mx || dt != dt) cn = mx + dt;                  // NaN
  else if (dt == 1.0 / 0.0) cn = (mn == 0.0) ? (0.0 / 0.0) : dt;
  else cn = dt * mx;
  if (F.is_float) cn = double(float(cn));
  // RungeKuttaTemporalScheme::do_timestep (RungeKutta.cpp:154-167), target as parameter
  const double tgt = F.cn_target;
  double nd;
  int rep;
  if (cn > tgt) {
    rep = 1;
    nd = (cn > 5.0 * tgt) ? dt / 5.0 : (dt * tgt) / (cn * 1.1);
  } else if (cn > 0.9 * tgt) {
    rep = 0; nd = dt;
  } else {
    rep = 0; nd = (dt * tgt) / cn;
  }
  if (F.max_dt > 0.0 && nd > F.max_dt) nd = F.max_dt;
  ctl->cn = cn;
  ctl->new_dt = nd;
  ctl->repeat = rep;
  ctl->pend_rain = rain;
  ctl->pend_out = outf;
  ctl->pend_wall = wall;
  ctl->pend_vol = vol;
  if (F.result) {
    F.result[0] = cn;
    F.result[1] = nd;
    F.result[2] = double(rep);
  }
  if (!F.auto_mode) return;
  // TypedTemporalScheme::step (TemporalScheme.hpp:119-146)
  double t = ctl->t_local;
  if (rep) {
    ctl->repeated++; ctl->step_repeated++;
  } else {
    ctl->accepted++; ctl->step_accepted++;
    ctl->rain_in += rain; ctl->outflow += outf; ctl->wall_in += wall; ctl->volume = vol;
    t = t + dt;
    ctl->cur ^= 1;
  }
  double ndt = nd;
  const double L = F.L;
  if (t >= L) {
    ctl->done = 1;
  } else if (t + ndt > L) {
    ndt = L - t;
  } else if (t + 2.0 * ndt > L) {
    ndt = (L - t) * 0.4;
  }
  if (!(t < L) && !(t >= L)) { ctl->done = 1; ctl->error = -5; }   // t became NaN
  ctl->t_local = t;
  ctl->dt = ndt;
  if (ctl->budget > 0 && --ctl->budget == 0 && !ctl->done) ctl->done = 2;  // paused, step not over
  if (F.q == nullptr || !ctl->done) return;
  // batch member: record the step that ended (or failed); start the next queued one
  StepQueue* q = F.q;
  const int k = q->k;
  q->acc[k] = ctl->step_accepted;
  q->rep[k] = ctl->step_repeated;
  q->rain[k] = ctl->rain_in;
  q->outflow[k] = ctl->outflow;
  q->wall[k] = ctl->wall_in;
  q->volume[k] = ctl->volume;
  q->cur = ctl->cur;
  if (ctl->error) { q->status = -5; return; }
  if (ctl->done == 2) { q->status = -7; return; }
  q->k = k + 1;
  if (k + 1 < q->n) {  // start_new_step of the next queued step; dt carries over as in step()
    *F.fc = q->f[k + 1];
    ctl->t_local = 0.0;
    ctl->step_accepted = 0;
    ctl->step_repeated = 0;
    ctl->budget = q->limit;
    ctl->done = 0;
  }
}

template <int CTAS> __global__ void __launch_bounds__(kFinalizeThreads) finalize_kernel(const __grid_constant__ FinalizeParams F) {
  chain_wait();
  finalize_body<CTAS>(F);
}

// Batched finalize: CTAS blocks per instance of a batch.
template <int CTAS>
__global__ void __launch_bounds__(kFinalizeThreads) finalize_batch_kernel(const FinalizeParams* __restrict__ Fs) {
  __shared__ FinalizeParams Fsh;
  chain_wait();
  if (threadIdx.x == 0) Fsh = Fs[blockIdx.x / CTAS];
  __syncthreads();
  finalize_body<CTAS>(Fsh);
}

// ---------------------------------------------------------------------------------------
// Persistent batch kernel. One cooperative launch advances every member of a batch through
// its queued steps (TypedTemporalScheme::solve / step for each member, TemporalScheme.hpp:
// 112-149, 244-276), each member at its own dt. A member's timestep is N stage phases of
// column-sweep strips followed by one finalize phase (reductions and the dt controller).
// A warp looks at 32 members at once (one per lane) for one whose open phase has unclaimed
// items and claims one with one atomicAdd on the member's word, which holds the open phase and
// the next item's number (no retry loop, so claims do not serialise when many warps work on one
// member). A claim past the phase's last item is void and its warp looks elsewhere: no warp
// ever waits for one member while another has work (claims that queued for a member's later
// phases instead held most warps of the GPU on members with nothing to do; 16 catchments of
// 6.2M cells ran 1.7 times slower than in one launch per stage). The warp that completes the last
// item of a phase opens the member's next phase. Phases are ordered by release fences before
// each completion count and acquire fences before each item, and the state buffers are read
// with coherent loads (ldst<true>, copies through L2).
// Every wait is bounded twice: a waiting warp gives up after spin_limit polls during which no
// warp completed an item (a global progress count), and every warp gives up once the launch
// has run max_ns; either records SV_E_TIMEOUT in the launch status, and every warp returns at
// its next poll.
// ---------------------------------------------------------------------------------------
struct PersistMember {
  unsigned long long word;    // open phase (stage 0 .. N-1, N = the finalize) * 2^32 + items claimed
  unsigned int done;          // items of the open phase completed
  int finished;               // 1: no more work for this member in this launch
  long long nstrips;          // column-sweep strips of one stage
};

template <typename T> struct PersistParams {
  const StageParams<T>* Ps;   // [nact]
  const FinalizeParams* Fs;   // [nact]
  PersistMember* mem;         // [nact]
  int nact, nstages;
  int* status;                // 0, or SV_E_TIMEOUT (-6) once a wait gave up
  unsigned long long* progress;   // items completed by all warps (zeroed before the launch)
  unsigned long long spin_limit;  // polls without any completed item before giving up
  unsigned long long max_ns;      // wall-clock bound of the launch, ns
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr int kPersistWarps = 4;   // warps per block

#ifdef SV_DEFINE_COMMON_KERNELS
// mark the members whose step queue starts with nothing to do (their controller is done)
__global__ void persist_init_kernel(const FinalizeParams* Fs, PersistMember* mem, const long long* warp_start,
                                    int nact) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nact) return;
  PersistMember m{};
  m.nstrips = warp_start[k + 1] - warp_start[k];
  m.finished = Fs[k].ctl->done != 0 ? 1 : 0;
  mem[k] = m;
}
#endif

// The finalize of one member by one warp: the same reductions over 32 strided chains (sums
// agree with the block's to rounding; the CFL max and min, which set dt, are the same values).
__device__ __forceinline__ void finalize_warp(const FinalizeParams& F) {
  Reduced r;
  r.slots(F, threadIdx.x & 31, 32);
  r.over_warp();
  if ((threadIdx.x & 31) == 0)
    finalize_control(F, r.mx, r.mn, r.vol, r.rain * F.cell_area, r.outf * F.cell_area, r.wall * F.cell_area);
  __syncwarp();
}

// The members' parameters as kernel parameters, for batches of up to kBatchMembers members
// (constant operands of the sweep, see sweep_batch_kernel); BANK = 1: a larger batch, whose
// warps copy an item's parameters to shared memory.
template <typename T, int BANK> struct MemberBank { StageParams<T> m[BANK]; };

template <typename T, int MINB, bool P2, bool EXTRA, int BANK>
__global__ void __launch_bounds__(32 * kPersistWarps, MINB)
    persist_batch_kernel(const __grid_constant__ PersistParams<T> PP, const __grid_constant__ MemberBank<T, BANK> bank) {
  __shared__ __align__(16) StageParams<T> Psh[BANK > 1 ? 1 : kPersistWarps];
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  const int lane = threadIdx.x, wib = uniform(threadIdx.y);
  const int N = PP.nstages, nact = PP.nact;
  const long long gwarp = (long long)blockIdx.x * kPersistWarps + wib;
  const int k0 = nact > 0 ? int(gwarp % nact) : 0;
  volatile int* status = PP.status;
  volatile unsigned long long* progress = PP.progress;
  const unsigned long long t_start = global_ns();
  unsigned long long idle = 0, seen = *progress;
  // one poll of a waiting warp; true when the warp must return (another warp gave up, the
  // launch ran out of time, or spin_limit polls passed with no item completed anywhere)
  auto poll_gives_up = [&]() -> bool {
    if (*status != 0) return true;
    if (global_ns() - t_start > PP.max_ns) {
      if (lane == 0) atomicExch((int*)PP.status, -6);
      return true;
    }
    const unsigned long long now = *progress;
    if (now != seen) {
      idle = 0;
      seen = now;
    } else if (++idle > PP.spin_limit) {
      if (lane == 0) atomicExch((int*)PP.status, -6);
      return true;
    } else {
      __nanosleep(256);
    }
    return false;
  };
  while (true) {
    if (*status != 0) return;  // whole warp: another warp gave up
    if (global_ns() - t_start > PP.max_ns) {
      if (lane == 0) atomicExch((int*)PP.status, -6);
      return;
    }
    // a member whose open phase has unclaimed items: the lanes look at 32 members at once,
    // starting from this warp's own member so that warps spread over the members
    int pick = -1;
    bool any_active = false;
    for (int j0 = 0; j0 < nact && pick < 0; j0 += 32) {
      const int j = j0 + lane;
      bool act = false, open = false;
      if (j < nact) {
        const PersistMember* m = PP.mem + (k0 + j) % nact;
        if (!*(volatile const int*)&m->finished) {
          act = true;
          const unsigned long long w = *(volatile const unsigned long long*)&m->word;
          open = (w & 0xffffffffull) < ((w >> 32) < (unsigned long long)N ? (unsigned long long)m->nstrips : 1ull);
        }
      }
      any_active = __any_sync(kFull, act) || any_active;
      const unsigned b = __ballot_sync(kFull, open);
      if (b) pick = (k0 + j0 + __ffs(b) - 1) % nact;
    }
    if (!any_active) return;  // every member has finished
    if (pick < 0) {
      if (poll_gives_up()) return;
      continue;
    }
    // claim the open phase's next item
    PersistMember* m = PP.mem + pick;
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(&m->word, 1ull);
    t = __shfl_sync(kFull, t, 0);
    const int s = int(t >> 32);
    const unsigned item = unsigned(t);
    const unsigned nwork = s < N ? unsigned(m->nstrips) : 1u;
    if (item >= nwork) continue;  // others took the last ones
    __threadfence();  // acquire: the previous phases' writes of every warp
    if (s < N) {
      // stage s, strip `item` of the member's list
      auto& sm = reinterpret_cast<SweepShared<T>*>(sweep_smem)[wib];
      const int pk = uniform(pick), st = uniform(s);
      if constexpr (BANK > 1) {
        const StageParams<T>& SP = bank.m[pk];
        sweep_strip<T, P2, EXTRA, false, true>(SP, st, SP.strips[item], sm);
      } else {
        static_assert(sizeof(StageParams<T>) % 4 == 0, "parameter block copied as 32-bit words");
        const unsigned* src = reinterpret_cast<const unsigned*>(PP.Ps + pk);
        unsigned* dst = reinterpret_cast<unsigned*>(&Psh[wib]);
        for (int i = lane; i < int(sizeof(StageParams<T>) / 4); i += 32) dst[i] = src[i];
        __syncwarp();
        const StageParams<T>& SP = Psh[wib];
        sweep_strip<T, P2, EXTRA, false, true>(SP, st, SP.strips[item], sm);
      }
      __syncwarp();
    } else {
      finalize_warp(PP.Fs[pick]);
    }
    __threadfence();  // release this item's writes before counting it
    int last = 0;
    if (lane == 0) {
      last = atomicAdd(&m->done, 1u) + 1u == nwork;
      atomicAdd(PP.progress, 1ull);
    }
    last = __shfl_sync(kFull, last, 0);
    if (last) {
      __threadfence();  // acquire the other items of the phase
      if (lane == 0) {
        m->done = 0;
        // after a finalize the member goes on while its controller has a step running
        const bool more = s < N || (*(volatile int*)&PP.Fs[pick].ctl->done == 0);
        __threadfence();
        if (more) atomicExch(&m->word, (unsigned long long)(s < N ? s + 1 : 0) << 32);
        else atomicExch(&m->finished, 1);
      }
      __syncwarp();
    }
    idle = 0;
    seen = *progress;
  }
}

#ifdef SV_DEFINE_COMMON_KERNELS
// Host-API accept (RungeKutta.hpp:428-431): flip the state parity, apply the pending tallies.
__global__ void accept_kernel(Ctl* ctl) {
  ctl->cur ^= 1;
  ctl->accepted++;
  ctl->rain_in += ctl->pend_rain;
  ctl->outflow += ctl->pend_out;
  ctl->wall_in += ctl->pend_wall;
  ctl->volume = ctl->pend_vol;
}
__global__ void begin_step_kernel(Ctl* ctl, int new_step, long long budget) {
  if (new_step) {
    ctl->t_local = 0.0;
    ctl->step_accepted = 0;
    ctl->step_repeated = 0;
  }
  ctl->done = 0;
  ctl->budget = budget;
}
// start a batched advance of queued steps: each member's first step (or, with no steps
// queued or a member that already failed, nothing: done at once)
__global__ void begin_queue_kernel(const FinalizeParams* Fs, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Ctl* c = Fs[i].ctl;
  StepQueue* q = Fs[i].q;
  c->t_local = 0.0;
  c->step_accepted = 0;
  c->step_repeated = 0;
  c->budget = q->limit;
  q->k = 0;
  q->status = 0;
  q->cur = c->cur;
  if (c->error) {
    q->status = -5;
    c->done = 1;
  } else if (q->n <= 0) {
    c->done = 1;
  } else {
    if (!q->keep_first) *Fs[i].fc = q->f[0];
    c->done = 0;
  }
}
// done flags of a batch into one array (1: step complete, nonzero error code: -1)
__global__ void gather_done_kernel(Ctl* const* ctls, int n, int* done) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  done[i] = ctls[i]->error ? -1 : ctls[i]->done;
}
#endif

// Volume of a cell field: per-CTA FP64 partials (same tiling and reduction as the stage
// kernel's last stage), then a fixed-order sum.
template <typename T, int TX, int TY>
__global__ void __launch_bounds__(TX * TY) volume_partials_kernel(const T* h, int nx, int ny, double area,
                                                                  double* part) {
  __shared__ double red[TX * TY / 32];
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int gx = blockIdx.x * TX + tx, gy = blockIdx.y * TY + ty;
  double v = 0.0;
  if (gx < nx && gy < ny) v = double(h[(long long)gy * nx + gx]) * area;
  double s = block_sum<TX * TY>(v, red);
  if (threadIdx.x == 0) part[(long long)blockIdx.y * gridDim.x + blockIdx.x] = s;
}
template <int NT> __global__ void __launch_bounds__(NT) sum_kernel(const double* p, long long n, double* out) {
  __shared__ double red[NT];
  double r = fixed_sum<NT>(p, n, red);
  if (threadIdx.x == 0) *out = r;
}

// ------------------------------- debug / per-function kernels -------------------------
template <typename T> struct DebugParams {
  int nx, ny;
  double dx, dy;
  const T *h, *u, *v, *z;
  T *dhdx, *dudx, *dvdx, *dzdx, *dhdy, *dudy, *dvdy, *dzdy;
  T *fh, *fu, *fv, *fz, *fb;
  T* k[3];
};

// SpatialDerivativeOperationKernel over global arrays (State.cpp:187-192, Constants.cpp:39-40)
template <typename T> __global__ void debug_slopes_kernel(const DebugParams<T> D) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)D.nx * D.ny;
  if (i >= n) return;
  int gx = int(i % D.nx), gy = int(i / D.nx);
  bool hasW = gx > 0, hasE = gx < D.nx - 1, hasN = gy < D.ny - 1, hasS = gy > 0;
  Div<T> divx = mkdiv<T>(D.dx), divy = mkdiv<T>(D.dy);
  const T* src[4] = {D.h, D.u, D.v, D.z};
  T* dx_[4] = {D.dhdx, D.dudx, D.dvdx, D.dzdx};
  T* dy_[4] = {D.dhdy, D.dudy, D.dvdy, D.dzdy};
  for (int f = 0; f < 4; ++f) {
    const T* a = src[f];
    T c = a[i];
    T l = hasW ? a[i - 1] : c, r = hasE ? a[i + 1] : c;
    dx_[f][i] = minmod3<T>(l, hasW, c, hasE, r, divx);
    T nn = hasN ? a[i + D.nx] : c, ss = hasS ? a[i - D.nx] : c;
    dy_[f][i] = minmod3<T>(nn, hasN, c, hasS, ss, divy);
  }
}

// SaintVenantFluxKernel over all faces (Fluxes.cpp:55-64)
template <typename T> __global__ void debug_flux_kernel(const DebugParams<T> D) {
  long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long nvf = (long long)(D.nx + 1) * D.ny;
  long long nf = nvf + (long long)(D.ny + 1) * D.nx;
  if (f >= nf) return;
  auto cell = [&](long long i) {
    CellV<T> c;
    c.h = D.h[i]; c.u = D.u[i]; c.v = D.v[i]; c.z = D.z[i];
    c.dhdx = D.dhdx[i]; c.dudx = D.dudx[i]; c.dvdx = D.dvdx[i]; c.dzdx = D.dzdx[i];
    c.dhdy = D.dhdy[i]; c.dudy = D.dudy[i]; c.dvdy = D.dvdy[i]; c.dzdy = D.dzdy[i];
    return c;
  };
  FaceF<T> F;
  T br;
  if (f < nvf) {
    long long fx = f % (D.nx + 1), fy = f / (D.nx + 1);
    int edge = fx == 0 ? -1 : (fx == D.nx ? 1 : 0);
    long long l = fy * D.nx + (edge == -1 ? 0 : fx - 1);
    long long r = fy * D.nx + (edge == 1 ? D.nx - 1 : fx);
    br = face_flux<T, 0>(cell(l), cell(r), edge, T(0.5) * T(D.dx), mkdiv<T>(D.dx), F);
  } else {
    long long f2 = f - nvf;
    long long fx = f2 % D.nx, fy = f2 / D.nx;
    int edge = fy == 0 ? -1 : (fy == D.ny ? 1 : 0);
    long long l = (edge == -1 ? 0 : fy - 1) * D.nx + fx;
    long long r = (edge == 1 ? D.ny - 1 : fy) * D.nx + fx;
    br = face_flux<T, 1>(cell(l), cell(r), edge, T(0.5) * T(D.dy), mkdiv<T>(D.dy), F);
  }
  D.fh[f] = F.h; D.fu[f] = F.u; D.fv[f] = F.v; D.fz[f] = F.z; D.fb[f] = br;
}

// temporal derivative + sources + boundaries per cell from the global face arrays
template <typename T>
__global__ void debug_cell_kernel(const StageParams<T> P, const DebugParams<T> D, T* nh, T* sf) {
  long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)P.nx * P.ny;
  if (g >= n) return;
  const Ctl* ctl = P.ctl;
  const double dt_d = ctl->dt;
  int gx = int(g % P.nx), gy = int(g / P.nx);
  CellCtx<T> c;
  c.divx = mkdiv<T>(P.dx); c.divy = mkdiv<T>(P.dy);
  c.divdt = mkdiv<T>(dt_d); c.divL = mkdiv<T>(P.L);
  c.dt = T(dt_d); c.dt_d = dt_d; c.tsub_d = ctl->t_local;
  c.manning = P.manning; c.rain_mode = P.rain_mode; c.head_first = P.head_first;
  long long w = (long long)gy * (P.nx + 1) + gx, e = w + 1;
  long long sf_ = (long long)(P.nx + 1) * P.ny + (long long)gy * P.nx + gx, nf_ = sf_ + P.nx;
  FaceF<T> fw{D.fh[w], D.fu[w], D.fv[w], D.fz[w]}, fe{D.fh[e], D.fu[e], D.fv[e], D.fz[e]};
  FaceF<T> fs{D.fh[sf_], D.fu[sf_], D.fv[sf_], D.fz[sf_]}, fn{D.fh[nf_], D.fu[nf_], D.fv[nf_], D.fz[nf_]};
  const DevForcing fc = *P.fc;
  T kh, ku, kv;
  double rain, removed, wall;
  EddyIn<T> ed{};
  if (P.eddy) {  // second derivatives from the mesh-wide slope fields
    const int nx = P.nx;
    const bool hasW = gx > 0, hasE = gx < nx - 1, hasN = gy < P.ny - 1, hasS = gy > 0;
    ed.ux = D.dudx[g]; ed.uy = D.dudy[g]; ed.vx = D.dvdx[g]; ed.vy = D.dvdy[g];
    ed.uxx = minmod3<T>(hasW ? D.dudx[g - 1] : ed.ux, hasW, ed.ux, hasE, hasE ? D.dudx[g + 1] : ed.ux, c.divx);
    ed.vxx = minmod3<T>(hasW ? D.dvdx[g - 1] : ed.vx, hasW, ed.vx, hasE, hasE ? D.dvdx[g + 1] : ed.vx, c.divx);
    ed.uyy = minmod3<T>(hasN ? D.dudy[g + nx] : ed.uy, hasN, ed.uy, hasS, hasS ? D.dudy[g - nx] : ed.uy, c.divy);
    ed.vyy = minmod3<T>(hasN ? D.dvdy[g + nx] : ed.vy, hasN, ed.vy, hasS, hasS ? D.dvdy[g - nx] : ed.vy, c.divy);
  }
  cell_dudt<T, CellCtx<T>, true>(P, fc, c, g, gx, gy, D.h[g], D.u[g], D.v[g], D.dhdx[g], D.dhdy[g], D.dzdx[g],
                                 D.dzdy[g], fw, fe, fs, fn, kh, ku, kv, rain, removed, wall, nh + g, sf + g, &ed);
  D.k[0][g] = kh; D.k[1][g] = ku; D.k[2][g] = kv;
}

}  // namespace svk
