// sv_launch.h -- host-callable launchers for the kernels in sv_kernels.cuh. They are
// explicitly instantiated per value type in sv_f64.cu (compiled with -fmad=false so every
// FP64 operation is separately rounded, as in the reference) and sv_f32.cu.
#pragma once
#include <cuda_runtime.h>

#include <cmath>

#include "sv_kernels.cuh"

namespace svk {

// Tile shapes compiled for the fused stage kernel (TX x TY cells per CTA, MINB resident
// CTAs per SM requested from the register allocator).
struct TileShape { int tx, ty, minb; };
constexpr TileShape kTiles[] = {{32, 8, 1}, {32, 8, 3}, {32, 4, 4}, {64, 4, 3}};
constexpr int kNumTiles = 4;

template <typename T> size_t stage_smem_bytes(int tile);
template <typename T> cudaError_t launch_stage(const StageParams<T>& P, int st, int tile, cudaStream_t s);

// Stage-kernel variants, in two schedules:
//  fused (one pass per RK stage): 0..3 the tiled shared-memory kernel with kTiles[v]; 4..10 and
//   12..15 the column sweep with the strip heights and register caps (resident 4-warp blocks per
//   SM) of kSweeps (12..15 FP32 only); variant 5 takes both from the mesh size;
//  split (two passes per RK stage): 11 the slopes pass (slopes_kernel) then the tiled 32 x 8
//   kernel at 3 CTAs/SM reading those slopes.
constexpr int kNumVariants = 16;
constexpr int kSplitVariant = 11;
constexpr int kAutoVariant = 5;
struct SweepShape { int rows, cap; };
constexpr SweepShape kSweeps[kNumVariants] = {{0, 0},  {0, 0},  {0, 0},  {0, 0},  {16, 4}, {32, 4},
                                              {64, 4}, {32, 3}, {32, 4}, {32, 5}, {32, 6}, {0, 0},
                                              {32, 3}, {32, 4}, {32, 7}, {32, 8}};
// the row-tile kernel (tile_rows_kernel): what variant 5 runs on small meshes
constexpr int kTileRowsVariant = kNumVariants;
// cell sizes within which the sweeps' FP64 quotients stay in the range of the exact division
inline bool exact_mesh(double dx, double dy, bool fp64) {
  auto fits = [](double d) { return d >= 0x1p-30 && d <= 0x1p40; };
  return !fp64 || (fits(dx) && fits(dy));
}
// dx and dy both powers of two: the mesh divisions are exact multiplies
inline bool pow2_mesh(double dx, double dy) {
  int e;
  return std::frexp(dx, &e) == 0.5 && std::frexp(dy, &e) == 0.5;
}
// resident blocks per SM of the batch kernels, and of the sweeps with every source term: FP32 at 4 and 5 blocks
// 526 and 457 us a stage at 3000 x 3000 with all terms (408 with two forms, splits_forms); FP64 at
// 3 and 4, which spills, 571 and 816 at 2048 x 2048
template <typename T> constexpr int kBatchCap = sizeof(T) == 8 ? 4 : 6;
template <typename T> constexpr int kBatchExtraCap = sizeof(T) == 8 ? 3 : 4;
template <typename T> constexpr int kExtraCap = sizeof(T) == 8 ? 3 : 5;
// variants compiled for FP32 solvers only
inline bool variant_is_fp32_only(int v) { return v >= 12 && v <= 15; }
inline bool variant_is_sweep(int v) { return v >= 0 && v < kNumVariants && kSweeps[v].rows > 0; }
inline bool variant_is_split(int v) { return v == kSplitVariant; }
// strips of `rows` rows of a mesh
inline long long strip_count(long long nx, long long ny, int rows) {
  return ((nx + kSweepOut - 1) / kSweepOut) * ((ny + rows - 1) / rows);
}
// Strips that are resident at once with one warp per scheduler: 148 SMs, 4-warp blocks.
constexpr long long kWaveStrips = 148 * 4;
constexpr long long kFillStrips = 4 * kWaveStrips;
// Strip height by mesh size, for variant 5. A strip marches its rows one after another, so a mesh
// of few strips waits for single warps (FP64 3.7 us a row, FP32 1.6); a short strip repeats more
// of its neighbours' rows; and a few strips more than are resident at once take a further wave.
// The height with the smallest estimate is taken: rows + 3 times the waves `x` of strips, where
// part of a wave is quicker a row than a full one, and a last wave that is nearly empty costs up
// to 0.3 of one in the first waves and less the more there are (strips of unequal duration fill
// in). Constants fitted to stage times of 4 to 64 rows on meshes of 0.3 to 17M cells; the choice
// is within 7 % of the best height on each. Microseconds per stage on B200, the tallest of 32, 16,
// 8 and 4 rows that fills the SMs / this choice: FP64 73 (8 rows) / 66 (10) at 900 x 700, 109 (16) /
// 98 (9) at 1100 x 1001, 311 (32) / 288 (34) at 2048 x 2048, 974 (32) / 945 (44) at 4096 x 4096; FP32
// 38 (8) / 31 (7) at 900 x 700, 130 (32) / 120 (43) at 2048 x 2048, 406 / 406 at 4096 x 4096; with
// every source term FP32 64 (16) / 58 (14) at 1200 x 900, FP64 65 (4) / 58 (6) at 601 x 433.
template <typename T> inline int auto_rows(long long nx, long long ny, bool extra) {
  constexpr bool F64 = sizeof(T) == 8;
  const double resident = double(kWaveStrips) * (extra ? kExtraCap<T> : F64 ? 4 : 6);
  int best = 4;
  double least = 0.0;
  for (int rows = 4; rows <= 44; ++rows) {
    const double x = double(strip_count(nx, ny, rows)) / resident;
    double waves;
    if (x <= 1.0) {
      waves = extra ? 0.7 + 0.3 * x : F64 ? 0.88 + 0.3 * x : 0.6 + 0.4 * x;
    } else {
      const double y = 1.02 * x;
      waves = x + 0.3 * (1.0 - (y - std::floor(y))) / std::floor(y);
    }
    const double cost = (rows + 3) * waves;
    if (rows == 4 || cost < least) { best = rows; least = cost; }
  }
  return best;
}
// Whether variant 5 runs the row-tile kernel on a mesh: while its blocks (12 warps; one resident per
// SM in FP64, two in FP32) take about two rounds. Per stage on B200, row tiles against 4-row
// strips: FP64 13 / 27 us at 100 x 100, 23 / 28 at 256 x 256, 38 / 31 at 400 x 400; FP32 11 / 17 at
// 64 x 64, 15 / 18 at 256 x 256, 20 / 20 at 400 x 400.
template <typename T> inline bool prefers_tile_rows(long long nx, long long ny) {
  return strip_count(nx, ny, kTileRows) <= (sizeof(T) == 8 ? 330 : 660);
}
// register caps compiled: FP64 3 and 4 blocks per SM, FP32 4 to 7 (tighter ones spill: FP64 stages at 4096 x 4096
// 1.3 ms at 5 blocks against 0.92 at 4, FP32 455 us at 8 against 408 at 6)
template <typename T> inline int clamp_cap(int cap) {
  const int lo = sizeof(T) == 8 ? 3 : 4, hi = sizeof(T) == 8 ? 4 : 7;
  return cap < lo ? lo : (cap > hi ? hi : cap);
}
// FP32, variant 5: the fewest blocks per SM, from 4, with which all strips are resident at once
// (each warp then runs fastest), else 6: at 900 x 700 and 8 rows (4.9 warps per scheduler) 38, 30 and 31
// us at 4, 5 and 6 blocks per SM; at 10 rows (3.9) 32, 33 and 34; 445 against 408 at 4096 x 4096 at 4 and 6
template <typename T> inline int variant_cap(int v, long long strips) {
  if (v == kAutoVariant && sizeof(T) == 4) return strips <= kFillStrips ? 4 : strips <= 5 * kWaveStrips ? 5 : 6;
  return clamp_cap<T>(kSweeps[v].cap);
}
// Whether interior strips run the form without edge tests. It is the faster one (FP64 10 % at
// 4096 x 4096, FP32 with every source term 11 % at 3000 x 3000), but while all strips are resident at
// once the SMs that hold both kinds evict one code with the other from the instruction cache: FP64 66 us
// with one form against 75 with two at 900 x 700 and 10 rows, 40 against 45 at 600 x 500 and 5 rows,
// FP32 with eddy viscosity 58 against 64 at 1200 x 900 and 14 rows. The lean FP32 sweep is small
// enough for two at any size; FP64 with every term is not at any (2 % either way).
template <typename T> inline bool splits_forms(long long strips, bool extra) {
  if (sizeof(T) == 8) return !extra && strips > kFillStrips;
  return !extra || strips > kExtraCap<T> * kWaveStrips;
}
// per-CTA partial count of the tiled variants
inline long long tiled_partials(int v, long long nx, long long ny) {
  if (v == kSplitVariant) v = 1;  // the split schedule's stage pass is the tiled 32 x 8 kernel
  return ((nx + kTiles[v].tx - 1) / kTiles[v].tx) * ((ny + kTiles[v].ty - 1) / kTiles[v].ty);
}
// a column-sweep variant with the shape of a lower one (the autotuner skips it)
template <typename T> inline bool variant_repeats(int v) {
  if (!variant_is_sweep(v) || v == kAutoVariant) return false;
  for (int u = 0; u < v; ++u)
    if (u != kAutoVariant && variant_is_sweep(u) && kSweeps[u].rows == kSweeps[v].rows &&
        clamp_cap<T>(kSweeps[u].cap) == clamp_cap<T>(kSweeps[v].cap))
      return true;
  return false;
}
// stage `st` of a timestep. extra: source terms, boundaries or a tableau that the lean sweep leaves out (sweep_rows)
template <typename T> cudaError_t launch_variant(const StageParams<T>& P, int st, int variant, bool extra, cudaStream_t s);
// classes of the column sweep's strips of `rows` rows (strip_class_kernel)
template <typename T> cudaError_t launch_strip_classes(const T* z, int nx, int ny, double dx, double dy, int rows,
                                                       long long nstrips, unsigned char* cls, cudaStream_t s);
template <typename T> cudaError_t launch_bed_slopes(const T* z, int nx, int ny, double dx, double dy, T* zx, T* zy,
                                                    cudaStream_t s);
// FP64 <-> T conversion of a field on the device
template <typename T> cudaError_t launch_from_f64(const double* src, T* dst, long long n, cudaStream_t s);
template <typename T> cudaError_t launch_to_f64(const T* src, double* dst, long long n, cudaStream_t s);
// *flag = 1 when T(src[i]) differs bit for bit from ref[i] for some i (flag left as it was otherwise)
template <typename T> cudaError_t launch_differs(const double* src, const T* ref, long long n, int* flag, cudaStream_t s);
// FP32 with tile datums, from an FP64 bed on the device: the tile datums, the FP32 offsets and
// the bed slopes (FP64, rounded once); and the absolute FP64 bed back from the offsets
cudaError_t launch_datum_bed(const double* z, int nx, int ny, double dx, double dy, int dtiles_x, int dtiles_y,
                             double* zdat, float* off, float* zx, float* zy, cudaStream_t s);
cudaError_t launch_datum_absolute(const float* off, int nx, int ny, int dtiles_x, const double* zdat, double* z,
                                  cudaStream_t s);
template <typename T> cudaError_t launch_volume(const T* h, int nx, int ny, double area, double* part, int tile,
                                                cudaStream_t s);
template <typename T> cudaError_t launch_debug(const StageParams<T>& P, const DebugParams<T>& D, T* nh, T* sf,
                                               cudaStream_t s);
// stage `st` of every one of n solvers (host array Ps) in one launch per kBatchMembers of them;
// p2 when every solver's dx and dy are powers of two, extra when any solver needs it
constexpr int kBatchVariant = 8;
template <typename T> cudaError_t launch_sweep_batch(const StageParams<T>* Ps, int n, int st, bool p2, bool extra,
                                                     cudaStream_t s);
// persistent batch kernel (persist_batch_kernel), cooperative launch filling the device; Ps: the
// members' parameters on the host (PP.Ps: the same on the device)
template <typename T> cudaError_t launch_persist(const PersistParams<T>& PP, const StageParams<T>* Ps, bool p2,
                                                 bool extra, cudaStream_t s);
cudaError_t launch_persist_init(const FinalizeParams* Fs, PersistMember* mem, const long long* warp_start, int nact,
                                cudaStream_t s);
cudaError_t launch_finalize(const FinalizeParams& F, cudaStream_t s);
cudaError_t launch_finalize_batch(const FinalizeParams* Fs, int ninst, long long max_nblk, cudaStream_t s);
cudaError_t launch_begin_queue(const FinalizeParams* Fs, int n, cudaStream_t s);
cudaError_t launch_gather_done(Ctl* const* ctls, int n, int* done, cudaStream_t s);
cudaError_t launch_sum(const double* p, long long n, double* out, cudaStream_t s);
cudaError_t launch_accept(Ctl* ctl, cudaStream_t s);
cudaError_t launch_begin_step(Ctl* ctl, int new_step, long long budget, cudaStream_t s);

}  // namespace svk
