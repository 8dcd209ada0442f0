// sv_inst.cuh -- launcher definitions, included once per value type by sv_f64.cu / sv_f32.cu
// with SV_T defined to the value type.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <memory>

#include "sv_launch.h"

namespace svk {

// cudaFuncSetAttribute applies to the device that is current when it is called, so the
// opt-in to more than 48 KB of dynamic shared memory is made once per device and kernel.
// `done` is a per-kernel table indexed by device number.
constexpr int kMaxAttrDevices = 64;
template <typename K>
static cudaError_t smem_optin(K kernel, int bytes, std::atomic<bool> (&done)[kMaxAttrDevices]) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < kMaxAttrDevices && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < kMaxAttrDevices) done[dev].store(true, std::memory_order_release);
  return cudaSuccess;
}

// a launch in a chain (chain_wait), with dynamic shared memory opted in above 48 KB
template <auto KERNEL, typename... Args>
static cudaError_t launch_chained(dim3 grid, dim3 block, int smem, cudaStream_t s, const Args&... args) {
  if (smem > 48 * 1024) {
    static std::atomic<bool> attr_set[kMaxAttrDevices];
    cudaError_t e = smem_optin(KERNEL, smem, attr_set);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, KERNEL, args...);
}

template <typename T, int TX, int TY, int MINB, bool P2, bool EDDY, bool PRE = false>
static cudaError_t launch_stage_p(const StageParams<T>& P, int st, cudaStream_t s) {
  using SM = StageSmem<T, TX, TY>;
  static std::atomic<bool> attr_set[kMaxAttrDevices];
  cudaError_t e = smem_optin(stage_kernel<T, TX, TY, MINB, P2, EDDY, PRE>, int(sizeof(SM)), attr_set);
  if (e != cudaSuccess) return e;
  dim3 grid((P.nx + TX - 1) / TX, (P.ny + TY - 1) / TY);
  stage_kernel<T, TX, TY, MINB, P2, EDDY, PRE><<<grid, TX * TY, sizeof(SM), s>>>(P, st);
  return cudaGetLastError();
}

// split schedule: the slopes pass, then the tiled 32 x 8 stage kernel reading its slopes
template <typename T> static cudaError_t launch_split_t(const StageParams<T>& P, int st, cudaStream_t s) {
  const bool p2 = pow2_mesh(P.dx, P.dy);
  const long long n = (long long)P.nx * P.ny;
  const unsigned blocks = unsigned((n + 255) / 256);
  if (p2) slopes_kernel<T, true><<<blocks, 256, 0, s>>>(P, st);
  else slopes_kernel<T, false><<<blocks, 256, 0, s>>>(P, st);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (P.eddy)
    return p2 ? launch_stage_p<T, 32, 8, 3, true, true, true>(P, st, s) : launch_stage_p<T, 32, 8, 3, false, true, true>(P, st, s);
  return p2 ? launch_stage_p<T, 32, 8, 3, true, false, true>(P, st, s) : launch_stage_p<T, 32, 8, 3, false, false, true>(P, st, s);
}
// kernels compiled with the eddy-viscosity term run only for solvers that have it
template <typename T, int TX, int TY, int MINB> static cudaError_t launch_stage_t(const StageParams<T>& P, int st, cudaStream_t s) {
  const bool p2 = pow2_mesh(P.dx, P.dy);
  if (P.eddy)
    return p2 ? launch_stage_p<T, TX, TY, MINB, true, true>(P, st, s) : launch_stage_p<T, TX, TY, MINB, false, true>(P, st, s);
  return p2 ? launch_stage_p<T, TX, TY, MINB, true, false>(P, st, s) : launch_stage_p<T, TX, TY, MINB, false, false>(P, st, s);
}

template <> size_t stage_smem_bytes<SV_T>(int tile) {
  switch (tile) {
    case 0: return sizeof(StageSmem<SV_T, 32, 8>);
    case 1: return sizeof(StageSmem<SV_T, 32, 8>);
    case 2: return sizeof(StageSmem<SV_T, 32, 4>);
    default: return sizeof(StageSmem<SV_T, 64, 4>);
  }
}

template <> cudaError_t launch_stage<SV_T>(const StageParams<SV_T>& P, int st, int tile, cudaStream_t s) {
  switch (tile) {
    case 0: return launch_stage_t<SV_T, 32, 8, 1>(P, st, s);
    case 1: return launch_stage_t<SV_T, 32, 8, 3>(P, st, s);
    case 2: return launch_stage_t<SV_T, 32, 4, 4>(P, st, s);
    default: return launch_stage_t<SV_T, 64, 4, 3>(P, st, s);
  }
}

// dynamic shared memory of the sweeps
constexpr int kRingBytes = kSweepWarps * int(sizeof(SweepShared<SV_T>));

// The column sweep of a stage: the strips in P.strips, P.rows rows each. `cap`: resident blocks
// per SM asked of the register allocator.
template <int MINB, bool EXTRA, bool SPLIT>
static cudaError_t launch_sweep_c(const StageParams<SV_T>& P, int st, cudaStream_t s) {
  if (P.n_strips <= 0) return cudaSuccess;
  const dim3 grid(unsigned((P.n_strips + kSweepWarps - 1) / kSweepWarps)), block(32, kSweepWarps);
  if (pow2_mesh(P.dx, P.dy))
    return launch_chained<sweep_kernel<SV_T, MINB, true, EXTRA, SPLIT>>(grid, block, kRingBytes, s, P, st);
  return launch_chained<sweep_kernel<SV_T, MINB, false, EXTRA, SPLIT>>(grid, block, kRingBytes, s, P, st);
}
static cudaError_t launch_sweep(const StageParams<SV_T>& P, int st, int cap, bool extra, cudaStream_t s) {
  const bool split = splits_forms<SV_T>(P.n_strips, extra);
  if constexpr (sizeof(SV_T) == 8) {
    if (extra) return launch_sweep_c<kExtraCap<SV_T>, true, false>(P, st, s);
    if (cap == 3) return launch_sweep_c<3, false, true>(P, st, s);
    return split ? launch_sweep_c<4, false, true>(P, st, s) : launch_sweep_c<4, false, false>(P, st, s);
  } else {
    if (extra)
      return split ? launch_sweep_c<kExtraCap<SV_T>, true, true>(P, st, s)
                   : launch_sweep_c<kExtraCap<SV_T>, true, false>(P, st, s);
    switch (cap) {
      case 4: return launch_sweep_c<4, false, true>(P, st, s);
      case 5: return launch_sweep_c<5, false, true>(P, st, s);
      case 6: return launch_sweep_c<6, false, true>(P, st, s);
      default: return launch_sweep_c<7, false, true>(P, st, s);
    }
  }
}

template <> cudaError_t launch_variant<SV_T>(const StageParams<SV_T>& P, int st, int variant, bool extra, cudaStream_t s) {
  if (variant == kTileRowsVariant) {
    if (P.nblk <= 0) return cudaSuccess;
    const dim3 grid{unsigned(P.nblk)}, block(32, kTileWarps);
    if (pow2_mesh(P.dx, P.dy)) return launch_chained<tile_rows_kernel<SV_T, true>>(grid, block, 0, s, P, st);
    return launch_chained<tile_rows_kernel<SV_T, false>>(grid, block, 0, s, P, st);
  }
  if (variant_is_split(variant)) return launch_split_t<SV_T>(P, st, s);
  if (variant_is_sweep(variant)) return launch_sweep(P, st, variant_cap<SV_T>(variant, P.n_strips), extra, s);
  return launch_stage<SV_T>(P, st, variant, s);
}

template <> cudaError_t launch_strip_classes<SV_T>(const SV_T* z, int nx, int ny, double dx, double dy, int rows,
                                                   long long nstrips, unsigned char* cls, cudaStream_t s) {
  if (nstrips <= 0) return cudaSuccess;
  strip_class_kernel<SV_T><<<unsigned((nstrips + 7) / 8), 256, 0, s>>>(z, nx, ny, rows, nstrips,
                                                                       exact_mesh(dx, dy, sizeof(SV_T) == 8), cls);
  return cudaGetLastError();
}

template <> cudaError_t launch_bed_slopes<SV_T>(const SV_T* z, int nx, int ny, double dx, double dy, SV_T* zx,
                                                SV_T* zy, cudaStream_t s) {
  long long n = (long long)nx * ny;
  bed_slopes_kernel<SV_T><<<unsigned((n + 255) / 256), 256, 0, s>>>(z, nx, ny, dx, dy, zx, zy);
  return cudaGetLastError();
}

static unsigned elementwise_blocks(long long n) {
  const long long b = (n + 255) / 256;
  return unsigned(b < 148 * 16 ? (b > 0 ? b : 1) : 148 * 16);  // grid-stride beyond 16 blocks per SM
}
template <> cudaError_t launch_from_f64<SV_T>(const double* src, SV_T* dst, long long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  convert_kernel<double, SV_T><<<elementwise_blocks(n), 256, 0, s>>>(src, dst, n);
  return cudaGetLastError();
}
template <> cudaError_t launch_differs<SV_T>(const double* src, const SV_T* ref, long long n, int* flag,
                                             cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  differs_kernel<SV_T><<<elementwise_blocks(n), 256, 0, s>>>(src, ref, n, flag);
  return cudaGetLastError();
}
template <> cudaError_t launch_to_f64<SV_T>(const SV_T* src, double* dst, long long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  convert_kernel<SV_T, double><<<elementwise_blocks(n), 256, 0, s>>>(src, dst, n);
  return cudaGetLastError();
}

template <bool EXTRA> static cudaError_t launch_batch_chunk(const BatchParams<SV_T>& B, int st, bool p2, cudaStream_t s) {
  constexpr int CAP = EXTRA ? kBatchExtraCap<SV_T> : kBatchCap<SV_T>;
  const dim3 block(32, kSweepWarps), grid(unsigned(B.first_block[B.n]));
  if (grid.x == 0) return cudaSuccess;
  if (p2) return launch_chained<sweep_batch_kernel<SV_T, CAP, true, EXTRA>>(grid, block, kRingBytes, s, B, st);
  return launch_chained<sweep_batch_kernel<SV_T, CAP, false, EXTRA>>(grid, block, kRingBytes, s, B, st);
}
template <> cudaError_t launch_sweep_batch<SV_T>(const StageParams<SV_T>* Ps, int n, int st, bool p2, bool extra,
                                                 cudaStream_t s) {
  for (int k0 = 0; k0 < n; k0 += kBatchMembers) {
    BatchParams<SV_T> B;
    B.n = std::min(n - k0, kBatchMembers);
    B.first_block[0] = 0;
    for (int k = 0; k < B.n; ++k) {
      B.m[k] = Ps[k0 + k];
      B.first_block[k + 1] = B.first_block[k] + (B.m[k].n_strips + kSweepWarps - 1) / kSweepWarps;
    }
    const cudaError_t e = extra ? launch_batch_chunk<true>(B, st, p2, s) : launch_batch_chunk<false>(B, st, p2, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Persistent batch kernel: one cooperative launch with as many 4-warp blocks as fit on the
// device at once (every block resident, so warps that wait for another warp's work always
// see it done).
template <int BANK>
static cudaError_t launch_persist_t(const PersistParams<SV_T>& PP, const StageParams<SV_T>* Ps, bool p2, bool extra,
                                    cudaStream_t s) {
  constexpr int CAP = kBatchCap<SV_T>, XCAP = kBatchExtraCap<SV_T>;
  void (*kern)(const PersistParams<SV_T>, const MemberBank<SV_T, BANK>) =
      extra ? (p2 ? persist_batch_kernel<SV_T, XCAP, true, true, BANK> : persist_batch_kernel<SV_T, XCAP, false, true, BANK>)
            : (p2 ? persist_batch_kernel<SV_T, CAP, true, false, BANK> : persist_batch_kernel<SV_T, CAP, false, false, BANK>);
  int dev = 0, nsm = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && kRingBytes > 48 * 1024)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRingBytes);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kPersistWarps, kRingBytes);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorCooperativeLaunchTooLarge;
  PersistParams<SV_T> arg = PP;
  auto bank = std::make_unique<MemberBank<SV_T, BANK>>();
  if (BANK > 1) std::copy(Ps, Ps + PP.nact, bank->m);
  void* args[] = {&arg, bank.get()};
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(unsigned(per_sm * nsm)), dim3(32, kPersistWarps), args,
                                     kRingBytes, s);
}
template <> cudaError_t launch_persist<SV_T>(const PersistParams<SV_T>& PP, const StageParams<SV_T>* Ps, bool p2,
                                             bool extra, cudaStream_t s) {
  if (PP.nact <= kBatchMembers) return launch_persist_t<kBatchMembers>(PP, Ps, p2, extra, s);
  return launch_persist_t<1>(PP, Ps, p2, extra, s);
}

template <typename T, int TX, int TY>
static cudaError_t launch_volume_t(const T* h, int nx, int ny, double area, double* part, cudaStream_t s) {
  dim3 grid((nx + TX - 1) / TX, (ny + TY - 1) / TY);
  volume_partials_kernel<T, TX, TY><<<grid, TX * TY, 0, s>>>(h, nx, ny, area, part);
  return cudaGetLastError();
}

template <> cudaError_t launch_volume<SV_T>(const SV_T* h, int nx, int ny, double area, double* part, int tile,
                                            cudaStream_t s) {
  (void)tile;  // one fixed decomposition: the volume must not depend on the stage-kernel variant
  return launch_volume_t<SV_T, 32, 8>(h, nx, ny, area, part, s);
}

template <> cudaError_t launch_debug<SV_T>(const StageParams<SV_T>& P, const DebugParams<SV_T>& D, SV_T* nh,
                                           SV_T* sf, cudaStream_t s) {
  long long n = (long long)D.nx * D.ny;
  long long nf = (long long)(D.nx + 1) * D.ny + (long long)(D.ny + 1) * D.nx;
  debug_slopes_kernel<SV_T><<<unsigned((n + 255) / 256), 256, 0, s>>>(D);
  debug_flux_kernel<SV_T><<<unsigned((nf + 255) / 256), 256, 0, s>>>(D);
  debug_cell_kernel<SV_T><<<unsigned((n + 255) / 256), 256, 0, s>>>(P, D, nh, sf);
  return cudaGetLastError();
}

}  // namespace svk
