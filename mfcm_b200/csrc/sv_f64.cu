// sv_f64.cu -- FP64 instantiation of the stage kernels. Compiled with -fmad=false: every
// FP64 multiply and add is rounded separately, as in the reference's CPU arithmetic, which
// is what makes the FP64 path bit-identical to the oracle. (Explicit fma() calls are kept:
// they implement the exact constant-divisor division in sv_device.cuh.)
#define SV_T double
#define SV_DEFINE_COMMON_KERNELS
#include "sv_inst.cuh"

namespace svk {

// The finalize kernels in the chain of a timestep's launches, with `ctas` blocks per solver (a
// cluster when there are several).
template <typename... KArgs, typename... Args>
static cudaError_t launch_clusters(void (*kern)(KArgs...), int solvers, int ctas, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(solvers * ctas));
  cfg.blockDim = dim3(kFinalizeThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = unsigned(ctas);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctas > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}
cudaError_t launch_finalize(const FinalizeParams& F, cudaStream_t s) {
  if (F.nblk > kFinalizeClusterSlots) return launch_clusters(finalize_kernel<kFinalizeCtas>, 1, kFinalizeCtas, s, F);
  return launch_clusters(finalize_kernel<1>, 1, 1, s, F);
}
cudaError_t launch_finalize_batch(const FinalizeParams* Fs, int ninst, long long max_nblk, cudaStream_t s) {
  if (ninst <= 0) return cudaSuccess;
  if (max_nblk > kFinalizeClusterSlots)
    return launch_clusters(finalize_batch_kernel<kFinalizeCtas>, ninst, kFinalizeCtas, s, Fs);
  return launch_clusters(finalize_batch_kernel<1>, ninst, 1, s, Fs);
}
cudaError_t launch_begin_queue(const FinalizeParams* Fs, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  begin_queue_kernel<<<(n + 127) / 128, 128, 0, s>>>(Fs, n);
  return cudaGetLastError();
}
cudaError_t launch_gather_done(Ctl* const* ctls, int n, int* done, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  gather_done_kernel<<<(n + 127) / 128, 128, 0, s>>>(ctls, n, done);
  return cudaGetLastError();
}
cudaError_t launch_sum(const double* p, long long n, double* out, cudaStream_t s) {
  sum_kernel<1024><<<1, 1024, 0, s>>>(p, n, out);
  return cudaGetLastError();
}
cudaError_t launch_accept(Ctl* ctl, cudaStream_t s) {
  accept_kernel<<<1, 1, 0, s>>>(ctl);
  return cudaGetLastError();
}
// In this unit (no contraction) so that the FP64 slopes round like those of the FP64 solver.
cudaError_t launch_datum_bed(const double* z, int nx, int ny, double dx, double dy, int dtiles_x, int dtiles_y,
                             double* zdat, float* off, float* zx, float* zy, cudaStream_t s) {
  const long long n = (long long)nx * ny, nt = (long long)dtiles_x * dtiles_y;
  if (n <= 0) return cudaSuccess;
  datum_tiles_kernel<<<unsigned((nt + 7) / 8), 256, 0, s>>>(z, nx, ny, dtiles_x, dtiles_y, zdat);
  datum_offsets_kernel<<<elementwise_blocks(n), 256, 0, s>>>(z, nx, ny, dtiles_x, zdat, off);
  bed_slopes_kernel<double, float><<<unsigned((n + 255) / 256), 256, 0, s>>>(z, nx, ny, dx, dy, zx, zy);
  return cudaGetLastError();
}
cudaError_t launch_datum_absolute(const float* off, int nx, int ny, int dtiles_x, const double* zdat, double* z,
                                  cudaStream_t s) {
  const long long n = (long long)nx * ny;
  if (n <= 0) return cudaSuccess;
  datum_absolute_kernel<<<elementwise_blocks(n), 256, 0, s>>>(off, nx, ny, dtiles_x, zdat, z);
  return cudaGetLastError();
}
cudaError_t launch_persist_init(const FinalizeParams* Fs, PersistMember* mem, const long long* warp_start, int nact,
                                cudaStream_t s) {
  if (nact <= 0) return cudaSuccess;
  persist_init_kernel<<<(nact + 127) / 128, 128, 0, s>>>(Fs, mem, warp_start, nact);
  return cudaGetLastError();
}
cudaError_t launch_begin_step(Ctl* ctl, int new_step, long long budget, cudaStream_t s) {
  begin_step_kernel<<<1, 1, 0, s>>>(ctl, new_step, budget);
  return cudaGetLastError();
}

}  // namespace svk
