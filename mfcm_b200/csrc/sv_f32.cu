// sv_f32.cu -- FP32 instantiation of the stage kernels. Compiled with -fmad=false: the sweeps
// write their fused multiply-adds out (sv_sweep.cuh, mad_).
#define SV_T float
#include "sv_inst.cuh"
