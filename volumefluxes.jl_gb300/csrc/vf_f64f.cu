// vf_f64f.cu -- Float64 per-step kernels held to a tolerance instead of to the
// reference's bits: the face fluxes use fused multiply-adds (madd, msub in
// vf_math.cuh). Every other operation, the order of the passes and every
// branch are the bitwise kernels' own (the same source): contraction in the
// pointwise updates as well measured 2.58 instead of 2.69 ms per two steps of
// 1500 x 1100 cells (start: 4.33), but moves cells across the dry threshold
// and with them the dt sequence of draining films.
//
// The kernels are instantiated from the same headers as vf_f64.cu, so they
// are renamed into their own namespace (vf_faithful): two units must not hold
// different bodies under one kernel name. The argument block has the same
// layout in both namespaces (one header text, VF_FP64_FAITHFUL changes
// arithmetic only, no type).
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#define VF_FP64_FAITHFUL 1
#define vf vf_faithful
#include "vf_step_impl.cuh"
#undef vf

namespace {
const vf_faithful::StepArgs<double>& args_of(const void* a) {
  return *static_cast<const vf_faithful::StepArgs<double>*>(a);
}
}  // namespace

cudaError_t vf_faithful_launch_step(const void* a, const double* Uin, double* Uout, int parity, cudaStream_t st) {
  return vf_faithful::launch_step_impl<double>(args_of(a), Uin, Uout, parity, st);
}
cudaError_t vf_faithful_launch_flux(const void* a, const double* Uin, int parity, cudaStream_t st) {
  return vf_faithful::launch_flux_impl<double>(args_of(a), Uin, parity, st);
}
cudaError_t vf_faithful_launch_stage(const void* a, const double* Uin, double* Uout, int parity, cudaStream_t st) {
  return vf_faithful::launch_stage_impl<double>(args_of(a), Uin, Uout, parity, st);
}
