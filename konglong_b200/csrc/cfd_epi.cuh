// cfd_epi.cuh - cell arithmetic of the compact-FD epilogues after the PML rounds,
// shared by the epilogue kernels and the line solves that carry them.
#pragma once
#include "kernel_api.h"
#include "rtm_device.cuh"

namespace rtm {
namespace {

// density division and VTI / TTI scaling of one cell's gradients after PML
// round 1 (KernelCPU::ScalarVTI / ScalarTTI), every rounding explicit so that
// each kernel inlining it gives the same bits
__device__ __forceinline__ void grad_finish(const CfdGradEpiArgs &a, bool do_y, float &gx, float &gy, float &gz,
                                            float ep, float dl, float ax, float ay, float r) {
  if (a.rho) divide_rho(r, do_y, gx, gy, gz);
  if (a.model == 3) aniso_scale<3>(make_float4(ep, dl, ax, ay), gx, gy, gz);
  else if (a.model == 2) aniso_scale<2>(make_float4(ep, dl, 0.f, 0.f), gx, gy, gz);
}

// accumulation w0 - vel (dx + dz + dy) (with density in the engine's form)
// and the update of MODE 0 (none) or 1 (leapfrog)
template <int MODE>
__device__ __forceinline__ float div_finish(const CfdDivEpiArgs &a, float dxv, float dyv, float dzv, float vel,
                                            float w0, float w1, float r) {
  float t;
  if (a.rho) {
    t = a.rho_form == 2   ? div_accumulate_rho<2>(w0, vel, r, dxv, dzv, dyv)
        : a.rho_form == 1 ? div_accumulate_rho<1>(w0, vel, r, dxv, dzv, dyv)
                          : div_accumulate_rho<0>(w0, vel, r, dxv, dzv, dyv);
  } else {
    t = __fmaf_rn(-dxv, vel, w0);
    t = __fmaf_rn(-dzv, vel, t);
    t = __fmaf_rn(-dyv, vel, t);
  }
  return MODE == 1 ? __fsub_rn(__fadd_rn(w1, w1), t) : t;
}

}  // namespace
}  // namespace rtm
