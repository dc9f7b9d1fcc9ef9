// cfd_rows.cuh - right-hand-side rows of the compact-FD line solves
// (FdEngine_cfd + Cfd_plan), shared by the line kernels.
#pragma once
#include <cuda_runtime.h>

namespace rtm {
namespace {

// One right-hand-side row of the 11-band A with every rounding explicit, so
// that each line kernel (staged, streamed, pipelined) gives the same bits:
// interior rows sum_d a[54 + d] (x[i + d] - x[i - d]), d = 1 .. 5, and the
// one-sided rows within 5 of a line end (banmul_dev_z_c,
// bgprtm/FdEngine_cfd.cpp:304-327) accumulated in the reference order.
struct RhsCoef {
  float c1, c2, c3, c4, c5;
};
__device__ __forceinline__ float rhs_interior(const RhsCoef &c, float m5, float m4, float m3, float m2, float m1,
                                              float p1, float p2, float p3, float p4, float p5) {
  float t = __fmul_rn(c.c1, __fsub_rn(p1, m1));
  t = __fmaf_rn(c.c2, __fsub_rn(p2, m2), t);
  t = __fmaf_rn(c.c3, __fsub_rn(p3, m3), t);
  t = __fmaf_rn(c.c4, __fsub_rn(p4, m4), t);
  return __fmaf_rn(c.c5, __fsub_rn(p5, m5), t);
}
// row i < 5 from x[i - 5 + j], j = 0 .. 10 (x[j] here)
__device__ __forceinline__ float rhs_low(const float (&a)[60], int i, const float *x) {
  float v = 0.f;
#pragma unroll
  for (int j = 0; j < 11; j++)
    if (j >= 5 - i) v = __fmaf_rn(a[j * 5 + i], x[j], v);
  return v;
}
// row i = n - t, t = 1 .. 5, from x[i - 5 + j], j = 0 .. 10
__device__ __forceinline__ float rhs_high(const float (&a)[60], int t, const float *x) {
  float v = 0.f;
#pragma unroll
  for (int j = 0; j < 11; j++)
    if (j < t + 5) v = __fmaf_rn(-a[t + 49 - 5 * j], x[j], v);
  return v;
}

}  // namespace
}  // namespace rtm
