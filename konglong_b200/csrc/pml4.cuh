// pml4.cuh - split-field PML pieces of the 4-z-cell tile kernels
// (kernels_iso4.cu, kernels_aniso4.cu): a thread owns 4 consecutive z cells of
// a 32 (z) x TX (x) column tile marching along y, so its x and z faces are
// fixed over the tile and every face array gives it one aligned float4 per
// plane (the z faces are whole float4s, see PmlFace).
#pragma once
#include "rtm_device.cuh"

namespace rtm {
namespace {

__device__ __forceinline__ float cmp4(const float4 &v, int c) { return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w; }
__device__ __forceinline__ void set4(float4 &v, int c, float x) {
  if (c == 0) v.x = x;
  else if (c == 1) v.y = x;
  else if (c == 2) v.z = x;
  else v.w = x;
}
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(__cvta_generic_to_global(p)));
}

// Recursion constants of a PML tile in shared memory (NC of the six per layer:
// 3 for the unscaled set, 6 with the pml3d-scaled one): for the z faces one
// float4 per constant and z quad (its 4 cells' layers), for the x faces the
// constants of the column.  Reading them from global memory per cell and plane
// cost up to 36 scalar loads with their address arithmetic.
template <int TX, int NC>
struct PmlCo {
  float4 z[NC][8];
  float x[TX][NC == 3 ? 4 : 8];
};
template <int TX, int NC>
__device__ __forceinline__ void fill_pml_co(PmlCo<TX, NC> &s, const PmlDev &P, const Grid3 &g, int iz0, int ix0,
                                            int tzq, int tx) {
  if (tx < NC) {
    float v[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int iz = iz0 + 4 * tzq + c, lo = P.f[DZ][0].w, hi = P.f[DZ][1].w;
      v[c] = iz < lo ? P.f[DZ][0].co[iz * 6 + tx]
                     : iz < g.nz && iz >= g.nz - hi ? P.f[DZ][1].co[(g.nz - 1 - iz) * 6 + tx] : 0.f;
    }
    s.z[tx][tzq] = make_float4(v[0], v[1], v[2], v[3]);
  }
  if (tzq < NC) {
    const int ix = ix0 + tx, lo = P.f[DX][0].w, hi = P.f[DX][1].w;
    s.x[tx][tzq] = ix < lo ? P.f[DX][0].co[ix * 6 + tzq]
                           : ix < g.nx && ix >= g.nx - hi ? P.f[DX][1].co[(g.nx - 1 - ix) * 6 + tzq] : 0.f;
  }
}

// one recursion of the 4 cells of an x / y face (one layer) and of a z face
// (a layer per cell; s: first constant of the set)
__device__ __forceinline__ void round4(const float *co, float (&p)[4], float4 &m) {
#pragma unroll
  for (int c = 0; c < 4; c++) {
    float q = cmp4(m, c);
    pml_round(co, p[c], &q);
    set4(m, c, q);
  }
}
template <int NC>
__device__ __forceinline__ void round4z(const float4 (&z)[NC][8], int tzq, int s, float (&p)[4], float4 &m) {
  const float4 a = z[s][tzq], b = z[s + 1][tzq], d = z[s + 2][tzq];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float co[3] = {cmp4(a, c), cmp4(b, c), cmp4(d, c)};
    float q = cmp4(m, c);
    pml_round(co, p[c], &q);
    set4(m, c, q);
  }
}

// Memory of the x and z faces that hold the thread's cells, at the current
// plane: round R, component 0 (component k is k * cs floats on), advancing by
// a constant stride per plane; null outside the faces.
template <int R>
struct TileFaces {
  float *fx = nullptr, *fz = nullptr;
  int sx = 0, sz = 0;  // plane strides (floats)
  __device__ __forceinline__ void init(const PmlDev &P, const Grid3 &g, int ix, int iz4, int y0, bool act) {
    const int nx = g.nx, nz = g.nz;
    if (act && (ix < P.f[DX][0].w || ix >= nx - P.f[DX][1].w)) {
      const int s = ix < P.f[DX][0].w ? 0 : 1, w = P.f[DX][s].w;
      fx = P.f[DX][s].q[R][0] + ((long long)y0 * w + (s ? ix - (nx - w) : ix)) * nz + iz4;
      sx = w * nz;
    }
    if (act && (iz4 < P.f[DZ][0].w || iz4 >= nz - P.f[DZ][1].w)) {
      const int s = iz4 < P.f[DZ][0].w ? 0 : 1, w = P.f[DZ][s].w;
      fz = P.f[DZ][s].q[R][0] + ((long long)y0 * nx + ix) * w + (s ? iz4 - (nz - w) : iz4);
      sz = nx * w;
    }
  }
  // memory of the y face holding plane iy (null when none) and its constants
  __device__ __forceinline__ float *yface(const PmlDev &P, const Grid3 &g, int ix, int iz4, int iy,
                                          const float *&co) const {
    const int lo = P.f[DY][0].w, hi = P.f[DY][1].w;
    if (iy >= lo && iy < g.ny - hi) return nullptr;
    const int s = iy < lo ? 0 : 1;
    co = P.f[DY][s].co + (s ? g.ny - 1 - iy : iy) * 6;
    return P.f[DY][s].q[R][0] + ((long long)(s ? iy - (g.ny - hi) : iy) * g.nx + ix) * g.nz + iz4;
  }
  __device__ __forceinline__ void advance() {
    if (fx) fx += sx;
    if (fz) fz += sz;
  }
  // L1 prefetch of N arrays (stride d per dimension) of the x / z faces k
  // planes ahead and of the y face of plane y
  template <int N>
  __device__ __forceinline__ void prefetch(const PmlDev &P, const Grid3 &g, int ix, int iz4, int y, int k, long long dx,
                                           long long dy, long long dz) const {
    auto pf = [&](const float *p, long long d) {
#pragma unroll
      for (int j = 0; j < N; j++, p += d) prefetch_l1(p);
    };
    if (fx) pf(fx + k * sx, dx);
    if (fz) pf(fz + k * sz, dz);
    const float *co;
    const float *fy = yface(P, g, ix, iz4, y, co);
    if (fy) pf(fy, dy);
  }
};

}  // namespace
}  // namespace rtm
