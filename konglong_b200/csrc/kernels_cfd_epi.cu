// kernels_cfd_epi.cu - pointwise epilogues of the line-derivative engines
// (compact FD, FFT and cosine / sine lines): PML round 1 and the VTI / TTI scaling
// on the raw gradient (FdEngine_cfd::d{x,y,z}1_2D, KernelCPU::ScalarVTI /
// ScalarTTI), PML round 2, accumulation and the update on the raw divergence
// parts (KernelCPU::applyVel_minus, Propagator::update2nd).
//
// One launch each over the whole grid.  A thread owns V consecutive z cells: 4
// when nz % 4 == 0 (128-bit accesses; a warp takes 32 z of 4 columns), else 1.
// What it does once per thread - face tests, addresses, the constants of the x
// and y faces - then serves 4 cells; the derivative components are damped in
// turn so that no more than two components' memory is held.
// Bound by HBM in the interior; the PML cells by issue.  Before, the PML cells
// were six launches of box kernels that located each cell in all faces (480
// instructions a cell in the y bands); one launch with a cell per thread issued
// 250 a cell and was slower than those on large grids.  Gradient / divergence:
// 911 -> 755 / 738 -> 683 us at 512 x 512 x 400, 125 -> 68 / 110 -> 60 us at
// 256 x 256 x 200 without cross terms, 68 -> 53 / 62 -> 53 us at 199 x 163 x 150.
#include "cfd_epi.cuh"
#include "kernel_api.h"
#include "rtm_device.cuh"

namespace rtm {
namespace {

template <int V>
struct Vec {
  float v[V];
};
template <int V>
__device__ __forceinline__ Vec<V> ld(const float *p) {
  Vec<V> r;
  if constexpr (V == 4) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    r.v[0] = q.x, r.v[1] = q.y, r.v[2] = q.z, r.v[3] = q.w;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int V>
__device__ __forceinline__ Vec<V> ldg(const float *p) {
  Vec<V> r;
  if constexpr (V == 4) {
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    r.v[0] = q.x, r.v[1] = q.y, r.v[2] = q.z, r.v[3] = q.w;
  } else {
    r.v[0] = __ldg(p);
  }
  return r;
}
template <int V>
__device__ __forceinline__ void st(float *p, const Vec<V> &r) {
  if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  else *p = r.v[0];
}

// one recursion of the cells of a y / x face (co: its layer's constants) and of
// a z face (c: the constants of the cells, [3] arrays w apart)
template <int V>
__device__ __forceinline__ void round_xy(const float *co, Vec<V> &p, float *mem, Vec<V> &m) {
  const float c[3] = {__ldg(co), __ldg(co + 1), __ldg(co + 2)};
#pragma unroll
  for (int k = 0; k < V; k++) pml_round(c, p.v[k], &m.v[k]);
  st<V>(mem, m);
}
template <int V>
__device__ __forceinline__ void round_z(const float *c, int w, Vec<V> &p, float *mem, Vec<V> &m) {
  const Vec<V> c0 = ldg<V>(c), c1 = ldg<V>(c + w), c2 = ldg<V>(c + 2 * w);
#pragma unroll
  for (int k = 0; k < V; k++) {
    const float ck[3] = {c0.v[k], c1.v[k], c2.v[k]};
    pml_round(ck, p.v[k], &m.v[k]);
  }
  st<V>(mem, m);
}

// PML round R of a thread's cells on the derivative components: pml1 for the z,
// x and y components in turn (own dimension unscaled, then the cross dimensions
// scaled; pml1_all's order).  Memory component k of a face, k * cs floats on,
// belongs to the derivative component: z faces z x y, x faces x z y, y faces
// y z x.  Returns whether a face holds the cells.
template <int R, int V, bool CROSS>
__device__ __forceinline__ bool epi_pml(const PmlDev &P, int nx, int ny, int nz, int ix, int iy, int iz, bool do_y,
                                        Vec<V> &pz, Vec<V> &px, Vec<V> &py) {
  const int yl = P.f[DY][0].w, yh = P.f[DY][1].w, xl = P.f[DX][0].w, xh = P.f[DX][1].w, zl = P.f[DZ][0].w,
            zh = P.f[DZ][1].w;
  const bool hy = iy < yl || iy >= ny - yh, hx = ix < xl || ix >= nx - xh, hz = iz < zl || iz >= nz - zh;
  if (!hy && !hx && !hz) return false;
  const long long cy = P.f[DY][0].cs, cx = P.f[DX][0].cs, cz = P.f[DZ][0].cs;
  float *fy = nullptr, *fx = nullptr, *fz = nullptr;
  const float *coy = nullptr, *cox = nullptr, *coz = nullptr;
  int wz = 0;
  if (hy) {
    const bool s = iy >= yl;
    fy = (s ? P.f[DY][1].q[R][0] : P.f[DY][0].q[R][0]) + ((long long)(s ? iy - (ny - yh) : iy) * nx + ix) * nz + iz;
    coy = s ? P.f[DY][1].co + (ny - 1 - iy) * 6 : P.f[DY][0].co + iy * 6;
  }
  if (hx) {
    const bool s = ix >= xl;
    fx = (s ? P.f[DX][1].q[R][0] : P.f[DX][0].q[R][0]) + ((long long)iy * (s ? xh : xl) + (s ? ix - (nx - xh) : ix)) * nz + iz;
    cox = s ? P.f[DX][1].co + (nx - 1 - ix) * 6 : P.f[DX][0].co + ix * 6;
  }
  if (hz) {
    const bool s = iz >= zl;
    const int k = s ? iz - (nz - zh) : iz;
    wz = s ? zh : zl;
    fz = (s ? P.f[DZ][1].q[R][0] : P.f[DZ][0].q[R][0]) + ((long long)iy * nx + ix) * wz + k;
    coz = (s ? P.f[DZ][1].cz : P.f[DZ][0].cz) + k;
  }
  Vec<V> yy, yz, yx, xx, xz, xy, zz, zx, zy;  // [face][component]
  if (hz) zz = ld<V>(fz);
  if (CROSS && hx) xz = ld<V>(fx + cx);
  if (CROSS && hy) yz = ld<V>(fy + cy);
  if (hx) xx = ld<V>(fx);
  if (CROSS && hz) zx = ld<V>(fz + cz);
  if (CROSS && hy) yx = ld<V>(fy + 2 * cy);
  if (hz) round_z<V>(coz, wz, pz, fz, zz);
  if (CROSS && hx) round_xy<V>(cox + 3, pz, fx + cx, xz);
  if (CROSS && hy) round_xy<V>(coy + 3, pz, fy + cy, yz);
  if (do_y) {
    if (hy) yy = ld<V>(fy);
    if (CROSS && hz) zy = ld<V>(fz + 2 * cz);
    if (CROSS && hx) xy = ld<V>(fx + 2 * cx);
  }
  if (hx) round_xy<V>(cox, px, fx, xx);
  if (CROSS && hz) round_z<V>(coz + 3 * wz, wz, px, fz + cz, zx);
  if (CROSS && hy) round_xy<V>(coy + 3, px, fy + 2 * cy, yx);
  if (do_y) {
    if (hy) round_xy<V>(coy, py, fy, yy);
    if (CROSS && hz) round_z<V>(coz + 3 * wz, wz, py, fz + 2 * cz, zy);
    if (CROSS && hx) round_xy<V>(cox + 3, py, fx + 2 * cx, xy);
  }
  return true;
}

// block: V == 4: 8 z quads x 32 x; V == 1: 32 z x 8 x; grid (z tiles, x tiles, y)
template <int V>
constexpr int kBx = V == 4 ? 8 : 32;
// resident CTAs of 256 threads the register allocation aims at: the fastest of
// those tried (512 x 512 x 400, V == 4, gradient / divergence: 2 CTAs 884 / 734
// us, 3 755 / 683, 4 782 / 735, the last with spills; 199 x 163 x 150, V == 1: 4
// 63 / 58 us, 5 57 / 53, 6 53 / 59)
template <int V>
constexpr int kGradCtas = V == 4 ? 3 : 6;
template <int V>
constexpr int kDivCtas = V == 4 ? 3 : 5;

template <int V, int MODEL, bool CROSS>
__global__ void __launch_bounds__(256, kGradCtas<V>) cfd_grad_epi_k(const __grid_constant__ CfdGradEpiArgs a, bool pml_only) {
  const int nx = a.nx, nz = a.nz, iz = (blockIdx.x * kBx<V> + threadIdx.x) * V,
            ix = blockIdx.y * (256 / kBx<V>)+threadIdx.y, iy = blockIdx.z;
  if (ix >= nx || iz >= nz) return;
  const bool do_y = a.ny > 1;
  const long long i = ((long long)iy * nx + ix) * nz + iz;
  Vec<V> gx = ld<V>(a.gx + i), gz = ld<V>(a.gz + i), gy{}, ep{}, dl{}, ax{}, ay{}, rho{};
  if (do_y) gy = ld<V>(a.gy + i);
  if (MODEL >= 2) ep = ldg<V>(a.eps + i), dl = ldg<V>(a.del + i);
  if (MODEL == 3) {
    ax = ldg<V>(a.pjx + i);
    if (do_y) ay = ldg<V>(a.pjy + i);
  }
  if (a.rho) rho = ldg<V>(a.rho + i);
  const bool in = epi_pml<0, V, CROSS>(a.pml, nx, a.ny, nz, ix, iy, iz, do_y, gz, gx, gy);
  if (!in && (pml_only || (MODEL < 2 && !a.rho))) return;  // unchanged
#pragma unroll
  for (int k = 0; k < V; k++) {
    if (a.rho) divide_rho(rho.v[k], do_y, gx.v[k], gy.v[k], gz.v[k]);
    if (MODEL >= 2)
      aniso_scale<MODEL>(make_float4(ep.v[k], dl.v[k], ax.v[k], ay.v[k]), gx.v[k], gy.v[k], gz.v[k]);
  }
  st<V>(a.gx + i, gx);
  if (do_y) st<V>(a.gy + i, gy);
  if (MODEL != 2 || in || a.rho) st<V>(a.gz + i, gz);  // the VTI scaling leaves z as it is
}

template <int V, int MODE, bool CROSS>
__global__ void __launch_bounds__(256, kDivCtas<V>) cfd_div_epi_k(const __grid_constant__ CfdDivEpiArgs a, bool pml_only) {
  const int nx = a.nx, nz = a.nz, iz = (blockIdx.x * kBx<V> + threadIdx.x) * V,
            ix = blockIdx.y * (256 / kBx<V>)+threadIdx.y, iy = blockIdx.z;
  if (ix >= nx || iz >= nz) return;
  const bool do_y = a.ny > 1 && a.dy;
  const long long i = ((long long)iy * nx + ix) * nz + iz, n = (long long)nx * a.ny * nz;
  Vec<V> dx = ld<V>(a.dx + i), dz = ld<V>(a.dz + i), vel = ldg<V>(a.vel + i), w0 = ld<V>(a.w0 + i), dy{}, w1{}, rho{};
  if (do_y) dy = ld<V>(a.dy + i);
  if (MODE != 0) w1 = ldg<V>(a.w1 + i);
  if (a.rho) rho = ldg<V>(a.rho + i);
  const bool in = epi_pml<1, V, CROSS>(a.pml, nx, a.ny, nz, ix, iy, iz, do_y, dz, dx, dy);
  if (!in && pml_only) return;
#pragma unroll
  for (int k = 0; k < V; k++) {
    if (MODE == 2)
      w0.v[k] = q_update(a.q, i + k, n, div_finish<0>(a, dx.v[k], dy.v[k], dz.v[k], vel.v[k], w0.v[k], w1.v[k], rho.v[k]),
                         w1.v[k]);
    else w0.v[k] = div_finish<MODE>(a, dx.v[k], dy.v[k], dz.v[k], vel.v[k], w0.v[k], w1.v[k], rho.v[k]);
  }
  st<V>(a.w0 + i, w0);
}

template <int V>
dim3 epi_grid(int nx, int ny, int nz) {
  return dim3((nz + kBx<V> * V - 1) / (kBx<V> * V), (nx + 256 / kBx<V> - 1) / (256 / kBx<V>), ny);
}

template <int V, int MODEL>
void grad_epi(const CfdGradEpiArgs &a, bool pml_only, cudaStream_t s) {
  const dim3 g = epi_grid<V>(a.nx, a.ny, a.nz), block(kBx<V>, 256 / kBx<V>);
  if (a.pml3d) cfd_grad_epi_k<V, MODEL, true><<<g, block, 0, s>>>(a, pml_only);
  else cfd_grad_epi_k<V, MODEL, false><<<g, block, 0, s>>>(a, pml_only);
}
template <int V>
void grad_epi(const CfdGradEpiArgs &a, bool pml_only, cudaStream_t s) {
  if (a.model == 3) grad_epi<V, 3>(a, pml_only, s);
  else if (a.model == 2) grad_epi<V, 2>(a, pml_only, s);
  else grad_epi<V, 1>(a, pml_only, s);
}
template <int V, int MODE>
void div_epi(const CfdDivEpiArgs &a, bool pml_only, cudaStream_t s) {
  const dim3 g = epi_grid<V>(a.nx, a.ny, a.nz), block(kBx<V>, 256 / kBx<V>);
  if (a.pml3d) cfd_div_epi_k<V, MODE, true><<<g, block, 0, s>>>(a, pml_only);
  else cfd_div_epi_k<V, MODE, false><<<g, block, 0, s>>>(a, pml_only);
}
template <int V>
void div_epi(const CfdDivEpiArgs &a, bool pml_only, cudaStream_t s) {
  if (a.mode == 0) div_epi<V, 0>(a, pml_only, s);
  else if (a.mode == 1) div_epi<V, 1>(a, pml_only, s);
  else div_epi<V, 2>(a, pml_only, s);
}

// rows and z faces are whole float4s
bool quads(const PmlDev &P, int nz) { return nz % 4 == 0 && P.f[DZ][0].w % 4 == 0 && P.f[DZ][1].w % 4 == 0; }

}  // namespace

void launch_cfd_grad_epi(const CfdGradEpiArgs &a, bool pml_only, cudaStream_t st) {
  if (quads(a.pml, a.nz)) grad_epi<4>(a, pml_only, st);
  else grad_epi<1>(a, pml_only, st);
}

void launch_cfd_div_epi(const CfdDivEpiArgs &a, bool pml_only, cudaStream_t st) {
  if (quads(a.pml, a.nz)) div_epi<4>(a, pml_only, st);
  else div_epi<1>(a, pml_only, st);
}

}  // namespace rtm
