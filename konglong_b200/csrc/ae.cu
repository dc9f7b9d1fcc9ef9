// ae.cu - learned snapshot compressor: a small 3-D convolutional autoencoder
// on 8^3-cell blocks, trained and run with hand-written tensor-core kernels.
//
// A block's cells are kept in Morton order (bit triples z y x from the least
// significant end), so the 8 children of every 2^3 cube are consecutive.
// With that layout every layer is one row-major GEMM on the previous layer's
// output memory, no reshaping:
//   E1  2^3 patch conv, stride 2   1 -> 16 ch   rows/block 64  K   8 N  16  leaky ReLU
//   E2  2^3 patch conv, stride 2  16 -> 16 ch              8   K 128 N  16  leaky ReLU
//   E3  pointwise                 16 -> 16 ch              8   K  16 N  16  leaky ReLU
//   E4  2^3 patch conv, stride 2  16 -> 64 ch (latent)     1   K 128 N  64  linear
//   D1  transposed 2^3, stride 2  64 -> 16 ch              1   K  64 N 128  leaky ReLU
//   D2  pointwise                 16 -> 16 ch              8   K  16 N  16  leaky ReLU
//   D3  transposed 2^3, stride 2  16 -> 16 ch              8   K  16 N 128  leaky ReLU
//   D4  transposed 2^3, stride 2  16 ->  1 ch              64  K  16 N   8  linear
// 512 cells -> 64 latent values stored as BF16 (the decoder's first GEMM rounds
// its operand to BF16, so BF16 storage keeps everything the decoder can use:
// 64 values in the bytes of 32 floats, 15.5:1 with the block's max |value|
// scale).
// GEMMs: mma.sync m16n8k16, BF16 operands (rounded from the FP32 activations
// and FP32 master weights), FP32 accumulation.  Training: MSE loss on the
// scale-normalised block, backward GEMMs, Adam on the FP32 master weights.
#include <cuda_bf16.h>
#include <stdint.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_fp16.h>

#include "kernel_api.h"
#include "rtm_b200.h"

namespace rtm {
namespace {

constexpr int kLayers = 8;
constexpr int kL_K[kLayers] = {8, 128, 16, 128, 64, 16, 16, 16};
constexpr int kL_N[kLayers] = {16, 16, 16, 64, 128, 16, 128, 8};
constexpr int kL_R[kLayers] = {64, 8, 8, 1, 1, 8, 8, 64};  // rows per block
constexpr int kL_ACT[kLayers] = {1, 1, 1, 0, 1, 1, 1, 0};
constexpr float kSlope = 0.1f;  // leaky ReLU
constexpr int kLatent = 64;
constexpr int kBlock = 512;

constexpr int w_off(int l) {
  int o = 0;
  for (int k = 0; k < l; k++) o += kL_K[k] * kL_N[k] + kL_N[k];
  return o;
}
constexpr int kNParams = w_off(kLayers);

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// C(m, n) [+]= sum_k A(m, k) B(k, n) over k in this block's split of [0, K),
// A(m, k) = A[m*sam + k*sak], B(k, n) = B[k*sbk + n*sbn]; operands rounded to
// BF16.  Epilogue: + bias[n], optional pre-activation copy, leaky ReLU; or an
// atomic add into C (split-K reductions, bias / activation not allowed).
struct Gemm {
  int M, N, K, ksplit;
  const float *A;
  long long sam, sak;
  const float *B;
  long long sbk, sbn;
  float *C;
  long long ldc;
  const float *bias;
  float *pre;
  int act, atomic;
};

// block: 4 warps, each a 16 x 32 tile; grid (M / 64, N / 32, ksplit)
__global__ void __launch_bounds__(128) gemm_bf16_k(Gemm g) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gr = lane >> 2, t = lane & 3;
  const int m0 = blockIdx.x * 64 + warp * 16, n0 = blockIdx.y * 32;
  const int kc = ((g.K + g.ksplit - 1) / g.ksplit + 15) / 16 * 16;
  const int kb = blockIdx.z * kc, ke = min(g.K, kb + kc);
  float acc[4][4] = {};
  auto a_at = [&](int m, int k) -> float { return (m < g.M && k < ke) ? g.A[m * g.sam + k * g.sak] : 0.f; };
  auto b_at = [&](int k, int n) -> float { return (n < g.N && k < ke) ? g.B[k * g.sbk + n * g.sbn] : 0.f; };
  for (int k0 = kb; k0 < ke; k0 += 16) {
    uint32_t a[4];
    const int r0 = m0 + gr, r1 = m0 + gr + 8, c0 = k0 + 2 * t, c1 = k0 + 2 * t + 8;
    a[0] = pack_bf16(a_at(r0, c0), a_at(r0, c0 + 1));
    a[1] = pack_bf16(a_at(r1, c0), a_at(r1, c0 + 1));
    a[2] = pack_bf16(a_at(r0, c1), a_at(r0, c1 + 1));
    a[3] = pack_bf16(a_at(r1, c1), a_at(r1, c1 + 1));
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const int n = n0 + nt * 8 + gr;
      const uint32_t b0 = pack_bf16(b_at(c0, n), b_at(c0 + 1, n));
      const uint32_t b1 = pack_bf16(b_at(c1, n), b_at(c1 + 1, n));
      mma_bf16(acc[nt], a, b0, b1);
    }
  }
#pragma unroll
  for (int nt = 0; nt < 4; nt++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int m = m0 + gr + (q >= 2 ? 8 : 0), n = n0 + nt * 8 + 2 * t + (q & 1);
      if (m >= g.M || n >= g.N) continue;
      float v = acc[nt][q];
      float *c = g.C + m * g.ldc + n;
      if (g.atomic) {
        atomicAdd(c, v);
        continue;
      }
      if (g.bias) v += g.bias[n];
      if (g.pre) g.pre[m * g.ldc + n] = v;
      if (g.act) v = v > 0.f ? v : kSlope * v;
      *c = v;
    }
}

void gemm(const Gemm &g0, cudaStream_t st) {
  Gemm g = g0;
  if (g.M <= 0 || g.N <= 0) return;
  if (!g.atomic) g.ksplit = 1;
  const dim3 grid((g.M + 63) / 64, (g.N + 31) / 32, std::max(1, g.ksplit));
  gemm_bf16_k<<<grid, 128, 0, st>>>(g);
}

// dP = dY * act'(pre) in place (leaky ReLU), for n elements
__global__ void act_back_k(float *dy, const float *pre, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (pre[i] <= 0.f) dy[i] *= kSlope;
}

// column sums of an R x N matrix into out[n] (atomic across row chunks)
__global__ void colsum_k(const float *dy, int R, int N, float *out) {
  const int n = blockIdx.y * 32 + (threadIdx.x & 31);
  if (n >= N) return;
  float s = 0.f;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < R; r += gridDim.x * 8) s += dy[(long long)r * N + n];
  atomicAdd(out + n, s);
}

// MSE loss on n values: loss += sum (y - x)^2 / n; dy = 2 (y - x) / n
__global__ void mse_k(const float *y, const float *x, long long n, float *dy, float *loss) {
  float s = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float d = y[i] - x[i];
    s += d * d;
    dy[i] = 2.f * d / (float)n;
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, s / (float)n);
}

// Adam (bias-corrected) on the FP32 master parameters
__global__ void adam_k(float *p, const float *g, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi, v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace
}  // namespace rtm

// ---- the compressor object ---------------------------------------------------
struct rtm_ae {
  int device = 0;
  cudaStream_t st = nullptr;
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // params, grads, Adam moments
  float *loss = nullptr;
  int step = 0;
  int wave_enc[2] = {1, 1}, wave_dec[2] = {1, 1};  // CTAs of one wave: cell by cell, 16-byte accesses
  // workspace for `cap` blocks: normalised input, per-layer outputs; training
  // also keeps pre-activations and gradients
  int cap = 0, cap_train = 0;
  float *x0 = nullptr, *y[8] = {}, *pre[8] = {}, *dy[8] = {}, *dx0 = nullptr, *sc = nullptr;
  std::string err;
};

namespace rtm {
namespace {

void ae_free_ws(rtm_ae *a) {
  auto fr = [](float *&q) {
    cudaFree(q);
    q = nullptr;
  };
  fr(a->x0), fr(a->dx0), fr(a->sc);
  for (int l = 0; l < kLayers; l++) fr(a->y[l]), fr(a->pre[l]), fr(a->dy[l]);
  a->cap = a->cap_train = 0;
}

// workspace for n blocks (train: also pre-activations and gradients)
int ae_reserve(rtm_ae *a, int n, bool train) {
  if (n <= a->cap && (!train || n <= a->cap_train)) return RTM_OK;
  const int cap = std::max(n, a->cap);
  const bool tr = train || a->cap_train > 0;
  ae_free_ws(a);
  bool ok = cudaMalloc(&a->x0, (size_t)cap * kBlock * 4) == cudaSuccess &&
            cudaMalloc(&a->sc, (size_t)cap * 4) == cudaSuccess;
  if (tr) ok = ok && cudaMalloc(&a->dx0, (size_t)cap * kBlock * 4) == cudaSuccess;
  for (int l = 0; l < kLayers && ok; l++) {
    const size_t e = (size_t)cap * kL_R[l] * kL_N[l] * 4;
    ok = cudaMalloc(&a->y[l], e) == cudaSuccess;
    if (tr) ok = ok && cudaMalloc(&a->pre[l], e) == cudaSuccess && cudaMalloc(&a->dy[l], e) == cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    ae_free_ws(a);
    a->err = "compressor workspace allocation failed";
    return RTM_ERR_NOMEM;
  }
  a->cap = cap, a->cap_train = tr ? cap : 0;
  return RTM_OK;
}

// forward of layers [l0, l1) for n blocks, input of layer l0 at `in`
void ae_forward(rtm_ae *a, int n, const float *in, int l0, int l1, bool keep_pre, cudaStream_t st) {
  const float *x = in;
  for (int l = l0; l < l1; l++) {
    Gemm g{};
    g.M = n * kL_R[l], g.N = kL_N[l], g.K = kL_K[l], g.ksplit = 1;
    g.A = x, g.sam = kL_K[l], g.sak = 1;
    g.B = a->p + w_off(l), g.sbk = kL_N[l], g.sbn = 1;
    g.C = a->y[l], g.ldc = kL_N[l];
    g.bias = a->p + w_off(l) + kL_K[l] * kL_N[l];
    g.pre = keep_pre ? a->pre[l] : nullptr;
    g.act = kL_ACT[l];
    gemm(g, st);
    x = a->y[l];
  }
}

// loss and parameter gradients (into a->g) of n normalised blocks at a->x0
void ae_loss_grad(rtm_ae *a, int n) {
  cudaStream_t st = a->st;
  ae_forward(a, n, a->x0, 0, kLayers, true, st);
  cudaMemsetAsync(a->loss, 0, 4, st);
  cudaMemsetAsync(a->g, 0, (size_t)kNParams * 4, st);
  const long long tot = (long long)n * kBlock;
  mse_k<<<(int)std::min<long long>((tot + 255) / 256, 1024), 256, 0, st>>>(a->y[kLayers - 1], a->x0, tot,
                                                                            a->dy[kLayers - 1], a->loss);
  for (int l = kLayers - 1; l >= 0; l--) {
    const int R = n * kL_R[l], K = kL_K[l], N = kL_N[l];
    const long long e = (long long)R * N;
    if (kL_ACT[l])
      act_back_k<<<(int)std::min<long long>((e + 255) / 256, 2048), 256, 0, st>>>(a->dy[l], a->pre[l], e);
    const float *xin = l == 0 ? a->x0 : a->y[l - 1];
    Gemm gw{};  // dW = X^T dP (K x N), reduction over the R rows, split-K
    gw.M = K, gw.N = N, gw.K = R, gw.ksplit = std::max(1, std::min(128, R / 256));
    gw.A = xin, gw.sam = 1, gw.sak = K;
    gw.B = a->dy[l], gw.sbk = N, gw.sbn = 1;
    gw.C = a->g + w_off(l), gw.ldc = N, gw.atomic = 1;
    gemm(gw, st);
    colsum_k<<<dim3(std::min(64, (R + 7) / 8), (N + 31) / 32), 256, 0, st>>>(a->dy[l], R, N,
                                                                            a->g + w_off(l) + K * N);
    Gemm gx{};  // dX = dP W^T (R x K)
    gx.M = R, gx.N = K, gx.K = N, gx.ksplit = 1;
    gx.A = a->dy[l], gx.sam = N, gx.sak = 1;
    gx.B = a->p + w_off(l), gx.sbk = 1, gx.sbn = N;
    gx.C = l == 0 ? a->dx0 : a->dy[l - 1], gx.ldc = K;
    gemm(gx, st);
  }
}

constexpr int kChunkBlocks = 8192;  // blocks per encode / decode pass over a volume

// ---- fused inference over a volume -------------------------------------------
// 16 blocks (consecutive in the latents' order, z fastest) are the 16 rows of
// every MMA, and a CTA's 8 warps are the 8 octants of the blocks (the row index
// of E2 / D2 within a block).  With a block a row, the 16 x 16 accumulator tile
// of one layer is, packed to BF16, the A fragment of the next: E1's tile of
// child j is k step j of E2, E2's tile is E3's operand, E3's tile of octant p is
// k step p of E4, and likewise D1 .. D4.  Cells go from memory to E1's fragments
// and from D4's accumulators to memory as float4s, each once; only the blocks'
// largest |value|, E3's tiles and D1's latents pass through shared memory.
// One warp per block with the layer outputs in shared memory, before, used 8 or
// 1 of the 16 rows in five layers of eight and moved every value through shared
// memory: encode + decode of 400 x 400 x 320 took 907 us, now 151 (84 + 65 us by
// events over repeated calls).  The MMAs with full rows take 27 us of tensor time and
// the volumes 67 us of memory time; what bounds the kernels is issue slots at 16
// warps an SM (half of them used) and, decoding, the half-sector stores.
// Each output element is the same mma.sync chain over k in steps of 16 as in
// gemm_bf16_k, with the same operand roundings, bias and activation, so the
// results equal the layer-by-layer path bit for bit.
constexpr int kAeWarps = 8, kAeRows = 16;

// the B fragment of rows [16 ks, 16 ks + 16) and columns [8 nt, 8 nt + 8) of layer L's weights
// (FP32 master, rounded to BF16); rows beyond K are zeros
template <int L>
__device__ __forceinline__ uint2 b_frag(const float *__restrict__ p, int ks, int nt, int lane) {
  constexpr int K = kL_K[L], N = kL_N[L];
  const float *w = p + w_off(L) + nt * 8 + (lane >> 2);
  const int k = ks * 16 + 2 * (lane & 3);
  uint2 b;
  b.x = pack_bf16(w[k * N], w[(k + 1) * N]);
  b.y = K > 8 ? pack_bf16(w[(k + 8) * N], w[(k + 9) * N]) : 0u;
  return b;
}
// the biases of a lane's columns 2t, 2t + 1 of tile nt and of the tile after it
template <int L>
__device__ __forceinline__ float4 b_bias(const float *__restrict__ p, int nt, int lane) {
  const float *b = p + w_off(L) + kL_K[L] * kL_N[L] + nt * 8 + 2 * (lane & 3);
  return make_float4(b[0], b[1], b[8], b[9]);
}
// (x + bx, y + by) under the leaky ReLU (slope < 1: the larger of v and slope v) as two BF16; the
// packed FP32 forms round as the scalar ones in half the issue slots
__device__ __forceinline__ uint32_t act2(float x, float y, float bx, float by) {
  float vx, vy, sx, sy;
  asm("{\n .reg .b64 v, b, s;\n"
      " mov.b64 v, {%4, %5};\n mov.b64 b, {%6, %7};\n mov.b64 s, {%8, %8};\n"
      " add.rn.f32x2 v, v, b;\n mul.rn.f32x2 s, v, s;\n"
      " mov.b64 {%0, %1}, v;\n mov.b64 {%2, %3}, s;\n}"
      : "=f"(vx), "=f"(vy), "=f"(sx), "=f"(sy)
      : "f"(x), "f"(y), "f"(bx), "f"(by), "f"(kSlope));
  return pack_bf16(fmaxf(vx, sx), fmaxf(vy, sy));
}
// bias and activation of a 16 x 16 accumulator, as the next layer's A fragment
__device__ __forceinline__ void next_a(uint32_t (&a)[4], const float (&d0)[4], const float (&d1)[4], const float4 &b) {
  a[0] = act2(d0[0], d0[1], b.x, b.y);
  a[1] = act2(d0[2], d0[3], b.x, b.y);
  a[2] = act2(d1[0], d1[1], b.z, b.w);
  a[3] = act2(d1[2], d1[3], b.z, b.w);
}
// The BF16 rounding of v / sc for four cells.  v * (1 / sc) lies within 2 units
// of the last FP32 place of v / sc, so the two round to the same BF16 unless the
// 16 bits that go are within 4 of half: then, or when 1 / sc may be subnormal
// (`far`), the cells are divided.  32 divisions a lane were a third of the
// encoder's instructions.
__device__ __forceinline__ uint2 scale4(const float4 &v, float sc, float inv, bool far) {
  float4 q = make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv);
  auto low = [](float f) { return (__float_as_uint(f) << 16) + 0x80040000u; };  // <= 8 << 16: near half
  const unsigned m = min(min(low(q.x), low(q.y)), min(low(q.z), low(q.w)));
  if (far || m <= 0x80000u) q = make_float4(v.x / sc, v.y / sc, v.z / sc, v.w / sc);
  return make_uint2(pack_bf16(q.x, q.y), pack_bf16(q.z, q.w));
}

// A lane's cells of the blocks of one row: octant `oct`, cube cells of column
// pair t; of child pair c (bits y1, x1) the 4 z cells from (x + 2 x1, y + 2 y1, z)
// on.  Starts at block `blk` and moves on by `step` blocks.
struct AeCells {
  int bz, bx, by, nbz, nbx, nby, sz, sx, sy;
  __device__ __forceinline__ AeCells(long long blk, long long step, int nbz_, int nbx_, int nby_)
      : nbz(nbz_), nbx(nbx_), nby(nby_) {
    const unsigned u = (unsigned)blk, q = u / nbz, v = (unsigned)step, w = v / nbz;
    bz = (int)(u - q * nbz), bx = (int)(q % nbx), by = (int)(q / nbx);
    sz = (int)(v - w * nbz), sx = (int)(w % nbx), sy = (int)(w / nbx);
  }
  __device__ __forceinline__ void next() {
    bz += sz, bx += sx, by += sy;
    if (bz >= nbz) bz -= nbz, bx++;
    if (bx >= nbx) bx -= nbx, by++;
  }
};
struct AeRow {
  int x, y, z;
  long long o;  // cell offset
  bool ok;      // there is such a block
  __device__ __forceinline__ AeRow(const AeCells &k, int nx, int nz, int oct, int t) {
    x = k.bx * 8 + (oct >> 2) * 4 + (t >> 1);
    y = k.by * 8 + ((oct >> 1) & 1) * 4 + (t & 1);
    z = k.bz * 8 + (oct & 1) * 4;
    ok = k.by < k.nby;
    o = ((long long)y * nx + x) * nz + z;
  }
  __device__ __forceinline__ bool in(int c, int nx, int ny, int nz) const {
    return ok && x + 2 * (c >> 1) < nx && y + 2 * (c & 1) < ny && z < nz;
  }
  __device__ __forceinline__ long long at(int c, int nx, int nz) const {
    return o + (long long)((c & 1) * nx + (c >> 1)) * 2 * nz;
  }
};

// VEC: the volume and the latents are 16-byte aligned and nz % 4 == 0; else cell by cell
template <bool VEC>
__device__ __forceinline__ float4 ae_load4(const float *__restrict__ vol, const AeRow &k, int c, int nx, int ny, int nz) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!k.in(c, nx, ny, nz)) return v;
  const float *s = vol + k.at(c, nx, nz);
  if (VEC) return __ldg(reinterpret_cast<const float4 *>(s));
  v.x = s[0];
  if (k.z + 1 < nz) v.y = s[1];
  if (k.z + 2 < nz) v.z = s[2];
  if (k.z + 3 < nz) v.w = s[3];
  return v;
}

// Persistent: the weights' fragments are made once, then groups of 16 blocks
// are taken until none is left, the next group's cells loaded before the last
// layer of the present one.
template <bool VEC>
__global__ void __launch_bounds__(32 * kAeWarps, 2) ae_encode_k(const float *__restrict__ p,
                                                                const float *__restrict__ vol, int nx, int ny, int nz,
                                                                __nv_bfloat16 *__restrict__ latent,
                                                                float *__restrict__ scales) {
  __shared__ uint4 w2[8][32];                // E2's fragments of k step j, both column tiles
  __shared__ uint4 h3[kAeWarps][32];         // E3's tile of an octant: E4's A fragment
  __shared__ float red[kAeWarps][kAeRows];   // largest |value| of a block's octants
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, t = lane & 3;
  const int nbz = (nz + 7) / 8, nbx = (nx + 7) / 8, nby = (ny + 7) / 8;
  const long long nb = (long long)nbz * nbx * nby, ngroups = (nb + kAeRows - 1) / kAeRows;
  {
    const uint2 f0 = b_frag<1>(p, warp, 0, lane), f1 = b_frag<1>(p, warp, 1, lane);
    w2[warp][lane] = make_uint4(f0.x, f0.y, f1.x, f1.y);
  }
  const uint32_t w10 = b_frag<0>(p, 0, 0, lane).x, w11 = b_frag<0>(p, 0, 1, lane).x;
  const uint2 w30 = b_frag<2>(p, 0, 0, lane), w31 = b_frag<2>(p, 0, 1, lane);
  uint2 w4[8];
#pragma unroll
  for (int k = 0; k < 8; k++) w4[k] = b_frag<3>(p, k, warp, lane);
  const float4 b1 = b_bias<0>(p, 0, lane), b2 = b_bias<1>(p, 0, lane), b3 = b_bias<2>(p, 0, lane);
  const float *b4 = p + w_off(3) + kL_K[3] * kL_N[3] + warp * 8 + 2 * t;
  const float b40 = b4[0], b41 = b4[1];
  float4 v[2][4];
  AeCells k0((long long)blockIdx.x * kAeRows + gr, (long long)gridDim.x * kAeRows, nbz, nbx, nby);
  AeCells k1((long long)blockIdx.x * kAeRows + gr + 8, (long long)gridDim.x * kAeRows, nbz, nbx, nby);
  auto load = [&]() {  // the cells of k0's and k1's blocks
    const AeRow r0(k0, nx, nz, warp, t), r1(k1, nx, nz, warp, t);
#pragma unroll
    for (int c = 0; c < 4; c++) v[0][c] = ae_load4<VEC>(vol, r0, c, nx, ny, nz);
#pragma unroll
    for (int c = 0; c < 4; c++) v[1][c] = ae_load4<VEC>(vol, r1, c, nx, ny, nz);
    k0.next(), k1.next();
  };
  load();
  for (long long grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    float sc[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      float a = 0.f;
#pragma unroll
      for (int c = 0; c < 4; c++)
        a = fmaxf(fmaxf(fmaxf(a, fabsf(v[r][c].x)), fabsf(v[r][c].y)), fmaxf(fabsf(v[r][c].z), fabsf(v[r][c].w)));
      a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 1));
      a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 2));
      if (t == 0) red[warp][gr + 8 * r] = a;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
      sc[r] = red[0][gr + 8 * r];
#pragma unroll
      for (int w = 1; w < kAeWarps; w++) sc[r] = fmaxf(sc[r], red[w][gr + 8 * r]);
    }
    uint2 x[2][4];  // E1's operands: [row][child pair] of z1 = 0, 1
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const float inv = 1.f / sc[r];
      const bool far = !(sc[r] > 1e-30f && sc[r] < 1e30f);
#pragma unroll
      for (int c = 0; c < 4; c++) x[r][c] = sc[r] > 0.f ? scale4(v[r][c], sc[r], inv, far) : make_uint2(0u, 0u);
    }
    float e0[4] = {0.f, 0.f, 0.f, 0.f}, e1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t a[4] = {j & 1 ? x[0][j >> 1].y : x[0][j >> 1].x, j & 1 ? x[1][j >> 1].y : x[1][j >> 1].x, 0u, 0u};
      float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
      mma_bf16(d0, a, w10, 0u);
      mma_bf16(d1, a, w11, 0u);
      uint32_t h[4];
      next_a(h, d0, d1, b1);
      const uint4 w = w2[j][lane];
      mma_bf16(e0, h, w.x, w.y);
      mma_bf16(e1, h, w.z, w.w);
    }
    {
      uint32_t h[4];
      next_a(h, e0, e1, b2);
      float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
      mma_bf16(d0, h, w30.x, w30.y);
      mma_bf16(d1, h, w31.x, w31.y);
      next_a(h, d0, d1, b3);
      h3[warp][lane] = make_uint4(h[0], h[1], h[2], h[3]);
    }
    if (grp + gridDim.x < ngroups) load();
    __syncthreads();
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const uint4 h = h3[k][lane];
      const uint32_t a[4] = {h.x, h.y, h.z, h.w};
      mma_bf16(d, a, w4[k].x, w4[k].y);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const long long blk = grp * kAeRows + gr + 8 * r;
      if (blk >= nb) continue;
      __nv_bfloat16 *l = latent + blk * kLatent + warp * 8 + 2 * t;
      const float l0 = d[2 * r] + b40, l1 = d[2 * r + 1] + b41;
      if (VEC) {
        *reinterpret_cast<uint32_t *>(l) = pack_bf16(l0, l1);
      } else {
        l[0] = __float2bfloat16_rn(l0), l[1] = __float2bfloat16_rn(l1);
      }
      if (warp == 0 && t == 0) scales[blk] = sc[r];
    }
  }
}

constexpr int kLdLat = kLatent + 8;  // row stride of the staged latents: a fragment's loads hit distinct banks

template <bool VEC>
__global__ void __launch_bounds__(32 * kAeWarps, 2) ae_decode_k(const float *__restrict__ p,
                                                                const __nv_bfloat16 *__restrict__ latent,
                                                                const float *__restrict__ scales, int nx, int ny, int nz,
                                                                float *__restrict__ vol) {
  __shared__ uint4 w3[8][32];                                       // D3's fragments of child j, both column tiles
  __shared__ float4 b3[8][4];                                       // D3's biases of child j by lane & 3
  __shared__ __align__(16) __nv_bfloat16 lat[2][kAeRows][kLdLat];   // D1's input, by parity of the group
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, t = lane & 3;
  const int nbz = (nz + 7) / 8, nbx = (nx + 7) / 8, nby = (ny + 7) / 8;
  const long long nb = (long long)nbz * nbx * nby, ngroups = (nb + kAeRows - 1) / kAeRows;
  {
    const uint2 f0 = b_frag<6>(p, 0, 2 * warp, lane), f1 = b_frag<6>(p, 0, 2 * warp + 1, lane);
    w3[warp][lane] = make_uint4(f0.x, f0.y, f1.x, f1.y);
    if (gr == 0) b3[warp][t] = b_bias<6>(p, 2 * warp, lane);
  }
  uint2 w1[4][2];
#pragma unroll
  for (int k = 0; k < 4; k++) w1[k][0] = b_frag<4>(p, k, 2 * warp, lane), w1[k][1] = b_frag<4>(p, k, 2 * warp + 1, lane);
  const uint2 w20 = b_frag<5>(p, 0, 0, lane), w21 = b_frag<5>(p, 0, 1, lane), w4 = b_frag<7>(p, 0, 0, lane);
  const float4 b1 = b_bias<4>(p, 2 * warp, lane), b2 = b_bias<5>(p, 0, lane);
  const float *b4 = p + w_off(7) + kL_K[7] * kL_N[7] + 2 * t;
  const float b40 = b4[0], b41 = b4[1];
  // a group's latents: 16 x 128 bytes, 16 to each of the first 128 threads
  const int lrow = threadIdx.x >> 3, lcol = (threadIdx.x & 7) * 8;
  uint4 ln = make_uint4(0u, 0u, 0u, 0u);
  auto fetch = [&](long long grp) {
    const long long blk = grp * kAeRows + lrow;
    ln = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x >= 8 * kAeRows || blk >= nb) return;
    const __nv_bfloat16 *l = latent + blk * kLatent + lcol;
    if (VEC) {
      ln = __ldg(reinterpret_cast<const uint4 *>(l));
    } else {
      const unsigned short *u = reinterpret_cast<const unsigned short *>(l);
      ln = make_uint4(u[0] | (unsigned)u[1] << 16, u[2] | (unsigned)u[3] << 16, u[4] | (unsigned)u[5] << 16,
                      u[6] | (unsigned)u[7] << 16);
    }
  };
  fetch(blockIdx.x);
  AeCells k0((long long)blockIdx.x * kAeRows + gr, (long long)gridDim.x * kAeRows, nbz, nbx, nby);
  AeCells k1((long long)blockIdx.x * kAeRows + gr + 8, (long long)gridDim.x * kAeRows, nbz, nbx, nby);
  int par = 0;
  for (long long grp = blockIdx.x; grp < ngroups; grp += gridDim.x, par ^= 1) {
    if (threadIdx.x < 8 * kAeRows) *reinterpret_cast<uint4 *>(&lat[par][lrow][lcol]) = ln;
    if (grp + gridDim.x < ngroups) fetch(grp + gridDim.x);
    float sc[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const long long blk = grp * kAeRows + gr + 8 * r;
      sc[r] = blk < nb ? scales[blk] : 0.f;
    }
    __syncthreads();
    float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const __nv_bfloat16 *l = &lat[par][gr][16 * k + 2 * t];
      const uint32_t a[4] = {
          *reinterpret_cast<const uint32_t *>(l), *reinterpret_cast<const uint32_t *>(l + 8 * kLdLat),
          *reinterpret_cast<const uint32_t *>(l + 8), *reinterpret_cast<const uint32_t *>(l + 8 * kLdLat + 8)};
      mma_bf16(d0, a, w1[k][0].x, w1[k][0].y);
      mma_bf16(d1, a, w1[k][1].x, w1[k][1].y);
    }
    uint32_t h[4];
    next_a(h, d0, d1, b1);
#pragma unroll
    for (int i = 0; i < 4; i++) d0[i] = d1[i] = 0.f;
    mma_bf16(d0, h, w20.x, w20.y);
    mma_bf16(d1, h, w21.x, w21.y);
    next_a(h, d0, d1, b2);
    const AeRow r0(k0, nx, nz, warp, t), r1(k1, nx, nz, warp, t);
    k0.next(), k1.next();
#pragma unroll
    for (int c = 0; c < 4; c++) {
      float o[2][4];  // [row][z]
#pragma unroll
      for (int z1 = 0; z1 < 2; z1++) {
        const int j = 2 * c + z1;
        const uint4 w = w3[j][lane];
        float f0[4] = {0.f, 0.f, 0.f, 0.f}, f1[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16(f0, h, w.x, w.y);
        mma_bf16(f1, h, w.z, w.w);
        uint32_t a[4];
        next_a(a, f0, f1, b3[j][t]);
        mma_bf16(e, a, w4.x, w4.y);
#pragma unroll
        for (int r = 0; r < 2; r++) {
          o[r][2 * z1] = sc[r] * (e[2 * r] + b40);
          o[r][2 * z1 + 1] = sc[r] * (e[2 * r + 1] + b41);
        }
      }
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const AeRow &k = r ? r1 : r0;
        if (!k.in(c, nx, ny, nz)) continue;
        float *q = vol + k.at(c, nx, nz);
        if (VEC) {
          *reinterpret_cast<float4 *>(q) = make_float4(o[r][0], o[r][1], o[r][2], o[r][3]);
        } else {
#pragma unroll
          for (int z = 0; z < 4; z++)
            if (k.z + z < nz) q[z] = o[r][z];
        }
      }
    }
  }
}

}  // namespace

long long ae_volume_blocks(int nx, int ny, int nz) {
  return (long long)((nx + 7) / 8) * ((ny + 7) / 8) * ((nz + 7) / 8);
}

int ae_prepare(rtm_ae *a) { return ae_reserve(a, kChunkBlocks, false); }

// CTAs of one wave of a persistent codec kernel on the current device
template <typename K>
static int ae_wave(K kernel) {
  int dev = 0, sms = 0, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 32 * kAeWarps, 0);
  return std::max(1, sms) * std::max(1, occ);
}
static void ae_waves(rtm_ae *a) {
  a->wave_enc[0] = ae_wave(ae_encode_k<false>), a->wave_enc[1] = ae_wave(ae_encode_k<true>);
  a->wave_dec[0] = ae_wave(ae_decode_k<false>), a->wave_dec[1] = ae_wave(ae_decode_k<true>);
}
static unsigned ae_grid(int wave, int nx, int ny, int nz) {
  return (unsigned)std::min<long long>((ae_volume_blocks(nx, ny, nz) + kAeRows - 1) / kAeRows, wave);
}
static bool ae_aligned(const void *vol, const void *latent, int nz) {
  return nz % 4 == 0 && ((reinterpret_cast<uintptr_t>(vol) | reinterpret_cast<uintptr_t>(latent)) & 15) == 0;
}

// volume -> latents [nb][64] (bfloat16) + scales [nb] (device), on stream st
int ae_compress(rtm_ae *a, const float *w, int nx, int ny, int nz, void *latent, float *scales, cudaStream_t st) {
  const bool vec = ae_aligned(w, latent, nz);
  auto *k = vec ? ae_encode_k<true> : ae_encode_k<false>;
  k<<<ae_grid(a->wave_enc[vec], nx, ny, nz), 32 * kAeWarps, 0, st>>>(a->p, w, nx, ny, nz, static_cast<__nv_bfloat16 *>(latent), scales);
  return cudaGetLastError() == cudaSuccess ? RTM_OK : RTM_ERR_CUDA;
}
// latents + scales -> volume (device), on stream st
int ae_decompress(rtm_ae *a, const void *latent, const float *scales, int nx, int ny, int nz, float *w,
                  cudaStream_t st) {
  const bool vec = ae_aligned(w, latent, nz);
  auto *k = vec ? ae_decode_k<true> : ae_decode_k<false>;
  k<<<ae_grid(a->wave_dec[vec], nx, ny, nz), 32 * kAeWarps, 0, st>>>(a->p, static_cast<const __nv_bfloat16 *>(latent), scales, nx, ny, nz, w);
  return cudaGetLastError() == cudaSuccess ? RTM_OK : RTM_ERR_CUDA;
}

// ---- FP16 fallback of the high-energy blocks of a learned snapshot ----------
// Per slot: a header, the indices of the stored blocks, and each stored block
// as 512 FP16 values of v / scale (natural z, x, y order).  The stored blocks
// are the candidates (scale > 0 and > tau x the largest) whose scale exceeds
// the (cap+1)-th largest candidate scale, all of them when there are at most
// cap: a deterministic choice, found by a radix select over the scales' IEEE
// bit patterns (positive floats order like their bits) in three levels of
// 11, 11 and 9 bits; thr ends as the smallest bit pattern stored.
namespace {

constexpr int kFbBins = 2048;
__host__ __device__ constexpr int fb_shift(int L) { return L == 0 ? 20 : L == 1 ? 9 : 0; }
__host__ __device__ constexpr int fb_width(int L) { return L == 2 ? 9 : 11; }

struct FbHdr {
  unsigned maxbits, prefix, thr;
  int count, rem, done;
  int hist[kFbBins];
};

__global__ void fb_max_k(const float *__restrict__ scales, long long nb, FbHdr *h) {
  float m = 0.f;
  for (long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += (long long)gridDim.x * blockDim.x)
    m = fmaxf(m, scales[b]);
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(&h->maxbits, __float_as_uint(m));
}

// histogram of the candidates inside the current prefix, by their next bits
template <int L>
__global__ void fb_hist_k(const float *__restrict__ scales, long long nb, float tau, FbHdr *h) {
  if (h->done) return;
  constexpr int hi = fb_shift(L) + fb_width(L);
  const float mx = __uint_as_float(h->maxbits);
  const unsigned pre = h->prefix >> hi;
  for (long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += (long long)gridDim.x * blockDim.x) {
    const float s = scales[b];
    const unsigned u = __float_as_uint(s);
    if (s > 0.f && s > tau * mx && (u >> hi) == pre)
      atomicAdd(&h->hist[(u >> fb_shift(L)) & ((1u << fb_width(L)) - 1)], 1);
  }
}

// the bin, from the top, where the running count passes the capacity left
template <int L>
__global__ void __launch_bounds__(256) fb_scan_k(FbHdr *h, int cap) {
  __shared__ int part[256];
  __shared__ int found;
  if (h->done) return;
  constexpr int nbin = 1 << fb_width(L), per = nbin / 256 > 0 ? nbin / 256 : 1;
  const int t = threadIdx.x;
  const int top = nbin - 1 - t * per;  // this thread's bins: top, top-1, ..., top-per+1 (t * per < nbin)
  int v[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = (i < per && t * per < nbin) ? h->hist[top - i] : 0;
    sum += v[i];
  }
  part[t] = sum;
  if (t == 0) found = 0;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {  // inclusive scan (Hillis-Steele)
    const int x = t >= o ? part[t - o] : 0;
    __syncthreads();
    part[t] += x;
    __syncthreads();
  }
  const int rem = L == 0 ? cap : h->rem;  // read by all before the one write below
  const int before = part[t] - sum;  // candidates in the bins above this thread's
  if (before <= rem && part[t] > rem) {  // the boundary bin is one of this thread's
    int cum = before, k = 0;
    while (cum + v[k] <= rem) cum += v[k++];
    const unsigned bin = (unsigned)(top - k);
    if (L == 2) {
      h->thr = h->prefix + (bin + 1);  // the bins above the boundary (bin + 1 may carry into the prefix)
      h->done = 1;
    } else {
      h->prefix |= bin << fb_shift(L);
      h->rem = rem - cum;
    }
    found = 1;
  }
  __syncthreads();
  if (t == 0 && !found) {  // every candidate inside the prefix fits
    h->thr = h->prefix;
    h->done = 1;
  }
  for (int i = t; i < kFbBins; i += 256) h->hist[i] = 0;  // for the next level
}

// the chosen blocks: index and FP16 copy of v / scale (one CTA of 512 per block)
__global__ void __launch_bounds__(512) fb_store_k(const float *__restrict__ w, const float *__restrict__ scales,
                                                  long long nb, float tau, int nx, int ny, int nz, FbHdr *h, int *idx,
                                                  __half *data) {
  __shared__ int slot;
  const float mx = __uint_as_float(h->maxbits);
  for (long long b = blockIdx.x; b < nb; b += gridDim.x) {
    const float s = scales[b];
    if (!(s > 0.f && s > tau * mx && __float_as_uint(s) >= h->thr)) continue;  // uniform over the CTA
    if (threadIdx.x == 0) {
      slot = atomicAdd(&h->count, 1);
      idx[slot] = (int)b;
    }
    __syncthreads();
    const int nbz = (nz + 7) / 8, nbx = (nx + 7) / 8;
    const int bz = (int)(b % nbz), bx = (int)((b / nbz) % nbx), by = (int)(b / ((long long)nbz * nbx));
    const int k = threadIdx.x & 7, i = (threadIdx.x >> 3) & 7, j = threadIdx.x >> 6;
    const int x = bx * 8 + i, y = by * 8 + j, z = bz * 8 + k;
    const float v = (x < nx && y < ny && z < nz) ? w[((long long)y * nx + x) * nz + z] : 0.f;
    data[(long long)slot * 512 + threadIdx.x] = __float2half_rn(v / s);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(512) fb_apply_k(const float *__restrict__ scales, const FbHdr *h, const int *idx,
                                                  const __half *data, int cap, int nx, int ny, int nz, float *w) {
  const int n = min(h->count, cap);  // a slot never stored holds no valid count: clamp, check each index
  const long long nb = (long long)((nx + 7) / 8) * ((ny + 7) / 8) * ((nz + 7) / 8);
  for (int t = blockIdx.x; t < n; t += gridDim.x) {
    const long long b = idx[t];
    if (b < 0 || b >= nb) continue;
    const int nbz = (nz + 7) / 8, nbx = (nx + 7) / 8;
    const int bz = (int)(b % nbz), bx = (int)((b / nbz) % nbx), by = (int)(b / ((long long)nbz * nbx));
    const int k = threadIdx.x & 7, i = (threadIdx.x >> 3) & 7, j = threadIdx.x >> 6;
    const int x = bx * 8 + i, y = by * 8 + j, z = bz * 8 + k;
    if (x < nx && y < ny && z < nz)
      w[((long long)y * nx + x) * nz + z] = __half2float(data[(long long)t * 512 + threadIdx.x]) * scales[b];
  }
}

}  // namespace

size_t ae_fallback_bytes(long long cap) { return sizeof(FbHdr) + (size_t)cap * 4 + (size_t)cap * 1024; }

void ae_fallback_store(const float *w, const float *scales, int nx, int ny, int nz, float tau, long long cap, void *fb,
                       cudaStream_t st) {
  const long long nb = ae_volume_blocks(nx, ny, nz);
  FbHdr *h = static_cast<FbHdr *>(fb);
  int *idx = reinterpret_cast<int *>(h + 1);
  __half *data = reinterpret_cast<__half *>(idx + cap);
  cudaMemsetAsync(h, 0, sizeof(FbHdr), st);
  const unsigned g = (unsigned)std::min<long long>((nb + 255) / 256, 1184);
  fb_max_k<<<g, 256, 0, st>>>(scales, nb, h);
  fb_hist_k<0><<<g, 256, 0, st>>>(scales, nb, tau, h);
  fb_scan_k<0><<<1, 256, 0, st>>>(h, (int)cap);
  fb_hist_k<1><<<g, 256, 0, st>>>(scales, nb, tau, h);
  fb_scan_k<1><<<1, 256, 0, st>>>(h, (int)cap);
  fb_hist_k<2><<<g, 256, 0, st>>>(scales, nb, tau, h);
  fb_scan_k<2><<<1, 256, 0, st>>>(h, (int)cap);
  fb_store_k<<<(unsigned)std::min<long long>(nb, 4096), 512, 0, st>>>(w, scales, nb, tau, nx, ny, nz, h, idx, data);
}

void ae_fallback_apply(const float *scales, int nx, int ny, int nz, long long cap, const void *fb, float *w,
                       cudaStream_t st) {
  const FbHdr *h = static_cast<const FbHdr *>(fb);
  const int *idx = reinterpret_cast<const int *>(h + 1);
  const __half *data = reinterpret_cast<const __half *>(idx + cap);
  fb_apply_k<<<(unsigned)std::max<long long>(1, std::min<long long>(cap, 4096)), 512, 0, st>>>(scales, h, idx, data,
                                                                                                  (int)cap, nx, ny, nz, w);
}

}  // namespace rtm

extern "C" {

int rtm_ae_nparams(void) { return rtm::kNParams; }

int rtm_ae_create(rtm_ae **out) {
  if (!out) return RTM_ERR_ARG;
  *out = nullptr;
  rtm_ae *a = new rtm_ae();
  cudaGetDevice(&a->device);
  const size_t b = (size_t)rtm::kNParams * 4;
  // a blocking stream: ordered after the parameter uploads (pageable cudaMemcpy)
  if (cudaStreamCreate(&a->st) || cudaMalloc(&a->p, b) || cudaMalloc(&a->g, b) ||
      cudaMalloc(&a->m, b) || cudaMalloc(&a->v, b) || cudaMalloc(&a->loss, 4) || cudaMemset(a->p, 0, b) ||
      cudaMemset(a->m, 0, b) || cudaMemset(a->v, 0, b)) {
    cudaGetLastError();
    rtm_ae_destroy(a);
    return RTM_ERR_NOMEM;
  }
  rtm::ae_waves(a);
  *out = a;
  return RTM_OK;
}

int rtm_ae_destroy(rtm_ae *a) {
  if (!a) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  if (a->st) cudaStreamSynchronize(a->st);
  rtm::ae_free_ws(a);
  cudaFree(a->p), cudaFree(a->g), cudaFree(a->m), cudaFree(a->v), cudaFree(a->loss);
  if (a->st) cudaStreamDestroy(a->st);
  delete a;
  return RTM_OK;
}

int rtm_ae_set_params(rtm_ae *a, const float *params) {
  if (!a || !params) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  if (cudaMemcpy(a->p, params, (size_t)rtm::kNParams * 4, cudaMemcpyHostToDevice)) return RTM_ERR_CUDA;
  cudaMemset(a->m, 0, (size_t)rtm::kNParams * 4), cudaMemset(a->v, 0, (size_t)rtm::kNParams * 4);
  a->step = 0;
  return RTM_OK;
}

int rtm_ae_get_params(rtm_ae *a, float *params) {
  if (!a || !params) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  cudaStreamSynchronize(a->st);
  return cudaMemcpy(params, a->p, (size_t)rtm::kNParams * 4, cudaMemcpyDeviceToHost) ? RTM_ERR_CUDA : RTM_OK;
}

int rtm_ae_loss_grad(rtm_ae *a, const float *blocks, int n, float *loss, float *grads) {
  if (!a || !blocks || n < 1 || !loss) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  if (int rc = rtm::ae_reserve(a, n, true)) return rc;
  if (cudaMemcpyAsync(a->x0, blocks, (size_t)n * rtm::kBlock * 4, cudaMemcpyHostToDevice, a->st)) return RTM_ERR_CUDA;
  rtm::ae_loss_grad(a, n);
  cudaMemcpyAsync(loss, a->loss, 4, cudaMemcpyDeviceToHost, a->st);
  if (grads) cudaMemcpyAsync(grads, a->g, (size_t)rtm::kNParams * 4, cudaMemcpyDeviceToHost, a->st);
  return cudaStreamSynchronize(a->st) == cudaSuccess ? RTM_OK : RTM_ERR_CUDA;
}

int rtm_ae_train_step(rtm_ae *a, const float *blocks, int n, float lr, float *loss) {
  if (!a || !blocks || n < 1 || !loss || !(lr > 0.f)) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  if (int rc = rtm::ae_reserve(a, n, true)) return rc;
  if (cudaMemcpyAsync(a->x0, blocks, (size_t)n * rtm::kBlock * 4, cudaMemcpyHostToDevice, a->st)) return RTM_ERR_CUDA;
  rtm::ae_loss_grad(a, n);
  a->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)a->step), c2 = 1.f - powf(b2, (float)a->step);
  rtm::adam_k<<<(rtm::kNParams + 255) / 256, 256, 0, a->st>>>(a->p, a->g, a->m, a->v, rtm::kNParams, lr, b1, b2, 1e-8f,
                                                            c1, c2);
  cudaMemcpyAsync(loss, a->loss, 4, cudaMemcpyDeviceToHost, a->st);
  return cudaStreamSynchronize(a->st) == cudaSuccess ? RTM_OK : RTM_ERR_CUDA;
}

int rtm_ae_reconstruct(rtm_ae *a, const float *blocks, int n, float *out, float *latent) {
  if (!a || !blocks || n < 1 || !out) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  if (int rc = rtm::ae_reserve(a, n, false)) return rc;
  if (cudaMemcpyAsync(a->x0, blocks, (size_t)n * rtm::kBlock * 4, cudaMemcpyHostToDevice, a->st)) return RTM_ERR_CUDA;
  rtm::ae_forward(a, n, a->x0, 0, rtm::kLayers, false, a->st);
  cudaMemcpyAsync(out, a->y[rtm::kLayers - 1], (size_t)n * rtm::kBlock * 4, cudaMemcpyDeviceToHost, a->st);
  if (latent) cudaMemcpyAsync(latent, a->y[3], (size_t)n * rtm::kLatent * 4, cudaMemcpyDeviceToHost, a->st);
  return cudaStreamSynchronize(a->st) == cudaSuccess ? RTM_OK : RTM_ERR_CUDA;
}

int rtm_ae_compress_volume(rtm_ae *a, const float *d_vol, int nx, int ny, int nz, void *d_latent, float *d_scales,
                           void *stream) {
  if (!a || !d_vol || !d_latent || !d_scales || nx < 1 || ny < 1 || nz < 1) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  return rtm::ae_compress(a, d_vol, nx, ny, nz, d_latent, d_scales, (cudaStream_t)stream);
}

int rtm_ae_decompress_volume(rtm_ae *a, const void *d_latent, const float *d_scales, int nx, int ny, int nz,
                             float *d_vol, void *stream) {
  if (!a || !d_vol || !d_latent || !d_scales || nx < 1 || ny < 1 || nz < 1) return RTM_ERR_ARG;
  cudaSetDevice(a->device);
  return rtm::ae_decompress(a, d_latent, d_scales, nx, ny, nz, d_vol, (cudaStream_t)stream);
}

}  // extern "C"
