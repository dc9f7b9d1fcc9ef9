// kernels_cfd_tile.cu - compact-FD line solves over shared-memory tiles, the
// default of every axis.  A derivative along one axis solves B f' = A f for
// every grid line (FdEngine_cfd::banmul_* / banbks_*,
// bgprtm/FdEngine_cfd.cpp:164-356).  A CTA holds 32 lines (lane = line), one HBM
// read and one write per cell:
//   1  its warps form the 11-point right-hand sides, a run of rows each;
//   2  one warp runs the two recurrences of the band LU.
//
// What bounds it: shared memory caps the lines in flight (three 512-point tiles
// a SM), so the launch takes (tiles / resident tiles) x (latency of one tile),
// and a tile's latency is the serial work of its warps.  Cycles of a 512-point
// tile, before this form and now: load 5 k / 4 k, right-hand sides 10.5 k / 5-7 k,
// elimination 12.5 k / 5.2 k, back substitution 15.7 k / 8.3 k, store 5 k / 2.5 k;
// a launch at 512 x 512 x 400: x / y lines 400 -> 240 us, z lines 410 -> 210 us
// (HBM copy rate: 130 us).  Every phase is written for the fewest instructions
// on its critical warp:
//   - lines live in shared memory as row quads (4 consecutive rows of a line in
//     one float4), so the recurrences move a quad per load / store instead of a
//     row; x / y tiles arrive row by row, and the right-hand-side pass, which
//     rewrites every value anyway, leaves them in quads (a quad row of the 32
//     lines takes the place of the 4 rows it came from), the back substitution
//     turns them back;
//   - each pivot is taken off the four following rows as soon as it is final
//     (the row's terms still arrive oldest pivot first, one FMA each, so the
//     bits are those of the row-by-row form): the row-to-row chain is one FMA
//     (elimination, 7.9 cycles a row alone on an SM, 18 before) or a multiply and
//     an FMA (back substitution, 12 cycles, 21 before);
//   - three quads are loaded ahead; the factors of the Toeplitz interior (rows
//     k0 .. k1 - 1, bitwise constant) come from the parameter bank, the others
//     from a table staged in shared memory while the tile loads (from global
//     memory these ~89 rows cost a third of both recurrences).  Loading a quad's
//     table rows one quad ahead was slower (z lines 232 us): the copies cost
//     more than the wait;
//   - resident CTAs solve on different schedulers (285 -> 259 us);
//   - four warps where four or more tiles fit an SM, eight where fewer do
//     (tile_threads);
//   - the tile that a resident CTA's successor will load is prefetched into L2
//     (250 -> 240 us).
#include <algorithm>

#include "cfd_rows.cuh"
#include "kernel_api.h"
#include "launch.cuh"
#include "rtm_device.cuh"
#include "tma.cuh"

namespace rtm {

namespace {

// How a tile reaches shared memory: x / y lines (32 consecutive z of one line
// set, row i of every line contiguous) by TMA boxes or plain copies, z lines
// (contiguous in memory) by bulk copies or plain copies
enum { IO_ROWS_TMA = 0, IO_ROWS = 1, IO_LINES_BULK = 2, IO_LINES = 3 };
constexpr bool io_rows(int io) { return io == IO_ROWS_TMA || io == IO_ROWS; }

struct TileArgs {
  const float *in;
  float *out;
  int nz;                  // rows: z extent
  long long es, other;     // rows: element stride of a line, stride of line sets
  int axis, R, nb;         // rows by TMA: box rows and count
  long long nlines;        // lines
  int lines, pitch;        // lines: per tile (<= 32), floats per line in shared memory
  int tab;                 // table rows
  int off;                 // byte offset of the tile
  int sms;                 // SMs of the device (CTAs of a wave)
  int ahead;               // CTAs resident at once: the tile that many on is prefetched into L2
};

// One lane's line in the tile: raw rows and quads
template <bool ROWS>
struct Line {
  float *r;
  float4 *q;
  __device__ __forceinline__ float &row(int i) const { return r[ROWS ? i * 32 : i]; }
  __device__ __forceinline__ float4 &quad(int k) const { return q[ROWS ? k * 32 : k]; }
  // 8 raw rows from i (a multiple of 8); the tile has room past its last row
  __device__ __forceinline__ void load8(float (&v)[8], int i) const {
    if (ROWS) {
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = row(i + k);
    } else {
      const float4 a = quad(i / 4), b = quad(i / 4 + 1);
      v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    }
  }
  // one value of row i in quad form
  __device__ __forceinline__ float &elem(int i) const { return reinterpret_cast<float *>(&quad(i / 4))[i % 4]; }
};

// Phase 1.  Warp w takes a run of 8-row chunks; the rows of the neighbouring
// runs that its windows reach are read before the barrier, so the runs can be
// rewritten in place as quads.  The loop forms every row as an interior one;
// the one-sided rows of the line's ends and the zero rows from n up to the next
// multiple of 4 are written over afterwards (selecting them inside the loop
// doubled its time).  act: the lane holds a line.
template <bool ROWS>
__device__ __forceinline__ void tile_rhs(const CfdPlanDev &p, const Line<ROWS> &L, int warp, int nw, bool act) {
  const int n = p.n, n4 = (n + 3) / 4 * 4;
  const int run = ((n4 + 7) / 8 + nw - 1) / nw * 8;
  const int p0 = min(n4, warp * run), p1 = min(n4, p0 + run);
  const bool own = act && p0 < p1;
  float prev[5], post[5], cur[8];
  // one-sided rows, every coefficient index a constant (indexed reads of the
  // parameter bank are slow): rows 0 .. 4 by the first run, rows n - 5 .. n - 1
  // by the runs that reach them (never the first: n >= 16)
  const bool lo = p0 == 0, hi = !lo && p1 > n - 5;
  float ends[5];
  if (own) {
    if (lo || hi) {
      float x[16];  // lo: rows -5 .. 10; hi: rows n - 11 .. n - 1
#pragma unroll
      for (int k = 0; k < 16; k++) x[k] = lo ? (k < 5 ? 0.f : L.row(k - 5)) : (k < 11 ? L.row(n - 11 + k) : 0.f);
#pragma unroll
      for (int k = 0; k < 5; k++) ends[k] = lo ? rhs_low(p.a, k, x + k) : rhs_high(p.a, 5 - k, x + 1 + k);
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {
      prev[k] = p0 - 5 + k >= 0 ? L.row(p0 - 5 + k) : 0.f;
      post[k] = p1 + k < n ? L.row(p1 + k) : 0.f;
    }
    L.load8(cur, p0);
  }
  __syncthreads();
  if (!own) return;
  const RhsCoef rc{p.a[55], p.a[56], p.a[57], p.a[58], p.a[59]};
  // rows i0 .. i0 + 7 from prev (i0 - 5 ..), cur and next (i0 + 8 ..)
  auto chunk = [&](int i0, const float *next, bool two) {
    float w[18];
#pragma unroll
    for (int k = 0; k < 18; k++) w[k] = k < 5 ? prev[k] : k < 13 ? cur[k - 5] : next[k - 13];
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; k++)
      v[k] = rhs_interior(rc, w[k], w[k + 1], w[k + 2], w[k + 3], w[k + 4], w[k + 6], w[k + 7], w[k + 8], w[k + 9],
                          w[k + 10]);
    if (ROWS) __syncwarp();  // a quad row replaces four rows of other lanes
    L.quad(i0 / 4) = make_float4(v[0], v[1], v[2], v[3]);
    if (two) L.quad(i0 / 4 + 1) = make_float4(v[4], v[5], v[6], v[7]);
  };
  int i0 = p0;
#pragma unroll 1
  for (; i0 + 8 < p1; i0 += 8) {
    float next[8];
    L.load8(next, i0 + 8);
    chunk(i0, next, true);
#pragma unroll
    for (int k = 0; k < 5; k++) prev[k] = cur[k + 3];
#pragma unroll
    for (int k = 0; k < 8; k++) cur[k] = next[k];
  }
  chunk(i0, post, i0 + 4 < n4);
  if (lo || hi)
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const int i = lo ? k : n - 5 + k;
      if (i >= p0 && i < p1) L.elem(i) = ends[k];
    }
  if (p1 == n4)
    for (int i = n; i < n4; i++) L.elem(i) = 0.f;
}

// Factors of the rows outside [k0, k1), in shared memory: per pivot row the
// multipliers to the next four rows, the upper-factor entries of the four rows
// before it, and the reciprocal pivot
struct TileTab {
  const float4 *l, *u;
  const float *rd;
};

// taking pivot value v of coefficients c off the four rows after it
#define CFD_TAKE(c, v, a0, a1, a2, a3) \
  a0 = __fmaf_rn(-c.x, v, a0), a1 = __fmaf_rn(-c.y, v, a1), a2 = __fmaf_rn(-c.z, v, a2), a3 = __fmaf_rn(-c.w, v, a3)

// Elimination of the quads [qb, qe): c / d / e hold quads q, q + 1, q + 2, the
// pivots before q already taken off; t: table row of quad qb's first pivot
template <bool ROWS, bool CST>
__device__ __forceinline__ void fwd_quads(const Line<ROWS> &L, const float4 *t, float4 mc, int qb, int qe, int last,
                                          float4 &c, float4 &d, float4 &e) {
#pragma unroll 4
  for (int q = qb; q < qe; q++) {
    const float4 f = L.quad(min(q + 3, last));
    const float4 m0 = CST ? mc : t[0], m1 = CST ? mc : t[1], m2 = CST ? mc : t[2], m3 = CST ? mc : t[3];
    CFD_TAKE(m0, c.x, c.y, c.z, c.w, d.x);
    CFD_TAKE(m1, c.y, c.z, c.w, d.x, d.y);
    CFD_TAKE(m2, c.z, c.w, d.x, d.y, d.z);
    CFD_TAKE(m3, c.w, d.x, d.y, d.z, d.w);
    L.quad(q) = c;
    c = d, d = e, e = f;
    if (!CST) t += 4;
  }
}

// Back substitution of the quads qe - 1 down to qb: c / d / e hold quads
// q, q - 1, q - 2; t / r: table rows of quad qe - 1's first row
template <bool ROWS, bool CST>
__device__ __forceinline__ void bwd_quads(const Line<ROWS> &L, const float4 *t, const float *r, float4 uc, float rc,
                                          int qb, int qe, float4 &c, float4 &d, float4 &e) {
#pragma unroll 4
  for (int q = qe - 1; q >= qb; q--) {
    const float4 f = L.quad(max(q - 3, 0));
    const float4 u0 = CST ? uc : t[0], u1 = CST ? uc : t[1], u2 = CST ? uc : t[2], u3 = CST ? uc : t[3];
    c.w = __fmul_rn(c.w, CST ? rc : r[3]);
    CFD_TAKE(u3, c.w, c.z, c.y, c.x, d.w);
    c.z = __fmul_rn(c.z, CST ? rc : r[2]);
    CFD_TAKE(u2, c.z, c.y, c.x, d.w, d.z);
    c.y = __fmul_rn(c.y, CST ? rc : r[1]);
    CFD_TAKE(u1, c.y, c.x, d.w, d.z, d.y);
    c.x = __fmul_rn(c.x, CST ? rc : r[0]);
    CFD_TAKE(u0, c.x, d.w, d.z, d.y, d.x);
    if (ROWS) {
      __syncwarp();  // rows replace the quad row of other lanes (all loaded three quads ago)
      L.row(4 * q) = c.x, L.row(4 * q + 1) = c.y, L.row(4 * q + 2) = c.z, L.row(4 * q + 3) = c.w;
    } else {
      L.quad(q) = c;
    }
    c = d, d = e, e = f;
    if (!CST) t -= 4, r -= 4;
  }
}
#undef CFD_TAKE

// Phase 2: both recurrences of one line (a whole warp calls it for ROWS)
template <bool ROWS>
__device__ __forceinline__ void tile_solve(const CfdPlanDev &p, const TileTab &tab, const Line<ROWS> &L) {
  const int Q = (p.n + 3) / 4, qa = p.k0 / 4, qz = p.k1 / 4;
  const float4 mc = make_float4(p.lmc[0], p.lmc[1], p.lmc[2], p.lmc[3]);
  const float4 uc = make_float4(p.buc[0], p.buc[1], p.buc[2], p.buc[3]);
  float4 c = L.quad(0), d = L.quad(1), e = L.quad(2);
  fwd_quads<ROWS, false>(L, tab.l, mc, 0, qa, Q - 1, c, d, e);
  fwd_quads<ROWS, true>(L, nullptr, mc, qa, qz, Q - 1, c, d, e);
  fwd_quads<ROWS, false>(L, tab.l + p.k0, mc, qz, Q, Q - 1, c, d, e);
  c = L.quad(Q - 1), d = L.quad(Q - 2), e = L.quad(Q - 3);
  const int tl = p.k0 + 4 * (Q - 1) - p.k1, ta = p.k0 - 4;  // table rows of quads Q - 1 and qa - 1
  bwd_quads<ROWS, false>(L, tab.u + tl, tab.rd + tl, uc, p.rdc, qz, Q, c, d, e);
  bwd_quads<ROWS, true>(L, nullptr, nullptr, uc, p.rdc, qa, qz, c, d, e);
  bwd_quads<ROWS, false>(L, tab.u + ta, tab.rd + ta, uc, p.rdc, 0, qa, c, d, e);
}

// registers for three resident CTAs of 256 threads or six of 128
template <int IO>
__global__ void __launch_bounds__(256, 3) cfd_tile_k(const __grid_constant__ CfdPlanDev p,
                                                     const __grid_constant__ CUtensorMap tin,
                                                     const __grid_constant__ CUtensorMap tout,
                                                     const __grid_constant__ TileArgs a, int *err) {
  constexpr bool ROWS = io_rows(IO), ASYNC = IO == IO_ROWS_TMA || IO == IO_LINES_BULK;
  extern __shared__ __align__(128) unsigned char smraw[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smraw);
  float4 *tl = reinterpret_cast<float4 *>(smraw + 128), *tu = tl + a.tab;
  float *tr = reinterpret_cast<float *>(tu + a.tab);
  float *sm = reinterpret_cast<float *>(smraw + a.off);
  const int n = p.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int iz0 = blockIdx.x * 32, o = blockIdx.y;                // rows
  const long long l0 = (long long)blockIdx.x * a.lines;           // lines
  const int nl = ROWS ? min(32, a.nz - iz0) : (int)min((long long)a.lines, a.nlines - l0);
  const long long base = ROWS ? (long long)o * a.other + iz0 : l0 * n;
  dep_launch();
  dep_wait();
  if (ASYNC) {
    if (threadIdx.x == 0) {
      mbar_init(bar, 1);
      mbar_fence_init();
      // the tile that one of the resident CTAs' successors will load
      const long long nx_ = (long long)blockIdx.x + (long long)blockIdx.y * gridDim.x + a.ahead;
      if (IO == IO_ROWS_TMA) {
        mbar_expect_tx(bar, (uint32_t)a.nb * (uint32_t)a.R * 32u * 4u);
        for (int b = 0; b < a.nb; b++) {
          if (a.axis == DX) tma_load_3d(sm + (size_t)b * a.R * 32, &tin, bar, iz0, b * a.R, o);
          else tma_load_3d(sm + (size_t)b * a.R * 32, &tin, bar, iz0, o, b * a.R);
        }
        const int zn = (int)(nx_ % gridDim.x) * 32, on = (int)(nx_ / gridDim.x);
        if (on < (int)gridDim.y)
          for (int b = 0; b < a.nb; b++) {
            if (a.axis == DX) tma_prefetch_3d(&tin, zn, b * a.R, on);
            else tma_prefetch_3d(&tin, zn, on, b * a.R);
          }
      } else {
        mbar_expect_tx(bar, (uint32_t)nl * (uint32_t)n * 4u);
        for (int l = 0; l < nl; l++)
          bulk_load(sm + (size_t)l * a.pitch, a.in + base + (long long)l * n, (uint32_t)n * 4u, bar);
        const long long ln = nx_ * a.lines;
        if (ln < a.nlines)
          bulk_prefetch(a.in + ln * n, (uint32_t)min((long long)a.lines, a.nlines - ln) * (uint32_t)n * 4u);
      }
    }
  } else if (IO == IO_ROWS) {
    for (int i = warp; i < n; i += nw) {
      if (lane < nl) cp_async4(sm + i * 32 + lane, a.in + base + lane + (long long)i * a.es);
      else sm[i * 32 + lane] = 0.f;
    }
  } else {
    for (int l = warp; l < nl; l += nw) {
      const float *src = a.in + base + (long long)l * n;
      float *dst = sm + l * a.pitch;
#pragma unroll 4
      for (int i = lane; i < n; i += 32) cp_async4(dst + i, src + i);
    }
  }
  // the factor table while the tile loads
  for (int k = threadIdx.x; k < a.tab; k += blockDim.x) {
    const int i = k < p.k0 ? k : k - p.k0 + p.k1;
    tl[k] = __ldg(reinterpret_cast<const float4 *>(p.tl) + i);
    tu[k] = __ldg(reinterpret_cast<const float4 *>(p.tu) + i);
    tr[k] = __ldg(p.tr + i);
  }
  // The solving warp.  Warp k of every CTA issues from scheduler k of its SM, so
  // one fixed warp would put all resident solvers on one scheduler (the fourth
  // of the right-hand sides that shares it then took twice as long, as did the
  // solvers); CTAs that are resident together differ in their wave, mostly.
  const int sw = (int)((blockIdx.x + (long long)blockIdx.y * gridDim.x) / a.sms) & 3;
  __syncthreads();  // the mbarrier is initialised
  if (ASYNC) {
    if (!__syncthreads_and(mbar_wait(bar, 0, err))) {
      if (threadIdx.x == 0) mbar_drain(bar, 0);
      return;
    }
  } else {
    cp_async_wait_all();
    __syncthreads();
  }
  Line<ROWS> L;
  L.r = ROWS ? sm + lane : sm + lane * a.pitch;
  L.q = ROWS ? reinterpret_cast<float4 *>(sm) + lane : reinterpret_cast<float4 *>(sm + lane * a.pitch);
  const bool act = ROWS || lane < nl;  // rows: lanes past nz hold zeros
  tile_rhs<ROWS>(p, L, warp, nw, act);
  __syncthreads();
  if (warp == sw && act) tile_solve<ROWS>(p, TileTab{tl, tu, tr}, L);
  if (ASYNC) {
    fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      if (IO == IO_ROWS_TMA) {
        for (int b = 0; b < a.nb; b++) {
          if (a.axis == DX) tma_store_3d(&tout, sm + (size_t)b * a.R * 32, iz0, b * a.R, o);
          else tma_store_3d(&tout, sm + (size_t)b * a.R * 32, iz0, o, b * a.R);
        }
      } else {
        for (int l = 0; l < nl; l++)
          bulk_store(a.out + base + (long long)l * n, sm + (size_t)l * a.pitch, (uint32_t)n * 4u);
      }
      bulk_commit();
      bulk_wait_read();
    }
  } else {
    __syncthreads();
    if (IO == IO_ROWS) {
      for (int i = warp; i < n; i += nw)
        if (lane < nl) __stcg(a.out + base + lane + (long long)i * a.es, sm[i * 32 + lane]);
    } else {
      for (int l = warp; l < nl; l += nw)
        for (int i = lane; i < n; i += 32) __stcg(a.out + base + (long long)l * n + i, sm[l * a.pitch + i]);
    }
  }
}

constexpr size_t kTileSmem = 227 * 1024;

// Tiles whose shared memory fits an SM together
int tiles_fit(size_t smem) { return (int)((228 * 1024) / (smem + 1024)); }

// Threads of a tile of `smem` bytes.  The registers let six CTAs of 128 threads or
// three of 256 onto an SM.  While four or more tiles fit, their number hides more
// than their warps: lines of 256 points, 512 x 400 of them, take 105 us (x) and 106
// us (z) with 128 threads, 144 and 127 with 256; of 400 points, 400 x 400, 142 and
// 136 against 158 and 136.  Where three fit, either way (512 points: 236 and 221
// against 236 and 223), eight warps copy faster if the copies are not asynchronous
// (512 points, depth 151: 95 and 63 against 79 and 61 us).  Plain copies already
// want them where four tiles fit: 320 points, five tiles, 150 us against 156, 330
// points, four tiles, 67 against 59.
int tile_threads(size_t smem, bool async) { return tiles_fit(smem) >= (async ? 4 : 5) ? 128 : 256; }

// byte offset of the tile after the barrier and the factor table of `tab` rows
int tile_off(int tab) { return (128 + tab * 36 + 127) / 128 * 128; }

// CTAs of `threads` threads and `smem` bytes resident on the device at once
int tiles_ahead(int sms, int threads, size_t smem) {
  return sms * std::max(1, std::min(768 / threads, tiles_fit(smem)));
}

template <int IO>
bool tile_attr() {
  return cudaFuncSetAttribute(cfd_tile_k<IO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem) ==
         cudaSuccess;
}

}  // namespace

bool cfd_tile_init() {
  return tile_attr<IO_ROWS_TMA>() && tile_attr<IO_ROWS>() && tile_attr<IO_LINES_BULK>() && tile_attr<IO_LINES>();
}

bool launch_cfd_tile(int axis, const CfdPlanDev &p, const float *in, float *out, int nx, int ny, int nz,
                     const CUtensorMap *tin, const CUtensorMap *tout, int sms, int *err, cudaStream_t st) {
  const int n4 = (p.n + 3) / 4 * 4;
  TileArgs a{};
  a.in = in, a.out = out, a.nz = nz, a.axis = axis, a.sms = sms;
  a.tab = p.k0 + n4 - p.k1;
  a.off = tile_off(a.tab);
  const CUtensorMap none{};
  if (axis == DZ) {
    a.nlines = (long long)nx * ny;
    // lines 4 floats (mod 32) apart: a quad load of eight lanes meets every bank once
    a.pitch = n4 + (36 - n4 % 32) % 32;
    // (a chunk read past n4 reaches up to 4 floats beyond the last line)
    auto bytes = [&](int lines) { return a.off + ((size_t)lines * a.pitch + 4) * 4; };
    for (a.lines = 32; a.lines > 1 && bytes(a.lines) > kTileSmem;) a.lines /= 2;
    const size_t smem = bytes(a.lines);
    if (smem > kTileSmem) return false;
    const unsigned grid = (unsigned)((a.nlines + a.lines - 1) / a.lines);
    const int threads = tile_threads(smem, nz % 4 == 0);
    a.ahead = tiles_ahead(sms, threads, smem);
    if (nz % 4 == 0) launch_dep(cfd_tile_k<IO_LINES_BULK>, grid, threads, smem, st, p, none, none, a, err);
    else launch_dep(cfd_tile_k<IO_LINES>, grid, threads, smem, st, p, none, none, a, err);
    return true;
  }
  const long long nxz = (long long)nx * nz;
  a.es = axis == DX ? nz : nxz, a.other = axis == DX ? nxz : nz;
  cfd_tma_box(p.n, &a.R, &a.nb);
  // (a chunk read past n4 reaches up to 4 rows beyond)
  const int rows = std::max(n4 + 4, (tin ? a.nb * a.R + 3 : 0) / 4 * 4);
  const size_t smem = a.off + (size_t)rows * 128;
  if (smem > kTileSmem) return false;
  const dim3 grid((nz + 31) / 32, axis == DX ? ny : nx);
  const int threads = tile_threads(smem, tin && tout);
  a.ahead = tiles_ahead(sms, threads, smem);
  if (tin && tout) launch_dep(cfd_tile_k<IO_ROWS_TMA>, grid, threads, smem, st, p, *tin, *tout, a, err);
  else launch_dep(cfd_tile_k<IO_ROWS>, grid, threads, smem, st, p, none, none, a, err);
  return true;
}

}  // namespace rtm
