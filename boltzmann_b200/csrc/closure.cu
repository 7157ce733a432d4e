// Learned subgrid closure (3-layer CNN on the coarse lattice) and on-device post-processing.
//
// No counterpart in the reference. The network: 3x3 convolutions 4 -> 32 -> 32 -> 1 with GELU
// (tanh form) after the first two layers, zero padding at the domain edges, channels-last
// activations.
//
//   layer   forward                       backward
//   1 (4->32)   CUDA cores (36 MAC/out)    weights: mma.sync; no input gradient
//   2 (32->32)  tcgen05 BF16, FP32 acc     data: tcgen05 (transposed conv, fused GELU');
//               (TMEM accumulators)        weights: tcgen05 (cells are the reduction axis)
//               mma.sync kept selectable (lbm_closure_set_layer2_kernel)
//   3 (32->1)   CUDA cores                 data: CUDA cores (fused GELU'); weights: mma.sync, dy
//                                          as the exact sum of three BF16 parts
//
// Every product sum takes BF16 operands (weights, activations, pre-activation gradients rounded
// to nearest even) and accumulates in FP32. Reductions over cells run per tile in a fixed order
// into per-CTA partial rows, which one kernel adds row by row: results are deterministic.
//
// Cell tiles are 4 rows (x) by 64 columns (y, the contiguous axis) unless a kernel says otherwise. Shared-memory tiles keep 40
// BF16 per cell (80 bytes): eight consecutive cells then start in eight different 16-byte bank
// groups, so ldmatrix reads them without conflicts. Weight rows (one per output channel) are
// padded from 288 to 296 BF16 (592 bytes) for the same reason.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>

#include "../../include/lbm_closure.h"
#include "device_once.h"
#include "sim.h"

namespace {

using bf16 = __nv_bfloat16;

constexpr int C = LBM_CLOSURE_CHANNELS;
constexpr int kTX = 4, kTY = 64;             // cell tile
constexpr int kHX = kTX + 2, kHY = kTY + 2;  // tile plus a one-cell halo
constexpr int kCS = 40;                      // shared-memory BF16 per cell (32 used)
constexpr int kWS = 296;                     // shared-memory BF16 per weight row (288 used)
constexpr int kPartialRows = 296;            // CTAs of the reducing kernels (2 per SM)
constexpr int kLossBlocks = 296;

int fail(int code, const std::string& msg) {
  lbm::set_last_error(msg);
  return code;
}

#define CL_CUDA(call)                                                    \
  do {                                                                   \
    cudaError_t e_ = (call);                                             \
    if (e_ != cudaSuccess)                                               \
      return fail(LBM_ERR_CUDA, std::string("CUDA error in " #call ": ") + \
                                    cudaGetErrorString(e_));             \
  } while (0)

struct Grid {
  int64_t nx, ny, batch;
  int64_t tx, ty;   // tiles along x and y
  int64_t tiles;    // all tiles of the batch
  __host__ __device__ void tile(int64_t t, int64_t& b, int64_t& x0, int64_t& y0) const {
    const int64_t per = tx * ty;
    b = t / per;
    const int64_t r = t - b * per;
    x0 = (r / ty) * kTX;
    y0 = (r % ty) * kTY;
  }
  __host__ __device__ int64_t cell(int64_t b, int64_t x, int64_t y) const {
    return (b * nx + x) * ny + y;
  }
};

// The domains of a batch in tiles of rows x cols cells.
Grid tiles_of(int64_t nx, int64_t ny, int64_t batch, int rows, int cols) {
  Grid g{nx, ny, batch, (nx + rows - 1) / rows, (ny + cols - 1) / cols, 0};
  g.tiles = g.tx * g.ty * batch;
  return g;
}
Grid make_grid(int64_t nx, int64_t ny, int64_t batch) { return tiles_of(nx, ny, batch, kTX, kTY); }

// ---------------------------------------------------------------------------------------------
// Scalar helpers

// GELU in its tanh form, 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))), written as
// z sigmoid(v) with v = z (a + b z^2), a = 2 sqrt(2/pi), b = 0.089430 sqrt(2/pi) (since
// 1 + tanh(u) = 2 sigmoid(2u)); evaluated with the fast exponential and division intrinsics
// (about 1e-6 relative, below the BF16 rounding every activation then takes). For v -> -inf the
// quotient goes to 0, as GELU does.
constexpr float kGeluA = 1.5957691216057308f;   // 2 sqrt(2/pi)
constexpr float kGeluB = 0.07135481627159709f;  // 2 sqrt(2/pi) 0.044715
__device__ __forceinline__ float gelu(float z) {
  const float v = z * fmaf(kGeluB, z * z, kGeluA);
  return __fdividef(z, 1.0f + __expf(-v));
}

// d/dz [z sigmoid(v(z))] = s (1 + z (1 - s) v'(z)), s = sigmoid(v), v' = a + 3 b z^2.
__device__ __forceinline__ float gelu_grad(float z) {
  const float z2 = z * z;
  const float v = z * fmaf(kGeluB, z2, kGeluA);
  const float sg = __fdividef(1.0f, 1.0f + __expf(-v));
  return sg * fmaf(z * (1.0f - sg), fmaf(3.0f * kGeluB, z2, kGeluA), 1.0f);
}

__device__ __forceinline__ float bf(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ bf16 to_bf(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ bool fluid_cell(int32_t flag) { return (flag & 7) == 0; }

// np.gradient along one axis (unit spacing, first-order edges): f[i+1]-f[i-1] halved inside,
// f[1]-f[0] and f[n-1]-f[n-2] at the ends.
__device__ __forceinline__ float np_gradient(float lo, float mid, float hi, int64_t i, int64_t n) {
  if (i == 0) return __fsub_rn(hi, mid);
  if (i == n - 1) return __fsub_rn(mid, lo);
  return __fmul_rn(__fsub_rn(hi, lo), 0.5f);
}

// ---------------------------------------------------------------------------------------------
// Tensor-core helpers (sm_80+ warp-level BF16 MMA, FP32 accumulate).

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const bf16* p) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const bf16* p) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// d += A * B with the running sum d kept by rounded FP32 additions. The tensor cores truncate what
// they add to, so a sum chained through them drifts with its length: over 4 M cells the gradients
// of layers 1 and 3 were 1.0e-6 and 2.4e-6 off, against 1.0e-7 and 2.6e-8 in FP32 on the CUDA
// cores. The 16 products of one instruction lose next to nothing.
__device__ __forceinline__ void mma_bf16_add(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                             uint32_t b1) {
  float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  mma_bf16(t, a, b0, b1);
  const float2 lo = __fadd2_rn(make_float2(d[0], d[1]), make_float2(t[0], t[1]));
  const float2 hi = __fadd2_rn(make_float2(d[2], d[3]), make_float2(t[2], t[3]));
  d[0] = lo.x, d[1] = lo.y, d[2] = hi.x, d[3] = hi.y;
}

// ---------------------------------------------------------------------------------------------
// Shared-memory tile loads (zero outside the domain).

// ROWS x COLS cells of a 32-channel BF16 field starting at (xs, ys), into dst[cell][kCS].
template <int ROWS, int COLS>
__device__ __forceinline__ void load_cells32(const bf16* __restrict__ src, const Grid& g,
                                             int64_t b, int64_t xs, int64_t ys, bf16* dst) {
  for (int i = threadIdx.x; i < ROWS * COLS * 4; i += blockDim.x) {
    const int chunk = i & 3, cell = i >> 2;
    const int r = cell / COLS, c = cell - r * COLS;
    const int64_t x = xs + r, y = ys + c;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (x >= 0 && x < g.nx && y >= 0 && y < g.ny)
      v = __ldg(reinterpret_cast<const uint4*>(src + g.cell(b, x, y) * C) + chunk);
    *reinterpret_cast<uint4*>(dst + cell * kCS + chunk * 8) = v;
  }
}

// A 16-byte asynchronous copy into shared memory, zeros when !valid (src is then not read).
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// load_cells32 by asynchronous copies (the caller commits and waits).
template <int ROWS, int COLS>
__device__ __forceinline__ void load_cells32_async(const bf16* __restrict__ src, const Grid& g,
                                                   int64_t b, int64_t xs, int64_t ys, bf16* dst) {
  for (int i = threadIdx.x; i < ROWS * COLS * 4; i += blockDim.x) {
    const int chunk = i & 3, cell = i >> 2;
    const int r = cell / COLS, c = cell - r * COLS;
    const int64_t x = xs + r, y = ys + c;
    const bool in = x >= 0 && x < g.nx && y >= 0 && y < g.ny;
    cp_async16(dst + cell * kCS + chunk * 8, in ? src + g.cell(b, x, y) * C + chunk * 8 : src, in);
  }
}

// A tile's 4-channel features with the halo in registers (zero outside the domain): loaded a tile
// ahead, then handed cell by cell (index in the kHX x kHY region) to `f`.
template <int THREADS>
struct FeatureTile {
  static constexpr int N = (kHX * kHY + THREADS - 1) / THREADS;
  uint2 v[N];
  __device__ __forceinline__ void load(const bf16* __restrict__ src, const Grid& g, int64_t t) {
    int64_t b, x0, y0;
    g.tile(t, b, x0, y0);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int i = threadIdx.x + k * THREADS;
      const int r = i / kHY, c = i - r * kHY;
      const int64_t x = x0 - 1 + r, y = y0 - 1 + c;
      v[k] = make_uint2(0, 0);
      if (i < kHX * kHY && x >= 0 && x < g.nx && y >= 0 && y < g.ny)
        v[k] = __ldg(reinterpret_cast<const uint2*>(src + g.cell(b, x, y) * 4));
    }
  }
  template <class F>
  __device__ __forceinline__ void each(F f) const {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int i = threadIdx.x + k * THREADS;
      if (i < kHX * kHY) f(i, v[k]);
    }
  }
};

// Two FP32 fused multiply-adds on one packed instruction, each rounded as fmaf.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// gelu of two values, its multiplications and additions on packed instructions (the same bits).
__device__ __forceinline__ float2 gelu2(float2 z) {
  const float2 zz = __fmul2_rn(z, z);
  const float2 v = __fmul2_rn(z, ffma2(make_float2(kGeluB, kGeluB), zz, make_float2(kGeluA, kGeluA)));
  const float2 d = __fadd2_rn(make_float2(1.0f, 1.0f), make_float2(__expf(-v.x), __expf(-v.y)));
  return make_float2(__fdividef(z.x, d.x), __fdividef(z.y, d.y));
}

// gelu_grad of two values, likewise.
__device__ __forceinline__ float2 gelu_grad2(float2 z) {
  const float2 one = make_float2(1.0f, 1.0f), a = make_float2(kGeluA, kGeluA);
  const float2 z2 = __fmul2_rn(z, z);
  const float2 v = __fmul2_rn(z, ffma2(make_float2(kGeluB, kGeluB), z2, a));
  const float2 d = __fadd2_rn(one, make_float2(__expf(-v.x), __expf(-v.y)));
  const float2 sg = make_float2(__fdividef(1.0f, d.x), __fdividef(1.0f, d.y));
  const float2 rest = __fadd2_rn(one, make_float2(-sg.x, -sg.y));
  const float2 slope = ffma2(make_float2(3.0f * kGeluB, 3.0f * kGeluB), z2, a);
  return __fmul2_rn(sg, ffma2(__fmul2_rn(z, rest), slope, one));
}

__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t pack_bf2(float2 v) { return pack_bf2(v.x, v.y); }
__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// The element-wise kernels of layers 1 and 3 give a cell to two neighbouring lanes (g2 = lane & 1),
// 16 channels each in four groups of four: channels 8 k + 4 g2 .. + 3, k = 0 .. 3. FP32 rows then
// move as full 32-byte sectors (two lanes x 16 bytes), and after a swap between the two lanes the
// BF16 rows too: `w` holds the lane's packed groups; afterwards lane g2 = 0 has channels 0-7 and
// 16-23, lane 1 channels 8-15 and 24-31, which it stores at 16-byte chunks g2 and g2 + 2.
__device__ __forceinline__ void store_bf16_row(bf16* row, uint32_t (&w)[4][2], int g2, bool valid) {
#pragma unroll
  for (int k = 0; k < 4; k += 2) {
    const uint32_t s0 = g2 ? w[k][0] : w[k + 1][0], s1 = g2 ? w[k][1] : w[k + 1][1];
    const uint32_t r0 = __shfl_xor_sync(0xffffffffu, s0, 1);
    const uint32_t r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
    const uint4 v = g2 ? make_uint4(r0, r1, w[k + 1][0], w[k + 1][1])
                       : make_uint4(w[k][0], w[k][1], r0, r1);
    if (valid) reinterpret_cast<uint4*>(row)[k + g2] = v;
  }
}

// Layer-2 weights [32 out][288] into rows of kWS.
__device__ __forceinline__ void load_w2(const bf16* __restrict__ w2, bf16* ws) {
  for (int i = threadIdx.x; i < C * 36; i += blockDim.x) {
    const int co = i / 36, ch = i - co * 36;
    *reinterpret_cast<uint4*>(ws + co * kWS + ch * 8) =
        __ldg(reinterpret_cast<const uint4*>(w2 + co * 288) + ch);
  }
}

// ---------------------------------------------------------------------------------------------
// Post-processing and features

__global__ void curl2d_kernel(const float* __restrict__ vel, int64_t nx, int64_t ny,
                              float* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nx * ny) return;
  const int64_t x = i / ny, y = i - x * ny;
  const int64_t xm = x > 0 ? x - 1 : x, xp = x < nx - 1 ? x + 1 : x;
  const int64_t ym = y > 0 ? y - 1 : y, yp = y < ny - 1 ? y + 1 : y;
  const float dux_dy = np_gradient(vel[(x * ny + ym) * 2], vel[i * 2], vel[(x * ny + yp) * 2], y, ny);
  const float duy_dx =
      np_gradient(vel[(xm * ny + y) * 2 + 1], vel[i * 2 + 1], vel[(xp * ny + y) * 2 + 1], x, nx);
  out[i] = __fsub_rn(dux_dy, duy_dx);
}

__global__ void curl3d_kernel(const float* __restrict__ vel, int64_t nx, int64_t ny, int64_t nz,
                              float* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nx * ny * nz) return;
  const int64_t x = i / (ny * nz), y = (i / nz) % ny, z = i % nz;
  const int64_t pos[3] = {x, y, z}, len[3] = {nx, ny, nz}, stride[3] = {ny * nz, nz, 1};
  float d[3][3];  // d[axis][component]
  for (int a = 0; a < 3; ++a) {
    const int64_t lo = pos[a] > 0 ? i - stride[a] : i;
    const int64_t hi = pos[a] < len[a] - 1 ? i + stride[a] : i;
    for (int c = 0; c < 3; ++c)
      d[a][c] = np_gradient(vel[lo * 3 + c], vel[i * 3 + c], vel[hi * 3 + c], pos[a], len[a]);
  }
  out[i * 3 + 0] = __fsub_rn(d[2][1], d[1][2]);
  out[i * 3 + 1] = __fsub_rn(d[0][2], d[2][0]);
  out[i * 3 + 2] = __fsub_rn(d[1][0], d[0][1]);
}

__global__ void vmag_kernel(const float* __restrict__ vel, int64_t n, int dim,
                            float* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = __fmul_rn(vel[i * dim], vel[i * dim]);
  for (int c = 1; c < dim; ++c) s = __fadd_rn(s, __fmul_rn(vel[i * dim + c], vel[i * dim + c]));
  out[i] = sqrtf(s);
}

struct Norm {
  float mean[4], inv_std[4];
};

// Velocity read for the closure's curl: walls count as the no-slip value 0.
__device__ __forceinline__ float vel_or_wall(const float* vel, const int32_t* flags, int64_t b,
                                             int64_t n, int64_t cell, int c) {
  return (flags[cell] & 1) ? 0.0f : vel[(b * n + cell) * 2 + c];
}

// The four BF16 features of cell (x, y) of batch entry b, packed in two words (0 on walls).
__device__ __forceinline__ uint2 cell_features(const float* __restrict__ rho,
                                               const float* __restrict__ vel,
                                               const int32_t* __restrict__ flags, int64_t nx,
                                               int64_t ny, int64_t b, int64_t x, int64_t y,
                                               const Norm& norm) {
  const int64_t n = nx * ny;
  const int64_t cell = x * ny + y, i = b * n + cell;
  uint2 packed = make_uint2(0, 0);
  if (!(flags[cell] & 1)) {
    const int64_t xm = x > 0 ? x - 1 : x, xp = x < nx - 1 ? x + 1 : x;
    const int64_t ym = y > 0 ? y - 1 : y, yp = y < ny - 1 ? y + 1 : y;
    const float dux_dy =
        np_gradient(vel_or_wall(vel, flags, b, n, x * ny + ym, 0), vel[i * 2],
                    vel_or_wall(vel, flags, b, n, x * ny + yp, 0), y, ny);
    const float duy_dx =
        np_gradient(vel_or_wall(vel, flags, b, n, xm * ny + y, 1), vel[i * 2 + 1],
                    vel_or_wall(vel, flags, b, n, xp * ny + y, 1), x, nx);
    const float v[4] = {__fsub_rn(rho[i], 1.0f), vel[i * 2], vel[i * 2 + 1],
                        __fsub_rn(dux_dy, duy_dx)};
    bf16 h[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) h[c] = to_bf(__fmul_rn(__fsub_rn(v[c], norm.mean[c]), norm.inv_std[c]));
    packed.x = (uint32_t)__bfloat16_as_ushort(h[0]) | ((uint32_t)__bfloat16_as_ushort(h[1]) << 16);
    packed.y = (uint32_t)__bfloat16_as_ushort(h[2]) | ((uint32_t)__bfloat16_as_ushort(h[3]) << 16);
  }
  return packed;
}

__global__ void features_kernel(const float* __restrict__ rho, const float* __restrict__ vel,
                                const int32_t* __restrict__ flags, int64_t nx, int64_t ny,
                                int64_t batch, Norm norm, bf16* __restrict__ x_out) {
  const int64_t n = nx * ny;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * batch) return;
  const int64_t b = i / n, cell = i - b * n;
  const int64_t x = cell / ny, y = cell - x * ny;
  reinterpret_cast<uint2*>(x_out)[i] = cell_features(rho, vel, flags, nx, ny, b, x, y, norm);
}

// ---------------------------------------------------------------------------------------------
// Layer 1 forward (CUDA cores): 36 MACs per output, in FP32 on packed instructions (two channels
// each). Bound by the FMA pipe (1152 a cell) beside 200 bytes a cell of traffic. A warp takes one row
// of the tile, two lanes a cell (store_bf16_row) and four cells a lane, so that each shared-memory
// weight load feeds eight FMAs; the inputs lie in shared memory as (v, v) pairs, the packed
// instruction's operand. Batch 8 x 1024 x 512: 635 -> 327 us (336 with the taps not unrolled).

constexpr int kC1Threads = 32 * kTX;
constexpr int kC1Cells = kTY / 16;  // cells a lane
constexpr int kC1PerSm = 3;

__global__ void __launch_bounds__(kC1Threads, kC1PerSm)
    conv1_fwd_kernel(Grid g, const bf16* __restrict__ x, const bf16* __restrict__ w1,
                     const float* __restrict__ b1, float* __restrict__ z1, bf16* __restrict__ a1) {
  __shared__ __align__(16) float xs[kHX * kHY * 8];  // [cell][ci] as (v, v)
  __shared__ __align__(16) float ws[9 * 4 * C];      // [tap][ci][co]
  for (int i = threadIdx.x; i < 9 * 4 * C; i += blockDim.x) {
    const int co = i / 36, r = i - co * 36;  // w1 is [co][tap][ci]
    ws[r * C + co] = bf(w1[i]);
  }
  const int ti = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g2 = lane & 1, lc = lane >> 1;
  float4 bias[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float* b = b1 + 8 * k + 4 * g2;
    bias[k] = make_float4(b[0], b[1], b[2], b[3]);
  }
  FeatureTile<kC1Threads> in;  // the next tile's features, loaded while this one is computed
  if ((int64_t)blockIdx.x < g.tiles) in.load(x, g, blockIdx.x);
  for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x) {
    int64_t b, x0, y0;
    g.tile(t, b, x0, y0);
    __syncthreads();
    in.each([&](int i, uint2 v) {
      float4* d = reinterpret_cast<float4*>(xs + i * 8);
      d[0] = make_float4(bf_lo(v.x), bf_lo(v.x), bf_hi(v.x), bf_hi(v.x));
      d[1] = make_float4(bf_lo(v.y), bf_lo(v.y), bf_hi(v.y), bf_hi(v.y));
    });
    __syncthreads();
    if (t + gridDim.x < g.tiles) in.load(x, g, t + gridDim.x);
    float2 acc[kC1Cells][8];
#pragma unroll
    for (int p = 0; p < kC1Cells; ++p)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[p][q] = make_float2(0.0f, 0.0f);
#pragma unroll 3
    for (int tap = 0; tap < 9; ++tap) {
      const int dx = tap / 3 - 1, dy = tap % 3 - 1;
      const float* xc = xs + ((ti + 1 + dx) * kHY + lc + 1 + dy) * 8;
      const float* wt = ws + tap * 4 * C + 4 * g2;
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // input channels 2 h, 2 h + 1
        float4 v[kC1Cells];
#pragma unroll
        for (int p = 0; p < kC1Cells; ++p)
          v[p] = *reinterpret_cast<const float4*>(xc + p * 16 * 8 + 4 * h);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 w = *reinterpret_cast<const float4*>(wt + (2 * h + e) * C + 8 * k);
#pragma unroll
            for (int p = 0; p < kC1Cells; ++p) {
              const float2 vv = e ? make_float2(v[p].z, v[p].w) : make_float2(v[p].x, v[p].y);
              acc[p][2 * k] = ffma2(vv, make_float2(w.x, w.y), acc[p][2 * k]);
              acc[p][2 * k + 1] = ffma2(vv, make_float2(w.z, w.w), acc[p][2 * k + 1]);
            }
          }
        }
      }
    }
    const int64_t xx = x0 + ti;
#pragma unroll
    for (int p = 0; p < kC1Cells; ++p) {
      const int64_t yy = y0 + lc + 16 * p;
      const bool valid = xx < g.nx && yy < g.ny;
      const int64_t cell = valid ? g.cell(b, xx, yy) : 0;
      uint32_t w[4][2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 z = make_float4(acc[p][2 * k].x + bias[k].x, acc[p][2 * k].y + bias[k].y,
                                     acc[p][2 * k + 1].x + bias[k].z, acc[p][2 * k + 1].y + bias[k].w);
        if (z1 != nullptr && valid) *reinterpret_cast<float4*>(z1 + cell * C + 8 * k + 4 * g2) = z;
        w[k][0] = pack_bf2(gelu2(make_float2(z.x, z.y)));
        w[k][1] = pack_bf2(gelu2(make_float2(z.z, z.w)));
      }
      store_bf16_row(a1 + cell * C, w, g2, valid);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Layer 2 on tensor cores: forward conv (BWD = false) or the transposed conv of the backward
// pass (BWD = true), as an implicit GEMM per tile: M = 64 cells of one row per warp (4 m-tiles
// of 16), N = 32 channels (4 n-tiles of 8), K = 9 taps x 32 channels (18 k-steps of 16).
//
// Forward:  z[p][co] = b[co] + sum_{tap,ci} W[co][tap][ci] a[p + tap][ci];  a2 = GELU(z) (BF16)
// Backward: d[q][ci] = sum_{tap,co} W[co][tap][ci] dz[q - tap][co];  dz1 = d GELU'(z1) (BF16).

constexpr int kConv32Threads = 128;
constexpr size_t kConv32Smem = (size_t)(kHX * kHY * kCS + C * kWS) * sizeof(bf16);

template <bool BWD>
__global__ void __launch_bounds__(kConv32Threads)
    conv32_kernel(Grid g, const bf16* __restrict__ in, const bf16* __restrict__ w2,
                  const float* __restrict__ bias, const float* __restrict__ zin,
                  float* __restrict__ zout, bf16* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* ins = reinterpret_cast<bf16*>(smem_raw);
  bf16* wsm = ins + kHX * kHY * kCS;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  load_w2(w2, wsm);

  for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x) {
    int64_t b, x0, y0;
    g.tile(t, b, x0, y0);
    __syncthreads();
    load_cells32<kHX, kHY>(in, g, b, x0 - 1, y0 - 1, ins);
    __syncthreads();

    float acc[4][4][4];
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[mt][nt][e] = 0.0f;

    const int mi = lane >> 3, rr = lane & 7;
#pragma unroll 1
    for (int tap = 0; tap < 9; ++tap) {
      const int dx = tap / 3 - 1, dy = tap % 3 - 1;
      const int sx = BWD ? -dx : dx, sy = BWD ? -dy : dy;
#pragma unroll
      for (int kc = 0; kc < 2; ++kc) {
        uint32_t bfrag[4][2];
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t r[4];
          if (!BWD) {
            const int co = (2 * np + (mi >> 1)) * 8 + rr;
            ldsm_x4(r, wsm + co * kWS + tap * 32 + kc * 16 + (mi & 1) * 8);
          } else {
            const int co = kc * 16 + (mi & 1) * 8 + rr;
            ldsm_x4_t(r, wsm + co * kWS + tap * 32 + (2 * np + (mi >> 1)) * 8);
          }
          bfrag[2 * np][0] = r[0];
          bfrag[2 * np][1] = r[1];
          bfrag[2 * np + 1][0] = r[2];
          bfrag[2 * np + 1][1] = r[3];
        }
        const int row = warp + 1 + sx;
        const int j = (lane & 7) + 8 * ((lane >> 3) & 1);
        const int koff = kc * 16 + 8 * (lane >> 4);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
          uint32_t a[4];
          ldsm_x4(a, ins + (row * kHY + mt * 16 + j + 1 + sy) * kCS + koff);
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) mma_bf16(acc[mt][nt], a, bfrag[nt][0], bfrag[nt][1]);
        }
      }
    }

    // Epilogue: thread holds cells (gq, gq + 8) of each m-tile, channels nt*8 + 2tq (+1).
    const int64_t xx = x0 + warp;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t yy = y0 + mt * 16 + gq + 8 * h;
        if (xx >= g.nx || yy >= g.ny) continue;
        const int64_t cell = g.cell(b, xx, yy);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const int ch = nt * 8 + 2 * tq;
          const float v0 = acc[mt][nt][2 * h], v1 = acc[mt][nt][2 * h + 1];
          __nv_bfloat162 o;
          if (!BWD) {
            const float z0 = v0 + bias[ch], z1v = v1 + bias[ch + 1];
            if (zout != nullptr)
              *reinterpret_cast<float2*>(zout + cell * C + ch) = make_float2(z0, z1v);
            o.x = to_bf(gelu(z0));
            o.y = to_bf(gelu(z1v));
          } else {
            const float2 z = *reinterpret_cast<const float2*>(zin + cell * C + ch);
            o.x = to_bf(v0 * gelu_grad(z.x));
            o.y = to_bf(v1 * gelu_grad(z.y));
          }
          *reinterpret_cast<__nv_bfloat162*>(out + cell * C + ch) = o;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Layer-2 weight gradient on tensor cores: dW[co][tap][ci] = sum_p dz[p][co] a1[p + tap][ci].
// M = 32 output channels (2 m-tiles), N = 32 input channels (4 n-tiles), K = the cells of the CTA's
// tiles, 16 per k-step. Warp (i, dx) takes tile row i and the three taps (dx, -1 .. 1): the dz
// fragments it loads serve 24 MMAs (one warp a tap loaded them for eight). The next tile's operands
// arrive (asynchronous copies) while this one's are multiplied. Bound by shared-memory reads (eight
// ldmatrix a 24 MMAs). Batch 8 x 1024 x 512: 366 -> 311 us. Runs with the warp-level layer-2 kernels,
// and where conv32_wgrad_tc_kernel (111 us) has no tensor map.

constexpr int kDw2Threads = 3 * kTX * 32;
constexpr int kDw2Stage = (kTX * kTY + kHX * kHY) * kCS;  // BF16 elements of one stage
constexpr size_t kDw2Smem = (size_t)2 * kDw2Stage * sizeof(bf16);
static_assert((size_t)C * 288 * 4 <= kDw2Smem, "the cross-row sums must fit the stages");

__global__ void __launch_bounds__(kDw2Threads, 1)
    conv32_wgrad_kernel(Grid g, const bf16* __restrict__ a1, const bf16* __restrict__ dz2,
                        float* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* stages = reinterpret_cast<bf16*>(smem_raw);  // [2][dz [kTX * kTY][kCS], a1 [kHX * kHY][kCS]]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dx = warp % 3 - 1, row = warp / 3;
  const int mi = lane >> 3, rr = lane & 7;

  float acc[3][2][4][4];
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[d][mt][nt][e] = 0.0f;

  auto fetch = [&](int64_t t, int s) {
    int64_t b, x0, y0;
    g.tile(t, b, x0, y0);
    bf16* st = stages + s * kDw2Stage;
    load_cells32_async<kTX, kTY>(dz2, g, b, x0, y0, st);
    load_cells32_async<kHX, kHY>(a1, g, b, x0 - 1, y0 - 1, st + kTX * kTY * kCS);
  };
  int s = 0;
  if ((int64_t)blockIdx.x < g.tiles) fetch(blockIdx.x, 0);
  cp_async_commit();
  for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, s ^= 1) {
    if (t + gridDim.x < g.tiles) fetch(t + gridDim.x, s ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const bf16* dzs = stages + s * kDw2Stage;
    const bf16* as = dzs + kTX * kTY * kCS;
#pragma unroll 1
    for (int c = 0; c < kTY / 16; ++c) {
      const int k0 = c * 16 + (mi >> 1) * 8 + rr, k1 = c * 16 + (mi & 1) * 8 + rr;
      uint32_t afrag[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
        ldsm_x4_t(afrag[mt], dzs + (row * kTY + k0) * kCS + mt * 16 + (mi & 1) * 8);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const bf16* ap = as + ((row + 1 + dx) * kHY + k1 + d) * kCS + (mi >> 1) * 8;
        uint32_t bfrag[4][2];
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t r[4];
          ldsm_x4_t(r, ap + np * 16);
          bfrag[2 * np][0] = r[0];
          bfrag[2 * np][1] = r[1];
          bfrag[2 * np + 1][0] = r[2];
          bfrag[2 * np + 1][1] = r[3];
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
            mma_bf16(acc[d][mt][nt], afrag[mt], bfrag[nt][0], bfrag[nt][1]);
      }
    }
    __syncthreads();  // stage s is free for the tile after the next
  }
  cp_async_wait<0>();
  __syncthreads();

  // The four tile rows' sums, added in row order, then this CTA's partial row.
  float* sums = reinterpret_cast<float*>(smem_raw);  // [co][288]
  const int gq = lane >> 2, tq = lane & 3;
  for (int r = 0; r < kTX; ++r) {
    if (row == r) {
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int co = mt * 16 + gq + 8 * h, ci = nt * 8 + 2 * tq;
              float2* p = reinterpret_cast<float2*>(sums + co * 288 + ((dx + 1) * 3 + d) * 32 + ci);
              float2 v = make_float2(acc[d][mt][nt][2 * h], acc[d][mt][nt][2 * h + 1]);
              if (r > 0) {
                const float2 o = *p;
                v = make_float2(o.x + v.x, o.y + v.y);
              }
              *p = v;
            }
    }
    __syncthreads();
  }
  float* out = partial + (int64_t)blockIdx.x * LBM_CLOSURE_PARAMS + LBM_CLOSURE_OFF_W2;
  for (int i = threadIdx.x; i < C * 288; i += blockDim.x) out[i] = sums[i];
}

// ---------------------------------------------------------------------------------------------
// Layer 3 (32 -> 1) forward: y[p] = b3 + sum_{tap,ci} w3[tap][ci] a2[p + tap][ci], as one product per
// cell, P[q][tap] = sum_ci w3[tap][ci] a2[q][ci], whose nine shifted values each output adds: every
// activation is read and widened once instead of nine times. FP32 on packed instructions (two
// channels each): tensor cores would do it for less, but their accumulation leans to one side, and
// the loss, an average over all cells, shows it. Two cells a thread, in three passes, so that each
// shared-memory weight load feeds four of them; on small batches in one pass on lower tiles (conv3_low).
// Batch 8 x 1024 x 512: 216 -> 118 us.

constexpr int kC3R = 30, kC3Low = 6;         // output rows of a tile (kTY columns)
constexpr int kC3RegC = kHY;                 // columns of the region with the halo
constexpr int kC3Per = 2, kC3Threads = 352;  // cells a thread takes in a pass
template <int R>
constexpr int kC3Cells = (R + 2) * kC3RegC;  // 2112 in three passes, 528 in one
template <int R>
constexpr size_t kConv3Smem = (size_t)9 * kC3Cells<R> * 4 + (size_t)9 * C * 4;

template <int R>
__global__ void __launch_bounds__(kC3Threads, 2)
    conv3_fwd_kernel(Grid g, const bf16* __restrict__ a2, const bf16* __restrict__ w3,
                     const float* __restrict__ b3, float* __restrict__ y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kCells = kC3Cells<R>;
  constexpr bool kWhole = kCells % (kC3Threads * kC3Per) == 0;  // no cell short in the last pass
  float* ps = reinterpret_cast<float*>(smem_raw);  // [9][kCells]
  float* ws = ps + 9 * kCells;                   // [tap][ci]
  for (int i = threadIdx.x; i < 9 * C; i += blockDim.x) ws[i] = bf(w3[i]);
  const float bias = b3[0];
  for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x) {
    int64_t b, x0, y0;
    {
      const int64_t per = g.tx * g.ty;  // this kernel's tiles are R x kTY (see the launcher)
      b = t / per;
      const int64_t r = t - b * per;
      x0 = (r / g.ty) * R;
      y0 = (r % g.ty) * kTY;
    }
    __syncthreads();  // the previous tile's P has been read (and, at first, ws written)
#pragma unroll 1
    for (int q0 = threadIdx.x; q0 < kCells; q0 += kC3Per * kC3Threads) {
      uint4 v[kC3Per][C / 8];
#pragma unroll
      for (int p = 0; p < kC3Per; ++p) {
        const int q = q0 + p * kC3Threads;
        const int r = q / kC3RegC, c = q - r * kC3RegC;
        const int64_t x = x0 - 1 + r, yy = y0 - 1 + c;
        const bool in = (kWhole || q < kCells) && x >= 0 && x < g.nx && yy >= 0 && yy < g.ny;
        const uint4* src = reinterpret_cast<const uint4*>(a2 + (in ? g.cell(b, x, yy) : 0) * C);
#pragma unroll
        for (int k = 0; k < C / 8; ++k) v[p][k] = in ? __ldg(src + k) : make_uint4(0, 0, 0, 0);
      }
      float2 acc[kC3Per][9];
#pragma unroll
      for (int p = 0; p < kC3Per; ++p)
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) acc[p][tap] = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int k = 0; k < C / 8; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float2 a[kC3Per][2];
#pragma unroll
          for (int p = 0; p < kC3Per; ++p) {
            const uint32_t u0 = h ? v[p][k].z : v[p][k].x, u1 = h ? v[p][k].w : v[p][k].y;
            a[p][0] = make_float2(bf_lo(u0), bf_hi(u0));
            a[p][1] = make_float2(bf_lo(u1), bf_hi(u1));
          }
#pragma unroll
          for (int tap = 0; tap < 9; ++tap) {
            const float4 w = *reinterpret_cast<const float4*>(ws + tap * C + k * 8 + 4 * h);
#pragma unroll
            for (int p = 0; p < kC3Per; ++p) {
              acc[p][tap] = ffma2(a[p][0], make_float2(w.x, w.y), acc[p][tap]);
              acc[p][tap] = ffma2(a[p][1], make_float2(w.z, w.w), acc[p][tap]);
            }
          }
        }
#pragma unroll
      for (int p = 0; p < kC3Per; ++p)
#pragma unroll
        for (int tap = 0; tap < 9; ++tap)
          if (kWhole || q0 + p * kC3Threads < kCells)
            ps[tap * kCells + q0 + p * kC3Threads] = acc[p][tap].x + acc[p][tap].y;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < R * kTY; i += kC3Threads) {
      const int r = i / kTY, c = i - r * kTY;
      const int64_t x = x0 + r, yy = y0 + c;
      if (x >= g.nx || yy >= g.ny) continue;
      float s = 0.0f;
#pragma unroll
      for (int tap = 0; tap < 9; ++tap)
        s += ps[tap * kCells + (r + tap / 3) * kC3RegC + c + tap % 3];
      y[g.cell(b, x, yy)] = s + bias;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Layer 3 backward. Per tile:
//   dz2[q][ci] = BF16( GELU'(z2[q][ci]) sum_tap w3[tap][ci] dy[q - tap] )
//   dW3[tap][ci] += sum_q a2[q][ci] dy[q - tap],  db3 += sum_q dy[q],  db2[ci] += sum_q dz2[q][ci]
// The first line in FP32 on packed instructions, two lanes a cell (store_bf16_row) and two cells a
// lane. The weight gradient on tensor cores: M = (part, tap), N = ci, K = cells, where dy enters as
// the exact sum of three BF16 parts (8 + 8 + 8 significant bits), so that every product is that of
// the FP32 value; the parts' sums are added at the end. (One thread an output over the tile's 256
// cells was the kernel's longest part by far.) Bound by 260 bytes a cell. Batch 8 x 1024 x 512: 978 -> 325 us.

constexpr int kB3Threads = 256;
constexpr int kDyS = kHY + 2;  // BF16 elements of a row of a dy part (a multiple of 2)
// A stage holds the tile's a2 [cell][kCS] and z2 [cell][C], whose 16-byte chunk c of cell p lies at
// chunk c ^ 2 (p % 4): four cells' chunks, which a quarter warp reads at once, in different banks.
constexpr size_t kB3OffZ = (size_t)kTX * kTY * kCS * 2;
constexpr size_t kB3Stage = kB3OffZ + (size_t)kTX * kTY * C * 4;
constexpr size_t kB3OffDy2 = 2 * kB3Stage;                             // dy as (v, v) pairs
constexpr size_t kB3OffPart = kB3OffDy2 + (size_t)kHX * kHY * 8;       // [part][shift][kHX][kDyS]
constexpr size_t kB3OffW = kB3OffPart + (size_t)3 * 2 * kHX * kDyS * 2;
constexpr size_t kConv3BwdSmem = kB3OffW + (size_t)9 * C * 4;
static_assert(kB3OffPart % 16 == 0 && kB3OffW % 16 == 0, "aligned parts");
constexpr int kB3Sums = 27 * C + C + 1;  // a warp's sums at the end: dW3 parts, db2, db3
static_assert((size_t)(kB3Threads / 32) * kB3Sums * 4 <= kConv3BwdSmem, "the sums must fit");

__global__ void __launch_bounds__(kB3Threads, 2)
    conv3_bwd_kernel(Grid g, const bf16* __restrict__ a2, const float* __restrict__ z2,
                     const bf16* __restrict__ w3, const float* __restrict__ dy,
                     bf16* __restrict__ dz2, float* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* dy2 = reinterpret_cast<float2*>(smem_raw + kB3OffDy2);     // [kHX * kHY]
  bf16* dyp = reinterpret_cast<bf16*>(smem_raw + kB3OffPart);
  float* ws = reinterpret_cast<float*>(smem_raw + kB3OffW);          // [tap][ci]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g2 = lane & 1, lc = lane >> 1, gq = lane >> 2, tq = lane & 3;
  const int mi = lane >> 3, rr = lane & 7;
  const int ti = warp >> 1, tj = (warp & 1) * 32;  // this warp's 32 cells: row ti, columns tj ..
  for (int i = threadIdx.x; i < 9 * C; i += blockDim.x) ws[i] = bf(w3[i]);
  for (int i = threadIdx.x; i < 3 * 2 * kHX * kDyS; i += blockDim.x) dyp[i] = to_bf(0.0f);

  // A fragments of the weight gradient: rows m = gq, gq + 8 of the two m-tiles, m = 9 part + tap
  // (rows 27 .. 31: none). Element k of row m is dy part `part` at column j - dyy + 1 (with the
  // halo) of tile row ti - dx + 1; pairs (k, k + 1) at an odd column come from the copy that is
  // shifted by one element.
  int aoff[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int m = gq + 8 * e;
    aoff[e] = -1;
    if (m < 27) {
      const int part = m / 9, tap = m % 9;
      const int col = tj + 1 - (tap % 3 - 1), r = ti + 1 - (tap / 3 - 1), odd = col & 1;
      aoff[e] = ((part * 2 + odd) * kHX + r) * kDyS + col - odd + 2 * tq;
    }
  }
  float acc[2][4][4];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[mt][nt][e] = 0.0f;
  float bsum[16];  // db2 of this lane's channels 8 k + 4 g2 + e
#pragma unroll
  for (int k = 0; k < 16; ++k) bsum[k] = 0.0f;
  float dsum = 0.0f;  // db3

  // The next tile's operands are in flight while this one is computed: a2 and z2 by asynchronous
  // copies, dy in registers.
  constexpr int kDyN = (kHX * kHY + kB3Threads - 1) / kB3Threads;
  float dyv[kDyN];
  auto fetch = [&](int64_t t, int s) {
    int64_t b, x0, y0;
    g.tile(t, b, x0, y0);
    unsigned char* st = smem_raw + (size_t)s * kB3Stage;
    load_cells32_async<kTX, kTY>(a2, g, b, x0, y0, reinterpret_cast<bf16*>(st));
    for (int i = threadIdx.x; i < kTX * kTY * 8; i += kB3Threads) {
      const int chunk = i & 7, p = i >> 3;
      const int64_t x = x0 + p / kTY, yv = y0 + p % kTY;
      const bool in = x < g.nx && yv < g.ny;
      cp_async16(st + kB3OffZ + p * 128 + ((chunk ^ (2 * (p & 3))) * 16),
                 in ? z2 + g.cell(b, x, yv) * C + chunk * 4 : z2, in);
    }
#pragma unroll
    for (int k = 0; k < kDyN; ++k) {
      const int i = threadIdx.x + k * kB3Threads;
      const int r = i / kHY, c = i - r * kHY;
      const int64_t x = x0 - 1 + r, yv = y0 - 1 + c;
      dyv[k] = (i < kHX * kHY && x >= 0 && x < g.nx && yv >= 0 && yv < g.ny)
                   ? dy[g.cell(b, x, yv)]
                   : 0.0f;
    }
  };
  int stage = 0;
  if ((int64_t)blockIdx.x < g.tiles) fetch(blockIdx.x, 0);
  cp_async_commit();
  for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, stage ^= 1) {
    int64_t b, x0, y0;
    g.tile(t, b, x0, y0);
    __syncthreads();  // the previous tile is done with dy2, dyp and its stage
    const bf16* as = reinterpret_cast<const bf16*>(smem_raw + (size_t)stage * kB3Stage);
    const unsigned char* zs = smem_raw + (size_t)stage * kB3Stage + kB3OffZ;
#pragma unroll
    for (int k3 = 0; k3 < kDyN; ++k3) {
      const int i = threadIdx.x + k3 * kB3Threads;
      if (i >= kHX * kHY) break;
      const int r = i / kHY, c = i - r * kHY;
      const float v = dyv[k3];
      dy2[i] = make_float2(v, v);
      // v = h + m + l exactly (a non-finite v stays in h)
      const bool fin = fabsf(v) <= 3.0e38f;
      const bf16 h = to_bf(v);
      const float vm = fin ? __fsub_rn(v, bf(h)) : 0.0f;
      const bf16 m = to_bf(vm);
      const bf16 l = to_bf(__fsub_rn(vm, bf(m)));
      const bf16 part[3] = {h, m, l};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        dyp[((k * 2) * kHX + r) * kDyS + c] = part[k];
        if (c > 0) dyp[((k * 2 + 1) * kHX + r) * kDyS + c - 1] = part[k];
      }
    }
    if (t + gridDim.x < g.tiles) fetch(t + gridDim.x, stage ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();

    const int64_t xx = x0 + ti;
    float2 d[2][8];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = 0; q < 8; ++q) d[p][q] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const int dx = tap / 3 - 1, dyy = tap % 3 - 1;
      const float2* vp = dy2 + (ti + 1 - dx) * kHY + tj + lc + 1 - dyy;
      const float2 v0 = vp[0], v1 = vp[16];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 w = *reinterpret_cast<const float4*>(ws + tap * C + 8 * k + 4 * g2);
        d[0][2 * k] = ffma2(make_float2(w.x, w.y), v0, d[0][2 * k]);
        d[0][2 * k + 1] = ffma2(make_float2(w.z, w.w), v0, d[0][2 * k + 1]);
        d[1][2 * k] = ffma2(make_float2(w.x, w.y), v1, d[1][2 * k]);
        d[1][2 * k + 1] = ffma2(make_float2(w.z, w.w), v1, d[1][2 * k + 1]);
      }
    }
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int64_t yy = y0 + tj + lc + 16 * p;
      const bool valid = xx < g.nx && yy < g.ny;
      const int64_t cell = valid ? g.cell(b, xx, yy) : 0;
      uint32_t w[4][2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int q = ti * kTY + tj + lc + 16 * p;
        const float4 z = *reinterpret_cast<const float4*>(
            zs + q * 128 + (((2 * k + g2) ^ (2 * (q & 3))) * 16));
        w[k][0] = pack_bf2(d[p][2 * k].x * gelu_grad(z.x), d[p][2 * k].y * gelu_grad(z.y));
        w[k][1] = pack_bf2(d[p][2 * k + 1].x * gelu_grad(z.z), d[p][2 * k + 1].y * gelu_grad(z.w));
        if (valid) {
          bsum[4 * k] += bf_lo(w[k][0]);
          bsum[4 * k + 1] += bf_hi(w[k][0]);
          bsum[4 * k + 2] += bf_lo(w[k][1]);
          bsum[4 * k + 3] += bf_hi(w[k][1]);
        }
      }
      store_bf16_row(dz2 + cell * C, w, g2, valid);
    }
    dsum += dy2[(ti + 1) * kHY + tj + 1 + lane].x;  // zero outside the domain

    // dW3: two k-steps of 16 cells.
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      uint32_t af[2][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(dyp + aoff[e] + ks * 16);
        af[e >> 1][e & 1] = aoff[e] >= 0 ? p[0] : 0u;
        af[e >> 1][(e & 1) + 2] = aoff[e] >= 0 ? p[4] : 0u;
      }
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        uint32_t r[4];
        const int cell = ti * kTY + tj + ks * 16 + (mi & 1) * 8 + rr;
        ldsm_x4_t(r, as + cell * kCS + (2 * np + (mi >> 1)) * 8);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          if (mt == 0) {  // rows of the first part, h; the others are below 2^-8 of it
            mma_bf16_add(acc[mt][2 * np], af[mt], r[0], r[1]);
            mma_bf16_add(acc[mt][2 * np + 1], af[mt], r[2], r[3]);
          } else {
            mma_bf16(acc[mt][2 * np], af[mt], r[0], r[1]);
            mma_bf16(acc[mt][2 * np + 1], af[mt], r[2], r[3]);
          }
        }
      }
    }
  }

  // Warp sums into shared memory, then the warps in order.
  cp_async_wait<0>();
  __syncthreads();
  float* sums = reinterpret_cast<float*>(smem_raw) + warp * kB3Sums;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = mt * 16 + gq + 8 * (e >> 1);
        if (m < 27) sums[m * C + nt * 8 + 2 * tq + (e & 1)] = acc[mt][nt][e];
      }
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    float v = bsum[k];
#pragma unroll
    for (int o = 2; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lc == 0) sums[27 * C + 8 * (k >> 2) + 4 * g2 + (k & 3)] = v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
  if (lane == 0) sums[28 * C] = dsum;
  __syncthreads();
  float* row = partial + (int64_t)blockIdx.x * LBM_CLOSURE_PARAMS;
  const float* all = reinterpret_cast<const float*>(smem_raw);
  for (int k = threadIdx.x; k < 10 * C + 1; k += blockDim.x) {
    float v = 0.0f;
    for (int w = 0; w < kB3Threads / 32; ++w) {
      const float* sw = all + w * kB3Sums;
      if (k < 9 * C)
        v += sw[18 * C + k] + sw[9 * C + k] + sw[k];  // smallest part first
      else
        v += sw[18 * C + k];  // db2, then db3
    }
    if (k < 9 * C)
      row[LBM_CLOSURE_OFF_W3 + k] = v;
    else if (k < 10 * C)
      row[LBM_CLOSURE_OFF_B2 + k - 9 * C] = v;
    else
      row[LBM_CLOSURE_OFF_B3] = v;
  }
}

// ---------------------------------------------------------------------------------------------
// Layer-1 weight gradient on tensor cores: dW1[co][tap][ci] = sum_p dz1[p][co] x[p + tap][ci].
// M = 32 output channels (2 m-tiles), N = 36 (tap, ci) columns and one of ones, whose sums are the
// bias gradient (5 n-tiles, the last three columns empty), K = cells. dz1 comes through ldmatrix; the features lie in shared memory as one plane a channel,
// twice (the second copy shifted by one cell), so that two consecutive cells of any tap are one
// aligned 32-bit word. Bound by reading dz1 and x; two CTAs an SM. Batch
// 8 x 1024 x 512: 870 -> 98 us (93 with the sums left in the tensor cores: mma_bf16_add).

constexpr int kW1Threads = 256;
constexpr int kXS = kHY + 2;  // BF16 elements of a row of a feature plane
constexpr size_t kW1Stage0 = (size_t)kTX * kTY * kCS * 2;  // dz1 of a tile
constexpr size_t kW1OffX = 2 * kW1Stage0;
constexpr size_t kW1Stage = kW1OffX + (size_t)4 * 2 * kHX * kXS * 2;
constexpr size_t kW1Smem = (size_t)(kW1Threads / 32) * 37 * C * 4 > kW1Stage
                               ? (size_t)(kW1Threads / 32) * 37 * C * 4
                               : kW1Stage;

__global__ void __launch_bounds__(kW1Threads, 2)
    conv1_wgrad_kernel(Grid g, const bf16* __restrict__ x, const bf16* __restrict__ dz1,
                       float* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* xp = reinterpret_cast<bf16*>(smem_raw + kW1OffX);  // [ci][shift][kHX][kXS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3, mi = lane >> 3, rr = lane & 7;
  const int ti = warp >> 1, tj = (warp & 1) * 32;
  // B fragments: column n = gq of n-tile nt is (tap, ci) = (n / 4, n % 4) of 8 nt + gq.
  int boff[5];
#pragma unroll
  for (int nt = 0; nt < 5; ++nt) {
    const int n = nt * 8 + gq, tap = n >> 2, ci = n & 3;
    boff[nt] = -1;
    if (tap < 9) {
      const int col = tj + 1 + tap % 3 - 1, r = ti + 1 + tap / 3 - 1, odd = col & 1;
      boff[nt] = ((ci * 2 + odd) * kHX + r) * kXS + col - odd + 2 * tq;
    }
  }
  // Column 36 holds ones: the sums of dz1, the bias gradient.
  const uint32_t none = gq == 4 ? 0x3f803f80u : 0u;
  float acc[2][5][4];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 5; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[mt][nt][e] = 0.0f;
  for (int i = threadIdx.x; i < 4 * 2 * kHX * kXS; i += blockDim.x) xp[i] = to_bf(0.0f);
  // The next tile's operands are in flight while this one is multiplied.
  FeatureTile<kW1Threads> in;
  auto fetch = [&](int64_t t, int s) {
    int64_t b, x0, y0;
    g.tile(t, b, x0, y0);
    load_cells32_async<kTX, kTY>(dz1, g, b, x0, y0,
                                 reinterpret_cast<bf16*>(smem_raw + (size_t)s * kW1Stage0));
    in.load(x, g, t);
  };
  int stage = 0;
  if ((int64_t)blockIdx.x < g.tiles) fetch(blockIdx.x, 0);
  cp_async_commit();
  for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, stage ^= 1) {
    __syncthreads();  // the previous tile is done with the planes and its stage
    in.each([&](int i, uint2 v) {
      const int r = i / kHY, c = i - r * kHY;
      const uint32_t h[4] = {v.x & 0xffffu, v.x >> 16, v.y & 0xffffu, v.y >> 16};
#pragma unroll
      for (int ci = 0; ci < 4; ++ci) {
        const bf16 e = __ushort_as_bfloat16((unsigned short)h[ci]);
        xp[((ci * 2) * kHX + r) * kXS + c] = e;
        if (c > 0) xp[((ci * 2 + 1) * kHX + r) * kXS + c - 1] = e;
      }
    });
    if (t + gridDim.x < g.tiles) fetch(t + gridDim.x, stage ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const bf16* dzs = reinterpret_cast<const bf16*>(smem_raw + (size_t)stage * kW1Stage0);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      uint32_t af[2][4];
      const int cell = ti * kTY + tj + ks * 16 + (mi >> 1) * 8 + rr;
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) ldsm_x4_t(af[mt], dzs + cell * kCS + mt * 16 + (mi & 1) * 8);
#pragma unroll
      for (int nt = 0; nt < 5; ++nt) {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(xp + boff[nt] + ks * 16);
        const uint32_t b0 = boff[nt] >= 0 ? p[0] : none, b1 = boff[nt] >= 0 ? p[4] : none;
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) mma_bf16_add(acc[mt][nt], af[mt], b0, b1);
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  float* sums = reinterpret_cast<float*>(smem_raw);  // [warp][co][37]
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 5; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int co = mt * 16 + gq + 8 * (e >> 1), n = nt * 8 + 2 * tq + (e & 1);
        if (n < 37) sums[(warp * C + co) * 37 + n] = acc[mt][nt][e];
      }
  __syncthreads();
  float* row = partial + (int64_t)blockIdx.x * LBM_CLOSURE_PARAMS;
  for (int i = threadIdx.x; i < 37 * C; i += blockDim.x) {
    float v = 0.0f;
    for (int w = 0; w < kW1Threads / 32; ++w) v += sums[w * 37 * C + i];
    const int co = i / 37, n = i - co * 37;
    row[n < 36 ? LBM_CLOSURE_OFF_W1 + co * 36 + n : LBM_CLOSURE_OFF_B1 + co] = v;
  }
}

// Column sums of the partial rows (double accumulation in a fixed order); the layer-2 weight
// gradient has rows_w2 of them, the rest `rows`. Eight threads a column, so that the rows are read
// by enough of the chip.
__global__ void __launch_bounds__(256)
    reduce_rows_kernel(const float* __restrict__ partial, int rows, int rows_w2,
                       float* __restrict__ out) {
  __shared__ double s[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + tx;
  double v = 0.0;
  if (j < LBM_CLOSURE_PARAMS) {
    const bool w2 = j >= LBM_CLOSURE_OFF_W2 && j < LBM_CLOSURE_OFF_W2 + C * 288;
    const int n = w2 ? rows_w2 : rows;
    for (int r = ty; r < n; r += 8) v += partial[(int64_t)r * LBM_CLOSURE_PARAMS + j];
  }
  s[ty][tx] = v;
  __syncthreads();
  if (ty == 0 && j < LBM_CLOSURE_PARAMS) {
    for (int k = 1; k < 8; ++k) v += s[k][tx];
    out[j] = (float)v;
  }
}

// ---------------------------------------------------------------------------------------------
// Loss

// Fluid cells, as kCountBlocks partial counts (one block alone took 77 us on 1024 x 512).
constexpr int kCountBlocks = 32;

__global__ void __launch_bounds__(1024)
    count_kernel(const int32_t* __restrict__ flags, int64_t n,
                 unsigned long long* __restrict__ counts) {
  __shared__ unsigned long long s[32];
  unsigned long long c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    c += fluid_cell(flags[i]) ? 1 : 0;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[w];
    counts[blockIdx.x] = t;
  }
}

__device__ __forceinline__ double total_count(const unsigned long long* counts, int64_t batch) {
  unsigned long long c = 0;
  for (int k = 0; k < kCountBlocks; ++k) c += counts[k];
  return (double)c * (double)batch;
}

// Each thread takes a cell through the whole batch: its flag is read once, and no index needs a
// division.
__global__ void __launch_bounds__(256)
    loss_kernel(const float* __restrict__ y, const float* __restrict__ target,
                const int32_t* __restrict__ flags, int64_t n, int64_t batch,
                const unsigned long long* __restrict__ counts, float* __restrict__ dy,
                double* __restrict__ partial) {
  __shared__ double s[32];
  const double total = total_count(counts, batch);
  const float scale = total > 0 ? (float)(2.0 / total) : 0.0f;
  double acc = 0.0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    const bool m = fluid_cell(flags[c]);
#pragma unroll 4
    for (int64_t b = 0; b < batch; ++b) {
      const int64_t i = b * n + c;
      const float d = y[i] - target[i];
      dy[i] = m ? scale * d : 0.0f;
      if (m) acc += (double)d * (double)d;
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[w];
    partial[blockIdx.x] = t;
  }
}

// One warp: the partial sums by lanes, then across them (a fixed order).
__global__ void __launch_bounds__(32)
    loss_final_kernel(const double* __restrict__ partial, int blocks,
                      const unsigned long long* __restrict__ counts, int64_t batch,
                      double* __restrict__ loss) {
  double t = 0.0;
  for (int i = threadIdx.x; i < blocks; i += 32) t += partial[i];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (threadIdx.x == 0) {
    const double total = total_count(counts, batch);
    *loss = total > 0 ? t / total : 0.0;
  }
}

// ---------------------------------------------------------------------------------------------
// Blackwell tensor cores (tcgen05): MMAs issued by one thread on shared-memory operands,
// accumulators in tensor memory (TMEM), completion signalled through an mbarrier.

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor, K-major without swizzle: rows (M or N) 16 bytes apart inside a
// group of 8 rows, `sbo` bytes between groups of 8 rows, `lbo` bytes between the two 8-element K
// halves of one MMA. Descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t umma_desc(unsigned start, unsigned lbo, unsigned sbo) {
  return (uint64_t)((start >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// The descriptor `bytes` (a multiple of 16) further on: one addition to its low word. One thread
// issues all of a CTA's products, and building a descriptor anew took it longer than the product.
__device__ __forceinline__ uint64_t umma_desc_at(uint64_t desc, unsigned bytes) {
  return (desc & ~0xffffffffull) | ((uint32_t)desc + (bytes >> 4));
}

// Instruction descriptor of kind::f16: BF16 A and B, FP32 accumulator, both K-major, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u), "r"(0u), "r"(0u),
      "r"(0u));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_addr(bar))
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
      "%30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Eight of them.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

constexpr unsigned kClosureSpinLimit = 1u << 22;

__device__ __forceinline__ void cl_mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

// Polls of a wait for tensor-core products before it gives up, in the fused kernel and in the epilogues
// of the training kernels (lbm_closure_set_spin_limit); the waits of the warps that copy and issue, and
// those that drain what is still in flight, keep the default.
__device__ unsigned g_closure_spin_limit = kClosureSpinLimit;

// Bounded wait for the phase with the given parity; false after `limit` polls.
__device__ __forceinline__ bool cl_mbar_wait(uint64_t* bar, unsigned parity,
                                             unsigned limit = kClosureSpinLimit) {
  const unsigned addr = smem_addr(bar);
  for (unsigned i = 0; i < limit; ++i) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void cl_mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// Bounded wait that also ends when another warp of the CTA has given up; whoever gives up stops the
// rest.
__device__ __forceinline__ bool cl_mbar_wait_or_stop(uint64_t* bar, unsigned parity, unsigned limit,
                                                     volatile int* stop) {
  constexpr unsigned kPolls = 64;
  for (unsigned k = 0; k < limit; k += kPolls) {
    if (cl_mbar_wait(bar, parity, kPolls)) return true;
    if (*stop) return false;
  }
  *stop = 1;
  return false;
}

// Set (bit 0) when a closure kernel gave up waiting for its tensor-core work; read and cleared
// by lbm_closure_status.
__device__ int g_closure_status;

// ---------------------------------------------------------------------------------------------
// Inference in one pass: features, the three layers and the relaxation field for a tile of
// kFR x kFC output cells, every intermediate in shared memory (~213 KB, one CTA of 16 warps per
// SM). The raw fields of the tile's neighbourhood are staged first with coalesced loads. Each
// layer is evaluated on its own halo-extended region -- layer 3 reads layer 2 one cell around
// the tile, layer 2 reads layer 1 two cells around, layer 1 reads the features three cells
// around -- and outside the domain every layer's output is 0, the zero padding the
// layer-by-layer kernels apply. All three layers run on tensor cores (mma.sync BF16 -> FP32):
// layer 1 with K = 48 (9 taps x 4 channels, zero-padded from 36), layer 2 with K = 288, layer 3
// with K = 288 and N = 8 (one real output column). A warp's
// 16-row MMA tile is any 16 consecutive cells of a region in row-major order (ldmatrix takes one
// row address per lane), so the regions need not be multiples of 16 wide. Bound by the instruction
// stream of the two GELU epilogues and layer 1's fragments, with the MMAs' reads of A behind it.
// 1024 x 512: 124 -> 105 us with GELU on packed pairs, the ninth block of layer 2 shared among the
// warps of a sub-partition and layer 3's chains in pairs; 99 us with descriptors advanced by one
// addition.

constexpr int kFR = 14, kFC = 64;               // output tile
constexpr int kA2R = kFR + 2, kA2C = kFC + 2;  // layer-2 region
constexpr int kA1R = kFR + 4, kA1C = kFC + 4;  // layer-1 region
constexpr int kXR = kFR + 6, kXC = kFC + 6;    // feature region
constexpr int kRawR = kFR + 8, kRawC = kFC + 8;  // raw fields (features read one cell around)
constexpr int kW1S = 56;                        // shared-memory BF16 per layer-1 weight row
constexpr int kFusedThreads = 512;
// Layer 1's output is stored "chunk-major" for the tensor-core descriptors: plane k (channels
// 8k .. 8k+7) holds 16 bytes per cell, cells in row-major order of the layer-1 region
// (kA1R x kA1C), padded so that every shifted 128-cell block stays inside the plane.
constexpr int kA1Pad = 1296;                    // >= 69 + 9 * 128 + 69 cells
constexpr int kL2Blocks = 9;                    // 128-cell blocks covering the layer-2 region
constexpr int kL2First = kA1C + 1;              // layer-1 flat index of layer-2 cell (0, 0)
constexpr size_t kFusedOffA1 = (size_t)kXR * kXC * 8;
constexpr size_t kFusedOffA2 = kFusedOffA1 + (size_t)4 * kA1Pad * 16;
constexpr size_t kFusedOffW1 = kFusedOffA2 + (size_t)kA2R * kA2C * kCS * 2;
constexpr size_t kFusedOffW2 = kFusedOffW1 + (size_t)C * kW1S * 2;
constexpr size_t kFusedOffW3 = kFusedOffW2 + (size_t)36 * C * 16;  // 36 K-chunks x 32 rows x 16 B
constexpr size_t kFusedOffB = kFusedOffW3 + (size_t)9 * C * 4;
constexpr size_t kFusedOffBar = kFusedOffB + (size_t)2 * C * 4;    // mbarrier + TMEM address
constexpr size_t kFusedSmem = kFusedOffBar + 16;
static_assert(kL2First + kL2Blocks * 128 + kA1C + 1 <= kA1Pad, "layer-1 planes too short");
static_assert(kL2First + kL2Blocks * 128 > (kA2R * kA1C) + kA2C, "blocks do not cover layer 2");
constexpr int kTmemCols = 512;  // 9 accumulators of 32 FP32 columns (power of two >= 288)
static_assert((size_t)kRawR * kRawC * 16 <= (size_t)kA2R * kA2C * kCS * 2,
              "the staged raw fields must fit in the layer-2 area");

struct FusedArgs {
  const float* params;
  const bf16* wb;
  const float* rho;
  const float* vel;
  const int32_t* flags;
  int64_t nx, ny;
  Norm norm;
  float tau0, gain, max_dtau;
  float* omega;
  int tiles_x, tiles_y;
};

__global__ void __launch_bounds__(kFusedThreads, 1)
    closure_fused_kernel(const __grid_constant__ FusedArgs f) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t* xs = reinterpret_cast<uint32_t*>(smem_raw);  // [cell][2 words]: channels 0-1, 2-3
  unsigned char* a1c = smem_raw + kFusedOffA1;  // [4 planes][kA1Pad cells][16 B]
  bf16* a2s = reinterpret_cast<bf16*>(smem_raw + kFusedOffA2);
  bf16* w1s = reinterpret_cast<bf16*>(smem_raw + kFusedOffW1);
  unsigned char* w2c = smem_raw + kFusedOffW2;  // [36 K-chunks][32 out channels][16 B]
  bf16* w3b = reinterpret_cast<bf16*>(smem_raw + kFusedOffW3);  // [9][32]
  float* bs = reinterpret_cast<float*>(smem_raw + kFusedOffB);  // b1 [32], b2 [32]
  uint64_t* mma_done = reinterpret_cast<uint64_t*>(smem_raw + kFusedOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + kFusedOffBar + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3, mi = lane >> 3, rr = lane & 7;
  constexpr int kWarps = kFusedThreads / 32;

  for (int i = threadIdx.x; i < C * kW1S; i += blockDim.x) {
    const int co = i / kW1S, k = i - co * kW1S;
    w1s[i] = k < 36 ? f.wb[LBM_CLOSURE_OFF_W1 + co * 36 + k] : __float2bfloat16(0.0f);
  }
  // Layer-2 weights as the MMA's B operand: K-chunk kk (k = 8 kk .. 8 kk + 7, k = tap*32 + ci)
  // of output channel co at (kk * 32 + co) * 16 bytes.
  for (int i = threadIdx.x; i < 36 * C; i += blockDim.x) {
    const int kk = i / C, co = i - kk * C;
    *reinterpret_cast<uint4*>(w2c + (size_t)i * 16) =
        __ldg(reinterpret_cast<const uint4*>(f.wb + LBM_CLOSURE_OFF_W2 + co * 288 + kk * 8));
  }
  for (int i = threadIdx.x; i < 9 * C; i += blockDim.x) w3b[i] = f.wb[LBM_CLOSURE_OFF_W3 + i];
  for (int i = threadIdx.x; i < 2 * C; i += blockDim.x)
    bs[i] = f.params[i < C ? LBM_CLOSURE_OFF_B1 + i : LBM_CLOSURE_OFF_B2 + i - C];
  const float b3 = f.params[LBM_CLOSURE_OFF_B3];
  // Padding cells of the layer-1 planes feed only discarded rows; keep them finite.
  for (int i = threadIdx.x; i < 4 * kA1Pad; i += blockDim.x) {
    if (i % kA1Pad >= kA1R * kA1C)
      *reinterpret_cast<uint4*>(a1c + (size_t)i * 16) = make_uint4(0, 0, 0, 0);
  }
  if (threadIdx.x == 0) {
    cl_mbar_init(mma_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t idesc = umma_idesc_bf16(128, 32);
  const uint64_t a1desc = umma_desc(smem_addr(a1c), kA1Pad * 16, 128);
  const uint64_t w2desc = umma_desc(smem_addr(w2c), C * 16, 128);
  bool healthy = true;
  const unsigned spin_limit = g_closure_spin_limit;
  // Layer-1 A fragments: element e of k-step kk holds input k = 16 kk + 2 tq + 8 (e >> 1), that
  // is tap k / 4 and the channel pair (k & 3) / 2 of the feature cell shifted by the tap. The
  // offset of that word from the cell's own (in 32-bit words of the feature region) depends on
  // the lane only; taps past 8 are the K padding (zero).
  int l1off[3][2];
  unsigned l1valid = 0;
#pragma unroll
  for (int kk = 0; kk < 3; ++kk)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int k = kk * 16 + 2 * tq + 8 * hi, tap = k >> 2;
      l1off[kk][hi] = 2 * ((tap / 3 - 1) * kXC + tap % 3 - 1) + ((k & 3) >> 1);
      if (tap < 9) l1valid |= 1u << (2 * kk + hi);
    }
  unsigned phase = 0;

  const int ntiles = f.tiles_x * f.tiles_y;
  // Raw fields and features of tile t (the raw fields pass through the layer-2 area, which is
  // free from a tile's layer 3 until the next tile's epilogue), by warps 1 .. 15: warp 0 issues
  // the layer-2 MMAs meanwhile. Named barrier 1 orders the staging before the features.
  constexpr int kStageThreads = kFusedThreads - 32;
  auto stage_features = [&](int t) {
    if (warp == 0) return;
    const int st = threadIdx.x - 32;
    const int64_t x0 = (int64_t)(t / f.tiles_y) * kFR, y0 = (int64_t)(t % f.tiles_y) * kFC;
    // Raw fields on [x0 - 4, x0 + kFR + 4) x [y0 - 4, y0 + kFC + 4), staged with coalesced loads
    // into the layer-2 area; velocities on walls read as 0.
    float* raw_rho = reinterpret_cast<float*>(a2s);
    float2* raw_vel = reinterpret_cast<float2*>(raw_rho + kRawR * kRawC);
    int* raw_flag = reinterpret_cast<int*>(raw_vel + kRawR * kRawC);
    for (int i = st; i < kRawR * kRawC; i += kStageThreads) {
      const int r = i / kRawC, c = i - r * kRawC;
      const int64_t x = x0 - 4 + r, y = y0 - 4 + c;
      float rv = 0.0f;
      float2 vv = make_float2(0.0f, 0.0f);
      int fl = 0;
      if (x >= 0 && x < f.nx && y >= 0 && y < f.ny) {
        const int64_t cell = x * f.ny + y;
        rv = f.rho[cell];
        vv = *reinterpret_cast<const float2*>(f.vel + 2 * cell);
        fl = f.flags[cell];
      }
      raw_rho[i] = rv;
      raw_vel[i] = vv;
      raw_flag[i] = fl;
    }
    asm volatile("bar.sync 1, %0;" ::"r"(kStageThreads) : "memory");
    // Features on [x0 - 3, x0 + kFR + 3) x [y0 - 3, y0 + kFC + 3), the arithmetic of
    // cell_features (np.gradient edges, walls at rest, normalise, BF16) on the staged fields.
    for (int i = st; i < kXR * kXC; i += kStageThreads) {
      const int r = i / kXC, c = i - r * kXC;
      const int64_t x = x0 - 3 + r, y = y0 - 3 + c;
      uint2 packed = make_uint2(0, 0);
      const int ri = (r + 1) * kRawC + c + 1;  // this cell in the raw region
      if (x >= 0 && x < f.nx && y >= 0 && y < f.ny && !(raw_flag[ri] & 1)) {
        const int im = x > 0 ? ri - kRawC : ri, ip = x < f.nx - 1 ? ri + kRawC : ri;
        const int jm = y > 0 ? ri - 1 : ri, jp = y < f.ny - 1 ? ri + 1 : ri;
        auto vx = [&](int k) { return (raw_flag[k] & 1) ? 0.0f : raw_vel[k].x; };
        auto vy = [&](int k) { return (raw_flag[k] & 1) ? 0.0f : raw_vel[k].y; };
        const float dux_dy = np_gradient(vx(jm), raw_vel[ri].x, vx(jp), y, f.ny);
        const float duy_dx = np_gradient(vy(im), raw_vel[ri].y, vy(ip), x, f.nx);
        const float v[4] = {__fsub_rn(raw_rho[ri], 1.0f), raw_vel[ri].x, raw_vel[ri].y,
                            __fsub_rn(dux_dy, duy_dx)};
        bf16 h[4];
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          h[ch] = to_bf(__fmul_rn(__fsub_rn(v[ch], f.norm.mean[ch]), f.norm.inv_std[ch]));
        packed.x = (uint32_t)__bfloat16_as_ushort(h[0]) | ((uint32_t)__bfloat16_as_ushort(h[1]) << 16);
        packed.y = (uint32_t)__bfloat16_as_ushort(h[2]) | ((uint32_t)__bfloat16_as_ushort(h[3]) << 16);
      }
      xs[2 * i] = packed.x;
      xs[2 * i + 1] = packed.y;
    }
  };
  // Tile t's layer-2 MMAs run while the CTA stages and featurises its next tile.
  if ((int)blockIdx.x < ntiles) stage_features(blockIdx.x);
  for (int t = blockIdx.x; t < ntiles && healthy; t += gridDim.x) {
    const int64_t x0 = (int64_t)(t / f.tiles_y) * kFR, y0 = (int64_t)(t % f.tiles_y) * kFC;
    tc_fence_before();
    __syncthreads();  // tile t's features are in place; the previous tile is done with a1c, a2s
                      // and every TMEM column
    tc_fence_after();

    // Layer 1 on [x0 - 2, ..) x [y0 - 2, ..): A fragments gathered from the features by tap.
    constexpr int n1 = kA1R * kA1C;
    for (int mt = warp; mt * 16 < n1; mt += kWarps) {
      int rq[2], cq[2], xw[2];  // xw: word index of the cell in the feature region
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int q = min(mt * 16 + gq + 8 * h, n1 - 1);
        rq[h] = q / kA1C;
        cq[h] = q - rq[h] * kA1C;
        xw[h] = 2 * ((rq[h] + 1) * kXC + cq[h] + 1);
      }
      float acc[4][4];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] = 0.0f;
#pragma unroll
      for (int kk = 0; kk < 3; ++kk) {
        uint32_t a[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int h = e & 1, hi = e >> 1;
          a[e] = (l1valid >> (2 * kk + hi)) & 1u ? xs[xw[h] + l1off[kk][hi]] : 0u;
        }
        uint32_t bfr[4][2];
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t r4[4];
          ldsm_x4(r4, w1s + ((2 * np + (mi >> 1)) * 8 + rr) * kW1S + kk * 16 + (mi & 1) * 8);
          bfr[2 * np][0] = r4[0];
          bfr[2 * np][1] = r4[1];
          bfr[2 * np + 1][0] = r4[2];
          bfr[2 * np + 1][1] = r4[3];
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) mma_bf16(acc[nt], a, bfr[nt][0], bfr[nt][1]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int q = mt * 16 + gq + 8 * h;
        if (q >= n1) continue;
        const int64_t x = x0 - 2 + rq[h], y = y0 - 2 + cq[h];
        const bool inside = x >= 0 && x < f.nx && y >= 0 && y < f.ny;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const int ch = nt * 8 + 2 * tq;
          const float2 z = __fadd2_rn(make_float2(acc[nt][2 * h], acc[nt][2 * h + 1]),
                                      *reinterpret_cast<const float2*>(bs + ch));
          *reinterpret_cast<uint32_t*>(a1c + ((size_t)nt * kA1Pad + q) * 16 + tq * 4) =
              inside ? pack_bf2(gelu2(z)) : 0u;
        }
      }
    }
    __syncthreads();

    // Layer 2 on tcgen05: nine blocks of 128 consecutive layer-1 cells (flat index from the
    // layer-1 cell of layer-2 cell (0, 0)), each an M = 128, N = 32, K = 288 product into its own
    // 32 TMEM columns. Tap (dx, dy) reads the block shifted by dx * kA1C + dy cells: with the
    // chunk-major planes that is an offset of the descriptor's start address (16 bytes a cell).
    // Rows that fall on the region's first or last column are computed and discarded.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // layer 1 visible to the MMAs
    __syncthreads();
    if (threadIdx.x == 0) {
      tc_fence_after();
      // K-slice outer, block inner: consecutive MMAs accumulate into different TMEM columns.
#pragma unroll 1
      for (int tap = 0; tap < 9; ++tap) {
        const int off = (tap / 3 - 1) * kA1C + (tap % 3 - 1);
#pragma unroll
        for (int kc = 0; kc < 2; ++kc) {
          const int sidx = tap * 2 + kc;
          const uint64_t bdesc = umma_desc_at(w2desc, (unsigned)(sidx * 1024));
          const uint64_t adesc =
              umma_desc_at(a1desc, (unsigned)((2 * kc * kA1Pad + kL2First + off) * 16));
#pragma unroll
          for (int m = 0; m < kL2Blocks; ++m)
            umma_bf16(tmem + (uint32_t)(m * 32), umma_desc_at(adesc, (unsigned)(m * 128 * 16)),
                      bdesc, idesc, sidx != 0);
        }
      }
      umma_commit(mma_done);
    }
    if (t + (int)gridDim.x < ntiles) stage_features(t + gridDim.x);
    const bool got = cl_mbar_wait(mma_done, phase, spin_limit);
    phase ^= 1u;
    if (!__syncthreads_and(got)) {
      healthy = false;
      break;
    }
    tc_fence_after();
    // Epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (its sub-partition) of blocks w / 4 and
    // w / 4 + 4, one thread per cell with its 32 channels, and channels 8 (w / 4) .. + 7 of the last
    // block: a sub-partition's four warps, which share a scheduler, end together (with one of them
    // on the whole last block they waited for it).
    const int sp = warp & 3, part = warp >> 2;
    auto activate = [&](int m, int ch0, const uint32_t* z, auto chunks) {
      const int p = kL2First + 128 * m + 32 * sp + lane;  // layer-1 flat index of this row
      const int r = p / kA1C - 1, c = p % kA1C - 1;      // layer-2 region coordinates
      if (r < 0 || r >= kA2R || c < 0 || c >= kA2C) return;
      const int64_t x = x0 - 1 + r, y = y0 - 1 + c;
      const bool inside = x >= 0 && x < f.nx && y >= 0 && y < f.ny;
      uint4* dst = reinterpret_cast<uint4*>(a2s + (r * kA2C + c) * kCS + ch0);
#pragma unroll
      for (int q = 0; q < decltype(chunks)::value; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int ch = 8 * q + 2 * e;
          const float2 v = __fadd2_rn(
              make_float2(__uint_as_float(z[ch]), __uint_as_float(z[ch + 1])),
              *reinterpret_cast<const float2*>(bs + C + ch0 + ch));
          w[e] = inside ? pack_bf2(gelu2(v)) : 0u;
        }
        dst[q] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    };
    const uint32_t lanes = (uint32_t)(32 * sp) << 16;
    static_assert(kL2Blocks == 9, "two blocks a warp and a quarter of the last");
#pragma unroll 1
    for (int m = part; m < 8; m += 4) {
      uint32_t z[32];
      __syncwarp();
      tmem_ld32(tmem + lanes + (uint32_t)(m * 32), z);
      activate(m, 0, z, std::integral_constant<int, 4>{});
    }
    {
      uint32_t z[8];
      __syncwarp();
      tmem_ld8(tmem + lanes + (uint32_t)(8 * 32 + 8 * part), z);
      activate(8, 8 * part, z, std::integral_constant<int, 1>{});
    }
    __syncthreads();

    // Layer 3 on tensor cores (N = 8 with only column 0 carrying w3; K = 288) and the relaxation
    // rate (the mapping of omega_kernel) on the output tile: 16 cells of one tile row per MMA tile.
    // A warp takes two of them side by side: their chains of 18 products hide each other's latency.
    constexpr int n3 = kFR * kFC, kTiles3 = n3 / 16;
    static_assert(n3 % 16 == 0, "whole tiles");
    for (int mt = warp; mt < kTiles3; mt += 2 * kWarps) {
      const int j = (lane & 7) + 8 * ((lane >> 3) & 1);
      const bf16* arow[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int qa = min(mt + u * kWarps, kTiles3 - 1) * 16 + j;
        const int ra = qa / kFC, ca = qa - ra * kFC;
        arow[u] = a2s + ((ra + 1) * kA2C + ca + 1) * kCS + 8 * (lane >> 4);
      }
      float acc[2][4] = {};
#pragma unroll 1
      for (int tap = 0; tap < 9; ++tap) {
        const int dx = tap / 3 - 1, dy = tap % 3 - 1;
        const int off = (dx * kA2C + dy) * kCS;
#pragma unroll
        for (int kc = 0; kc < 2; ++kc) {
          // B column 0 = w3[tap][kc*16 + k]; lanes of the other columns hold zeros.
          uint32_t b0 = 0u, b1 = 0u;
          if (gq == 0) {
            const int k0 = tap * C + kc * 16 + 2 * tq;
            b0 = *reinterpret_cast<const uint32_t*>(w3b + k0);
            b1 = *reinterpret_cast<const uint32_t*>(w3b + k0 + 8);
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            uint32_t a[4];
            ldsm_x4(a, arow[u] + off + kc * 16);
            mma_bf16(acc[u], a, b0, b1);
          }
        }
      }
      if (tq == 0) {  // column 0: rows gq and gq + 8 of each tile
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int u = k >> 1, h = k & 1;
          if (mt + u * kWarps >= kTiles3) continue;
          const int q = (mt + u * kWarps) * 16 + gq + 8 * h;
          const int r = q / kFC, c = q - r * kFC;
          const int64_t x = x0 + r, y = y0 + c;
          if (x >= f.nx || y >= f.ny) continue;
          const float yv = acc[u][2 * h] + b3;
          const int64_t cell = x * f.ny + y;
          float tau = f.tau0;
          if (fluid_cell(f.flags[cell])) tau += fminf(f.max_dtau, f.gain * fmaxf(yv, 0.0f));
          f.omega[cell] = 1.0f / tau;
        }
      }
    }
  }
  if (!healthy) {
    if (threadIdx.x == 0) {
      atomicOr(&g_closure_status, 1);
      cl_mbar_wait(mma_done, phase ^ 1u);  // give MMAs still in flight a bounded chance to end
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// Layer 2 of the training path on tcgen05: the forward conv (BWD = false: z2 = b2 + W * a1,
// a2 = GELU(z2) in BF16) and the transposed conv of the backward pass (BWD = true:
// d = W^T * dz2, dz1 = BF16(d GELU'(z1))). Same products as conv32_kernel, on the fifth-generation
// tensor cores:
//   - the input of a tile of kTR x kTC output cells is three copies of kTR + 2 rows of kTC cells,
//     shifted by -1, 0 and 1 cells along the row by the tensor engine (zero outside the domain),
//     64 bytes a cell, swizzled: a tap (dx, dy) of the 3x3 stencil reads copy dy + 1 from row
//     1 + dx on (both negated for the transposed conv), and a row's 2 KB keep the swizzle's phase;
//   - kTBlocks blocks of 128 consecutive cells, each an M = 128, N = 32, K = 288 product into its
//     own 32 TMEM columns;
//   - the B operand is the weights as K-chunks of 8: [k chunk][n][8] with k = (tap, ci) and
//     n = co for the forward conv, k = (tap, co) and n = ci for the transposed one.
// One warp copies (a ring of kTStages tiles), one issues the products, and two groups of eight warps
// take the tiles in turn in the epilogue, which reads each cell's 32 accumulators with tcgen05.ld.
// Bound by shared memory (the products read A anew for each tap: 720 bytes a cell, of 1300 in all)
// close to DRAM (256 bytes a cell, 166 us over batch 8 x 1024 x 512): 199 us forward and backward
// there. With copies, products and epilogue in turn in three CTAs an SM, on regions with a halo whose
// discarded rows are an eighth of the products, it took 290 and 278 us; side by side 279 and 276; on
// whole rows 241 and 232, 120 cycles a product, most of them the issuing thread's descriptors.

constexpr int kTR = 8, kTC = 32;                    // output tile
constexpr int kTBlocks = kTR * kTC / 128;           // 128-cell blocks
constexpr int kTGroup = 4 * kTBlocks;               // epilogue warps of a tile
constexpr int kTEpilogue = 2 * kTGroup;             // warps of the epilogue
constexpr int kTThreads = (kTEpilogue + 2) * 32;    // and one each for the copies and the products
constexpr int kTStages = 2;
constexpr int kTTmemCols = 2 * kTBlocks * 32;       // two tiles' accumulators of 32 FP32 columns
constexpr unsigned kTRow = kTC * C * 2;             // bytes of a row of cells
constexpr unsigned kTCopy = (kTR + 2) * kTRow;      // one shifted copy
constexpr unsigned kTStage = 3 * kTCopy;
constexpr size_t kTOffW = (size_t)kTStages * kTStage;
constexpr size_t kTOffRows = kTOffW + (size_t)36 * C * 16;
constexpr int kTStageBytes = 32 * 128;              // an epilogue warp's rows
constexpr size_t kTOffBias = kTOffRows + (size_t)kTEpilogue * kTStageBytes;
constexpr size_t kTOffBar = kTOffBias + (size_t)C * 4;
constexpr int kTBars = 2 * kTStages + 5;            // full, empty; done[2], read[2]; drained
constexpr size_t kTSmem = kTOffBar + kTBars * 8 + 8 + 1024;  // the stages start on 1 KB
static_assert(kTR * kTC == kTBlocks * 128 && (kTTmemCols & (kTTmemCols - 1)) == 0, "whole blocks");
static_assert(kTRow % 512 == 0, "a row keeps the swizzle's phase");

__device__ __forceinline__ void tc_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

// A box of whole cells of the activations (tc_rows_map) at row x, column y of sample b; cells outside
// the domain read as zero.
__device__ __forceinline__ void tc_rows_copy(void* dst, const CUtensorMap* map, int y, int x, int b,
                                             uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(y), "r"(x), "r"(b), "r"(smem_addr(bar))
      : "memory");
}

// For umma_desc: rows of 64 bytes, swizzled.
constexpr uint64_t kSwizzle64 = 4ull << 61;

template <bool BWD>
__global__ void __launch_bounds__(kTThreads, 1)
    conv32_tc_kernel(Grid g, const __grid_constant__ CUtensorMap in_map,
                     const bf16* __restrict__ w2, const float* __restrict__ bias,
                     const float* __restrict__ zin, float* __restrict__ zout,
                     bf16* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  unsigned char* wc = base + kTOffW;                // [36 K-chunks][32 n][16 B]
  float* bs = reinterpret_cast<float*>(base + kTOffBias);  // forward: b2
  uint64_t* full = reinterpret_cast<uint64_t*>(base + kTOffBar);
  uint64_t* empty = full + kTStages;
  uint64_t* done = empty + kTStages;
  uint64_t* read = done + 2;
  uint64_t* drained = read + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  volatile int* stop = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // The B operand. Forward: chunk kk = (tap, ci chunk) of output channel co, 8 consecutive
  // weights of the [co][288] row. Transposed: chunk kk = (tap, co chunk) of input channel ci,
  // weights W[8 cc .. 8 cc + 7][tap][ci].
  for (int i = threadIdx.x; i < 36 * C; i += blockDim.x) {
    const int kk = i / C, n = i - kk * C;
    if (!BWD) {
      *reinterpret_cast<uint4*>(wc + (size_t)i * 16) =
          __ldg(reinterpret_cast<const uint4*>(w2 + n * 288 + kk * 8));
    } else {
      const int tap = kk >> 2, cc = kk & 3;
      bf16 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = w2[(cc * 8 + j) * 288 + tap * 32 + n];
      *reinterpret_cast<uint4*>(wc + (size_t)i * 16) = *reinterpret_cast<const uint4*>(v);
    }
  }
  if (!BWD && threadIdx.x < C) bs[threadIdx.x] = bias[threadIdx.x];
  // The weights, written here, are read by the MMAs (async proxy).
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (threadIdx.x == 0) {
    for (int k = 0; k < kTStages; ++k) cl_mbar_init(full + k, 1), cl_mbar_init(empty + k, 1);
    for (int k = 0; k < 2; ++k) cl_mbar_init(done + k, 1), cl_mbar_init(read + k, kTGroup);
    cl_mbar_init(drained, 1);
    *stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(tmem_slot)),
                 "r"(kTTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const unsigned spin_limit = g_closure_spin_limit;
  auto wait = [&](uint64_t* bar, unsigned parity, unsigned limit) {
    return cl_mbar_wait_or_stop(bar, parity, limit, stop);
  };
  auto tile_of = [&](int64_t t, int64_t& b, int64_t& x0, int64_t& y0) {
    const int64_t per = g.tx * g.ty;  // this kernel's tiles are kTR x kTC (see the launcher)
    b = t / per;
    const int64_t r = t - b * per;
    x0 = (r / g.ty) * kTR;
    y0 = (r % g.ty) * kTC;
  };

  if (warp == kTEpilogue) {
    if (lane == 0) {
      unsigned n = 0;
      for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, ++n) {
        const unsigned s = n % kTStages, lap = n / kTStages;
        if (lap > 0 && !wait(empty + s, (lap - 1) & 1u, kClosureSpinLimit)) break;
        int64_t b, x0, y0;
        tile_of(t, b, x0, y0);
        tc_expect_tx(full + s, kTStage);
#pragma unroll
        for (int d = 0; d < 3; ++d)
          tc_rows_copy(base + s * kTStage + d * kTCopy, &in_map, (int)y0 + d - 1, (int)x0 - 1, (int)b,
                       full + s);
      }
      // Every copy has landed before the CTA ends, whoever gave up.
      for (unsigned k = n > kTStages ? n - kTStages : 0; k < n; ++k)
        cl_mbar_wait(full + k % kTStages, (k / kTStages) & 1u);
    }
  } else if (warp == kTEpilogue + 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_bf16(128, 32);
      const uint64_t bdesc = umma_desc(smem_addr(wc), C * 16, 128);
      unsigned n = 0;
      for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, ++n) {
        const unsigned s = n % kTStages, h = n & 1u;
        if (!wait(full + s, (n / kTStages) & 1u, kClosureSpinLimit)) break;
        if (n >= 2 && !wait(read + h, (n / 2 - 1) & 1u, kClosureSpinLimit)) break;
        tc_fence_after();
        const uint64_t adesc =
            umma_desc(smem_addr(base) + s * kTStage, 16, 8 * C * 2) | kSwizzle64;
        // K-slice outer, block inner: consecutive MMAs accumulate into different TMEM columns.
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) {
          const int dx = BWD ? 1 - tap / 3 : tap / 3 - 1, d = BWD ? 2 - tap % 3 : tap % 3;
#pragma unroll
          for (int kc = 0; kc < 2; ++kc) {
            const int sidx = tap * 2 + kc;
#pragma unroll
            for (int m = 0; m < kTBlocks; ++m)
              umma_bf16(tmem + h * (kTBlocks * 32) + (uint32_t)(m * 32),
                        umma_desc_at(adesc, d * kTCopy + (1 + dx) * kTRow + kc * 32 +
                                                (unsigned)(m * 128 * C * 2)),
                        umma_desc_at(bdesc, (unsigned)(sidx * 1024)), idesc, sidx != 0);
          }
        }
        umma_commit(empty + s);
        umma_commit(done + h);
      }
      umma_commit(drained);  // before tensor memory is given back
      cl_mbar_wait(drained, 0);
    }
  } else {
    // Epilogue: warp w of a group reads TMEM lanes 32 (w % 4) .. + 31 (its sub-partition) of block
    // w / 4; one thread per cell, its 32 channels in registers. Rows of cells pass through shared
    // memory, so that global accesses are whole 128-byte lines: a lane's own row of 128 bytes at a
    // time is a quarter of that. Chunk c of the row of lane l lies at chunk c ^ (l % 8).
    const unsigned h = warp / kTGroup;  // tiles h, h + 2, ... of this CTA
    const int sp = warp & 3, m = (warp % kTGroup) >> 2;
    unsigned char* buf = base + kTOffRows + warp * kTStageBytes;  // 32 rows x 128 bytes
    const int q = 128 * m + 32 * sp + lane, r = q / kTC, c = q % kTC;  // this lane's cell of a tile
    unsigned n = h;
    for (int64_t t = blockIdx.x + (int64_t)h * gridDim.x; t < g.tiles; t += 2 * gridDim.x, n += 2) {
      int64_t b, x0, y0;
      tile_of(t, b, x0, y0);
      const int64_t cell = x0 + r < g.nx && y0 + c < g.ny ? g.cell(b, x0 + r, y0 + c) : -1;
      if (BWD) {  // this block's rows of z1, while its products are computed
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int l = 4 * k + (lane >> 3), ch = lane & 7;
          const int64_t cl = __shfl_sync(0xffffffffu, cell, l);
          cp_async16(buf + l * 128 + ((ch ^ (l & 7)) * 16), cl >= 0 ? zin + cl * C + ch * 4 : zin,
                     cl >= 0);
        }
        cp_async_commit();
      }
      if (!__all_sync(0xffffffffu, wait(done + h, (n / 2) & 1u, spin_limit))) {
        *stop = 1;
        break;
      }
      tc_fence_after();
      uint32_t r32[32];
      tmem_ld32(tmem + h * (kTBlocks * 32) + ((uint32_t)(32 * sp) << 16) + (uint32_t)(m * 32), r32);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) cl_mbar_arrive(read + h);
      if (BWD) {
        cp_async_wait<0>();
        __syncwarp();
      }
      uint4* mine = reinterpret_cast<uint4*>(buf + lane * 128);
      uint32_t packed[C / 2];
      if (!BWD) {
#pragma unroll
        for (int k = 0; k < C / 4; ++k) {
          float z[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) z[e] = __uint_as_float(r32[4 * k + e]) + bs[4 * k + e];
          if (zout != nullptr)
            mine[k ^ (lane & 7)] = make_uint4(__float_as_uint(z[0]), __float_as_uint(z[1]),
                                              __float_as_uint(z[2]), __float_as_uint(z[3]));
          packed[2 * k] = pack_bf2(gelu2(make_float2(z[0], z[1])));
          packed[2 * k + 1] = pack_bf2(gelu2(make_float2(z[2], z[3])));
        }
        if (zout != nullptr) {
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int l = 4 * k + (lane >> 3), ch = lane & 7;
            const int64_t cl = __shfl_sync(0xffffffffu, cell, l);
            const uint4 v = *reinterpret_cast<const uint4*>(buf + l * 128 + ((ch ^ (l & 7)) * 16));
            if (cl >= 0) reinterpret_cast<uint4*>(zout + cl * C)[ch] = v;
          }
          __syncwarp();
        }
      } else {
#pragma unroll
        for (int k = 0; k < C / 4; ++k) {
          const uint4 zz = mine[k ^ (lane & 7)];
          const float zv[4] = {__uint_as_float(zz.x), __uint_as_float(zz.y), __uint_as_float(zz.z),
                               __uint_as_float(zz.w)};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const int ch = 4 * k + e;
            packed[ch / 2] = pack_bf2(
                __fmul2_rn(make_float2(__uint_as_float(r32[ch]), __uint_as_float(r32[ch + 1])),
                           gelu_grad2(make_float2(zv[e], zv[e + 1]))));
          }
        }
        __syncwarp();
      }
      // BF16 rows of 64 bytes, eight cells an access.
      const int swz = (lane >> 1) & 3;
#pragma unroll
      for (int k = 0; k < C / 8; ++k)
        reinterpret_cast<uint4*>(buf + lane * 64)[k ^ swz] =
            make_uint4(packed[4 * k], packed[4 * k + 1], packed[4 * k + 2], packed[4 * k + 3]);
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int l = 8 * k + (lane >> 2), ch = lane & 3;
        const int64_t cl = __shfl_sync(0xffffffffu, cell, l);
        const uint4 v = *reinterpret_cast<const uint4*>(buf + l * 64 + ((ch ^ ((l >> 1) & 3)) * 16));
        if (cl >= 0) reinterpret_cast<uint4*>(out + cl * C)[ch] = v;
      }
      __syncwarp();
    }
    if (BWD) cp_async_wait<0>();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTTmemCols)
                 : "memory");
  }
  if (*stop && threadIdx.x == 0) atomicOr(&g_closure_status, 1);
}

// ---------------------------------------------------------------------------------------------
// Layer-2 weight gradient on tcgen05: dW[co][tap][ci] = sum_p dz[p][co] a1[p + tap][ci], the products
// of conv32_wgrad_kernel. The cells are the contraction (K), so both operands lie as they do in
// memory, 32 channels (64 bytes, swizzled) a cell: M and N are the contiguous directions. One product
// of 128 x 96 x 16 serves all nine taps of 16 cells of a1 row i:
//   - M = (r, co): the rows i - 1 + r of dz, r = 0 .. 2, which lie one behind the other in shared
//     memory (the stride between groups of 32 rows of A is a row of the tile). r = 3 is what M = 128
//     adds; its results are dropped, so it may read anything;
//   - N = (d, ci): three copies of the a1 row, shifted by d - 1 cells by the tensor engine.
// Cells outside the domain read as zero. Warp 4 copies (a ring of kDtStages tiles), warp 3 issues,
// warps 0 .. 2 (r) add each tile's accumulators to running sums in registers while the next tile's
// products go to the other half of tensor memory: a chain in the truncating accumulators ends with
// its tile.
// Bound by the copies: 128 bytes a cell of DRAM traffic take 83 us over batch 8 x 1024 x 512, and
// 288 bytes a cell come out of L2. 111 us, where conv32_wgrad_kernel, at the rate of mma.sync, takes
// 311; the gradient is 2.1e-7 off its float64 sums at any batch, 6.8e-6 there.

constexpr int kDtThreads = 160;
constexpr int kDtStages = 3;
constexpr unsigned kDtRow = kTY * C * 2;               // bytes of a tile row of 64 cells
constexpr unsigned kDtDz = kHX * kDtRow;               // dz rows -1 .. kTX
constexpr unsigned kDtCopy = kTX * kDtRow;             // one shifted copy of the a1 rows
constexpr unsigned kDtStage = kDtDz + 3 * kDtCopy;
constexpr size_t kDtOffBar = (size_t)kDtStages * kDtStage;
constexpr int kDtBars = 2 * kDtStages + 5;             // full, empty; done[2], read[2]; drained
constexpr size_t kDtSmem = kDtOffBar + kDtBars * 8 + 16 + 1024;  // the stages start on 1 KB
constexpr int kDtTmemCols = 256;                       // two accumulators of 96 columns, 128 apart
static_assert(kTX + 3 <= kHX + 3 * kTX, "the dropped rows stay inside the stage");

__global__ void __launch_bounds__(kDtThreads, 1)
    conv32_wgrad_tc_kernel(Grid g, const __grid_constant__ CUtensorMap dz_map,
                           const __grid_constant__ CUtensorMap a1_map,
                           float* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + kDtOffBar);
  uint64_t* empty = full + kDtStages;
  uint64_t* done = empty + kDtStages;
  uint64_t* read = done + 2;
  uint64_t* drained = read + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  volatile int* stop = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int k = 0; k < kDtStages; ++k) cl_mbar_init(full + k, 1), cl_mbar_init(empty + k, 1);
    for (int k = 0; k < 2; ++k) cl_mbar_init(done + k, 1), cl_mbar_init(read + k, 3);
    cl_mbar_init(drained, 1);
    *stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(tmem_slot)),
                 "r"(kDtTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const unsigned spin_limit = g_closure_spin_limit;
  auto wait = [&](uint64_t* bar, unsigned parity, unsigned limit) {
    return cl_mbar_wait_or_stop(bar, parity, limit, stop);
  };

  float acc[3][C];  // warps 0 .. 2: row co = lane of tap row 2 - warp, columns (d, ci)
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int k = 0; k < C; ++k) acc[d][k] = 0.0f;

  if (warp == 4) {
    if (lane == 0) {
      unsigned n = 0;
      for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, ++n) {
        const unsigned s = n % kDtStages, lap = n / kDtStages;
        if (lap > 0 && !wait(empty + s, (lap - 1) & 1u, kClosureSpinLimit)) break;
        int64_t b, x0, y0;
        g.tile(t, b, x0, y0);
        unsigned char* st = base + (size_t)s * kDtStage;
        tc_expect_tx(full + s, kDtStage);
        tc_rows_copy(st, &dz_map, (int)y0, (int)x0 - 1, (int)b, full + s);
#pragma unroll
        for (int d = 0; d < 3; ++d)
          tc_rows_copy(st + kDtDz + d * kDtCopy, &a1_map, (int)y0 + d - 1, (int)x0, (int)b, full + s);
      }
      // Every copy has landed before the CTA ends, whoever gave up.
      for (unsigned k = n > kDtStages ? n - kDtStages : 0; k < n; ++k)
        cl_mbar_wait(full + k % kDtStages, (k / kDtStages) & 1u);
    }
  } else if (warp == 3) {
    if (lane == 0) {
      // Both operands with M / N contiguous (bits 15 and 16): the descriptor's strides are between
      // groups of 32 of M or N and between groups of eight cells.
      const uint32_t idesc = umma_idesc_bf16(128, 96) | (1u << 15) | (1u << 16);
      unsigned n = 0;
      for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, ++n) {
        const unsigned s = n % kDtStages, h = n & 1u;
        if (!wait(full + s, (n / kDtStages) & 1u, kClosureSpinLimit)) break;
        if (n >= 2 && !wait(read + h, (n / 2 - 1) & 1u, kClosureSpinLimit)) break;
        tc_fence_after();
        const unsigned dz = smem_addr(base) + s * kDtStage;
        const uint64_t adesc = umma_desc(dz, kDtRow, 8 * C * 2) | kSwizzle64;
        const uint64_t bdesc = umma_desc(dz + kDtDz, kDtCopy, 8 * C * 2) | kSwizzle64;
#pragma unroll
        for (int i = 0; i < kTX; ++i)
#pragma unroll
          for (int k = 0; k < kTY / 16; ++k) {
            const unsigned off = i * kDtRow + k * 16 * C * 2;
            umma_bf16(tmem + h * 128, umma_desc_at(adesc, off), umma_desc_at(bdesc, off), idesc,
                      i + k != 0);
          }
        umma_commit(empty + s);
        umma_commit(done + h);
      }
      umma_commit(drained);  // before tensor memory is given back
      cl_mbar_wait(drained, 0);
    }
  } else {
    unsigned n = 0;
    for (int64_t t = blockIdx.x; t < g.tiles; t += gridDim.x, ++n) {
      const unsigned h = n & 1u;
      if (!__all_sync(0xffffffffu, wait(done + h, (n / 2) & 1u, spin_limit))) {
        *stop = 1;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        uint32_t v[32];
        tmem_ld32(tmem + h * 128 + ((uint32_t)(warp * 32) << 16) + d * 32, v);
#pragma unroll
        for (int k = 0; k < C; ++k) acc[d][k] += __uint_as_float(v[k]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) cl_mbar_arrive(read + h);
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kDtTmemCols)
                 : "memory");
  }
  if (*stop && threadIdx.x == 0) atomicOr(&g_closure_status, 1);
  if (warp < 3) {
    float* row = partial + (int64_t)blockIdx.x * LBM_CLOSURE_PARAMS + LBM_CLOSURE_OFF_W2 +
                 lane * 288 + (2 - warp) * 3 * C;
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int k = 0; k < C; ++k) row[d * C + k] = acc[d][k];
  }
}

// The runtime's driver entry point (no link against libcuda), or null.
PFN_cuTensorMapEncodeTiled_v12000 tc_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return encode;
}

// The [batch][nx][ny][32] BF16 activations as a tensor map with boxes of rows x cols whole cells,
// swizzled over 64 bytes. False when it cannot be encoded.
bool tc_rows_map(CUtensorMap* map, const void* base, int64_t nx, int64_t ny, int64_t batch, int rows,
                 int cols) {
  const auto encode = tc_encoder();
  if (encode == nullptr || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
  if (nx >= (1ll << 31) || ny >= (1ll << 31) || batch >= (1ll << 31)) return false;
  const cuuint64_t dims[4] = {C, (cuuint64_t)ny, (cuuint64_t)nx, (cuuint64_t)batch};
  const cuuint64_t strides[3] = {64, (cuuint64_t)ny * 64, (cuuint64_t)(nx * ny) * 64};
  const cuuint32_t box[4] = {C, (cuuint32_t)cols, (cuuint32_t)rows, 1};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides,
                box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tiles of kTR x kTC cells for conv32_tc_kernel.
Grid tc_grid(int64_t nx, int64_t ny, int64_t batch) { return tiles_of(nx, ny, batch, kTR, kTC); }

// Which kernel runs layer 2 of the training path (lbm_closure_set_layer2_kernel).
int g_layer2_kernel = LBM_CLOSURE_LAYER2_TCGEN05;

// ---------------------------------------------------------------------------------------------
// Optimiser, relaxation field, coarsening

__global__ void adam_kernel(float* __restrict__ p, bf16* __restrict__ pb, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, float lr, float beta1,
                            float beta2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= LBM_CLOSURE_PARAMS) return;
  const float gi = g[i];
  const float mi = beta1 * m[i] + (1.0f - beta1) * gi;
  const float vi = beta2 * v[i] + (1.0f - beta2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  p[i] = pi;
  pb[i] = to_bf(pi);
}

__global__ void sync_bf16_kernel(const float* __restrict__ p, bf16* __restrict__ pb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < LBM_CLOSURE_PARAMS) pb[i] = to_bf(p[i]);
}

__global__ void omega_kernel(const float* __restrict__ y, const int32_t* __restrict__ flags,
                             int64_t n, float tau0, float gain, float max_dtau,
                             float* __restrict__ omega) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float tau = tau0;
  if (fluid_cell(flags[i])) tau += fminf(max_dtau, gain * fmaxf(y[i], 0.0f));
  omega[i] = 1.0f / tau;
}

__global__ void coarsen_kernel(const float* __restrict__ rho, const float* __restrict__ vel,
                               const float* __restrict__ c, int64_t nx, int64_t ny, int f,
                               float* __restrict__ rho_c, float* __restrict__ vel_c,
                               float* __restrict__ c_c, float* __restrict__ sgs) {
  const int64_t cx_n = nx / f, cy_n = ny / f;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= cx_n * cy_n) return;
  const int64_t cx = i / cy_n, cy = i - cx * cy_n;
  float sr = 0.0f, su = 0.0f, sv = 0.0f, sc = 0.0f;
  for (int a = 0; a < f; ++a)
    for (int b = 0; b < f; ++b) {
      const int64_t j = (cx * f + a) * ny + cy * f + b;
      sr += rho[j];
      su += vel[2 * j];
      sv += vel[2 * j + 1];
      if (c != nullptr) sc += c[j];
    }
  const float inv = 1.0f / (float)(f * f);
  const float mu = su * inv, mv = sv * inv;
  float k = 0.0f;
  for (int a = 0; a < f; ++a)
    for (int b = 0; b < f; ++b) {
      const int64_t j = (cx * f + a) * ny + cy * f + b;
      const float du = vel[2 * j] - mu, dv = vel[2 * j + 1] - mv;
      k = fmaf(du, du, fmaf(dv, dv, k));
    }
  if (rho_c != nullptr) rho_c[i] = sr * inv;
  if (vel_c != nullptr) {
    vel_c[2 * i] = mu;
    vel_c[2 * i + 1] = mv;
  }
  if (c_c != nullptr && c != nullptr) c_c[i] = sc * inv;
  if (sgs != nullptr) sgs[i] = sqrtf(0.5f * k * inv);
}

// ---------------------------------------------------------------------------------------------

int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }

int device_sms() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

bool shape_ok(int64_t nx, int64_t ny, int64_t batch) {
  return nx >= 2 && ny >= 2 && batch >= 1 && nx * ny * batch < (int64_t(1) << 40);
}

// Whether layer 3 takes its low tiles: where they need no more than twice the turns of the high ones at
// two CTAs an SM, that is on small and thin batches. us, low / high: 32 x 32 3.8 / 8.2, 64 x 512 x 2
// 6.5 / 9.5, 3 x 4000 x 8 9.7 / 23.5, 128 x 256 x 4 8.8 / 9.7, 300 x 200 x 4 15.6 / 16.3, 512 x 256 x 2
// 13.0 / 10.1, 1024 x 512 24.8 / 17.3. The same bits.
bool conv3_low(int64_t nx, int64_t ny, int64_t batch, int sms) {
  auto turns = [&](int rows) {
    return (tiles_of(nx, ny, batch, rows, kTY).tiles + 2 * sms - 1) / (2 * sms);
  };
  return turns(kC3Low) <= 2 * turns(kC3R);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

cudaError_t set_smem(const void* fn, size_t bytes) {
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Workspace: [kCountBlocks counts (256 B)][loss partials (kLossBlocks doubles, padded)]
//            [dz2 BF16 [cells][32]][dz1 BF16 [cells][32]][partial rows FP32 [kPartialRows][P]]
constexpr int64_t kWsCount = 0;
constexpr int64_t kWsLoss = 256;
static_assert(kCountBlocks * 8 <= kWsLoss, "the counts must fit");
constexpr int64_t kWsDz = kWsLoss + ((kLossBlocks * 8 + 255) / 256) * 256;

int64_t round256(int64_t v) { return (v + 255) / 256 * 256; }

}  // namespace

extern "C" {

int lbm_postproc_curl2d(const float* vel, int64_t nx, int64_t ny, float* out, void* stream) {
  if (!vel || !out || nx < 2 || ny < 2) return fail(LBM_ERR_ARGUMENT, "curl2d: bad arguments");
  curl2d_kernel<<<blocks_for(nx * ny, 256), 256, 0, (cudaStream_t)stream>>>(vel, nx, ny, out);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_postproc_curl3d(const float* vel, int64_t nx, int64_t ny, int64_t nz, float* out,
                        void* stream) {
  if (!vel || !out || nx < 2 || ny < 2 || nz < 2)
    return fail(LBM_ERR_ARGUMENT, "curl3d: bad arguments");
  curl3d_kernel<<<blocks_for(nx * ny * nz, 256), 256, 0, (cudaStream_t)stream>>>(vel, nx, ny, nz,
                                                                                 out);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_postproc_vmag(const float* vel, int64_t n, int dim, float* out, void* stream) {
  if (!vel || !out || n < 0 || dim < 1 || dim > 3) return fail(LBM_ERR_ARGUMENT, "vmag: bad arguments");
  if (n == 0) return LBM_OK;
  vmag_kernel<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(vel, n, dim, out);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_features(const float* rho, const float* vel, const int32_t* flags, int64_t nx,
                         int64_t ny, int64_t batch, const float* norm, uint16_t* x, void* stream) {
  if (!rho || !vel || !flags || !norm || !x || !shape_ok(nx, ny, batch))
    return fail(LBM_ERR_ARGUMENT, "closure features: bad arguments");
  if (!aligned16(x)) return fail(LBM_ERR_ARGUMENT, "closure features: x must be 16-byte aligned");
  Norm nm;
  for (int c = 0; c < 4; ++c) {
    nm.mean[c] = norm[c];
    nm.inv_std[c] = norm[4 + c];
  }
  features_kernel<<<blocks_for(nx * ny * batch, 256), 256, 0, (cudaStream_t)stream>>>(
      rho, vel, flags, nx, ny, batch, nm, reinterpret_cast<bf16*>(x));
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_forward(const float* params, const uint16_t* params_bf16, const uint16_t* x,
                        int64_t nx, int64_t ny, int64_t batch, float* z1, uint16_t* a1, float* z2,
                        uint16_t* a2, float* y, void* stream) {
  if (!params || !params_bf16 || !x || !a1 || !a2 || !y || !shape_ok(nx, ny, batch))
    return fail(LBM_ERR_ARGUMENT, "closure forward: bad arguments");
  if (!aligned16(params_bf16) || !aligned16(x) || !aligned16(a1) || !aligned16(a2) ||
      (z1 && !aligned16(z1)) || (z2 && !aligned16(z2)))
    return fail(LBM_ERR_ARGUMENT, "closure forward: arrays must be 16-byte aligned");
  static lbm::DeviceOnce once;
  const cudaError_t setup = once([] {
    if (cudaError_t e = set_smem((const void*)conv32_kernel<false>, kConv32Smem)) return e;
    if (cudaError_t e = set_smem((const void*)conv32_kernel<true>, kConv32Smem)) return e;
    if (cudaError_t e = set_smem((const void*)conv32_tc_kernel<false>, kTSmem)) return e;
    if (cudaError_t e = set_smem((const void*)conv3_fwd_kernel<kC3R>, kConv3Smem<kC3R>)) return e;
    if (cudaError_t e = set_smem((const void*)conv3_fwd_kernel<kC3Low>, kConv3Smem<kC3Low>)) return e;
    return cudaSuccess;
  });
  CL_CUDA(setup);
  const Grid g = make_grid(nx, ny, batch);
  const cudaStream_t s = (cudaStream_t)stream;
  const int sms = device_sms();
  const auto* wb = reinterpret_cast<const bf16*>(params_bf16);
  const int grid1 = (int)std::min<int64_t>(g.tiles, (int64_t)sms * kC1PerSm);
  conv1_fwd_kernel<<<grid1, kC1Threads, 0, s>>>(g, reinterpret_cast<const bf16*>(x),
                                              wb + LBM_CLOSURE_OFF_W1, params + LBM_CLOSURE_OFF_B1,
                                              z1, reinterpret_cast<bf16*>(a1));
  CL_CUDA(cudaGetLastError());
  CUtensorMap a1_map;
  if (g_layer2_kernel == LBM_CLOSURE_LAYER2_TCGEN05 && tc_rows_map(&a1_map, a1, nx, ny, batch, kTR + 2, kTC)) {
    const Grid gt = tc_grid(nx, ny, batch);
    const int grid_tc = (int)std::min<int64_t>(gt.tiles, (int64_t)sms);
    conv32_tc_kernel<false><<<grid_tc, kTThreads, kTSmem, s>>>(
        gt, a1_map, wb + LBM_CLOSURE_OFF_W2, params + LBM_CLOSURE_OFF_B2, nullptr, z2,
        reinterpret_cast<bf16*>(a2));
  } else {
    const int grid32 = (int)std::min<int64_t>(g.tiles, (int64_t)sms * 4);
    conv32_kernel<false><<<grid32, kConv32Threads, kConv32Smem, s>>>(
        g, reinterpret_cast<const bf16*>(a1), wb + LBM_CLOSURE_OFF_W2,
        params + LBM_CLOSURE_OFF_B2, nullptr, z2, reinterpret_cast<bf16*>(a2));
  }
  CL_CUDA(cudaGetLastError());
  auto conv3 = [&](auto rows) {
    constexpr int R = decltype(rows)::value;
    const Grid g3 = tiles_of(nx, ny, batch, R, kTY);
    const int grid3 = (int)std::min<int64_t>(g3.tiles, (int64_t)sms * 2);
    conv3_fwd_kernel<R><<<grid3, kC3Threads, kConv3Smem<R>, s>>>(
        g3, reinterpret_cast<const bf16*>(a2), wb + LBM_CLOSURE_OFF_W3, params + LBM_CLOSURE_OFF_B3, y);
  };
  if (conv3_low(nx, ny, batch, sms))
    conv3(std::integral_constant<int, kC3Low>{});
  else
    conv3(std::integral_constant<int, kC3R>{});
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int64_t lbm_closure_workspace_bytes(int64_t nx, int64_t ny, int64_t batch) {
  if (!shape_ok(nx, ny, batch)) return -1;
  const int64_t dz = round256(nx * ny * batch * C * 2);
  return kWsDz + 2 * dz + (int64_t)kPartialRows * LBM_CLOSURE_PARAMS * 4;
}

int lbm_closure_loss(const float* y, const float* target, const int32_t* flags, int64_t nx,
                     int64_t ny, int64_t batch, float* dy, double* loss, void* workspace,
                     void* stream) {
  if (!y || !target || !flags || !dy || !loss || !workspace || !shape_ok(nx, ny, batch))
    return fail(LBM_ERR_ARGUMENT, "closure loss: bad arguments");
  const cudaStream_t s = (cudaStream_t)stream;
  auto* base = static_cast<unsigned char*>(workspace);
  auto* count = reinterpret_cast<unsigned long long*>(base + kWsCount);
  auto* partial = reinterpret_cast<double*>(base + kWsLoss);
  const int64_t n = nx * ny;
  count_kernel<<<kCountBlocks, 1024, 0, s>>>(flags, n, count);
  CL_CUDA(cudaGetLastError());
  loss_kernel<<<kLossBlocks, 256, 0, s>>>(y, target, flags, n, batch, count, dy, partial);
  CL_CUDA(cudaGetLastError());
  loss_final_kernel<<<1, 32, 0, s>>>(partial, kLossBlocks, count, batch, loss);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_backward(const float* params, const uint16_t* params_bf16, const uint16_t* x,
                         const float* z1, const uint16_t* a1, const float* z2, const uint16_t* a2,
                         const float* dy, int64_t nx, int64_t ny, int64_t batch, float* grad,
                         void* workspace, void* stream) {
  if (!params || !params_bf16 || !x || !z1 || !a1 || !z2 || !a2 || !dy || !grad || !workspace ||
      !shape_ok(nx, ny, batch))
    return fail(LBM_ERR_ARGUMENT, "closure backward: bad arguments");
  if (!aligned16(workspace) || !aligned16(params_bf16) || !aligned16(x) || !aligned16(z1) ||
      !aligned16(a1) || !aligned16(z2) || !aligned16(a2))
    return fail(LBM_ERR_ARGUMENT, "closure backward: arrays must be 16-byte aligned");
  static lbm::DeviceOnce once;
  const cudaError_t setup = once([] {
    if (cudaError_t e = set_smem((const void*)conv32_kernel<false>, kConv32Smem)) return e;
    if (cudaError_t e = set_smem((const void*)conv32_kernel<true>, kConv32Smem)) return e;
    if (cudaError_t e = set_smem((const void*)conv32_tc_kernel<true>, kTSmem)) return e;
    if (cudaError_t e = set_smem((const void*)conv32_wgrad_kernel, kDw2Smem)) return e;
    if (cudaError_t e = set_smem((const void*)conv32_wgrad_tc_kernel, kDtSmem)) return e;
    if (cudaError_t e = set_smem((const void*)conv3_bwd_kernel, kConv3BwdSmem)) return e;
    if (cudaError_t e = set_smem((const void*)conv1_wgrad_kernel, kW1Smem)) return e;
    return cudaSuccess;
  });
  CL_CUDA(setup);
  const Grid g = make_grid(nx, ny, batch);
  const cudaStream_t s = (cudaStream_t)stream;
  auto* base = static_cast<unsigned char*>(workspace);
  const int64_t dzb = round256(nx * ny * batch * C * 2);
  auto* dz2 = reinterpret_cast<bf16*>(base + kWsDz);
  auto* dz1 = reinterpret_cast<bf16*>(base + kWsDz + dzb);
  auto* partial = reinterpret_cast<float*>(base + kWsDz + 2 * dzb);
  const auto* wb = reinterpret_cast<const bf16*>(params_bf16);
  const int rows = (int)std::min<int64_t>(g.tiles, kPartialRows);
  const int rows_w2 = (int)std::min<int64_t>(rows, device_sms());
  conv3_bwd_kernel<<<rows, kB3Threads, kConv3BwdSmem, s>>>(g, reinterpret_cast<const bf16*>(a2), z2,
                                                    wb + LBM_CLOSURE_OFF_W3, dy, dz2, partial);
  CL_CUDA(cudaGetLastError());
  CUtensorMap dz2_rows, a1_rows;
  if (g_layer2_kernel == LBM_CLOSURE_LAYER2_TCGEN05 &&
      tc_rows_map(&dz2_rows, dz2, nx, ny, batch, kHX, kTY) &&
      tc_rows_map(&a1_rows, a1, nx, ny, batch, kTX, kTY)) {
    conv32_wgrad_tc_kernel<<<rows_w2, kDtThreads, kDtSmem, s>>>(g, dz2_rows, a1_rows, partial);
  } else {
    conv32_wgrad_kernel<<<rows_w2, kDw2Threads, kDw2Smem, s>>>(g, reinterpret_cast<const bf16*>(a1),
                                                            dz2, partial);
  }
  CL_CUDA(cudaGetLastError());
  CUtensorMap dz2_map;
  if (g_layer2_kernel == LBM_CLOSURE_LAYER2_TCGEN05 && tc_rows_map(&dz2_map, dz2, nx, ny, batch, kTR + 2, kTC)) {
    const Grid gt = tc_grid(nx, ny, batch);
    const int ctas = (int)std::min<int64_t>(gt.tiles, (int64_t)device_sms());
    conv32_tc_kernel<true><<<ctas, kTThreads, kTSmem, s>>>(
        gt, dz2_map, wb + LBM_CLOSURE_OFF_W2, nullptr, z1, nullptr, dz1);
  } else {
    conv32_kernel<true><<<rows, kConv32Threads, kConv32Smem, s>>>(
        g, dz2, wb + LBM_CLOSURE_OFF_W2, nullptr, z1, nullptr, dz1);
  }
  CL_CUDA(cudaGetLastError());
  conv1_wgrad_kernel<<<rows, kW1Threads, kW1Smem, s>>>(
      g, reinterpret_cast<const bf16*>(x), dz1, partial);
  CL_CUDA(cudaGetLastError());
  reduce_rows_kernel<<<blocks_for(LBM_CLOSURE_PARAMS, 32), 256, 0, s>>>(partial, rows, rows_w2, grad);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_adam(float* params, uint16_t* params_bf16, const float* grad, float* m, float* v,
                     float lr, float beta1, float beta2, float eps, int64_t step, void* stream) {
  if (!params || !params_bf16 || !grad || !m || !v || step < 1)
    return fail(LBM_ERR_ARGUMENT, "closure adam: bad arguments");
  const float c1 = (float)(1.0 / (1.0 - std::pow((double)beta1, (double)step)));
  const float c2 = (float)(1.0 / (1.0 - std::pow((double)beta2, (double)step)));
  adam_kernel<<<blocks_for(LBM_CLOSURE_PARAMS, 256), 256, 0, (cudaStream_t)stream>>>(
      params, reinterpret_cast<bf16*>(params_bf16), grad, m, v, lr, beta1, beta2, eps, c1, c2);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_sync_bf16(const float* params, uint16_t* params_bf16, void* stream) {
  if (!params || !params_bf16) return fail(LBM_ERR_ARGUMENT, "closure sync: bad arguments");
  sync_bf16_kernel<<<blocks_for(LBM_CLOSURE_PARAMS, 256), 256, 0, (cudaStream_t)stream>>>(
      params, reinterpret_cast<bf16*>(params_bf16));
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_omega(const float* y, const int32_t* flags, int64_t nx, int64_t ny, float tau0,
                      float gain, float max_dtau, float* omega, void* stream) {
  if (!y || !flags || !omega || nx < 1 || ny < 1 || !(tau0 > 0.5f) || !(max_dtau >= 0.0f))
    return fail(LBM_ERR_ARGUMENT, "closure omega: bad arguments");
  omega_kernel<<<blocks_for(nx * ny, 256), 256, 0, (cudaStream_t)stream>>>(y, flags, nx * ny, tau0,
                                                                         gain, max_dtau, omega);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_relaxation(const float* params, const uint16_t* params_bf16, const float* rho,
                           const float* vel, const int32_t* flags, int64_t nx, int64_t ny,
                           const float* norm, float tau0, float gain, float max_dtau,
                           float* omega, void* stream) {
  if (!params || !params_bf16 || !rho || !vel || !flags || !norm || !omega || nx < 2 || ny < 2 ||
      !(tau0 > 0.5f) || !(max_dtau >= 0.0f))
    return fail(LBM_ERR_ARGUMENT, "closure relaxation: bad arguments");
  if (!aligned16(params_bf16))
    return fail(LBM_ERR_ARGUMENT, "closure relaxation: params_bf16 must be 16-byte aligned");
  static lbm::DeviceOnce once;
  const cudaError_t setup =
      once([] { return set_smem((const void*)closure_fused_kernel, kFusedSmem); });
  CL_CUDA(setup);
  FusedArgs fa;
  fa.params = params;
  fa.wb = reinterpret_cast<const bf16*>(params_bf16);
  fa.rho = rho;
  fa.vel = vel;
  fa.flags = flags;
  fa.nx = nx;
  fa.ny = ny;
  for (int c = 0; c < 4; ++c) {
    fa.norm.mean[c] = norm[c];
    fa.norm.inv_std[c] = norm[4 + c];
  }
  fa.tau0 = tau0;
  fa.gain = gain;
  fa.max_dtau = max_dtau;
  fa.omega = omega;
  fa.tiles_x = (int)((nx + kFR - 1) / kFR);
  fa.tiles_y = (int)((ny + kFC - 1) / kFC);
  const int64_t ntiles = (int64_t)fa.tiles_x * fa.tiles_y;
  const int grid = (int)std::min<int64_t>(ntiles, (int64_t)device_sms());
  closure_fused_kernel<<<grid, kFusedThreads, kFusedSmem, (cudaStream_t)stream>>>(fa);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

int lbm_closure_set_layer2_kernel(int kind) {
  if (kind != LBM_CLOSURE_LAYER2_TCGEN05 && kind != LBM_CLOSURE_LAYER2_WARP_MMA)
    return fail(LBM_ERR_ARGUMENT, "unknown layer-2 kernel");
  g_layer2_kernel = kind;
  return LBM_OK;
}

int lbm_closure_set_spin_limit(int64_t polls) {
  const unsigned v = polls < 0 ? kClosureSpinLimit
                               : (unsigned)std::min<int64_t>(polls, (int64_t)kClosureSpinLimit);
  CL_CUDA(cudaMemcpyToSymbol(g_closure_spin_limit, &v, sizeof(unsigned)));
  return LBM_OK;
}

int lbm_closure_status(void) {
  int word = 0;
  CL_CUDA(cudaMemcpyFromSymbol(&word, g_closure_status, sizeof(int)));
  if (word == 0) return LBM_OK;
  const int zero = 0;
  CL_CUDA(cudaMemcpyToSymbol(g_closure_status, &zero, sizeof(int)));
  return fail(LBM_ERR_STATE,
              "closure: a kernel gave up waiting for its copies or tensor-core products");
}

int lbm_closure_coarsen(const float* rho, const float* vel, const float* c, int64_t nx, int64_t ny,
                        int factor, float* rho_c, float* vel_c, float* c_c, float* sgs,
                        void* stream) {
  if (!rho || !vel || factor < 1 || nx % factor != 0 || ny % factor != 0 || nx < 1 || ny < 1)
    return fail(LBM_ERR_ARGUMENT, "closure coarsen: nx and ny must be multiples of the factor");
  const int64_t n = (nx / factor) * (ny / factor);
  coarsen_kernel<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(rho, vel, c, nx, ny, factor,
                                                                       rho_c, vel_c, c_c, sgs);
  CL_CUDA(cudaGetLastError());
  return LBM_OK;
}

}  // extern "C"
