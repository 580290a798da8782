// Learned initial guess for the Newton inversion: a small MLP
// (3 (P+1)^3 + 3 -> 128 -> 128 -> 3, GELU) mapping an order-P hex element's
// control points plus a physical point to a reference-space guess: 84
// inputs at order 2 (27 control points), 195 at order 3 (64).  No counterpart
// in the reference; it feeds DRB_GUESS_GIVEN, with plain Newton from the
// element centre as the fallback whenever the guessed solve fails.
//
// Tensor-core kernels (tcgen05 / UMMA, BF16 operands, FP32 accumulation in
// tensor memory):
//   net_kernel        forward pass or a whole training step (forward, loss,
//                     backward, weight gradients) per tile of 128 rows, one
//                     launch; reduce_kernel adds the CTAs' gradients
//   mlp_guess_kernel  fused inference: per tile of 128 (point, element)
//                     pairs, features are built in shared memory, two UMMA
//                     GEMMs run with the weights resident in shared memory,
//                     the 128 -> 3 head runs on the CUDA cores
// Every mbarrier wait is bounded; on timeout the kernel records an error
// flag, frees its tensor memory and returns.
#include <cuda_bf16.h>

#include <cstdio>

#include "bernstein.cuh"
#include "drb_common.cuh"
#include "drb_internal.h"
#include "umma.cuh"

namespace drb
{
namespace mlp
{

constexpr int kHid = 128;
constexpr int kOut = 3;

// Dimensions and parameter layout of the network for order-P hex elements.
// Inputs: the (P+1)^3 control points' 3 coordinates, then the point; K
// padded to a multiple of 16 for the UMMA K steps.  Parameters, in one fp32
// vector: W1 [128 x kIn], b1, W2 [128 x 128], b2, W3 [3 x 128], b3.  bf16
// operand copies: W1 [128 x kInPad], W2 (the kernels read it both ways).
template <int P> struct Net
{
  static constexpr int kNd = (P + 1) * (P + 1) * (P + 1);
  static constexpr int kCoords = 3 * kNd;
  static constexpr int kIn = kCoords + 3;
  static constexpr int kInPad = (kIn + 15) / 16 * 16;
  static constexpr int kW1 = 0;
  static constexpr int kB1 = kW1 + kHid * kIn;
  static constexpr int kW2 = kB1 + kHid;
  static constexpr int kB2 = kW2 + kHid * kHid;
  static constexpr int kW3 = kB2 + kHid;
  static constexpr int kB3 = kW3 + kOut * kHid;
  static constexpr int kParams = kB3 + kOut;
  static constexpr int kBW1 = 0;
  static constexpr int kBW2 = kBW1 + kHid * kInPad;
  static constexpr int kBf16 = kBW2 + kHid * kHid;
  // packed geometry rows: kCoords relative coordinates, then the origin
  static constexpr int kRowF4 = packed_stride (kNd, 3) / 4;
  // activation tile width: the layer-1 input, then the layer-2 input in
  // the same bytes
  static constexpr int kActW = kInPad > kHid ? kInPad : kHid;
  // 128-row tiles in flight per CTA in the fused inference (shared memory:
  // W1, W2 and one activation tile per group within 227 KB)
  static constexpr int kGroups = kActW > kHid ? 2 : 4;
};
static_assert (Net<2>::kIn == 84 && Net<2>::kInPad == 96 && Net<3>::kIn == 195 &&
               Net<3>::kInPad == 208, "network input widths");
static_assert (packed_origin (27) == 81 && packed_origin (64) == 192,
               "geometry rows: relative coordinates, then the origin");

constexpr uint32_t kWaitTries = 1u << 22;

// tanh on the special-function unit (PTX tanh.approx.f32, relative error
// about 2^-11): one instruction instead of a libm-style evaluation, and
// well below the bf16 rounding the activations go through.
DRB_D float tanh_sfu (float x)
{
  float y;
  asm ("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// GELU, tanh form: 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3)))
DRB_D float gelu (float x)
{
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.f + tanh_sfu (u));
}
DRB_D float gelu_grad (float x)
{
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  const float t = tanh_sfu (u);
  const float du = 0.7978845608028654f * (1.f + 3.f * 0.044715f * x * x);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}

// Features of one (element, point) pair: control points and point relative
// to the centre of the element's control-point box, scaled by its largest
// half-extent.  (P+1)^3 x 3 control coordinates, then the point, then zeros.
// The packed row holds the relative coordinates, then the origin O, 16-byte
// aligned, so it is read as float4.

// Centre and inverse largest half-extent of the control-point box.
template <int P> DRB_D void pair_frame (const float *__restrict__ row, float (&c)[3], float &inv)
{
  const float4 *r4 = reinterpret_cast<const float4 *> (row);
  float mn[3] = { INFINITY, INFINITY, INFINITY }, mx[3] = { -INFINITY, -INFINITY, -INFINITY };
#pragma unroll
  for (int j = 0; j < Net<P>::kRowF4; ++j)
  {
    const float4 v4 = __ldg (r4 + j);
    const float v[4] = { v4.x, v4.y, v4.z, v4.w };
#pragma unroll
    for (int t = 0; t < 4; ++t)
    {
      const int q = 4 * j + t;
      if (q < Net<P>::kCoords)
      {
        mn[q % 3] = fminf (mn[q % 3], v[t]);
        mx[q % 3] = fmaxf (mx[q % 3], v[t]);
      }
    }
  }
  float h = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    c[k] = 0.5f * (mn[k] + mx[k]);
    h = fmaxf (h, 0.5f * (mx[k] - mn[k]));
  }
  inv = h > 0.f ? 1.f / h : 0.f;
}

// Features [8 k8, 8 k8 + 8) of one pair as eight packed bf16.  The point
// enters in the row's frame, pt - O (O follows the coordinates in the row).
template <int P>
DRB_D uint4 pair_features8 (const float *__restrict__ row, const float (&pt)[3], const float (&c)[3],
                            float inv, int k8)
{
  constexpr int RF = 4 * Net<P>::kRowF4;
  const int f0 = 8 * k8;
  const float4 z4 = make_float4 (0.f, 0.f, 0.f, 0.f);
  const float4 a = f0 < RF ? __ldg (reinterpret_cast<const float4 *> (row) + 2 * k8) : z4;
  const float4 b = f0 + 4 < RF ? __ldg (reinterpret_cast<const float4 *> (row) + 2 * k8 + 1) : z4;
  float v[8] = { a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w };
#pragma unroll
  for (int t = 0; t < 8; ++t)
  {
    const int q = f0 + t;
    if (q >= Net<P>::kIn) v[t] = 0.f;
    else if (q >= Net<P>::kCoords) v[t] = __fsub_rn (pt[q - Net<P>::kCoords], v[t]);
  }
#pragma unroll
  for (int t = 0; t < 8; ++t)
  {
    const int q = f0 + t;
    if (q < Net<P>::kIn) v[t] = (v[t] - c[q % 3]) * inv;
  }
  uint4 out;
  __nv_bfloat162 p0 = __floats2bfloat162_rn (v[0], v[1]), p1 = __floats2bfloat162_rn (v[2], v[3]);
  __nv_bfloat162 p2 = __floats2bfloat162_rn (v[4], v[5]), p3 = __floats2bfloat162_rn (v[6], v[7]);
  out.x = *reinterpret_cast<uint32_t *> (&p0);
  out.y = *reinterpret_cast<uint32_t *> (&p1);
  out.z = *reinterpret_cast<uint32_t *> (&p2);
  out.w = *reinterpret_cast<uint32_t *> (&p3);
  return out;
}

// ------------------------------------------------------------ prepare --

template <int P>
__global__ void prepare_kernel (const float *__restrict__ p, __nv_bfloat16 *__restrict__ wb)
{
  using N = Net<P>;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < kHid * N::kInPad)
  {
    const int r = t / N::kInPad, k = t - r * N::kInPad;
    wb[N::kBW1 + t] = __float2bfloat16_rn (k < N::kIn ? p[N::kW1 + r * N::kIn + k] : 0.f);
  }
  if (t < kHid * kHid) wb[N::kBW2 + t] = __float2bfloat16_rn (p[N::kW2 + t]);
}

// ----------------------------------------------------------- features --

template <int P>
__global__ void features_kernel (const float *__restrict__ packed, int stride,
                                 const int *__restrict__ elem, const float *__restrict__ pts, int n,
                                 int n_pad, __nv_bfloat16 *__restrict__ X)
{
  using N = Net<P>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pad) return;
  const int e = i < n ? elem[i] : -1;
  uint4 *dst = reinterpret_cast<uint4 *> (X + (size_t)i * N::kInPad);
  if (e < 0)
  {
#pragma unroll
    for (int k8 = 0; k8 < N::kInPad / 8; ++k8) dst[k8] = make_uint4 (0u, 0u, 0u, 0u);
    return;
  }
  const float *row = packed + (size_t)e * stride;
  const float pt[3] = { pts[3 * (size_t)i], pts[3 * (size_t)i + 1], pts[3 * (size_t)i + 2] };
  float c[3], inv;
  pair_frame<P> (row, c, inv);
#pragma unroll
  for (int k8 = 0; k8 < N::kInPad / 8; ++k8) dst[k8] = pair_features8<P> (row, pt, c, inv, k8);
}

// ---------------------------------------------- fused network evaluation --
//
// One kernel for the forward pass and for a training step.  A CTA of 16
// warps takes tiles of 128 rows.  The activations of a tile never leave the
// SM: the layer outputs are one accumulator of 128 TMEM columns, read by four
// warpgroups (32 columns each, a thread per row), and every matrix operand
// is a bf16 tile in shared memory that is used both ways, as it lies
// (K-major) and transposed (MN-major), so no transposes are made:
//   Z1 = X W1^T              H1 = gelu (Z1 + b1)
//   Z2 = H1 W2^T             head, loss, dY, dZ2 = (W3^T dY) gelu'(Z2 + b2)
//   dH1 = dZ2 W2             dZ1 = dH1 gelu'(Z1 + b1)
//   dW2 += dZ2^T H1          dW1 += dZ1^T X
// dW1 and dW2 stay in TMEM over the CTA's tiles; at its end every CTA
// writes its sums to a slot of its own and reduce_kernel adds the slots in
// order, so the gradients do not depend on the schedule.  The first form
// (a GEMM kernel per product, 15 launches a step) kept Z and H in DRAM with
// row-per-thread stores and transposed four matrices for the weight
// gradients.
// 16,384 rows at order 2: 27 us with the reduction, against 363; bound by
// the chain of one tile per CTA (loads, four MMA groups, four epilogues).

struct NetArgs
{
  const float *params;
  const __nv_bfloat16 *wb;
  const __nv_bfloat16 *X;
  const float *target;
  const float *weight;
  int n, tiles;
  float inv_count;
  float *y_out;
  float *partials; // partial_stride<P> () floats per CTA: the gradient, then the loss
  int *err;
};

constexpr int kNetThreads = 512;
constexpr int kNetGroups = 4; // warpgroups, 32 columns each

template <int P> constexpr int partial_stride () { return (Net<P>::kParams + 1 + 3) / 4 * 4; }
template <int P> constexpr size_t net_smem ()
{
  return (size_t)2 * 2 * 128 * Net<P>::kInPad + (size_t)3 * 2 * 128 * kHid;
}
static_assert (net_smem<1> () <= 200 * 1024 && net_smem<2> () <= 200 * 1024 &&
               net_smem<3> () <= 200 * 1024, "the network's tiles fit beside the static arrays");
static_assert (2 * kHid + Net<3>::kInPad <= 512, "accumulators fit in tensor memory");

// Sums of 16 values over the warp's lanes: the sum of v[c] for c = lane & 15
// (halving the columns a lane keeps at each step: 16 shuffles, not 80).
DRB_D float column_sums (float (&v)[16], int lane)
{
#pragma unroll
  for (int s = 8; s > 0; s >>= 1)
#pragma unroll
    for (int k = 0; k < s; ++k)
    {
      const bool upper = lane & s;
      const float give = upper ? v[k] : v[k + s];
      const float keep = upper ? v[k + s] : v[k];
      v[k] = keep + __shfl_xor_sync (0xffffffffu, give, s);
    }
  return v[0] + __shfl_xor_sync (0xffffffffu, v[0], 16);
}

DRB_D uint32_t pack_bf16 (float a, float b)
{
  __nv_bfloat162 h = __floats2bfloat162_rn (a, b);
  return *reinterpret_cast<uint32_t *> (&h);
}

// Columns [c0, c0 + 16) of a row of a 128-wide operand tile.
DRB_D void store_row16 (unsigned char *tile, int row, int c0, const float (&v)[16])
{
#pragma unroll
  for (int q = 0; q < 2; ++q)
    *reinterpret_cast<uint4 *> (tile + umma::tile_offset (row, c0 + 8 * q, kHid)) =
    make_uint4 (pack_bf16 (v[8 * q], v[8 * q + 1]), pack_bf16 (v[8 * q + 2], v[8 * q + 3]),
                pack_bf16 (v[8 * q + 4], v[8 * q + 5]), pack_bf16 (v[8 * q + 6], v[8 * q + 7]));
}

// A 128-row operand tile from row-major bf16 rows.  Consecutive lanes take
// consecutive rows, so their 16-byte stores fill whole core matrices.
template <int W> DRB_D void load_tile (unsigned char *tile, const __nv_bfloat16 *__restrict__ rows, int tid)
{
  for (int v = tid; v < 128 * (W / 8); v += kNetThreads)
  {
    const int r = v & 127, j = v >> 7;
    *reinterpret_cast<uint4 *> (tile + umma::tile_offset (r, 8 * j, W)) =
    __ldg (reinterpret_cast<const uint4 *> (rows + (size_t)r * W) + j);
  }
}

template <int P, bool TRAIN>
__global__ void __launch_bounds__ (kNetThreads, 1) net_kernel (NetArgs a)
{
  using N = Net<P>;
  constexpr int kInPad = N::kInPad;
  extern __shared__ __align__ (1024) unsigned char smem[];
  unsigned char *sX = smem;
  unsigned char *sW1 = sX + 2 * 128 * kInPad;
  unsigned char *sW2 = sW1 + 2 * 128 * kInPad;
  unsigned char *sH = sW2 + 2 * 128 * kHid; // H1, then dZ1
  unsigned char *sZ = sH + 2 * 128 * kHid;  // dZ2
  __shared__ float s_b1[kHid], s_b2[kHid], s_w3[kOut * kHid], s_b3[kOut];
  __shared__ float s_y[kNetGroups][128][kOut];
  __shared__ float s_sum[kNetThreads / 32][5][32];
  __shared__ __align__ (8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = warp >> 2;   // this warpgroup's columns: [32 g, 32 g + 32)
  const int row = tid & 127; // this thread's row = TMEM lane
  load_tile<kInPad> (sW1, a.wb + N::kBW1, tid);
  load_tile<kHid> (sW2, a.wb + N::kBW2, tid);
  if (tid < kHid)
  {
    s_b1[tid] = a.params[N::kB1 + tid];
    s_b2[tid] = a.params[N::kB2 + tid];
  }
  if (tid < kOut * kHid) s_w3[tid] = a.params[N::kW3 + tid];
  if (tid < kOut) s_b3[tid] = a.params[N::kB3 + tid];
  if (warp == 0) umma::tmem_alloc (&tmem_base, 512);
  if (tid == 0) umma::mbar_init (&mbar, 1);
  umma::fence_before_sync ();
  __syncthreads ();
  umma::fence_after_sync ();
  const uint32_t tD = tmem_base, tW2 = tD + kHid, tW1 = tD + 2 * kHid;
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t tmine = tD + lane_off + 32 * g;
  const uint32_t aX = umma::smem_addr (sX), aW1 = umma::smem_addr (sW1), aW2 = umma::smem_addr (sW2),
                 aH = umma::smem_addr (sH), aZ = umma::smem_addr (sZ);
  constexpr uint32_t kD = umma::idesc_bf16_f32 (128, kHid);
  uint32_t phase = 0;
  bool ok = true;
  // running column sums: dZ2 and the three dY x H2 products, then dZ1, per
  // 16-column half (this lane's column is lane & 15)
  float sums[2][5] = { { 0.f, 0.f, 0.f, 0.f, 0.f }, { 0.f, 0.f, 0.f, 0.f, 0.f } };
  float db3[kOut] = { 0.f, 0.f, 0.f };
  float loss = 0.f;
  bool first = true;

  for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x)
  {
    const int i = tile * 128 + row;
    load_tile<kInPad> (sX, a.X + (size_t)tile * 128 * kInPad, tid);
    umma::fence_async_smem ();
    __syncthreads ();
    if (tid == 0)
    {
      umma::fence_after_sync ();
#pragma unroll
      for (int kk = 0; kk < kInPad / 16; ++kk)
        umma::mma_bf16 (tD, umma::desc_rows (aX, kInPad, kk), umma::desc_rows (aW1, kInPad, kk), kD,
                        kk > 0 ? 1u : 0u);
      umma::mma_commit (&mbar);
    }
    ok = __syncthreads_and (umma::mbar_wait (&mbar, phase, kWaitTries));
    phase ^= 1u;
    umma::fence_after_sync ();
    if (!ok) break;
    // H1 = gelu (Z1 + b1); gelu'(Z1 + b1) is kept for the backward pass
    float dg1[2][16];
#pragma unroll
    for (int half = 0; half < 2; ++half)
    {
      const int c0 = 32 * g + 16 * half;
      float d[16];
      umma::tmem_ld16 (tmine + 16 * half, d);
#pragma unroll
      for (int j = 0; j < 16; ++j)
      {
        const float z = d[j] + s_b1[c0 + j];
        d[j] = gelu (z);
        if (TRAIN) dg1[half][j] = gelu_grad (z);
      }
      store_row16 (sH, row, c0, d);
    }
    umma::fence_async_smem ();
    umma::fence_before_sync ();
    __syncthreads ();
    if (tid == 0)
    {
      umma::fence_after_sync ();
#pragma unroll
      for (int kk = 0; kk < kHid / 16; ++kk)
        umma::mma_bf16 (tD, umma::desc_rows (aH, kHid, kk), umma::desc_rows (aW2, kHid, kk), kD,
                        kk > 0 ? 1u : 0u);
      umma::mma_commit (&mbar);
    }
    ok = __syncthreads_and (umma::mbar_wait (&mbar, phase, kWaitTries));
    phase ^= 1u;
    umma::fence_after_sync ();
    if (!ok) break;
    // head: y = W3 gelu (Z2 + b2) + b3, a part per warpgroup
    float y[kOut] = { 0.f, 0.f, 0.f };
#pragma unroll
    for (int half = 0; half < 2; ++half)
    {
      const int c0 = 32 * g + 16 * half;
      float d[16];
      umma::tmem_ld16 (tmine + 16 * half, d);
#pragma unroll
      for (int j = 0; j < 16; ++j)
      {
        const float h = gelu (d[j] + s_b2[c0 + j]);
#pragma unroll
        for (int o = 0; o < kOut; ++o) y[o] = fmaf (s_w3[o * kHid + c0 + j], h, y[o]);
      }
    }
#pragma unroll
    for (int o = 0; o < kOut; ++o) s_y[g][row][o] = y[o];
    __syncthreads ();
    const float w = TRAIN && i < a.n ? (a.weight ? __ldg (a.weight + i) : 1.f) : 0.f;
    float dy[kOut];
#pragma unroll
    for (int o = 0; o < kOut; ++o)
    {
      const float yo = ((s_y[0][row][o] + s_y[1][row][o]) + (s_y[2][row][o] + s_y[3][row][o])) + s_b3[o];
      const float e = TRAIN && i < a.n ? yo - __ldg (a.target + 3 * (size_t)i + o) : 0.f;
      dy[o] = 2.f * w * e * a.inv_count;
      if (g == 0)
      {
        loss += w * e * e * a.inv_count;
        db3[o] += dy[o];
        if (!TRAIN && i < a.n) a.y_out[3 * (size_t)i + o] = yo;
      }
    }
    if (TRAIN)
    {
      // dZ2 and its sums
#pragma unroll
      for (int half = 0; half < 2; ++half)
      {
        const int c0 = 32 * g + 16 * half;
        float h[16], v[16];
        umma::tmem_ld16 (tmine + 16 * half, h);
#pragma unroll
        for (int j = 0; j < 16; ++j)
        {
          const float z = h[j] + s_b2[c0 + j];
          float dh = 0.f;
#pragma unroll
          for (int o = 0; o < kOut; ++o) dh = fmaf (s_w3[o * kHid + c0 + j], dy[o], dh);
          v[j] = dh * gelu_grad (z);
          h[j] = gelu (z);
        }
        store_row16 (sZ, row, c0, v);
        sums[half][0] += column_sums (v, lane);
#pragma unroll
        for (int o = 0; o < kOut; ++o)
        {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = dy[o] * h[j];
          sums[half][1 + o] += column_sums (v, lane);
        }
      }
      umma::fence_async_smem ();
      umma::fence_before_sync ();
      __syncthreads ();
      if (tid == 0)
      {
        umma::fence_after_sync ();
#pragma unroll
        for (int kk = 0; kk < kHid / 16; ++kk)
          umma::mma_bf16 (tD, umma::desc_rows (aZ, kHid, kk), umma::desc_cols (aW2, kHid, kk),
                          umma::idesc_bf16_f32 (128, kHid, false, true), kk > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < 128 / 16; ++kk)
          umma::mma_bf16 (tW2, umma::desc_cols (aZ, kHid, kk), umma::desc_cols (aH, kHid, kk),
                          umma::idesc_bf16_f32 (128, kHid, true, true), first && kk == 0 ? 0u : 1u);
        umma::mma_commit (&mbar);
      }
      ok = __syncthreads_and (umma::mbar_wait (&mbar, phase, kWaitTries));
      phase ^= 1u;
      umma::fence_after_sync ();
      if (!ok) break;
      // dZ1 over H1, which dW2 has read
#pragma unroll
      for (int half = 0; half < 2; ++half)
      {
        const int c0 = 32 * g + 16 * half;
        float d[16];
        umma::tmem_ld16 (tmine + 16 * half, d);
#pragma unroll
        for (int j = 0; j < 16; ++j) d[j] *= dg1[half][j];
        store_row16 (sH, row, c0, d);
        sums[half][4] += column_sums (d, lane);
      }
      umma::fence_async_smem ();
      umma::fence_before_sync ();
      __syncthreads ();
      if (tid == 0)
      {
        umma::fence_after_sync ();
#pragma unroll
        for (int kk = 0; kk < 128 / 16; ++kk)
          umma::mma_bf16 (tW1, umma::desc_cols (aH, kHid, kk), umma::desc_cols (aX, kInPad, kk),
                          umma::idesc_bf16_f32 (128, kInPad, true, true), first && kk == 0 ? 0u : 1u);
        umma::mma_commit (&mbar);
      }
      ok = __syncthreads_and (umma::mbar_wait (&mbar, phase, kWaitTries));
      phase ^= 1u;
      umma::fence_after_sync ();
      if (!ok) break;
    }
    else
    {
      // the next tile writes s_y and the accumulator again
      umma::fence_before_sync ();
      __syncthreads ();
      umma::fence_after_sync ();
    }
    first = false;
  }
  if (!ok && tid == 0 && a.err) atomicExch (a.err, 1);
  if (TRAIN)
  {
    // this CTA's sums to its slot; where a wait ran out, zeros for the matrices and
    // the finished tiles' sums for the rest (*err says that the step is void)
    float *out = a.partials + (size_t)blockIdx.x * partial_stride<P> ();
#pragma unroll 1
    for (int c0 = 32 * g; c0 < kHid + kInPad; c0 += 32 * kNetGroups)
    {
      // W2's columns, then W1's
      float d[32];
      umma::tmem_ld32 (tW2 + lane_off + c0, d);
      const bool w2 = c0 < kHid;
      float *dst = out + (w2 ? N::kW2 + row * kHid + c0 : N::kW1 + row * N::kIn + c0 - kHid);
      const int limit = w2 ? 32 : min (32, N::kIn - (c0 - kHid));
      if (w2 || N::kIn % 4 == 0) // 16-byte aligned: every offset is a multiple of 4
      {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          if (j < limit)
            *reinterpret_cast<float4 *> (dst + j) =
            ok ? make_float4 (d[j], d[j + 1], d[j + 2], d[j + 3]) : make_float4 (0.f, 0.f, 0.f, 0.f);
      }
      else
      {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < limit) dst[j] = ok ? d[j] : 0.f;
      }
    }
    // sums over the four warps of a warpgroup, rows in order
#pragma unroll
    for (int q = 0; q < 5; ++q) s_sum[warp][q][lane] = lane < 16 ? sums[0][q] : sums[1][q];
    float *s_tail = &s_y[0][0][0]; // loss, db3 per warp of group 0
    __syncthreads ();
    if (g == 0)
    {
      float t[4] = { loss, db3[0], db3[1], db3[2] };
#pragma unroll
      for (int q = 0; q < 4; ++q)
      {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t[q] += __shfl_xor_sync (0xffffffffu, t[q], o);
        if (lane == 0) s_tail[4 * warp + q] = t[q];
      }
    }
    __syncthreads ();
    if (tid < kHid)
    {
      const int w0 = 4 * (tid >> 5); // the warps that hold this column
      float t[5];
#pragma unroll
      for (int q = 0; q < 5; ++q)
        t[q] = (s_sum[w0][q][lane] + s_sum[w0 + 1][q][lane]) + (s_sum[w0 + 2][q][lane] + s_sum[w0 + 3][q][lane]);
      out[N::kB2 + tid] = t[0];
#pragma unroll
      for (int o = 0; o < kOut; ++o) out[N::kW3 + o * kHid + tid] = t[1 + o];
      out[N::kB1 + tid] = t[4];
    }
    if (tid < 4)
    {
      const float t = (s_tail[tid] + s_tail[4 + tid]) + (s_tail[8 + tid] + s_tail[12 + tid]);
      out[tid == 0 ? N::kParams : N::kB3 + tid - 1] = t;
    }
  }
  umma::fence_before_sync ();
  __syncthreads ();
  if (warp == 0) umma::tmem_dealloc (tmem_base, 512);
}

// Gradient and loss: the sum of the CTAs' slots.  A block takes 128
// consecutive values; 32 threads read them as float4, 8 rows of threads
// share the slots.
__global__ void __launch_bounds__ (256)
reduce_kernel (const float *__restrict__ partials, int slots, int stride, int n_params,
               float *__restrict__ grad, float *__restrict__ loss)
{
  __shared__ float4 s[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int at = blockIdx.x * 128 + 4 * tx;
  float4 acc = make_float4 (0.f, 0.f, 0.f, 0.f);
  if (at < stride)
  {
#pragma unroll 8
    for (int q = ty; q < slots; q += 8)
    {
      const float4 v = __ldg (reinterpret_cast<const float4 *> (partials + (size_t)q * stride + at));
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
  }
  s[ty][tx] = acc;
  __syncthreads ();
  if (threadIdx.x < 128)
  {
    const int v = blockIdx.x * 128 + threadIdx.x;
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += reinterpret_cast<const float *> (s[q])[threadIdx.x];
    if (v < n_params) grad[v] = t;
    else if (v == n_params && loss) loss[0] = t;
  }
}

__global__ void adam_kernel (float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                             float *__restrict__ v, int n, float lr, float b1, float b2, float eps,
                             float c1, float c2)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi * c1) / (sqrtf (vi * c2) + eps);
}

// ------------------------------------------------------ fused inference --

struct GuessArgs
{
  const float *params;
  const __nv_bfloat16 *wb;
  const float *packed;
  int stride;
  const int *elem;
  const float *pts;
  const int *order;
  int n;
  float *guess;
  int *err;
};

// Fused inference keeps Net<P>::kGroups 128-row tiles in flight per CTA
// (four at orders 1-2, two at order 3, whose 208-wide layer-1 input needs
// wider tiles), one per warpgroup, with the bf16 weights resident once per
// CTA.  Each warpgroup owns one activation tile (the layer-1 input, then
// the 128-wide layer-2 input in the same bytes) and 128 TMEM columns (D1,
// then D2 in the same columns), and synchronises only with itself (named
// barrier 1 + g), so one group's gathers and epilogues overlap the others'
// MMAs.
template <int P> constexpr size_t guess_w1_bytes () { return (size_t)kHid * Net<P>::kInPad * 2; }
constexpr size_t guess_w2_bytes () { return (size_t)kHid * kHid * 2; }
template <int P> constexpr size_t guess_act_bytes () { return (size_t)128 * Net<P>::kActW * 2; }
template <int P> constexpr size_t guess_smem ()
{
  return guess_w1_bytes<P> () + guess_w2_bytes () + Net<P>::kGroups * guess_act_bytes<P> ();
}
static_assert (guess_smem<3> () <= 227 * 1024 && guess_smem<2> () <= 227 * 1024 &&
               guess_smem<1> () <= 227 * 1024, "fused inference fits in shared memory");

DRB_D void group_sync (int g)
{
  asm volatile ("bar.sync %0, %1;" ::"r"(1 + g), "r"(128) : "memory");
}
// AND of a predicate over the 128 threads of warpgroup g.
DRB_D bool group_and (int g, bool v)
{
  uint32_t r;
  asm volatile ("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\t"
                "bar.red.and.pred p, %2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                : "=r"(r)
                : "r"((uint32_t)v), "r"(1 + g)
                : "memory");
  return r != 0;
}

template <int P>
__global__ void __launch_bounds__ (128 * Net<P>::kGroups, 1) mlp_guess_kernel (GuessArgs a)
{
  using N = Net<P>;
  constexpr int kGuessGroups = N::kGroups;
  constexpr int kGuessThreads = 128 * kGuessGroups;
  constexpr int kInPad = N::kInPad;
  constexpr size_t kGuessW1 = guess_w1_bytes<P> ();
  constexpr size_t kGuessW2 = guess_w2_bytes ();
  constexpr size_t kGuessAct = guess_act_bytes<P> ();
  extern __shared__ __align__ (1024) unsigned char smem[];
  unsigned char *sW1 = smem;                     // 128 x 96
  unsigned char *sW2 = sW1 + kGuessW1;           // 128 x 128
  __shared__ float s_b1[kHid], s_b2[kHid], s_w3[kOut * kHid], s_b3[kOut];
  __shared__ __align__ (8) uint64_t mbar[kGuessGroups];
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int g = warp >> 2;              // warpgroup = tile slot
  const int row = tid & 127;            // row of the tile = TMEM lane
  unsigned char *sAct = sW2 + kGuessW2 + (size_t)g * kGuessAct;
  for (int v = tid; v < kHid * (kInPad / 8); v += kGuessThreads)
  {
    const int r = v / (kInPad / 8), j = v - r * (kInPad / 8);
    *reinterpret_cast<uint4 *> (sW1 + umma::tile_offset (r, 8 * j, kInPad)) =
    *reinterpret_cast<const uint4 *> (a.wb + N::kBW1 + (size_t)r * kInPad + 8 * j);
  }
  for (int v = tid; v < kHid * (kHid / 8); v += kGuessThreads)
  {
    const int r = v / (kHid / 8), j = v - r * (kHid / 8);
    *reinterpret_cast<uint4 *> (sW2 + umma::tile_offset (r, 8 * j, kHid)) =
    *reinterpret_cast<const uint4 *> (a.wb + N::kBW2 + (size_t)r * kHid + 8 * j);
  }
  for (int q = tid; q < kHid; q += kGuessThreads)
  {
    s_b1[q] = a.params[N::kB1 + q];
    s_b2[q] = a.params[N::kB2 + q];
  }
  for (int q = tid; q < kOut * kHid; q += kGuessThreads) s_w3[q] = a.params[N::kW3 + q];
  if (tid < kOut) s_b3[tid] = a.params[N::kB3 + tid];
  if (warp == 0) umma::tmem_alloc (&tmem_base, kGuessGroups * kHid);
  if (tid < kGuessGroups) umma::mbar_init (&mbar[tid], 1);
  umma::fence_before_sync ();
  __syncthreads ();
  umma::fence_after_sync ();
  // warp w reads TMEM lanes [32 (w % 4), +32); its group's columns start at 128 g
  const uint32_t tacc = tmem_base + (uint32_t)(g * kHid) + ((uint32_t)((warp & 3) * 32) << 16);
  const uint32_t tmma = tmem_base + (uint32_t)(g * kHid);
  const uint32_t idesc = umma::idesc_bf16_f32 (128, kHid);
  uint32_t phase = 0;
  bool ok = true;
  const int tiles = (a.n + 127) / 128;
  for (int tile = blockIdx.x * kGuessGroups + g; tile < tiles; tile += gridDim.x * kGuessGroups)
  {
    const int i = tile * 128 + row;
    const int q = i < a.n ? (a.order ? __ldg (a.order + i) : i) : -1;
    const int e = q >= 0 ? __ldg (a.elem + q) : -1;
    float pt[3] = { 0.f, 0.f, 0.f };
    // layer-1 input row: features in the 96-wide interleaved layout
    if (e >= 0)
    {
      pt[0] = __ldg (a.pts + 3 * (size_t)q);
      pt[1] = __ldg (a.pts + 3 * (size_t)q + 1);
      pt[2] = __ldg (a.pts + 3 * (size_t)q + 2);
      const float *er = a.packed + (size_t)e * a.stride;
      float c[3], inv;
      pair_frame<P> (er, c, inv);
#pragma unroll
      for (int k8 = 0; k8 < kInPad / 8; ++k8)
        *reinterpret_cast<uint4 *> (sAct + umma::tile_offset (row, 8 * k8, kInPad)) =
        pair_features8<P> (er, pt, c, inv, k8);
    }
    else
    {
#pragma unroll
      for (int k8 = 0; k8 < kInPad / 8; ++k8)
        *reinterpret_cast<uint4 *> (sAct + umma::tile_offset (row, 8 * k8, kInPad)) =
        make_uint4 (0u, 0u, 0u, 0u);
    }
    umma::fence_async_smem ();
    group_sync (g);
    if (row == 0)
    {
      umma::fence_after_sync ();
      const uint32_t a0 = umma::smem_addr (sAct), b0 = umma::smem_addr (sW1);
#pragma unroll
      for (int kk = 0; kk < kInPad / 16; ++kk)
        umma::mma_bf16 (tmma, umma::desc_kmajor (a0 + kk * 256, 128, (kInPad / 8) * 128),
                        umma::desc_kmajor (b0 + kk * 256, 128, (kInPad / 8) * 128), idesc,
                        kk > 0 ? 1u : 0u);
      umma::mma_commit (&mbar[g]);
    }
    ok = group_and (g, umma::mbar_wait (&mbar[g], phase, kWaitTries));
    phase ^= 1u;
    umma::fence_after_sync ();
    if (!ok) break;
    // layer-1 epilogue: GELU(D1 + b1) as bf16 -> layer-2 input (same bytes)
#pragma unroll 1
    for (int c0 = 0; c0 < kHid; c0 += 32)
    {
      float d[32];
      umma::tmem_ld32 (tacc + c0, d);
#pragma unroll
      for (int k8 = 0; k8 < 4; ++k8)
      {
        uint4 o;
        uint32_t *ow = reinterpret_cast<uint32_t *> (&o);
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
          const int cc = 8 * k8 + 2 * j;
          __nv_bfloat162 h2 = __floats2bfloat162_rn (gelu (d[cc] + s_b1[c0 + cc]),
                                                     gelu (d[cc + 1] + s_b1[c0 + cc + 1]));
          ow[j] = *reinterpret_cast<uint32_t *> (&h2);
        }
        *reinterpret_cast<uint4 *> (sAct + umma::tile_offset (row, c0 + 8 * k8, kHid)) = o;
      }
    }
    umma::fence_async_smem ();
    umma::fence_before_sync ();
    group_sync (g);
    if (row == 0)
    {
      umma::fence_after_sync ();
      const uint32_t a0 = umma::smem_addr (sAct), b0 = umma::smem_addr (sW2);
#pragma unroll
      for (int kk = 0; kk < kHid / 16; ++kk)
        umma::mma_bf16 (tmma, umma::desc_kmajor (a0 + kk * 256, 128, (kHid / 8) * 128),
                        umma::desc_kmajor (b0 + kk * 256, 128, (kHid / 8) * 128), idesc,
                        kk > 0 ? 1u : 0u);
      umma::mma_commit (&mbar[g]);
    }
    ok = group_and (g, umma::mbar_wait (&mbar[g], phase, kWaitTries));
    phase ^= 1u;
    umma::fence_after_sync ();
    if (!ok) break;
    // layer-2 epilogue + 128 -> 3 head on the CUDA cores
    float y[kOut] = { s_b3[0], s_b3[1], s_b3[2] };
#pragma unroll 1
    for (int c0 = 0; c0 < kHid; c0 += 32)
    {
      float d[32];
      umma::tmem_ld32 (tacc + c0, d);
#pragma unroll
      for (int j = 0; j < 32; ++j)
      {
        const float h = gelu (d[j] + s_b2[c0 + j]);
#pragma unroll
        for (int o = 0; o < kOut; ++o) y[o] = fmaf (s_w3[o * kHid + c0 + j], h, y[o]);
      }
    }
    if (q >= 0)
    {
#pragma unroll
      for (int o = 0; o < kOut; ++o)
        a.guess[3 * (size_t)q + o] = (e >= 0) ? fminf (1.f, fmaxf (0.f, y[o])) : 0.5f;
    }
    // D2 and the activation tile are reused by the next tile of this group
    umma::fence_before_sync ();
    group_sync (g);
  }
  if (!ok && row == 0 && a.err) atomicExch (a.err, 1);
  umma::fence_before_sync ();
  __syncthreads ();
  if (warp == 0) umma::tmem_dealloc (tmem_base, kGuessGroups * kHid);
}

} // namespace mlp
} // namespace drb

using namespace drb;
using namespace drb::mlp;

namespace
{

bool mlp_order_ok (int order)
{
  if (order >= 1 && order <= 3) return true;
  set_last_error ("mlp: the network is defined for hex orders 1..3");
  return false;
}

template <int P> int prepare_p (const float *params, void *wbf16, cudaStream_t s)
{
  const int n = kHid * (Net<P>::kInPad > kHid ? Net<P>::kInPad : kHid);
  prepare_kernel<P><<<div_up (n, 256), 256, 0, s>>> (params, (__nv_bfloat16 *)wbf16);
  return check_launch ("prepare_kernel");
}

template <int P>
int features_p (const drb_mesh *mesh, const int *elem, const float *pts, int n, int n_pad, void *X,
                cudaStream_t s)
{
  features_kernel<P><<<div_up (n_pad, 128), 128, 0, s>>> (
  mesh->packed, packed_stride (Net<P>::kNd, 3), elem, pts, n, n_pad, (__nv_bfloat16 *)X);
  return check_launch ("features_kernel");
}

// Slots of a training step: one per CTA of net_kernel.
int net_ctas (int n_pad) { return min (n_pad / 128, sm_count ()); }

// Large enough for every device's slots: a tile has one CTA at most.
template <int P> long long workspace_p (int n_pad)
{
  return (long long)(n_pad / 128) * partial_stride<P> () * 4 + 4096;
}

template <int P, bool TRAIN> int launch_net (const NetArgs &a, int ctas, cudaStream_t s)
{
  constexpr size_t smem = net_smem<P> ();
  cudaFuncSetAttribute (net_kernel<P, TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  net_kernel<P, TRAIN><<<ctas, kNetThreads, smem, s>>> (a);
  return check_launch ("net_kernel");
}

template <int P>
int forward_p (const float *params, const void *wbf16, const void *X, int n, int n_pad, float *y,
               int *err, cudaStream_t s)
{
  NetArgs a{};
  a.params = params;
  a.wb = (const __nv_bfloat16 *)wbf16;
  a.X = (const __nv_bfloat16 *)X;
  a.n = n;
  a.tiles = n_pad / 128;
  a.y_out = y;
  a.err = err;
  return launch_net<P, false> (a, net_ctas (n_pad), s);
}

template <int P>
int train_step_p (const float *params, const void *wbf16, const void *X, const float *target,
                  const float *weight, int n, int n_pad, float *grad, float *loss, void *workspace,
                  int *err, cudaStream_t s)
{
  NetArgs a{};
  a.params = params;
  a.wb = (const __nv_bfloat16 *)wbf16;
  a.X = (const __nv_bfloat16 *)X;
  a.target = target;
  a.weight = weight;
  a.n = n;
  a.tiles = n_pad / 128;
  a.inv_count = 1.f / (float)n;
  a.partials = (float *)workspace;
  a.err = err;
  const int ctas = net_ctas (n_pad);
  int st = launch_net<P, true> (a, ctas, s);
  if (st) return st;
  constexpr int stride = partial_stride<P> ();
  reduce_kernel<<<div_up (stride, 128), 256, 0, s>>> (a.partials, ctas, stride, Net<P>::kParams, grad, loss);
  return check_launch ("reduce_kernel");
}

template <int P>
int guess_p (const float *params, const void *wbf16, const drb_mesh *mesh, const int *elem,
             const float *pts, const int *order, int n, float *guess, int *err, cudaStream_t s)
{
  GuessArgs a;
  a.params = params;
  a.wb = (const __nv_bfloat16 *)wbf16;
  a.packed = mesh->packed;
  a.stride = packed_stride (Net<P>::kNd, 3);
  a.elem = elem;
  a.pts = pts;
  a.order = order;
  a.n = n;
  a.guess = guess;
  a.err = err;
  constexpr size_t smem = guess_smem<P> ();
  cudaFuncSetAttribute (mlp_guess_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int tiles = div_up (n, 128);
  const int grid = min (div_up (tiles, Net<P>::kGroups), sm_count ());
  mlp_guess_kernel<P><<<grid, 128 * Net<P>::kGroups, smem, s>>> (a);
  return check_launch ("mlp_guess_kernel");
}

bool mesh_ok (const drb_mesh *mesh, const char *what)
{
  if (mesh && mesh->packed && mesh->dim == 3 && mesh->order >= 1 && mesh->order <= 3 &&
      mesh->ncomp == 3 && mesh->shape == DRB_SHAPE_TENSOR)
    return true;
  char buf[160];
  std::snprintf (buf, sizeof (buf), "%s: needs a packed hex geometry mesh of order 1..3", what);
  set_last_error (buf);
  return false;
}

} // namespace

extern "C" int drb_mlp_param_count (int order)
{
  return !mlp_order_ok (order) ? -1 : order == 1 ? Net<1>::kParams : order == 2 ? Net<2>::kParams
                                                                                  : Net<3>::kParams;
}
extern "C" int drb_mlp_bf16_count (int order)
{
  return !mlp_order_ok (order) ? -1 : order == 1 ? Net<1>::kBf16 : order == 2 ? Net<2>::kBf16
                                                                                : Net<3>::kBf16;
}
extern "C" int drb_mlp_input_width (int order)
{
  return !mlp_order_ok (order) ? -1 : order == 1 ? Net<1>::kInPad : order == 2 ? Net<2>::kInPad
                                                                                 : Net<3>::kInPad;
}

extern "C" int drb_mlp_prepare (int order, const float *params, void *wbf16, void *stream)
{
  if (!mlp_order_ok (order)) return DRB_ERR_INVALID_ARG;
  if (!params || !wbf16)
  {
    set_last_error ("mlp_prepare: bad arguments");
    return DRB_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  return order == 1 ? prepare_p<1> (params, wbf16, s) : order == 2 ? prepare_p<2> (params, wbf16, s)
                                                                   : prepare_p<3> (params, wbf16, s);
}

extern "C" int drb_mlp_features (const drb_mesh *mesh, const int *elem, const float *pts, int n,
                                 int n_pad, void *X, void *stream)
{
  if (!mesh_ok (mesh, "mlp_features")) return DRB_ERR_INVALID_ARG;
  if (n < 0 || n_pad < n || (n_pad > 0 && !X) || (n > 0 && (!elem || !pts)))
  {
    set_last_error ("mlp_features: bad arguments (n <= n_pad)");
    return DRB_ERR_INVALID_ARG;
  }
  if (n_pad == 0) return DRB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int o = mesh->order;
  return o == 1 ? features_p<1> (mesh, elem, pts, n, n_pad, X, s)
         : o == 2 ? features_p<2> (mesh, elem, pts, n, n_pad, X, s)
                  : features_p<3> (mesh, elem, pts, n, n_pad, X, s);
}

// Workspace of one training step over n_pad rows (multiple of 128): a slot of
// partial gradients per CTA.
extern "C" long long drb_mlp_workspace_bytes (int order, int n_pad)
{
  if (!mlp_order_ok (order) || n_pad < 0) return -1;
  return order == 1 ? workspace_p<1> (n_pad) : order == 2 ? workspace_p<2> (n_pad)
                                                          : workspace_p<3> (n_pad);
}

extern "C" int drb_mlp_forward (int order, const float *params, const void *wbf16, const void *X,
                                int n, int n_pad, float *y, void *workspace, int *err,
                                void *stream)
{
  if (!mlp_order_ok (order)) return DRB_ERR_INVALID_ARG;
  if (!params || !wbf16 || !X || !y || !workspace || n < 0 || n_pad < n || (n_pad % 128))
  {
    set_last_error ("mlp_forward: bad arguments (n_pad must be a multiple of 128 and >= n)");
    return DRB_ERR_INVALID_ARG;
  }
  if (n_pad == 0) return DRB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  return order == 1 ? forward_p<1> (params, wbf16, X, n, n_pad, y, err, s)
         : order == 2 ? forward_p<2> (params, wbf16, X, n, n_pad, y, err, s)
                      : forward_p<3> (params, wbf16, X, n, n_pad, y, err, s);
}

extern "C" int drb_mlp_train_step (int order, const float *params, const void *wbf16, const void *X,
                                   const float *target, const float *weight, int n, int n_pad,
                                   float *grad, float *loss, void *workspace, int *err,
                                   void *stream)
{
  if (!mlp_order_ok (order)) return DRB_ERR_INVALID_ARG;
  if (!params || !wbf16 || !X || !target || !grad || !workspace || n < 1 || n_pad < n ||
      (n_pad % 128))
  {
    set_last_error ("mlp_train_step: bad arguments (n_pad must be a multiple of 128 and >= n)");
    return DRB_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  return order == 1 ? train_step_p<1> (params, wbf16, X, target, weight, n, n_pad, grad, loss,
                                       workspace, err, s)
         : order == 2 ? train_step_p<2> (params, wbf16, X, target, weight, n, n_pad, grad, loss,
                                         workspace, err, s)
                      : train_step_p<3> (params, wbf16, X, target, weight, n, n_pad, grad, loss,
                                         workspace, err, s);
}

extern "C" int drb_mlp_adam (int order, float *params, const float *grad, float *m, float *v,
                             float lr, float beta1, float beta2, float eps, int step, void *stream)
{
  if (!mlp_order_ok (order)) return DRB_ERR_INVALID_ARG;
  if (!params || !grad || !m || !v || step < 1)
  {
    set_last_error ("mlp_adam: bad arguments");
    return DRB_ERR_INVALID_ARG;
  }
  const int np = drb_mlp_param_count (order);
  const float c1 = 1.f / (1.f - powf (beta1, (float)step));
  const float c2 = 1.f / (1.f - powf (beta2, (float)step));
  adam_kernel<<<div_up (np, 256), 256, 0, (cudaStream_t)stream>>> (params, grad, m, v, np, lr, beta1,
                                                                   beta2, eps, c1, c2);
  return check_launch ("adam_kernel");
}

extern "C" int drb_mlp_guess (const float *params, const void *wbf16, const drb_mesh *mesh,
                              const int *elem, const float *pts, const int *order, int n,
                              float *guess, int *err, void *stream)
{
  if (!mesh_ok (mesh, "mlp_guess")) return DRB_ERR_INVALID_ARG;
  if (!params || !wbf16 || n < 0 || (n > 0 && (!elem || !pts || !guess)))
  {
    set_last_error ("mlp_guess: bad arguments");
    return DRB_ERR_INVALID_ARG;
  }
  if (n == 0) return DRB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int o = mesh->order;
  return o == 1 ? guess_p<1> (params, wbf16, mesh, elem, pts, order, n, guess, err, s)
         : o == 2 ? guess_p<2> (params, wbf16, mesh, elem, pts, order, n, guess, err, s)
                  : guess_p<3> (params, wbf16, mesh, elem, pts, order, n, guess, err, s);
}
