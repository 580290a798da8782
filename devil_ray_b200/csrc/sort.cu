// Stable LSD radix sort of (uint32 key, int32 value) pairs and an int32
// exclusive scan, hand-written for sm_100a.  Replaces the host std::sort of
// the reference's LBVH build (linear_bvh_builder.cpp:120-135) and the RAJA
// exclusive_scan of its compactions (array_utils.hpp:171-270).
//
// Sort pass (8-bit digit): 20 bytes per pair, 0.34 ms of 30M pairs (1.8 TB/s):
// bound by the latency of a tile's chain, three blocks an SM (36 % of the issue
// slots, 12 % of DRAM at 8.65M pairs), not by the memory.
//   hist_kernel     per-tile digit histogram in shared memory, written
//                   digit-major
//   digit_kernel    a block per digit scans its tiles' counts in place and
//                   leaves the digit's total
//   scatter_kernel  a tile of 4096 pairs (1024 of few) per block.  Every warp
//                   ranks its eighth of them on its own (eight ballots a
//                   row of 32 give the peers with the same digit, unless
//                   the row is one run; a per-warp counter in shared
//                   memory gives the rank), so the block synchronises
//                   only three times a tile; the pairs
//                   are then put in digit order in shared memory and leave
//                   as runs of consecutive addresses.  Equal keys keep their
//                   input order (stability), which makes the result
//                   deterministic run to run.
// Four passes over 8.65M pairs and three over 109M: 5.5 -> 4.0 ms.  30M random
// keys of 30 bits 2.24 -> 1.34 ms, all of them equal 1.02 -> 1.21: runs as long as
// a tile were coalesced without being put in order.
#include "drb_common.cuh"
#include "drb_internal.h"

#include <cstdint>

namespace drb
{
namespace
{
constexpr int kSortBlock = 256;
// Keys per thread: 16, or 4 where tiles of 4096 would leave SMs without one: the
// chain of a tile's rows is then what a pass waits for (30-bit keys, 16 / 4 a
// thread: 100 of them 90 / 75 us, 10,000 106 / 80, 600,000 111 / 93).
constexpr int kSortItems = 16;
constexpr int kSortItemsFew = 4;
constexpr int kSortWarps = kSortBlock / kWarp;
constexpr int kRadix = 256;
static_assert (kRadix == kSortBlock, "a thread per digit");

template <int ITEMS>
__global__ void __launch_bounds__ (kSortBlock)
hist_kernel (const unsigned *__restrict__ keys, int n, int shift, int ntiles, int *__restrict__ counts)
{
  __shared__ int hist[kRadix];
  hist[threadIdx.x] = 0;
  __syncthreads ();
  const long long base = (long long)blockIdx.x * (kSortBlock * ITEMS);
  unsigned key[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
  {
    const long long idx = base + (long long)j * kSortBlock + threadIdx.x;
    key[j] = idx < n ? __ldg (keys + idx) : 0u;
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if (base + (long long)j * kSortBlock + threadIdx.x < n) atomicAdd (&hist[(key[j] >> shift) & 0xffu], 1);
  __syncthreads ();
  counts[(size_t)threadIdx.x * ntiles + blockIdx.x] = hist[threadIdx.x];
}

// Exclusive scan of one value per thread over the block (blockDim.x a
// multiple of 32); total: the sum over the block.
DRB_D int block_exclusive_scan (int v, int *total)
{
  __shared__ int warp_sums[32];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const int y = __shfl_up_sync (0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads ();
  if (warp == 0)
  {
    int s = (lane < warps) ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const int y = __shfl_up_sync (0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < warps) warp_sums[lane] = s;
  }
  __syncthreads ();
  const int warp_prefix = (warp > 0) ? warp_sums[warp - 1] : 0;
  *total = warp_sums[warps - 1];
  __syncthreads ();
  return warp_prefix + x - v;
}

// Exclusive scan of a row of n values by one block, in place; returns the
// row's sum.  A thread takes four consecutive values a round.
DRB_D int scan_row (int *row, int n)
{
  int carry = 0;
  for (int b = 0; b < n; b += 4 * blockDim.x)
  {
    const int i = b + 4 * threadIdx.x;
    int v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = i + q < n ? row[i + q] : 0;
    int total;
    int at = carry + block_exclusive_scan (v[0] + v[1] + v[2] + v[3], &total);
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
      if (i + q < n) row[i + q] = at;
      at += v[q];
    }
    carry += total;
  }
  return carry;
}

__global__ void __launch_bounds__ (1024)
digit_kernel (int *__restrict__ counts, int ntiles, int *__restrict__ totals)
{
  const int total = scan_row (counts + (size_t)blockIdx.x * ntiles, ntiles);
  if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

// vals_in NULL: the values are the input positions.
template <int ITEMS>
__global__ void __launch_bounds__ (kSortBlock, 3)
scatter_kernel (const unsigned *__restrict__ keys_in, const int *__restrict__ vals_in,
                unsigned *__restrict__ keys_out, int *__restrict__ vals_out, int n, int shift,
                int ntiles, const int *__restrict__ counts, const int *__restrict__ totals)
{
  constexpr int kTile = kSortBlock * ITEMS;
  __shared__ unsigned s_key[kTile];
  __shared__ int s_val[kTile];
  __shared__ int wcnt[kSortWarps][kRadix];
  __shared__ int out_base[kRadix]; // digit's place in the output minus its place in the tile
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  const long long base = (long long)blockIdx.x * kTile;
  const int tile_n = (int)min ((long long)kTile, n - base);
  unsigned key[ITEMS];
  unsigned short rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
  {
    const int i = warp * kWarp * ITEMS + j * kWarp + lane;
    key[j] = i < tile_n ? __ldg (keys_in + base + i) : 0u;
  }
#pragma unroll
  for (int q = 0; q < kRadix / kWarp; ++q) wcnt[warp][lane + q * kWarp] = 0;
  __syncwarp ();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
  {
    const bool valid = warp * kWarp * ITEMS + j * kWarp + lane < tile_n;
    const int digit = (key[j] >> shift) & 0xffu;
    unsigned peers = __ballot_sync (0xffffffffu, valid);
    const int digit0 = __shfl_sync (0xffffffffu, digit, 0);
    if (!__all_sync (0xffffffffu, digit == digit0)) // else the row is one run
    {
#pragma unroll
      for (int b = 0; b < 8; ++b)
      {
        const bool set = (digit >> b) & 1;
        const unsigned m = __ballot_sync (0xffffffffu, set);
        peers &= set ? m : ~m;
      }
    }
    int before = 0;
    if (valid) before = wcnt[warp][digit];
    __syncwarp ();
    rank[j] = (unsigned short)(before + __popc (peers & lt_mask));
    if (valid && (peers & lt_mask) == 0u) wcnt[warp][digit] = before + __popc (peers);
    __syncwarp ();
  }
  __syncthreads ();
  // thread = digit: the warps' counts to their places in the tile
  {
    int sum = 0, c[kSortWarps];
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w)
    {
      c[w] = sum;
      sum += wcnt[w][tid];
    }
    int all;
    const int start = block_exclusive_scan (sum, &all);
    const int digit_start = block_exclusive_scan (totals[tid], &all);
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) wcnt[w][tid] = start + c[w];
    out_base[tid] = digit_start + counts[(size_t)tid * ntiles + blockIdx.x] - start;
  }
  __syncthreads ();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
  {
    const int i = warp * kWarp * ITEMS + j * kWarp + lane;
    if (i < tile_n)
    {
      const int at = wcnt[warp][(key[j] >> shift) & 0xffu] + rank[j];
      s_key[at] = key[j];
      s_val[at] = vals_in ? __ldg (vals_in + base + i) : (int)(base + i);
    }
  }
  __syncthreads ();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
  {
    const int i = j * kSortBlock + tid;
    if (i < tile_n)
    {
      const unsigned k = s_key[i];
      const int pos = out_base[(k >> shift) & 0xffu] + i;
      keys_out[pos] = k;
      vals_out[pos] = s_val[i];
    }
  }
}

// ---- exclusive scan: tile sums, one block over them, apply ----
constexpr int kScanBlock = 256;
constexpr int kScanRows = 4;                              // rows of int4 per thread
constexpr int kScanTile = kScanBlock * kScanRows * 4;

// Row j of this thread's values: four consecutive ones, coalesced over the
// warp.  VEC: the array is 16-byte aligned.
template <bool VEC> DRB_D void scan_load (const int *in, long long at, int n, int (&v)[4])
{
  if (VEC && at + 3 < n)
  {
    const int4 q = *reinterpret_cast<const int4 *> (in + at);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  }
  else
  {
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = at + q < n ? in[at + q] : 0;
  }
}

template <bool VEC>
__global__ void __launch_bounds__ (kScanBlock)
scan_reduce_kernel (const int *__restrict__ in, int n, int *__restrict__ block_sums)
{
  int s = 0;
#pragma unroll
  for (int j = 0; j < kScanRows; ++j)
  {
    int v[4];
    scan_load<VEC> (in, (long long)blockIdx.x * kScanTile + 4 * (j * kScanBlock + (int)threadIdx.x), n, v);
    s += v[0] + v[1] + v[2] + v[3];
  }
  int total;
  block_exclusive_scan (s, &total);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__ (1024) scan_sums_kernel (int *sums, int n) { scan_row (sums, n); }

template <bool VEC>
__global__ void __launch_bounds__ (kScanBlock)
scan_apply_kernel (const int *in, int *out, int n, const int *__restrict__ block_offsets,
                   int *d_total, int nblocks)
{
  __shared__ int warp_sums[kScanBlock / kWarp];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  // a warp's values are contiguous: its rows follow one another
  const long long base = (long long)blockIdx.x * kScanTile + warp * (kWarp * 4 * kScanRows);
  int v[kScanRows][4], before[kScanRows];
  int carry = 0;
#pragma unroll
  for (int j = 0; j < kScanRows; ++j) scan_load<VEC> (in, base + 4 * (j * kWarp + lane), n, v[j]);
#pragma unroll
  for (int j = 0; j < kScanRows; ++j)
  {
    const int s = v[j][0] + v[j][1] + v[j][2] + v[j][3];
    int x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const int y = __shfl_up_sync (0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    before[j] = carry + x - s;
    carry += __shfl_sync (0xffffffffu, x, 31);
  }
  if (lane == 0) warp_sums[warp] = carry;
  __syncthreads ();
  int prefix = block_offsets ? block_offsets[blockIdx.x] : 0;
  for (int w = 0; w < warp; ++w) prefix += warp_sums[w];
#pragma unroll
  for (int j = 0; j < kScanRows; ++j)
  {
    const long long at = base + 4 * (j * kWarp + lane);
    int o[4];
    o[0] = prefix + before[j];
    o[1] = o[0] + v[j][0];
    o[2] = o[1] + v[j][1];
    o[3] = o[2] + v[j][2];
    if (VEC && at + 3 < n) *reinterpret_cast<int4 *> (out + at) = make_int4 (o[0], o[1], o[2], o[3]);
    else
    {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (at + q < n) out[at + q] = o[q];
    }
    // values past n count as zero, so the last row of the last block ends
    // at the total
    if (d_total && blockIdx.x == nblocks - 1 && threadIdx.x == kScanBlock - 1 && j == kScanRows - 1)
      *d_total = o[3] + v[j][3];
  }
}

template <bool VEC>
int scan_launch (const int *in, int *out, int n, int *d_total, int *tmp, int nblocks, cudaStream_t s)
{
  if (nblocks > 1)
  {
    scan_reduce_kernel<VEC><<<nblocks, kScanBlock, 0, s>>> (in, n, tmp);
    int st = check_launch ("scan_reduce_kernel");
    if (st) return st;
    scan_sums_kernel<<<1, 1024, 0, s>>> (tmp, nblocks);
    if ((st = check_launch ("scan_sums_kernel"))) return st;
  }
  scan_apply_kernel<VEC><<<nblocks, kScanBlock, 0, s>>> (in, out, n, nblocks > 1 ? tmp : nullptr,
                                                         d_total, nblocks);
  return check_launch ("scan_apply_kernel");
}

} // namespace

int scan_ws_ints (int n) { return div_up (n, kScanTile) + 1; }

int exclusive_scan_i32_ws (const int *in, int *out, int n, int *d_total, int *tmp, cudaStream_t s)
{
  if (n <= 0)
  {
    if (d_total) cudaMemsetAsync (d_total, 0, sizeof (int), s);
    return DRB_OK;
  }
  const int nblocks = div_up (n, kScanTile);
  const bool vec = (reinterpret_cast<uintptr_t> (in) | reinterpret_cast<uintptr_t> (out)) % 16 == 0;
  return vec ? scan_launch<true> (in, out, n, d_total, tmp, nblocks, s)
             : scan_launch<false> (in, out, n, d_total, tmp, nblocks, s);
}

int exclusive_scan_i32 (const int *in, int *out, int n, int *d_total, cudaStream_t s)
{
  Scratch scr (s);
  int *tmp = n > kScanTile ? scr.alloc<int> (scan_ws_ints (n)) : nullptr;
  if (scr.err != cudaSuccess) return status_from (scr.err);
  return exclusive_scan_i32_ws (in, out, n, d_total, tmp, s);
}

int radix_sort_pairs (const unsigned *keys_in, const int *vals_in, unsigned *keys_out,
                      int *vals_out, int n, int bits, cudaStream_t s)
{
  if (n <= 0) return DRB_OK;
  const bool few = n < kSortBlock * kSortItems * sm_count ();
  const int ntiles = div_up (n, kSortBlock * (few ? kSortItemsFew : kSortItems));
  const int passes = (bits + 7) / 8;
  Scratch scr (s);
  int *counts = scr.alloc<int> ((size_t)kRadix * (ntiles + 1)); // and the digits' totals
  int *totals = counts + (size_t)kRadix * ntiles;
  unsigned *kbuf = passes > 1 ? scr.alloc<unsigned> (n) : nullptr;
  int *vbuf = passes > 1 ? scr.alloc<int> (n) : nullptr;
  if (scr.err != cudaSuccess) return status_from (scr.err);
  // Ping-pong so that the last pass lands in keys_out/vals_out.
  const unsigned *ksrc = keys_in;
  const int *vsrc = vals_in;
  for (int p = 0; p < passes; ++p)
  {
    const bool to_out = ((passes - 1 - p) % 2) == 0;
    unsigned *kdst = to_out ? keys_out : kbuf;
    int *vdst = to_out ? vals_out : vbuf;
    if (few) hist_kernel<kSortItemsFew><<<ntiles, kSortBlock, 0, s>>> (ksrc, n, 8 * p, ntiles, counts);
    else hist_kernel<kSortItems><<<ntiles, kSortBlock, 0, s>>> (ksrc, n, 8 * p, ntiles, counts);
    int st = check_launch ("hist_kernel");
    if (st) return st;
    digit_kernel<<<kRadix, min (1024, div_up (div_up (ntiles, 4), 32) * 32), 0, s>>> (counts, ntiles, totals);
    if ((st = check_launch ("digit_kernel"))) return st;
    if (few)
      scatter_kernel<kSortItemsFew><<<ntiles, kSortBlock, 0, s>>> (ksrc, vsrc, kdst, vdst, n, 8 * p, ntiles,
                                                                   counts, totals);
    else
      scatter_kernel<kSortItems><<<ntiles, kSortBlock, 0, s>>> (ksrc, vsrc, kdst, vdst, n, 8 * p, ntiles,
                                                                counts, totals);
    if ((st = check_launch ("scatter_kernel"))) return st;
    ksrc = kdst;
    vsrc = vdst;
  }
  return DRB_OK;
}

} // namespace drb

extern "C" int drb_radix_sort_pairs (const unsigned *keys_in, const int *vals_in,
                                     unsigned *keys_out, int *vals_out, int n, int bits,
                                     void *stream)
{
  if (n < 0 || bits < 1 || bits > 32 ||
      (n > 0 && (!keys_in || !vals_in || !keys_out || !vals_out)))
  {
    drb::set_last_error ("radix_sort_pairs: bad arguments");
    return DRB_ERR_INVALID_ARG;
  }
  if (n > 0 && (keys_in == keys_out || vals_in == vals_out))
  {
    drb::set_last_error ("radix_sort_pairs: in-place sort is not supported");
    return DRB_ERR_INVALID_ARG;
  }
  return drb::radix_sort_pairs (keys_in, vals_in, keys_out, vals_out, n, bits,
                                (cudaStream_t)stream);
}
