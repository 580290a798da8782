// Uniform-grid candidate lists over the leaves of a built BVH.
//
// The batched locate spends about half of its time walking the tree to the
// first candidate leaf (12 wide-node visits of 112 bytes per query on the
// 64^3 mesh).  Because a leaf is a traversal candidate exactly when its own
// box holds the point, and the left-first traversal meets leaves in index
// order, a list per grid cell of the leaves whose boxes overlap the cell,
// sorted by leaf index, yields the same candidates in the same order: the
// point's cell gives a short contiguous run of leaf indices whose boxes
// (a 32-byte record per leaf) are tested instead of a chain of dependent
// node loads.  No reference counterpart (the reference traverses its binary
// nodes, data_model/device_mesh.hpp:262-318).
//
// Build: the leaf boxes are read back out of their parents' node records
// (the same floats the traversal tests) into the box table, and each leaf is
// filed under every cell its box overlaps (grid_axis of its corners): a
// counting sort over the cells, whose short lists are then put in leaf order.
// 8.65M leaves, 109M entries, 13.4M cells: count 0.29 ms, fill 0.82 ms (both
// bound by atomics and scattered 4-byte stores in L2), order 0.57 ms; emitting
// the pairs and sorting them by three radix passes took 4.7 ms.
#include "drb_common.cuh"
#include "drb_internal.h"
#include "locate.cuh"

#include <algorithm>
#include <cmath>

namespace drb
{
namespace
{

constexpr long long kMaxCells = 1ll << 28;
constexpr int kMaxDim = 4096;
// The counting sort's lists are ordered by comparing every entry with its
// list, so it is taken while an entry meets at most kOrderWork others on
// average (on ordinary meshes about ten: 1.7 ms a 109M entries against 4.7 ms
// of radix passes, whose time does not depend on the lists' length) and while
// the longest list does not keep its warp, whose 32 cells are neighbours and
// likely as long, busy for longer than the passes would take: L^2 rounds of
// about 2.2 ns against 34 ps an entry, L^2 * kOrderTail entries.  Graded 24^3
// order-2 meshes (us a build, counting / passes): longest list 118 of 3.7M
// entries 351 / 437, 251 of 2.1M 427 / 357, 854 of 3.7M 957 / 440.
constexpr unsigned long long kOrderWork = 64;
constexpr unsigned long long kOrderTail = 64;

struct GridGeom
{
  int dims[3];
  float origin[3];
  float inv[3];
};

GridGeom geom_of (const drb_bvh *b)
{
  GridGeom g;
  for (int d = 0; d < 3; ++d)
  {
    g.dims[d] = b->grid_dims[d];
    g.origin[d] = b->grid_origin[d];
    g.inv[d] = b->grid_inv[d];
  }
  return g;
}

// The leaf children of a binary node record (4 x float4: left box lo.xyz
// hi.xyz, right box lo.xyz hi.xyz, child codes; a leaf child is -(leaf + 1)):
// calls f (leaf, box) for each.
template <class F> DRB_D void for_leaf_boxes (const float4 *__restrict__ nodes, int i, F f)
{
  const float4 d = __ldg (nodes + 4 * (size_t)i + 3);
  const int l = __float_as_int (d.x), r = __float_as_int (d.y);
  if (l >= 0 && r >= 0) return;
  const float4 a = __ldg (nodes + 4 * (size_t)i);
  const float4 b = __ldg (nodes + 4 * (size_t)i + 1);
  const float4 c = __ldg (nodes + 4 * (size_t)i + 2);
  if (l < 0)
  {
    const float box[6] = { a.x, a.y, a.z, a.w, b.x, b.y };
    f (-l - 1, box);
  }
  if (r < 0)
  {
    const float box[6] = { b.z, b.w, c.x, c.y, c.z, c.w };
    f (-r - 1, box);
  }
}

// Sum of the leaf extents per axis (double atomics, one per warp and axis).
__global__ void extent_sum_kernel (const float4 *__restrict__ nodes, int n_inner,
                                   double *__restrict__ sum)
{
  double s[3] = { 0.0, 0.0, 0.0 };
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_inner; i += gridDim.x * blockDim.x)
    for_leaf_boxes (nodes, i, [&] (int, const float (&b)[6]) {
      for (int d = 0; d < 3; ++d) s[d] += (double)b[3 + d] - (double)b[d];
    });
  for (int d = 0; d < 3; ++d)
  {
    for (int o = 16; o > 0; o >>= 1) s[d] += __shfl_down_sync (0xffffffffu, s[d], o);
    if ((threadIdx.x & 31) == 0) atomicAdd (sum + d, s[d]);
  }
}

DRB_D void cell_range (const GridGeom &g, const float *b, int (&c0)[3], int (&c1)[3])
{
  for (int d = 0; d < 3; ++d)
  {
    c0[d] = grid_axis (b[d], g.origin[d], g.inv[d], g.dims[d]);
    c1[d] = grid_axis (b[3 + d], g.origin[d], g.inv[d], g.dims[d]);
  }
}

// Number of cells in a range; none where it is empty (a box with a NaN).
DRB_D unsigned long long cells_in (const int (&c0)[3], const int (&c1)[3])
{
  return (unsigned long long)max (c1[0] - c0[0] + 1, 0) * (unsigned)max (c1[1] - c0[1] + 1, 0) *
         (unsigned)max (c1[2] - c0[2] + 1, 0);
}

// Cells of all leaves together (64-bit).
__global__ void pair_total_kernel (GridGeom g, const float4 *__restrict__ nodes, int n_inner,
                                   unsigned long long *__restrict__ total)
{
  unsigned long long c = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_inner; i += gridDim.x * blockDim.x)
    for_leaf_boxes (nodes, i, [&] (int, const float (&b)[6]) {
      int c0[3], c1[3];
      cell_range (g, b, c0, c1);
      c += cells_in (c0, c1);
    });
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync (0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd (total, c);
}

// Box table: per leaf its box and element (32 bytes, float4 aligned).
__global__ void box_table_kernel (const float4 *__restrict__ nodes, int n_inner,
                                  const int *__restrict__ leaf_nodes, float4 *__restrict__ table)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_inner) return;
  for_leaf_boxes (nodes, i, [&] (int k, const float (&b)[6]) {
    table[2 * (size_t)k] = make_float4 (b[0], b[1], b[2], __int_as_float (__ldg (leaf_nodes + k)));
    table[2 * (size_t)k + 1] = make_float4 (b[3], b[4], b[5], 0.f);
  });
}

DRB_D void table_range (const GridGeom &g, const float4 *__restrict__ table, int k, int (&c0)[3],
                        int (&c1)[3])
{
  const float4 lo = __ldg (table + 2 * (size_t)k), hi = __ldg (table + 2 * (size_t)k + 1);
  const float b[6] = { lo.x, lo.y, lo.z, hi.x, hi.y, hi.z };
  cell_range (g, b, c0, c1);
}

// Whether a graded mesh crowds its leaves into few cells: one warp of leaves
// in kSampleWarps counts them into their first cells and raises *crowded when a
// cell gets more than kSampleCrowd, so that it holds about a thousand.  The
// lists will then take the radix passes whatever the counts are, and the
// counting is left out: of 8.65M leaves, a quarter of them in one cell, it took
// 5 ms of a build of 12.3, most of it atomics on that one counter and the few
// leaves that cover thousands of cells each.  About 5 us where no cell is
// crowded.
constexpr int kSampleWarps = 16;
constexpr int kSampleCrowd = 64;

__global__ void cell_sample_kernel (GridGeom g, const float4 *__restrict__ table, int n,
                                    int *__restrict__ counts, int *crowded)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const long long k = (long long)(t >> 5) * (32 * kSampleWarps) + (t & 31);
  if (k >= n || *(volatile int *)crowded) return;
  int c0[3], c1[3];
  table_range (g, table, (int)k, c0, c1);
  const int cell = (c0[2] * g.dims[1] + c0[1]) * g.dims[0] + c0[0];
  if (atomicAdd (counts + cell, 1) >= kSampleCrowd) *(volatile int *)crowded = 1;
}

// Leaves per cell; with `sampled`, cell_sample_kernel has counted its leaves'
// first cells.
__global__ void cell_count_kernel (GridGeom g, const float4 *__restrict__ table, int n, bool sampled,
                                   const int *__restrict__ crowded, int *__restrict__ counts)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || *crowded) return;
  const int counted = sampled && (k >> 5) % kSampleWarps == 0 ? 1 : 0;
  int c0[3], c1[3];
  table_range (g, table, k, c0, c1);
  for (int z = c0[2]; z <= c1[2]; ++z)
    for (int y = c0[1]; y <= c1[1]; ++y)
    {
      int *row = counts + (size_t)(z * g.dims[1] + y) * g.dims[0];
      const bool first = z == c0[2] && y == c0[1];
      for (int x = c0[0] + (first ? counted : 0); x <= c1[0]; ++x) atomicAdd (row + x, 1);
    }
}

// Of the cells' counts: the sum, the sum of squares and the maximum.
__global__ void count_stats_kernel (const int *__restrict__ counts, long long n_cells,
                                    unsigned long long *__restrict__ stats)
{
  unsigned long long sum = 0, sq = 0, top = 0;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n_cells;
       c += (long long)gridDim.x * blockDim.x)
  {
    const unsigned long long k = (unsigned)__ldg (counts + c);
    sum += k;
    sq += k * k;
    top = max (top, k);
  }
  for (int o = 16; o > 0; o >>= 1)
  {
    sum += __shfl_down_sync (0xffffffffu, sum, o);
    sq += __shfl_down_sync (0xffffffffu, sq, o);
    top = max (top, __shfl_down_sync (0xffffffffu, top, o));
  }
  if ((threadIdx.x & 31) == 0 && sum)
  {
    atomicAdd (stats, sum);
    atomicAdd (stats + 1, sq);
    atomicMax (stats + 2, top);
  }
}

// Every leaf into the lists of its cells, in whatever order the atomics give;
// counts runs down to zero.
__global__ void cell_fill_kernel (GridGeom g, const float4 *__restrict__ table, int n,
                                  const int *__restrict__ start, int *__restrict__ counts,
                                  int *__restrict__ lists)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int c0[3], c1[3];
  table_range (g, table, k, c0, c1);
  for (int z = c0[2]; z <= c1[2]; ++z)
    for (int y = c0[1]; y <= c1[1]; ++y)
    {
      const size_t row = (size_t)(z * g.dims[1] + y) * g.dims[0];
      for (int x = c0[0]; x <= c1[0]; ++x)
        lists[__ldg (start + row + x) + atomicSub (counts + row + x, 1) - 1] = k;
    }
}

// The lists in leaf order: a warp takes 32 consecutive cells, a lane an
// entry, whose place is the number of smaller ones in its cell's list (a
// leaf occurs once in a list).  The list is re-read through L1.  Entry indices
// are unsigned: the last round's reach past the end, which is below 2^31.
__global__ void cell_order_kernel (const int *__restrict__ start, long long n_cells,
                                   const int *__restrict__ lists, int *__restrict__ entries)
{
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const long long c0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) - lane;
  if (c0 >= n_cells) return;
  const unsigned lo = __ldg (start + min (c0 + lane, n_cells));
  const unsigned end = __ldg (start + min (c0 + 32, n_cells));
  const unsigned begin = __shfl_sync (FULL, lo, 0);
  for (unsigned base = begin; base < end; base += 32)
  {
    const unsigned e = base + lane;
    int j = 0; // the last cell that starts at or before e
#pragma unroll
    for (int h = 16; h; h >>= 1)
      if (__shfl_sync (FULL, lo, j + h) <= e) j += h;
    const unsigned first = __shfl_sync (FULL, lo, j);
    const unsigned next = __shfl_sync (FULL, lo, (j + 1) & 31);
    const unsigned last = j == 31 ? end : next;
    if (e < end)
    {
      const int v = __ldg (lists + e);
      int rank = 0;
      for (unsigned q = first; q < last; ++q) rank += __ldg (lists + q) < v;
      entries[first + rank] = v;
    }
  }
}

// --- grids with long lists: the pairs sorted by radix passes ---

// Cells per leaf, and their sum (64-bit).
__global__ void pair_count_kernel (GridGeom g, const float4 *__restrict__ table, int n,
                                   int *__restrict__ counts, unsigned long long *__restrict__ total)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long c = 0;
  if (k < n)
  {
    int c0[3], c1[3];
    table_range (g, table, k, c0, c1);
    c = cells_in (c0, c1);
    counts[k] = (int)c;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync (0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd (total, c);
}

// (cell, leaf) pairs of every leaf, written from its offset in leaf order.
__global__ void pair_emit_kernel (GridGeom g, const float4 *__restrict__ table, int n,
                                  const int *__restrict__ offsets, unsigned *__restrict__ keys,
                                  int *__restrict__ vals)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int c0[3], c1[3];
  table_range (g, table, k, c0, c1);
  int o = offsets[k];
  for (int z = c0[2]; z <= c1[2]; ++z)
    for (int y = c0[1]; y <= c1[1]; ++y)
      for (int x = c0[0]; x <= c1[0]; ++x)
      {
        keys[o] = (unsigned)((z * g.dims[1] + y) * g.dims[0] + x);
        vals[o] = k;
        ++o;
      }
}

// start[c] = first sorted pair whose cell is >= c (lower bound), and
// start[n_cells] = m.
__global__ void cell_start_kernel (const unsigned *__restrict__ keys, int m, long long n_cells,
                                   int *__restrict__ start)
{
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c > n_cells) return;
  unsigned lo = 0, hi = (unsigned)m;
  while (lo < hi)
  {
    const unsigned mid = (lo + hi) >> 1;
    if (__ldg (keys + mid) < c) lo = mid + 1;
    else hi = mid;
  }
  start[c] = (int)lo;
}

int check_bvh (const drb_bvh *b, const char *what)
{
  if (!b || b->n_leaf < 2 || !b->inner_nodes || !b->leaf_nodes)
  {
    set_last_error (what);
    return DRB_ERR_INVALID_ARG;
  }
  return DRB_OK;
}

int too_many_entries ()
{
  set_last_error ("bvh_grid_build: 2^31 entries or more; use a larger cell_scale");
  return DRB_ERR_UNSUPPORTED;
}

// Starts and entries by a stable radix sort of the (cell, leaf) pairs on the
// cell; the box table is there.
int sort_entries (const drb_bvh *bvh, const GridGeom &g, long long n_cells, Scratch &scr, cudaStream_t s)
{
  const int n = bvh->n_leaf;
  const float4 *table = (const float4 *)bvh->grid_boxes;
  int *counts = scr.alloc<int> (n);
  int *offsets = scr.alloc<int> (n);
  unsigned long long *total = scr.alloc<unsigned long long> (1);
  if (scr.err != cudaSuccess) return status_from (scr.err);
  cudaMemsetAsync (total, 0, sizeof (unsigned long long), s);
  pair_count_kernel<<<div_up (n, 256), 256, 0, s>>> (g, table, n, counts, total);
  if (int st = check_launch ("pair_count_kernel")) return st;
  unsigned long long h_total = 0;
  cudaMemcpyAsync (&h_total, total, sizeof h_total, cudaMemcpyDeviceToHost, s);
  if (cudaError_t e = cudaStreamSynchronize (s))
  {
    set_last_error ("bvh_grid_build: pair count failed");
    return status_from (e);
  }
  if (h_total >= (1ull << 31)) return too_many_entries ();
  const int m = (int)h_total;
  unsigned *keys = scr.alloc<unsigned> (m);
  int *vals = scr.alloc<int> (m);
  unsigned *keys_s = scr.alloc<unsigned> (m);
  if (scr.err != cudaSuccess) return status_from (scr.err);
  if (int st = exclusive_scan_i32 (counts, offsets, n, nullptr, s)) return st;
  pair_emit_kernel<<<div_up (n, 256), 256, 0, s>>> (g, table, n, offsets, keys, vals);
  if (int st = check_launch ("pair_emit_kernel")) return st;
  int bits = 1;
  while ((1ll << bits) < n_cells) ++bits;
  if (int st = radix_sort_pairs (keys, vals, keys_s, bvh->grid_entries, m, bits, s)) return st;
  cell_start_kernel<<<div_up (n_cells + 1, 256), 256, 0, s>>> (keys_s, m, n_cells, bvh->grid_start);
  return check_launch ("cell_start_kernel");
}

} // namespace
} // namespace drb

using namespace drb;

extern "C" int drb_bvh_grid_size (drb_bvh *bvh, float cell_scale, long long *n_entries, void *stream)
{
  if (int st = check_bvh (bvh, "bvh_grid_size: needs a built BVH with at least two leaves")) return st;
  if (!n_entries || !(cell_scale > 0.f) || !std::isfinite (cell_scale))
  {
    set_last_error ("bvh_grid_size: bad arguments");
    return DRB_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int n = bvh->n_leaf, n_inner = bvh->n_inner;
  const float4 *nodes = (const float4 *)bvh->inner_nodes;
  const int blocks = std::min (div_up (n_inner, 256), 8 * sm_count ());
  Scratch scr (s);
  double *sum = scr.alloc<double> (3);
  unsigned long long *total = scr.alloc<unsigned long long> (1);
  if (!sum || !total) return status_from (scr.err);
  cudaMemsetAsync (sum, 0, 3 * sizeof (double), s);
  cudaMemsetAsync (total, 0, sizeof (unsigned long long), s);
  extent_sum_kernel<<<blocks, 256, 0, s>>> (nodes, n_inner, sum);
  if (int st = check_launch ("extent_sum_kernel")) return st;
  double h_sum[3];
  cudaMemcpyAsync (h_sum, sum, sizeof h_sum, cudaMemcpyDeviceToHost, s);
  if (cudaError_t e = cudaStreamSynchronize (s))
  {
    set_last_error ("bvh_grid_size: extent reduction failed");
    return status_from (e);
  }
  // cells about cell_scale times the mean leaf extent per axis
  double ext[3], want[3];
  for (int d = 0; d < 3; ++d)
  {
    ext[d] = (double)bvh->bounds[2 * d + 1] - (double)bvh->bounds[2 * d];
    const double mean = h_sum[d] / n;
    want[d] = (ext[d] > 0.0 && mean > 0.0) ? std::ceil (ext[d] / (cell_scale * mean)) : 1.0;
    want[d] = std::min (std::max (want[d], 1.0), (double)kMaxDim);
  }
  double cells = want[0] * want[1] * want[2];
  if (cells > (double)kMaxCells)
  {
    const double f = std::cbrt ((double)kMaxCells / cells);
    for (int d = 0; d < 3; ++d) want[d] = std::max (1.0, std::floor (want[d] * f));
  }
  GridGeom g;
  for (int d = 0; d < 3; ++d)
  {
    g.dims[d] = (int)want[d];
    g.origin[d] = bvh->bounds[2 * d];
    g.inv[d] = ext[d] > 0.0 ? (float)(g.dims[d] / ext[d]) : 0.f;
    bvh->grid_dims[d] = g.dims[d];
    bvh->grid_origin[d] = g.origin[d];
    bvh->grid_inv[d] = g.inv[d];
  }
  pair_total_kernel<<<blocks, 256, 0, s>>> (g, nodes, n_inner, total);
  if (int st = check_launch ("pair_total_kernel")) return st;
  unsigned long long h_total = 0;
  cudaMemcpyAsync (&h_total, total, sizeof h_total, cudaMemcpyDeviceToHost, s);
  if (cudaError_t e = cudaStreamSynchronize (s))
  {
    set_last_error ("bvh_grid_size: pair count failed");
    return status_from (e);
  }
  *n_entries = (long long)h_total;
  return DRB_OK;
}

extern "C" int drb_bvh_grid_build (const drb_bvh *bvh, void *stream)
{
  if (int st = check_bvh (bvh, "bvh_grid_build: needs a built BVH with at least two leaves")) return st;
  if (!bvh->grid_start || !bvh->grid_entries || !bvh->grid_boxes)
  {
    set_last_error ("bvh_grid_build: grid_start, grid_entries and grid_boxes must be set");
    return DRB_ERR_INVALID_ARG;
  }
  const GridGeom g = geom_of (bvh);
  const long long n_cells = (long long)g.dims[0] * g.dims[1] * g.dims[2];
  if (g.dims[0] < 1 || g.dims[1] < 1 || g.dims[2] < 1 || n_cells > kMaxCells)
  {
    set_last_error ("bvh_grid_build: call drb_bvh_grid_size first");
    return DRB_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int n = bvh->n_leaf;
  float4 *table = (float4 *)bvh->grid_boxes;
  Scratch scr (s);
  box_table_kernel<<<div_up (bvh->n_inner, 256), 256, 0, s>>> (
      (const float4 *)bvh->inner_nodes, bvh->n_inner, bvh->leaf_nodes, table);
  if (int st = check_launch ("box_table_kernel")) return st;
  // with this many leaves a cell, each in two or more lists while cells are a
  // few leaves wide, the lists are too long on average, and counting them would
  // only crowd the atomics on a few counters
  if (n > (long long)kOrderWork / 2 * n_cells) return sort_entries (bvh, g, n_cells, scr, s);
  int *counts = scr.alloc<int> (n_cells + 1);
  unsigned long long *stats = scr.alloc<unsigned long long> (4);
  if (!counts || !stats) return status_from (scr.err);
  int *crowded = reinterpret_cast<int *> (stats + 3);
  cudaMemsetAsync (counts, 0, sizeof (int) * (n_cells + 1), s);
  cudaMemsetAsync (stats, 0, 4 * sizeof (unsigned long long), s);
  // (few leaves are counted in no time)
  const bool sampled = n > 32768;
  if (sampled)
  {
    cell_sample_kernel<<<div_up (n, 256 * kSampleWarps), 256, 0, s>>> (g, table, n, counts, crowded);
    if (int st = check_launch ("cell_sample_kernel")) return st;
  }
  cell_count_kernel<<<div_up (n, 256), 256, 0, s>>> (g, table, n, sampled, crowded, counts);
  if (int st = check_launch ("cell_count_kernel")) return st;
  count_stats_kernel<<<std::min (div_up (n_cells, 256), 8 * sm_count ()), 256, 0, s>>> (counts, n_cells,
                                                                                 stats);
  if (int st = check_launch ("count_stats_kernel")) return st;
  unsigned long long h_stats[4] = { 0, 0, 0, 0 };
  cudaMemcpyAsync (h_stats, stats, sizeof h_stats, cudaMemcpyDeviceToHost, s);
  if (cudaError_t e = cudaStreamSynchronize (s))
  {
    set_last_error ("bvh_grid_build: pair count failed");
    return status_from (e);
  }
  if (h_stats[3]) return sort_entries (bvh, g, n_cells, scr, s);
  if (h_stats[0] >= (1ull << 31)) return too_many_entries ();
  if (h_stats[1] > kOrderWork * h_stats[0] || h_stats[2] * h_stats[2] * kOrderTail > h_stats[0])
    return sort_entries (bvh, g, n_cells, scr, s);
  int *lists = scr.alloc<int> ((size_t)h_stats[0]);
  if (!lists) return status_from (scr.err);
  // (a list of n_cells + 1 counts, the last one zero: the last start is their sum)
  if (int st = exclusive_scan_i32 (counts, bvh->grid_start, (int)n_cells + 1, nullptr, s)) return st;
  cell_fill_kernel<<<div_up (n, 256), 256, 0, s>>> (g, table, n, bvh->grid_start, counts, lists);
  if (int st = check_launch ("cell_fill_kernel")) return st;
  cell_order_kernel<<<div_up (n_cells, 256), 256, 0, s>>> (bvh->grid_start, n_cells, lists,
                                                           bvh->grid_entries);
  return check_launch ("cell_order_kernel");
}
