// 4-wide collapse of the reference-layout binary LBVH, for traversal only.
//
// Every binary inner node at even depth becomes one 128-byte wide node whose
// (up to) four children are its grandchildren, or its children where those
// are leaves, in left-to-right order.  A query then makes one dependent
// 128-byte load per two binary levels.  The child boxes are copied bit for
// bit from the binary records, and a parent box is the exact union of its
// children's, so a leaf is reached in the wide tree exactly when its own box
// holds the point, as in the binary tree (linear_bvh_builder.cpp:253-397,
// device_mesh.hpp:262-318); visiting the hit children lowest first keeps
// the binary traversal's left-first leaf order.  Point location over the
// wide tree therefore tries the same candidates in the same order and
// returns the same result.
//
//   parent_kernel    parent index of every binary inner node
//   depth_kernel     depth of every node, even -> wide
//   (exclusive scan of the flags gives each wide node its index)
//   wide_emit_kernel one thread per wide node gathers its children
// 8.65M leaves: 0.45 ms in all (HBM and the gathers), 1.3 ms when every node
// walked to the root, every thread stored its own 128 bytes and the size
// query ran the first two steps once more.
#include "drb_common.cuh"
#include "drb_internal.h"
#include "locate.cuh"

namespace drb
{
namespace
{

constexpr int kMaxWalk = 1024; // depth bound of the parent walk

__global__ void parent_kernel (const float4 *__restrict__ nodes, int n_inner, int *__restrict__ parent)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_inner) return;
  if (i == 0) parent[0] = -1;
  const float4 d = nodes[4 * (size_t)i + 3];
  const int l = __float_as_int (d.x), r = __float_as_int (d.y);
  if (l >= 0 && l / 4 < n_inner) parent[l / 4] = i;
  if (r >= 0 && r / 4 < n_inner) parent[r / 4] = i;
}

// Depth of every node.  A block takes kDepthNodes consecutive nodes.  A
// node's index is an end of its leaf range, so most parents lie in the
// block: only the nodes whose parent does not (some tens of a block) walk
// the parents through global memory, and the others walk to one of those in
// shared memory.  (Every node walking to the root took 25 dependent loads a
// node.)  Walks are bounded by kMaxWalk.
constexpr int kDepthBlock = 256;
constexpr int kDepthNodes = 4 * kDepthBlock;

__global__ void __launch_bounds__ (kDepthBlock)
depth_kernel (const int *__restrict__ parent, int n_inner, int *__restrict__ wide_flag,
              int *__restrict__ max_depth)
{
  __shared__ int s_parent[kDepthNodes];
  __shared__ int s_depth[kDepthNodes]; // of nodes whose parent is elsewhere, else -1
  __shared__ int s_max;
  const int b0 = blockIdx.x * kDepthNodes;
  const int count = min (kDepthNodes, n_inner - b0);
  if (threadIdx.x == 0) s_max = 0;
  for (int q = threadIdx.x; q < count; q += kDepthBlock)
  {
    const int p = parent[b0 + q];
    s_parent[q] = p - b0;
    int d = -1;
    if (p < b0 || p >= b0 + count)
    {
      d = 0;
      for (int j = p; j >= 0 && d < kMaxWalk; j = __ldg (parent + j)) ++d;
    }
    s_depth[q] = d;
  }
  __syncthreads ();
  int deepest = 0;
  for (int q = threadIdx.x; q < count; q += kDepthBlock)
  {
    int j = q, d = 0;
    while (s_depth[j] < 0 && d < kMaxWalk)
    {
      j = s_parent[j];
      ++d;
    }
    d += max (s_depth[j], 0);
    wide_flag[b0 + q] = (d & 1) == 0 ? 1 : 0;
    deepest = max (deepest, d);
  }
  deepest = __reduce_max_sync (0xffffffffu, deepest);
  if ((threadIdx.x & 31) == 0) atomicMax (&s_max, deepest);
  __syncthreads ();
  if (threadIdx.x == 0) atomicMax (max_depth, s_max);
}

// box c (0 left, 1 right) of a binary record: lo xyz, hi xyz
DRB_D void record_box (const float4 *__restrict__ rec, int c, float (&b)[6])
{
  const float4 a = rec[0], bb = rec[1], cc = rec[2];
  if (c == 0)
  {
    b[0] = a.x; b[1] = a.y; b[2] = a.z; b[3] = a.w; b[4] = bb.x; b[5] = bb.y;
  }
  else
  {
    b[0] = bb.z; b[1] = bb.w; b[2] = cc.x; b[3] = cc.y; b[4] = cc.z; b[5] = cc.w;
  }
}

// Child k of a wide row: its box (lo xyz, hi xyz) into the six SoA float4,
// its code into the seventh.
DRB_D void put_child (float *row, int k, const float (&box)[6], int code)
{
#pragma unroll
  for (int f = 0; f < 6; ++f) row[4 * f + k] = box[f];
  row[24 + k] = __int_as_float (code);
}

// wide_id: exclusive scan of the wide flags (n_wide in all), so node i is
// wide when the next value is larger.  The wide nodes of a block are
// consecutive: they are put together in shared memory and written as one
// run (a thread storing its own 128 bytes touched 32 lines a store).
constexpr int kEmitBlock = 128;
constexpr int kEmitRow = 33; // floats a row: 32 and a pad against bank conflicts

__global__ void __launch_bounds__ (kEmitBlock)
wide_emit_kernel (const float4 *__restrict__ nodes, int n_inner, const int *__restrict__ wide_id,
                  int n_wide, float4 *__restrict__ wide)
{
  __shared__ float s_row[kEmitBlock * kEmitRow];
  const int b0 = blockIdx.x * kEmitBlock;
  const int i = b0 + threadIdx.x;
  const int first = __ldg (wide_id + b0);
  const int end = b0 + kEmitBlock < n_inner ? __ldg (wide_id + b0 + kEmitBlock) : n_wide;
  const int id = i < n_inner ? __ldg (wide_id + i) : n_wide;
  const int next = i + 1 < n_inner ? __ldg (wide_id + i + 1) : n_wide;
  if (next > id)
  {
    float *row = s_row + (id - first) * kEmitRow;
    const float4 *rec = nodes + 4 * (size_t)i;
    const float4 d = rec[3];
    const int ch[2] = { __float_as_int (d.x), __float_as_int (d.y) };
    int k = 0;
#pragma unroll
    for (int c = 0; c < 2; ++c)
    {
      float box[6];
      if (ch[c] < 0)
      {
        record_box (rec, c, box);
        put_child (row, k++, box, ch[c]);
      }
      else
      {
        const float4 *rj = nodes + ch[c];
        const float4 dj = rj[3];
        const int gc[2] = { __float_as_int (dj.x), __float_as_int (dj.y) };
#pragma unroll
        for (int g = 0; g < 2; ++g)
        {
          record_box (rj, g, box);
          put_child (row, k++, box, gc[g] < 0 ? gc[g] : __ldg (wide_id + gc[g] / 4));
        }
      }
    }
    row[28] = __int_as_float (k);
    row[29] = row[30] = row[31] = 0.f;
    const float none[6] = { INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY };
    for (; k < 4; ++k) put_child (row, k, none, kWideEmpty);
  }
  __syncthreads ();
  float *out = reinterpret_cast<float *> (wide) + 32 * (size_t)first;
  for (int q = threadIdx.x; q < 32 * (end - first); q += kEmitBlock)
    out[q] = s_row[(q >> 5) * kEmitRow + (q & 31)];
}

// Wide index of every binary node (scan of the even-depth flags) into ids,
// n_wide and wide_depth of the BVH; synchronises for the two numbers.
int plan_wide (drb_bvh *bvh, int *ids, cudaStream_t s)
{
  const int n = bvh->n_inner;
  Scratch scr (s);
  int *parent = scr.alloc<int> (n);
  int *stat = scr.alloc<int> (2); // [0] max depth, [1] wide count
  if (!stat) return status_from (scr.err);
  cudaMemsetAsync (stat, 0, 2 * sizeof (int), s);
  parent_kernel<<<div_up (n, 256), 256, 0, s>>> ((const float4 *)bvh->inner_nodes, n, parent);
  int st = check_launch ("parent_kernel");
  if (st) return st;
  depth_kernel<<<div_up (n, kDepthNodes), kDepthBlock, 0, s>>> (parent, n, ids, stat);
  if ((st = check_launch ("depth_kernel"))) return st;
  if ((st = exclusive_scan_i32 (ids, ids, n, stat + 1, s))) return st;
  int h[2] = { 0, 0 };
  cudaError_t e = cudaMemcpyAsync (h, stat, sizeof (h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize (s);
  if (e != cudaSuccess)
  {
    set_last_error (cudaGetErrorString (e));
    return status_from (e);
  }
  bvh->n_wide = h[1];
  bvh->wide_depth = h[0] / 2 + 1;
  if (h[0] >= kMaxWalk || 3 * bvh->wide_depth + 1 > kWideStack)
  {
    set_last_error ("bvh_widen: tree too deep for the wide traversal stack");
    bvh->wide_nodes = nullptr;
    return DRB_ERR_UNSUPPORTED;
  }
  return DRB_OK;
}

int emit_wide (drb_bvh *bvh, const int *ids, float *wide_nodes, cudaStream_t s)
{
  const int n = bvh->n_inner;
  wide_emit_kernel<<<div_up (n, kEmitBlock), kEmitBlock, 0, s>>> ((const float4 *)bvh->inner_nodes, n,
                                                                  ids, bvh->n_wide, (float4 *)wide_nodes);
  int st = check_launch ("wide_emit_kernel");
  if (st == DRB_OK) bvh->wide_nodes = wide_nodes;
  return st;
}

bool widen_args_ok (const drb_bvh *bvh)
{
  if (bvh && bvh->inner_nodes && bvh->n_inner >= 1) return true;
  set_last_error ("bvh_widen: needs a built BVH");
  return false;
}

} // namespace
} // namespace drb

using namespace drb;

extern "C" int drb_bvh_widen (drb_bvh *bvh, float *wide_nodes, int capacity, void *stream)
{
  if (!widen_args_ok (bvh)) return DRB_ERR_INVALID_ARG;
  if (wide_nodes && capacity < 1)
  {
    set_last_error ("bvh_widen: needs a built BVH");
    return DRB_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  Scratch scr (s);
  int *ids = scr.alloc<int> (bvh->n_inner);
  if (!ids) return status_from (scr.err);
  int st = plan_wide (bvh, ids, s);
  if (st || !wide_nodes) return st; // size query
  if (capacity < bvh->n_wide)
  {
    set_last_error ("bvh_widen: wide node array too small (query the count first)");
    return DRB_ERR_INVALID_ARG;
  }
  return emit_wide (bvh, ids, wide_nodes, s);
}

extern "C" int drb_bvh_widen_plan (drb_bvh *bvh, int *wide_ids, void *stream)
{
  if (!widen_args_ok (bvh)) return DRB_ERR_INVALID_ARG;
  if (!wide_ids)
  {
    set_last_error ("bvh_widen_plan: wide_ids is NULL");
    return DRB_ERR_INVALID_ARG;
  }
  return plan_wide (bvh, wide_ids, (cudaStream_t)stream);
}

extern "C" int drb_bvh_widen_emit (drb_bvh *bvh, const int *wide_ids, float *wide_nodes, int capacity,
                                   void *stream)
{
  if (!widen_args_ok (bvh)) return DRB_ERR_INVALID_ARG;
  if (!wide_ids || !wide_nodes || capacity < bvh->n_wide || bvh->n_wide < 1)
  {
    set_last_error ("bvh_widen_emit: needs the plan's ids and n_wide wide nodes");
    return DRB_ERR_INVALID_ARG;
  }
  return emit_wide (bvh, wide_ids, wide_nodes, (cudaStream_t)stream);
}
