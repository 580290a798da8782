// LBVH construction over Bernstein element sub-boxes, B200-native.
//
// Pipeline (one stream, no host round trip until the final bounds copy):
//   subbox_kernel   warp per element, 32/16 de Casteljau splits held in shared
//                   memory (the reference spills them to a num_els*33*nd
//                   global scratch, data_model/mesh_utils.cpp:552-569), hull
//                   AABBs, x1.000001 scale, block-reduced scene bounds
//   morton_kernel   30-bit codes of the scaled-box centroids
//   radix sort      stable 4-pass LSD sort of (code, sub-box id)  (sort.cu)
//   tree_kernel     Karras 2012 radix tree with index tie-break, AABB union
//                   and 4 x float4 node records in one bottom-up pass
//
// Bit-exactness: the sub-box, scale, measure and Morton arithmetic use
// explicitly rounded intrinsics (__fadd_rn/__fmul_rn/__fsub_rn) in the same
// operation order as the reference so that no FMA contraction changes a
// bit; min/max and the integer tree steps are exact by construction.
#include "bernstein.cuh"
#include "drb_common.cuh"
#include "drb_internal.h"
#include "simplex.cuh"

#include <cstdio>
#include <cstring>
#include <vector>

namespace drb
{

namespace
{

constexpr int kSubboxWarps = 4;

template <int DIM> struct SplitCount
{
  // construct_bvh: splits = 2 * (2 << dim)  (mesh_utils.cpp:527)
  static constexpr int splits = 2 * (2 << DIM);
  static constexpr int boxes = splits + 1;
};

DRB_D float warp_min (float v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf (v, __shfl_xor_sync (0xffffffffu, v, o));
  return v;
}
DRB_D float warp_max (float v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf (v, __shfl_xor_sync (0xffffffffu, v, o));
  return v;
}

// Warp minimum and maximum of a float: one redux instruction (sm_100a has
// the f32 forms) in place of five shuffle steps.  NaN lanes are ignored, as
// fminf and fmaxf ignore them.
DRB_D float redux_min (float v)
{
  float r;
  asm volatile ("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
DRB_D float redux_max (float v)
{
  float r;
  asm volatile ("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// AABB::volume, falling back to AABB::surface_area when the volume is 0
// (aabb.hpp:173-195, mesh_utils.cpp:587-603).  Explicit rounding, same order.
DRB_D float box_measure (const float *b)
{
  const float l0 = __fsub_rn (b[1], b[0]);
  const float l1 = __fsub_rn (b[3], b[2]);
  const float l2 = __fsub_rn (b[5], b[4]);
  float vol = __fmul_rn (__fmul_rn (__fmul_rn (1.f, l0), l1), l2);
  if (vol == 0.f)
  {
    float area = __fmul_rn (__fmul_rn (2.f, l0), l1);
    area = __fadd_rn (area, __fmul_rn (__fmul_rn (2.f, l1), l2));
    area = __fadd_rn (area, __fmul_rn (__fmul_rn (2.f, l2), l0));
    vol = area;
  }
  return vol;
}

// Range::scale about the centre (range.hpp:162-172) with the float value of
// the double constant 1.000001 (mesh_utils.cpp:517, aabb.hpp:105-111).
DRB_D void scale_range (float &mn, float &mx, float s)
{
  if (mn > mx) return;
  const float c = __fmul_rn (0.5f, __fadd_rn (mn, mx));
  const float delta = __fmul_rn (__fmul_rn (s, 0.5f), __fsub_rn (mx, mn));
  mn = fminf (mn, __fsub_rn (c, delta));
  mx = fmaxf (mx, __fadd_rn (c, delta));
}

// Key of a box's measure for the warp's argmax: ordered as the floats are,
// so that the largest key, lowest lane first, is the box that the
// reference's scan picks (mesh_utils.cpp:586-603: replace on >, from box 0).
// A NaN never replaces, and a NaN in box 0 is never replaced.
DRB_D unsigned measure_key (const float (&b)[6], int lane)
{
  const float m = box_measure (b);
  if (m != m) return lane == 0 ? 0xffffffffu : 0u;
  return float_to_ordered (__fadd_rn (m, 0.f)); // -0 compares equal to +0
}

DRB_D int largest_box (unsigned key)
{
  const unsigned best = __reduce_max_sync (0xffffffffu, key);
  return __ffs (__ballot_sync (0xffffffffu, key == best)) - 1;
}

// Both halves of one line of a binary split at 0.5 by a single de Casteljau
// triangle: the first values of its rows are the [0, 0.5] half, the last
// ones the [0.5, 1] half.  The reference runs two in-place sweeps
// (split_inplace, data_model/elem_ops.hpp:1216-1405); each of their sums is
// one of the triangle's, of the same two products, so the bits are equal.
// m: the line's degree (m <= P); d: its m + 1 values, first half on return.
template <int P> DRB_D void split_line (float (&d)[P + 1], float (&second)[P + 1], int m)
{
#pragma unroll
  for (int a = 0; a <= P; ++a) second[a] = d[a];
#pragma unroll
  for (int row = 1; row <= P; ++row)
  {
    if (row > m) break;
#pragma unroll
    for (int a = 0; a + row <= P; ++a)
      if (a + row <= m) second[a] = __fadd_rn (__fmul_rn (second[a], 0.5f), __fmul_rn (second[a + 1], 0.5f));
    // second[0 .. m - row] is row `row`; its first value ends the first half
    d[row] = second[0];
  }
}

// Hulls of the two halves of a split box, from each lane's extremes of the
// values it holds (component comp[r] in round r, no values: +-INF).
template <int ROUNDS>
DRB_D void half_hulls (const int (&comp)[ROUNDS], const float (&lo1)[ROUNDS], const float (&hi1)[ROUNDS],
                       const float (&lo2)[ROUNDS], const float (&hi2)[ROUNDS], float (&b1)[6],
                       float (&b2)[6])
{
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    float l1 = INFINITY, h1 = -INFINITY, l2 = INFINITY, h2 = -INFINITY;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
      if (comp[r] == k)
      {
        l1 = fminf (l1, lo1[r]);
        h1 = fmaxf (h1, hi1[r]);
        l2 = fminf (l2, lo2[r]);
        h2 = fmaxf (h2, hi2[r]);
      }
    b1[2 * k] = redux_min (l1);
    b1[2 * k + 1] = redux_max (h1);
    b2[2 * k] = redux_min (l2);
    b2[2 * k + 1] = redux_max (h2);
  }
}

// Hull of ND control points in shared memory, the same in every lane
// (Element::get_bounds via positive_get_bounds, data_model/element.hpp:150-160).
template <int ND> DRB_D void warp_hull (const float *cps, float (&box)[6], int lane)
{
  float mn[3] = { INFINITY, INFINITY, INFINITY };
  float mx[3] = { -INFINITY, -INFINITY, -INFINITY };
  for (int i = lane; i < ND; i += kWarp)
  {
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      const float q = cps[3 * i + k];
      mn[k] = fminf (mn[k], q);
      mx[k] = fmaxf (mx[k], q);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    box[2 * k] = redux_min (mn[k]);
    box[2 * k + 1] = redux_max (mx[k]);
  }
}

// One finished sub-box: the scaled box, its element and reference box (R
// floats) to slot o, and its box into the block's scene bounds.
template <int R>
DRB_D void write_subbox (size_t o, int el, const float (&box)[6], const float *ref,
                         float *__restrict__ aabbs6, int *__restrict__ prim_ids,
                         float *__restrict__ ref_out, float (&bmn)[3], float (&bmx)[3])
{
  const float s = (float)1.000001;
  float bx[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) bx[q] = box[q];
#pragma unroll
  for (int k = 0; k < 3; ++k) scale_range (bx[2 * k], bx[2 * k + 1], s);
#pragma unroll
  for (int q = 0; q < 6; ++q) aabbs6[6 * o + q] = bx[q];
  if (prim_ids) prim_ids[o] = el;
#pragma unroll
  for (int q = 0; q < R; ++q) ref_out[R * o + q] = ref[q];
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    bmn[k] = fminf (bmn[k], bx[2 * k]);
    bmx[k] = fmaxf (bmx[k], bx[2 * k + 1]);
  }
}

// Scene bounds (reduce, linear_bvh_builder.cpp:19-58) of the boxes a block
// wrote: warp, then block, then ordered-integer atomics into bounds_ord.
DRB_D void reduce_scene_bounds (float (&bmn)[3], float (&bmx)[3], float (*s_bounds)[6], int warp,
                                int lane, unsigned *bounds_ord)
{
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    bmn[k] = warp_min (bmn[k]);
    bmx[k] = warp_max (bmx[k]);
  }
  if (lane == 0)
  {
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      s_bounds[warp][2 * k] = bmn[k];
      s_bounds[warp][2 * k + 1] = bmx[k];
    }
  }
  __syncthreads ();
  if (threadIdx.x < 6)
  {
    const int q = threadIdx.x;
    float v = s_bounds[0][q];
    for (int w = 1; w < kSubboxWarps; ++w)
      v = (q & 1) ? fmaxf (v, s_bounds[w][q]) : fminf (v, s_bounds[w][q]);
    if (!isinf (v))
    {
      if (q & 1) atomicMax (bounds_ord + q, float_to_ordered (v));
      else atomicMin (bounds_ord + q, float_to_ordered (v));
    }
  }
}

// A warp per element.  Lane b owns box b: its hull and measure key in
// registers, its reference box as the low corner and the number of halvings
// per axis (the reference boxes are dyadic, so low + 2^-halvings is exact).
// Only the control points live in shared memory.  A split is then an argmax
// over the lanes' keys (the first form scanned all measures again in every
// lane, 528 measures an element), one de Casteljau triangle per line that
// gives both halves, and twelve redux for the two hulls (the first form ran
// 60 shuffles).  Box NB - 1 = 32 of a hex is the last one made and never a
// candidate, so 32 lanes suffice.  Bound by instruction issue and the latency
// of the split's chain.  262,144 order-2 hexes: 8.0 -> 1.87 ms; 32,768 of
// order 3: 2.0 -> 0.47 ms.
template <int DIM, int P>
__global__ void __launch_bounds__ (kSubboxWarps * kWarp)
subbox_kernel (const int *__restrict__ ctrl_idx, const float *__restrict__ xyz, int n_elem,
               float *__restrict__ aabbs6, int *__restrict__ prim_ids, float *__restrict__ ref_out,
               unsigned *__restrict__ bounds_ord)
{
  constexpr int ND = (DIM == 3) ? (P + 1) * (P + 1) * (P + 1) : (P + 1) * (P + 1);
  constexpr int NB = SplitCount<DIM>::boxes;
  constexpr int NL = (DIM == 3) ? (P + 1) * (P + 1) : (P + 1);
  constexpr int CPW = NB * ND * 3; // control point floats per warp
  constexpr int ROUNDS = (3 * NL + kWarp - 1) / kWarp;
  extern __shared__ float smem[];
  __shared__ float s_bounds[kSubboxWarps][6];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  float *cps = smem + warp * CPW;

  const int el = blockIdx.x * kSubboxWarps + warp;
  float bmn[3] = { INFINITY, INFINITY, INFINITY };
  float bmx[3] = { -INFINITY, -INFINITY, -INFINITY };

  if (el < n_elem)
  {
    // box 0: the element itself, ref universe [0,1]^dim
    for (int t = lane; t < ND * 3; t += kWarp)
    {
      const int i = t / 3;
      const int k = t - 3 * i;
      cps[t] = __ldg (xyz + 3 * (size_t)__ldg (ctrl_idx + (size_t)el * ND + i) + k);
    }
    // this lane's (line, component) items: component major, and the float
    // offset of each item's first value for a split along each axis
    int comp[ROUNDS], first[ROUNDS][DIM];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
    {
      const int item = lane + r * kWarp;
      const int line = item % NL;
      comp[r] = item < 3 * NL ? item / NL : -1;
      int stride = 1;
#pragma unroll
      for (int d = 0; d < DIM; ++d)
      {
        const int chunk = line / stride;
        first[r][d] = 3 * (chunk * stride * (P + 1) + line - chunk * stride) + comp[r];
        stride *= P + 1;
      }
    }
    float box[6], low[DIM];
    int halvings = 0; // 8 bits per axis
#pragma unroll
    for (int d = 0; d < DIM; ++d) low[d] = 0.f;
    __syncwarp ();
    warp_hull<ND> (cps, box, lane);
    unsigned key = lane == 0 ? measure_key (box, lane) : 0u;
    float last_box[6], last_low[DIM];
    int last_halvings = 0;

    for (int count = 1; count < NB; ++count)
    {
      // largest-measure box, first one on ties
      const int mother_id = largest_box (key);
      // pick_binary_split: longest reference axis, first on ties
      // (mesh_utils.cpp:482-506), here the one with the fewest halvings
      int hv = __shfl_sync (0xffffffffu, halvings, mother_id);
      int axis = 0, fewest = hv & 255;
#pragma unroll
      for (int d = 1; d < DIM; ++d)
      {
        const int h = (hv >> (8 * d)) & 255;
        if (h < fewest)
        {
          axis = d;
          fewest = h;
        }
      }
      // split_subref<Tensor> (data_model/ref_space.hpp:148-171): the
      // daughter starts at the mother's middle
      float dlow[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d)
      {
        dlow[d] = __shfl_sync (0xffffffffu, low[d], mother_id);
        if (d == axis) dlow[d] = __fadd_rn (dlow[d], __int_as_float ((126 - fewest) << 23));
      }
      hv += 1 << (8 * axis);
      float *mother = cps + mother_id * ND * 3;
      float *dghter = cps + count * ND * 3;
      const int step = axis == 0 ? 3 : (axis == 1 ? 3 * (P + 1) : 3 * (P + 1) * (P + 1));
      float lo1[ROUNDS], hi1[ROUNDS], lo2[ROUNDS], hi2[ROUNDS];
#pragma unroll
      for (int r = 0; r < ROUNDS; ++r)
      {
        lo1[r] = lo2[r] = INFINITY;
        hi1[r] = hi2[r] = -INFINITY;
        if (comp[r] >= 0)
        {
          int at = first[r][0];
#pragma unroll
          for (int d = 1; d < DIM; ++d)
            if (axis == d) at = first[r][d];
          float d1[P + 1], d2[P + 1];
#pragma unroll
          for (int a = 0; a <= P; ++a) d1[a] = mother[at + a * step];
          split_line<P> (d1, d2, P);
#pragma unroll
          for (int a = 0; a <= P; ++a)
          {
            mother[at + a * step] = d1[a];
            dghter[at + a * step] = d2[a];
            lo1[r] = fminf (lo1[r], d1[a]);
            hi1[r] = fmaxf (hi1[r], d1[a]);
            lo2[r] = fminf (lo2[r], d2[a]);
            hi2[r] = fmaxf (hi2[r], d2[a]);
          }
        }
      }
      float b1[6], b2[6];
      half_hulls<ROUNDS> (comp, lo1, hi1, lo2, hi2, b1, b2);
      const bool is_daughter = lane == count;
      if (lane == mother_id || is_daughter)
      {
#pragma unroll
        for (int q = 0; q < 6; ++q) box[q] = is_daughter ? b2[q] : b1[q];
        key = measure_key (box, lane);
        halvings = hv;
        if (is_daughter)
        {
#pragma unroll
          for (int d = 0; d < DIM; ++d) low[d] = dlow[d];
        }
      }
      if (NB > kWarp && count == NB - 1)
      {
#pragma unroll
        for (int q = 0; q < 6; ++q) last_box[q] = b2[q];
#pragma unroll
        for (int d = 0; d < DIM; ++d) last_low[d] = dlow[d];
        last_halvings = hv;
      }
      __syncwarp ();
    }

    const size_t o = (size_t)el * NB;
    float ref[2 * DIM];
    if (lane < NB)
    {
#pragma unroll
      for (int d = 0; d < DIM; ++d)
      {
        ref[d] = low[d];
        ref[DIM + d] = __fadd_rn (low[d], __int_as_float ((127 - ((halvings >> (8 * d)) & 255)) << 23));
      }
      write_subbox<2 * DIM> (o + lane, el, box, ref, aabbs6, prim_ids, ref_out, bmn, bmx);
    }
    if (NB > kWarp && lane == 0)
    {
#pragma unroll
      for (int d = 0; d < DIM; ++d)
      {
        ref[d] = last_low[d];
        ref[DIM + d] = __fadd_rn (last_low[d], __int_as_float ((127 - ((last_halvings >> (8 * d)) & 255)) << 23));
      }
      write_subbox<2 * DIM> (o + NB - 1, el, last_box, ref, aabbs6, prim_ids, ref_out, bmn, bmx);
    }
  }
  reduce_scene_bounds (bmn, bmx, s_bounds, warp, lane, bounds_ord);
}

// ---- simplex (tet) sub-boxes -------------------------------------------
//
// Same forall as the tensor case (mesh_utils.cpp:557-670, 33 boxes per tet)
// with the simplex split: the reference sub-simplex is four vertices (u, v,
// w axis vertices, then the origin; ref_space.hpp:36-46); the split halves
// its longest edge (first pair v1 < v2 on ties, mesh_utils.cpp:455-480) and
// moves the `displaced` vertex to the midpoint (split_subref<Simplex>,
// ref_space.hpp:133-146); the control points of both halves come from
// de Casteljau along that edge (split_inplace<3,Simplex>,
// elem_ops.hpp:1270-1311).  The reference linearises the dof multi-index
// there with cartesian_to_tet_idx (elem_ops.hpp:32-47), whose in-layer term
// uses the full edge length instead of the layer's: for orders >= 2 it
// addresses the wrong dofs (e.g. order 2 maps (0,1,1) and (0,0,2) both to
// 9) and order 3 reaches index 20 of a 20-dof element.  The layout every
// evaluator uses (the general-order eval_d walk, elem_ops.hpp:945-1030) is
// the layered one of tet_index, which this kernel uses, so its sub-boxes
// bound the split geometry at every order; at order 1 the two indexings
// coincide and the boxes are bit-identical to the reference's.

constexpr int kTetRefFloats = 12; // SubRef<3,Simplex>: four vertices
constexpr int kTriRefFloats = 6;  // SubRef<2,Simplex>: three vertices

// ---- simplex faces (triangles): 17 sub-boxes per triangle ----
//
// The same split with dim 2: the reference sub-triangle is three vertices
// (u and v axis vertices, then the origin), the longest of its three edges
// is halved, and split_inplace<2,Simplex> (elem_ops.hpp:1216-1250) runs de
// Casteljau along it on the rows parallel to it.  Its triangle index
// (cartesian_to_tri_idx) is the evaluators' layout, so these boxes match the
// reference's at every order.

// Lines of a simplex split: for each pair of vertices (displaced v0 <
// tradeoff v1, in the order of the edge search) and each line (the dofs with
// fixed exponents of the other vertices), the dof with exponent a of v0 in
// byte a.  Line l is the same (exponents, degree) for every pair.
template <int DIM, int P> struct SimplexLines
{
  static constexpr int kPairs = DIM == 3 ? 6 : 3;
  static constexpr int kLines = DIM == 3 ? (P + 1) * (P + 2) / 2 : P + 1;
  unsigned ids[kPairs][kLines];
  int degree[kLines];
};

template <int DIM, int P> constexpr SimplexLines<DIM, P> simplex_lines ()
{
  SimplexLines<DIM, P> t{};
  int pair = 0;
  for (int v0 = 0; v0 < DIM; ++v0)
    for (int v1 = v0 + 1; v1 <= DIM; ++v1, ++pair)
    {
      int v2 = 0;
      while (v2 == v0 || v2 == v1) ++v2;
      const int v3 = DIM == 3 ? 6 - v0 - v1 - v2 : 0;
      int line = 0;
      for (int h = 0; h <= (DIM == 3 ? P : 0); ++h)
        for (int g = 0; g + h <= P; ++g, ++line)
        {
          const int m = P - g - h;
          unsigned packed = 0;
          for (int a = 0; a <= m; ++a)
          {
            int b[4] = { 0, 0, 0, 0 };
            b[v0] = a;
            b[v1] = m - a;
            b[v2] = g;
            if (DIM == 3) b[v3] = h;
            const int id = DIM == 3 ? tet_index (b[0], b[1], b[2], P) : tri_index (b[0], b[1], P);
            packed |= (unsigned)id << (8 * a);
          }
          t.ids[pair][line] = packed;
          t.degree[line] = m;
        }
    }
  return t;
}

template <int DIM, int P> __device__ const SimplexLines<DIM, P> kSimplexLines = simplex_lines<DIM, P> ();

// The tensor kernel's scheme for tets (33 sub-boxes) and triangles (17).
// The reference sub-simplices stay in shared memory (their vertices are
// read by every lane for the edge search); every item (line, component) has
// a lane of its own, degree-0 lines among them, which both halves share.
template <int DIM, int P>
__global__ void __launch_bounds__ (kSubboxWarps * kWarp)
simplex_subbox_kernel (const int *__restrict__ ctrl_idx, const float *__restrict__ xyz, int n_elem,
                       float *__restrict__ aabbs6, int *__restrict__ prim_ids,
                       float *__restrict__ ref_out, unsigned *__restrict__ bounds_ord)
{
  using Lines = SimplexLines<DIM, P>;
  constexpr int ND = DIM == 3 ? tet_dofs<P> () : tri_dofs<P> ();
  constexpr int NB = SplitCount<DIM>::boxes;
  constexpr int R = DIM == 3 ? kTetRefFloats : kTriRefFloats;
  constexpr int CPW = NB * ND * 3;
  static_assert (3 * Lines::kLines <= kWarp, "one item per lane");
  extern __shared__ float smem[];
  __shared__ float s_bounds[kSubboxWarps][6];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  float *cps = smem + warp * CPW;
  float *refs = smem + kSubboxWarps * CPW + warp * NB * R;

  const int el = blockIdx.x * kSubboxWarps + warp;
  float bmn[3] = { INFINITY, INFINITY, INFINITY };
  float bmx[3] = { -INFINITY, -INFINITY, -INFINITY };

  if (el < n_elem)
  {
    for (int t = lane; t < ND * 3; t += kWarp)
    {
      const int i = t / 3;
      const int k = t - 3 * i;
      cps[t] = __ldg (xyz + 3 * (size_t)__ldg (ctrl_idx + (size_t)el * ND + i) + k);
    }
    // ref_universe<Simplex>: unit axis vertices, then the origin
    if (lane < R) refs[lane] = (lane < DIM * DIM && lane % (DIM + 1) == 0) ? 1.f : 0.f;
    const int line = lane % Lines::kLines;
    const int comp[1] = { lane < 3 * Lines::kLines ? lane / Lines::kLines : -1 };
    const int degree = kSimplexLines<DIM, P>.degree[line];
    unsigned ids[Lines::kPairs];
#pragma unroll
    for (int q = 0; q < Lines::kPairs; ++q) ids[q] = kSimplexLines<DIM, P>.ids[q][line];
    float box[6];
    __syncwarp ();
    warp_hull<ND> (cps, box, lane);
    unsigned key = lane == 0 ? measure_key (box, lane) : 0u;
    float last_box[6];

    for (int count = 1; count < NB; ++count)
    {
      const int mother_id = largest_box (key);
      // pick_binary_split<Simplex>: longest reference edge (squared length
      // summed in component order), first pair on ties
      float *rm = refs + mother_id * R;
      int dv = 0, tv = 1, pair = 0, q = 0;
      float max_l2 = 0.f;
#pragma unroll
      for (int a = 0; a < DIM; ++a)
#pragma unroll
        for (int b = a + 1; b <= DIM; ++b, ++q)
        {
          float l2 = 0.f;
#pragma unroll
          for (int d = 0; d < DIM; ++d)
          {
            const float e = __fsub_rn (rm[DIM * a + d], rm[DIM * b + d]);
            l2 = d == 0 ? __fmul_rn (e, e) : __fadd_rn (l2, __fmul_rn (e, e));
          }
          if (l2 > max_l2)
          {
            dv = a;
            tv = b;
            pair = q;
            max_l2 = l2;
          }
        }
      __syncwarp ();
      if (lane < R)
      {
        // split_subref<Simplex> (ref_space.hpp:133-146): the mother's
        // displaced vertex and the daughter's tradeoff vertex move to the
        // edge's middle
        const int v = lane / DIM, d = lane - v * DIM;
        const float sp = __fadd_rn (__fmul_rn (rm[DIM * tv + d], 0.5f), __fmul_rn (rm[DIM * dv + d], 0.5f));
        const float keep = rm[lane];
        __syncwarp (R == 32 ? 0xffffffffu : (1u << R) - 1u);
        refs[count * R + lane] = v == tv ? sp : keep;
        if (v == dv) rm[lane] = sp;
      }
      // mother: split (displaced dv, tradeoff tv); daughter: the complement
      float *mother = cps + mother_id * ND * 3;
      float *dghter = cps + count * ND * 3;
      float lo1[1] = { INFINITY }, hi1[1] = { -INFINITY }, lo2[1] = { INFINITY }, hi2[1] = { -INFINITY };
      if (comp[0] >= 0)
      {
        unsigned packed = ids[0];
#pragma unroll
        for (int p = 1; p < Lines::kPairs; ++p)
          if (pair == p) packed = ids[p];
        // from the tradeoff end: the daughter's half is the second one
        float d1[P + 1], d2[P + 1];
#pragma unroll
        for (int a = 0; a <= P; ++a)
          d1[a] = a <= degree ? mother[3 * ((packed >> (8 * a)) & 255) + comp[0]] : 0.f;
        split_line<P> (d1, d2, degree);
#pragma unroll
        for (int a = 0; a <= P; ++a)
          if (a <= degree)
          {
            const int at = 3 * ((packed >> (8 * a)) & 255) + comp[0];
            mother[at] = d1[a];
            dghter[at] = d2[a];
            lo1[0] = fminf (lo1[0], d1[a]);
            hi1[0] = fmaxf (hi1[0], d1[a]);
            lo2[0] = fminf (lo2[0], d2[a]);
            hi2[0] = fmaxf (hi2[0], d2[a]);
          }
      }
      float b1[6], b2[6];
      half_hulls<1> (comp, lo1, hi1, lo2, hi2, b1, b2);
      const bool is_daughter = lane == count;
      if (lane == mother_id || is_daughter)
      {
#pragma unroll
        for (int p = 0; p < 6; ++p) box[p] = is_daughter ? b2[p] : b1[p];
        key = measure_key (box, lane);
      }
      if (NB > kWarp && count == NB - 1)
      {
#pragma unroll
        for (int p = 0; p < 6; ++p) last_box[p] = b2[p];
      }
      __syncwarp ();
    }

    const size_t o = (size_t)el * NB;
    if (lane < NB) write_subbox<R> (o + lane, el, box, refs + lane * R, aabbs6, prim_ids, ref_out, bmn, bmx);
    if (NB > kWarp && lane == 0)
      write_subbox<R> (o + NB - 1, el, last_box, refs + (NB - 1) * R, aabbs6, prim_ids, ref_out, bmn, bmx);
  }
  reduce_scene_bounds (bmn, bmx, s_bounds, warp, lane, bounds_ord);
}

__global__ void bounds_init_kernel (unsigned *bounds_ord)
{
  const int q = threadIdx.x;
  if (q < 6) bounds_ord[q] = (q & 1) ? float_to_ordered (-INFINITY) : float_to_ordered (INFINITY);
}

__global__ void bounds_finish_kernel (const unsigned *bounds_ord, float *bounds6)
{
  const int q = threadIdx.x;
  if (q < 6) bounds6[q] = ordered_to_float (bounds_ord[q]);
}

// get_mcodes + morton_3d (linear_bvh_builder.cpp:60-90, morton_codes.hpp:16-53)
DRB_D unsigned expand_bits32 (unsigned x)
{
  x = (x | (x << 16)) & 0x030000FFu;
  x = (x | (x << 8)) & 0x0300F00Fu;
  x = (x | (x << 4)) & 0x030C30C3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

__global__ void morton_kernel (const float *__restrict__ aabbs6, int n,
                               const float *__restrict__ bounds6, unsigned *__restrict__ codes)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float mn[3], inv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    mn[k] = bounds6[2 * k];
    const float ext = __fsub_rn (bounds6[2 * k + 1], bounds6[2 * k]);
    inv[k] = (ext == 0.f) ? 0.f : __fdiv_rn (1.f, ext);
  }
  unsigned e[3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    const float lo = aabbs6[6 * (size_t)i + 2 * k];
    const float hi = aabbs6[6 * (size_t)i + 2 * k + 1];
    // Range::center returns NaN for an empty range (range.hpp:130-137)
    const float c = (lo > hi) ? __int_as_float (0x7fc00000) : __fmul_rn (0.5f, __fadd_rn (lo, hi));
    float x = __fmul_rn (__fsub_rn (c, mn[k]), inv[k]);
    x = fminf (fmaxf (__fmul_rn (x, 1024.0f), 0.0f), 1023.0f);
    e[k] = expand_bits32 ((unsigned)x);
  }
  codes[i] = (e[2] << 2) | (e[1] << 1) | e[0];
}

// ---- tree: Karras topology, refit and node records in one bottom-up pass --
//
// The reference builds the Karras 2012 radix tree top-down per node
// (linear_bvh_builder.cpp:149-251), then refits (:253-317) and emits
// (:319-397).  The same tree forms bottom-up (Apetrei 2014): the node over
// the sorted leaves [l, r] joins the neighbour across its closer end, where
// closeness is the reference's delta (common prefix of the 30-bit codes, the
// index breaking ties), which is a strict order along any node's ends.  Of
// the two children the second to arrive builds the parent: it has the whole
// range, both boxes and both child codes, so the final 64-byte record is
// written at once, and the topology arrays, the sorted box copy and two of
// the three passes over them are not needed.  A node's index is Karras': r
// for a left child, l for a right child, 0 for the root.  Nothing waits: the
// first arrival leaves its box and ends.
//
// A block takes kTreeBlock consecutive leaves.  Joins whose result lies
// inside the block (known beforehand from prefix and suffix minima of the
// deltas: the result ends where the delta drops below the join's) go through
// shared memory; only the nodes that cross a block border, a few dozen per
// block, use global memory and its atomics.
// 8.65M leaves: 0.67 ms, against 1.41 ms for the four kernels it replaces
// (gather, top-down Karras, refit with global atomics, emit).  Bound by the
// scattered 64-byte records and the box gather.
constexpr int kTreeBlock = 256;

// delta of the sorted leaves j and j + 1 (linear_bvh_builder.cpp:149-167)
DRB_D int adjacent_delta (const unsigned *__restrict__ codes, int j, int n)
{
  if (j < 0 || j >= n - 1) return -1;
  const unsigned x = __ldg (codes + j) ^ __ldg (codes + j + 1);
  return x ? __clz (x) : 32 + __clz ((unsigned)j ^ (unsigned)(j + 1));
}

// Exchange with release and acquire at device scope: what a thread wrote
// before its exchange is visible to the one that gets its value.
DRB_D int exchange_acq_rel (int *p, int v)
{
  int old;
  asm volatile ("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

// Node record (bvh.hpp:16-37): left box, right box, child codes (4 x node
// for an inner child, -(leaf + 1) for a leaf).  Boxes are x0 x1 y0 y1 z0 z1.
DRB_D void write_record (float4 *__restrict__ nodes, int id, const float (&lb)[6], const float (&rb)[6],
                         int lcode, int rcode)
{
  float4 *o = nodes + 4 * (size_t)id;
  o[0] = make_float4 (lb[0], lb[2], lb[4], lb[1]);
  o[1] = make_float4 (lb[3], lb[5], rb[0], rb[2]);
  o[2] = make_float4 (rb[4], rb[1], rb[3], rb[5]);
  o[3] = make_float4 (__int_as_float (lcode), __int_as_float (rcode), 0.f, 0.f);
}

// inner_box: 8 floats per inner node (32-byte sectors), met: n - 1 ints of -1.
__global__ void __launch_bounds__ (kTreeBlock)
tree_kernel (const unsigned *__restrict__ codes, const int *__restrict__ perm,
             const float *__restrict__ aabbs6, int n, int boxes_per_elem, int *__restrict__ leaf_nodes,
             float *inner_box, int *met, float4 *__restrict__ nodes)
{
  __shared__ int s_delta[kTreeBlock + 1];  // of leaf pairs (b0 - 1 + q, b0 + q)
  __shared__ float s_leaf[kTreeBlock][7];  // odd stride: no bank conflicts
  __shared__ float s_inner[kTreeBlock][7]; // by node index - b0
  __shared__ int s_met[kTreeBlock];
  __shared__ bool s_inside[kTreeBlock];    // join at b0 + q stays in the block
  __shared__ int s_warp_min[2][kTreeBlock / kWarp];
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.x * kTreeBlock;
  const int b1 = min (b0 + kTreeBlock, n);
  const int i = b0 + tid;
  constexpr int kFar = 1 << 20;

  float box[6];
  const int here = i < n ? adjacent_delta (codes, i, n) : kFar;
  if (tid == 0) s_delta[0] = adjacent_delta (codes, b0 - 1, n);
  s_delta[tid + 1] = here;
  s_met[tid] = -1;
  if (i < n)
  {
    const int src = perm[i];
    leaf_nodes[i] = src / boxes_per_elem;
#pragma unroll
    for (int q = 0; q < 6; ++q)
    {
      box[q] = __ldg (aabbs6 + 6 * (size_t)src + q);
      s_leaf[tid][q] = box[q];
    }
  }
  // minima of the deltas before and after each join
  int before = here, after = here;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const int u = __shfl_up_sync (0xffffffffu, before, o);
    const int d = __shfl_down_sync (0xffffffffu, after, o);
    if (lane >= o) before = min (before, u);
    if (lane + o < 32) after = min (after, d);
  }
  if (lane == 31) s_warp_min[0][warp] = before;
  if (lane == 0) s_warp_min[1][warp] = after;
  before = __shfl_up_sync (0xffffffffu, before, 1);
  after = __shfl_down_sync (0xffffffffu, after, 1);
  if (lane == 0) before = kFar;
  if (lane == 31) after = kFar;
  __syncthreads ();
  before = min (before, s_delta[0]);
  for (int w = 0; w < warp; ++w) before = min (before, s_warp_min[0][w]);
  for (int w = warp + 1; w < kTreeBlock / kWarp; ++w) after = min (after, s_warp_min[1][w]);
  s_inside[tid] = i < b1 - 1 && before < here && after < here;
  __syncthreads ();
  if (i >= n) return;

  int l = i, r = i, code = -(i + 1);
  int dl = s_delta[tid], dr = here;
  while (true)
  {
    if (l == 0 && r == n - 1) return; // the root is written
    const bool left = dr > dl; // a left child: the parent joins at r
    const int p = left ? r : l - 1;
    const bool inside = p >= b0 && p < b1 - 1 && s_inside[p - b0];
    const int id = left ? r : l; // this node's index, if it is an inner one
    int other;
    if (inside)
    {
      if (l != r)
      {
#pragma unroll
        for (int q = 0; q < 6; ++q) s_inner[id - b0][q] = box[q];
      }
      __threadfence_block ();
      other = atomicExch (&s_met[p - b0], left ? l : r);
      if (other < 0) return;
      __threadfence_block ();
    }
    else
    {
      if (l != r)
      {
        float4 *o = reinterpret_cast<float4 *> (inner_box + 8 * (size_t)id);
        __stcg (o, make_float4 (box[0], box[1], box[2], box[3]));
        __stcg (o + 1, make_float4 (box[4], box[5], 0.f, 0.f));
      }
      other = exchange_acq_rel (met + p, left ? l : r);
      if (other < 0) return;
    }
    // the sibling: [p + 1, other] of a left child, [other, p] of a right one
    const int sib_id = left ? p + 1 : p;
    const bool sib_leaf = other == sib_id;
    float sib[6];
    if (inside)
    {
      const volatile float *sb = sib_leaf ? s_leaf[sib_id - b0] : s_inner[sib_id - b0];
#pragma unroll
      for (int q = 0; q < 6; ++q) sib[q] = sb[q];
    }
    else if (sib_leaf)
    {
      const size_t src = __ldg (perm + sib_id);
#pragma unroll
      for (int q = 0; q < 6; ++q) sib[q] = __ldg (aabbs6 + 6 * src + q);
    }
    else
    {
      const float4 *o = reinterpret_cast<const float4 *> (inner_box + 8 * (size_t)sib_id);
      const float4 a = __ldcg (o), b = __ldcg (o + 1);
      sib[0] = a.x, sib[1] = a.y, sib[2] = a.z, sib[3] = a.w, sib[4] = b.x, sib[5] = b.y;
    }
    const int sib_code = sib_leaf ? -(sib_id + 1) : 4 * sib_id;
    if (left)
    {
      r = other;
      dr = inside ? s_delta[r - b0 + 1] : adjacent_delta (codes, r, n);
    }
    else
    {
      l = other;
      dl = inside ? s_delta[l - b0] : adjacent_delta (codes, l - 1, n);
    }
    const int parent = (l == 0 && r == n - 1) ? 0 : (dr > dl ? r : l);
    if (left) write_record (nodes, parent, box, sib, code, sib_code);
    else write_record (nodes, parent, sib, box, sib_code, code);
    code = 4 * parent;
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      box[2 * k] = fminf (box[2 * k], sib[2 * k]);
      box[2 * k + 1] = fmaxf (box[2 * k + 1], sib[2 * k + 1]);
    }
  }
}

template <int NC>
__global__ void pack_kernel (const int *__restrict__ ctrl_idx, const float *__restrict__ vals,
                             int n_elem, int nd, int stride, float *__restrict__ packed)
{
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)n_elem * stride;
  if (t >= total) return;
  const int e = (int)(t / stride);
  const int r = (int)(t - (long long)e * stride);
  float v = 0.f;
  if (r < nd * NC)
  {
    const int i = r / NC;
    const int k = r - NC * i;
    v = __ldg (vals + (size_t)NC * __ldg (ctrl_idx + (size_t)e * nd + i) + k);
    // geometry rows: relative to the first control point (packed_stride)
    if (NC == 3) v = __fsub_rn (v, __ldg (vals + (size_t)NC * __ldg (ctrl_idx + (size_t)e * nd) + k));
  }
  else if (NC == 3 && r < nd * NC + 3)
  {
    v = __ldg (vals + (size_t)NC * __ldg (ctrl_idx + (size_t)e * nd) + (r - nd * NC));
  }
  packed[t] = v;
}

template <int DIM, int P>
int launch_subbox (const drb_mesh *m, float *aabbs6, int *prim_ids, float *ref_boxes,
                   unsigned *bounds_ord, cudaStream_t s)
{
  constexpr int ND = (DIM == 3) ? (P + 1) * (P + 1) * (P + 1) : (P + 1) * (P + 1);
  constexpr size_t smem = sizeof (float) * kSubboxWarps * SplitCount<DIM>::boxes * ND * 3;
  cudaFuncSetAttribute (subbox_kernel<DIM, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                        (int)smem);
  const int blocks = div_up (m->n_elem, kSubboxWarps);
  if (blocks > 0)
    subbox_kernel<DIM, P><<<blocks, kSubboxWarps * kWarp, smem, s>>> (
    m->ctrl_idx, m->values, m->n_elem, aabbs6, prim_ids, ref_boxes, bounds_ord);
  return check_launch ("subbox_kernel");
}

template <int DIM, int P>
int launch_simplex_subbox (const drb_mesh *m, float *aabbs6, int *prim_ids, float *ref_boxes,
                           unsigned *bounds_ord, cudaStream_t s)
{
  constexpr int ND = DIM == 3 ? tet_dofs<P> () : tri_dofs<P> ();
  constexpr int R = DIM == 3 ? kTetRefFloats : kTriRefFloats;
  constexpr size_t smem = sizeof (float) * kSubboxWarps * SplitCount<DIM>::boxes * (ND * 3 + R);
  cudaFuncSetAttribute (simplex_subbox_kernel<DIM, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                        (int)smem);
  const int blocks = div_up (m->n_elem, kSubboxWarps);
  if (blocks > 0)
    simplex_subbox_kernel<DIM, P><<<blocks, kSubboxWarps * kWarp, smem, s>>> (
    m->ctrl_idx, m->values, m->n_elem, aabbs6, prim_ids, ref_boxes, bounds_ord);
  return check_launch ("simplex_subbox_kernel");
}

int dispatch_subbox (const drb_mesh *m, float *aabbs6, int *prim_ids, float *ref_boxes,
                     unsigned *bounds_ord, cudaStream_t s)
{
  if (m->shape == DRB_SHAPE_SIMPLEX && m->dim == 3)
  {
    if (m->order == 1) return launch_simplex_subbox<3, 1> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 2) return launch_simplex_subbox<3, 2> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 3) return launch_simplex_subbox<3, 3> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
  }
  else if (m->shape == DRB_SHAPE_SIMPLEX && m->dim == 2)
  {
    if (m->order == 1) return launch_simplex_subbox<2, 1> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 2) return launch_simplex_subbox<2, 2> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 3) return launch_simplex_subbox<2, 3> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
  }
  else if (m->shape != DRB_SHAPE_TENSOR)
  {
    set_last_error ("subbox: unknown element shape");
    return DRB_ERR_UNSUPPORTED;
  }
  else if (m->dim == 3)
  {
    if (m->order == 1) return launch_subbox<3, 1> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 2) return launch_subbox<3, 2> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 3) return launch_subbox<3, 3> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
  }
  else if (m->dim == 2)
  {
    if (m->order == 1) return launch_subbox<2, 1> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 2) return launch_subbox<2, 2> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
    if (m->order == 3) return launch_subbox<2, 3> (m, aabbs6, prim_ids, ref_boxes, bounds_ord, s);
  }
  set_last_error ("subbox: dim must be 2 or 3 and order 1..3");
  return DRB_ERR_UNSUPPORTED;
}

int validate_mesh (const drb_mesh *m, int want_ncomp)
{
  if (!m) { set_last_error ("mesh is NULL"); return DRB_ERR_INVALID_ARG; }
  if (m->dim != 2 && m->dim != 3) { set_last_error ("mesh dim must be 2 or 3"); return DRB_ERR_INVALID_ARG; }
  if (m->shape != DRB_SHAPE_TENSOR && m->shape != DRB_SHAPE_SIMPLEX)
  {
    set_last_error ("mesh shape must be tensor or simplex");
    return DRB_ERR_UNSUPPORTED;
  }
  if (m->order < 1 || m->order > 3) { set_last_error ("mesh order must be 1..3"); return DRB_ERR_UNSUPPORTED; }
  if (m->ncomp != want_ncomp) { set_last_error ("mesh ncomp mismatch"); return DRB_ERR_INVALID_ARG; }
  if (m->n_elem < 0 || m->n_ctrl < 0) { set_last_error ("negative mesh size"); return DRB_ERR_INVALID_ARG; }
  if (m->n_elem > 0 && (!m->ctrl_idx || !m->values)) { set_last_error ("mesh arrays are NULL"); return DRB_ERR_INVALID_ARG; }
  const long long nb = (m->dim == 3) ? 33 : 17;
  if ((long long)m->n_elem * nb >= (1ll << 31) - 1) { set_last_error ("too many sub-boxes for int32 leaf ids"); return DRB_ERR_INVALID_ARG; }
  return DRB_OK;
}

} // namespace

int mesh_nd (int dim, int order)
{
  int nd = 1;
  for (int d = 0; d < dim; ++d) nd *= (order + 1);
  return nd;
}

int mesh_nd (const drb_mesh *m)
{
  if (m->shape == DRB_SHAPE_SIMPLEX) return m->dim == 2 ? tri_dofs (m->order) : tet_dofs (m->order);
  return mesh_nd (m->dim, m->order);
}

} // namespace drb

using namespace drb;

extern "C" int drb_packed_stride (int dim, int order, int ncomp)
{
  if ((dim != 2 && dim != 3) || order < 1 || order > 3 || ncomp < 1) return -1;
  return packed_stride (mesh_nd (dim, order), ncomp);
}

extern "C" int drb_elem_dofs (int shape, int dim, int order)
{
  if (order < 1 || order > 3) return -1;
  if (shape == DRB_SHAPE_TENSOR && (dim == 2 || dim == 3)) return mesh_nd (dim, order);
  if (shape == DRB_SHAPE_SIMPLEX && dim == 3) return tet_dofs (order);
  if (shape == DRB_SHAPE_SIMPLEX && dim == 2) return tri_dofs (order);
  return -1;
}

extern "C" int drb_packed_stride_shape (int shape, int dim, int order, int ncomp)
{
  const int nd = drb_elem_dofs (shape, dim, order);
  if (nd < 0 || ncomp < 1) return -1;
  return packed_stride (nd, ncomp);
}

extern "C" int drb_ref_box_floats (int shape, int dim)
{
  if (dim != 2 && dim != 3) return -1;
  if (shape == DRB_SHAPE_TENSOR) return 2 * dim;
  if (shape == DRB_SHAPE_SIMPLEX) return dim * (dim + 1);
  return -1;
}

extern "C" int drb_pack_elements (const drb_mesh *mesh, float *packed, void *stream)
{
  if (!mesh || (mesh->ncomp != 1 && mesh->ncomp != 3)) { set_last_error ("pack: bad mesh"); return DRB_ERR_INVALID_ARG; }
  int st = validate_mesh (mesh, mesh->ncomp);
  if (st) return st;
  if (mesh->n_elem == 0) return DRB_OK;
  if (!packed) { set_last_error ("pack: output NULL"); return DRB_ERR_INVALID_ARG; }
  const int nd = mesh_nd (mesh);
  const int stride = packed_stride (nd, mesh->ncomp);
  const long long total = (long long)mesh->n_elem * stride;
  cudaStream_t s = (cudaStream_t)stream;
  const int blocks = div_up (total, 256);
  if (mesh->ncomp == 3)
    pack_kernel<3><<<blocks, 256, 0, s>>> (mesh->ctrl_idx, mesh->values, mesh->n_elem, nd, stride, packed);
  else
    pack_kernel<1><<<blocks, 256, 0, s>>> (mesh->ctrl_idx, mesh->values, mesh->n_elem, nd, stride, packed);
  return check_launch ("pack_kernel");
}

extern "C" int drb_bvh_sizes (int dim, int n_elem, int *n_inner, int *n_leaf)
{
  if ((dim != 2 && dim != 3) || n_elem < 0 || !n_inner || !n_leaf)
  {
    set_last_error ("bvh_sizes: bad arguments");
    return DRB_ERR_INVALID_ARG;
  }
  const long long nb = (dim == 3) ? SplitCount<3>::boxes : SplitCount<2>::boxes;
  long long leaves = nb * n_elem;
  if (leaves >= (1ll << 31) - 1) { set_last_error ("bvh_sizes: too many leaves"); return DRB_ERR_INVALID_ARG; }
  // 0 primitives: the reference inserts two dummy leaves (linear_bvh_builder.cpp:411-433)
  if (leaves == 0) leaves = 2;
  *n_leaf = (int)leaves;
  *n_inner = (int)leaves - 1;
  return DRB_OK;
}

extern "C" int drb_elem_subboxes (const drb_mesh *mesh, float *aabbs6, int *prim_ids,
                                  float *ref_boxes, float *bounds6, void *stream)
{
  int st = validate_mesh (mesh, 3);
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  Scratch scr (s);
  unsigned *bord = scr.alloc<unsigned> (6);
  if (!bord) return status_from (scr.err);
  bounds_init_kernel<<<1, 32, 0, s>>> (bord);
  if ((st = check_launch ("bounds_init_kernel"))) return st;
  st = dispatch_subbox (mesh, aabbs6, prim_ids, ref_boxes, bord, s);
  if (st) return st;
  bounds_finish_kernel<<<1, 32, 0, s>>> (bord, bounds6);
  return check_launch ("bounds_finish");
}

extern "C" int drb_morton_codes (const float *aabbs6, int n, const float *bounds6,
                                 unsigned *codes, void *stream)
{
  if (n < 0 || (n > 0 && (!aabbs6 || !bounds6 || !codes)))
  {
    set_last_error ("morton: bad arguments");
    return DRB_ERR_INVALID_ARG;
  }
  if (n == 0) return DRB_OK;
  morton_kernel<<<div_up (n, 256), 256, 0, (cudaStream_t)stream>>> (aabbs6, n, bounds6, codes);
  return check_launch ("morton_kernel");
}

extern "C" int drb_lbvh_build (const drb_mesh *mesh, drb_bvh *bvh, unsigned *sorted_codes,
                               void *stream)
{
  int st = validate_mesh (mesh, 3);
  if (st) return st;
  if (!bvh || !bvh->inner_nodes || !bvh->leaf_nodes || !bvh->aabb_ids || !bvh->ref_boxes)
  {
    set_last_error ("lbvh_build: bvh arrays must be allocated (see drb_bvh_sizes)");
    return DRB_ERR_INVALID_ARG;
  }
  int n_inner, n_leaf;
  st = drb_bvh_sizes (mesh->dim, mesh->n_elem, &n_inner, &n_leaf);
  if (st) return st;
  if (bvh->n_leaf != n_leaf || bvh->n_inner != n_inner)
  {
    set_last_error ("lbvh_build: bvh sizes do not match drb_bvh_sizes");
    return DRB_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;

  if (mesh->n_elem == 0)
  {
    // Zero-primitive special case (linear_bvh_builder.cpp:411-433): two
    // point boxes at the origin, both leaves refer to primitive 0, and the
    // bounds stay empty because the reduction is skipped.
    float node[16] = { 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0 };
    const int kids[2] = { -1, -2 };
    std::memcpy (node + 12, kids, sizeof (kids));
    const int leaf[2] = { 0, 0 };
    const int ids[2] = { 0, 1 };
    const float ref3[12] = { 0, 0, 0, 1, 1, 1, 0, 0, 0, 1, 1, 1 };
    // ref_universe<Simplex>: axis vertices, then the origin
    const float tet_ref[24] = { 1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0 };
    const float tri_ref[12] = { 1, 0, 0, 1, 0, 0, 1, 0, 0, 1, 0, 0 };
    const bool simplex = mesh->shape == DRB_SHAPE_SIMPLEX;
    cudaMemcpyAsync (bvh->inner_nodes, node, sizeof (node), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync (bvh->leaf_nodes, leaf, sizeof (leaf), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync (bvh->aabb_ids, ids, sizeof (ids), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync (bvh->ref_boxes, simplex ? (mesh->dim == 3 ? tet_ref : tri_ref) : ref3,
                     sizeof (float) * (simplex ? 4 * mesh->dim * (mesh->dim + 1) / 2 : 4 * mesh->dim),
                     cudaMemcpyHostToDevice, s);
    if (sorted_codes) cudaMemsetAsync (sorted_codes, 0, sizeof (unsigned) * 2, s);
    const float empty[6] = { INFINITY, -INFINITY, INFINITY, -INFINITY, INFINITY, -INFINITY };
    for (int q = 0; q < 6; ++q) bvh->bounds[q] = empty[q];
    cudaError_t e = cudaStreamSynchronize (s);
    return status_from (e);
  }

  Scratch scr (s);
  const int n = n_leaf;
  float *aabbs = scr.alloc<float> ((size_t)6 * n);
  unsigned *codes = scr.alloc<unsigned> (n);
  unsigned *codes_sorted = sorted_codes ? sorted_codes : scr.alloc<unsigned> (n);
  float *inner_box = scr.alloc<float> ((size_t)8 * n_inner);
  int *met = scr.alloc<int> (n_inner);
  unsigned *bord = scr.alloc<unsigned> (8);
  float *bounds6 = scr.alloc<float> (8);
  if (scr.err != cudaSuccess) return status_from (scr.err);

  bounds_init_kernel<<<1, 32, 0, s>>> (bord);
  if ((st = check_launch ("bounds_init_kernel"))) return st;
  st = dispatch_subbox (mesh, aabbs, nullptr, bvh->ref_boxes, bord, s);
  if (st) return st;
  bounds_finish_kernel<<<1, 32, 0, s>>> (bord, bounds6);
  if ((st = check_launch ("bounds_finish_kernel"))) return st;
  morton_kernel<<<div_up (n, 256), 256, 0, s>>> (aabbs, n, bounds6, codes);
  if ((st = check_launch ("morton_kernel"))) return st;
  st = radix_sort_pairs (codes, nullptr, codes_sorted, bvh->aabb_ids, n, 30, s);
  if (st) return st;
  cudaMemsetAsync (met, 0xff, sizeof (int) * (size_t)n_inner, s);
  tree_kernel<<<div_up (n, kTreeBlock), kTreeBlock, 0, s>>> (codes_sorted, bvh->aabb_ids, aabbs, n,
                                                             n / mesh->n_elem, bvh->leaf_nodes, inner_box,
                                                             met, (float4 *)bvh->inner_nodes);
  if ((st = check_launch ("tree_kernel"))) return st;
  float hb[8];
  cudaError_t e = cudaMemcpyAsync (hb, bounds6, sizeof (float) * 6, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize (s);
  if (e != cudaSuccess) { set_last_error (cudaGetErrorString (e)); return status_from (e); }
  for (int q = 0; q < 6; ++q) bvh->bounds[q] = hb[q];
  return DRB_OK;
}
