// SPDX-License-Identifier: Apache-2.0
// On-device BVH construction, replacing the driver's BLAS/TLAS builds. Two
// builders: a SAH builder of many BVHs at once (all of a scene's BLASes in
// three launches, and the TLAS), and, for larger meshes, a linear BVH
// (Karras, "Maximizing Parallelism in the Construction of BVHs, Octrees, and
// k-d Trees", HPG 2012) over 63-bit Morton codes of the primitives'
// centroids, sorted by CUB's radix sort, with bounds fitted bottom-up. The
// reference's builds are (backend/vulkan/gpu_scene.cpp:1899-1950, 2240-2322
// in hydra-lotus).
#include "bvh_build.cuh"

#include <algorithm>

#include <cub/device/device_radix_sort.cuh>

namespace lotus {

namespace {

constexpr int kBuildBlock = 256;

__device__ __forceinline__ uint32_t ordered(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float unordered(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Folds a warp's primitive centroids into the centroid bounds with one
// atomic per bound (lanes without a primitive add the identities); every
// lane of the warp takes part.
__device__ __forceinline__ void warp_centroid_bounds(uint32_t* bounds, bool valid, const float* l,
    const float* h) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const uint32_t o = ordered(0.5f * (l[a] + h[a]));
    const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, valid ? o : 0xFFFFFFFFu);
    const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, valid ? o : 0u);
    if ((threadIdx.x & 31u) == 0) {
      atomicMin(&bounds[a], lo);
      atomicMax(&bounds[3 + a], hi);
    }
  }
}

// Triangle boxes in object space from the geometry's positions.
__global__ void k_triangle_boxes(const float* __restrict__ positions,
    const uint32_t* __restrict__ triangles, uint32_t n, float4* __restrict__ lo,
    float4* __restrict__ hi, uint32_t* __restrict__ centroid_bounds) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < n;
  float l[3] = {kFloatMax, kFloatMax, kFloatMax}, h[3] = {-kFloatMax, -kFloatMax, -kFloatMax};
  if (valid) {
    for (int k = 0; k < 3; ++k) {
      const uint32_t v = triangles[3 * i + k];
      for (int a = 0; a < 3; ++a) {
        const float p = positions[3 * (size_t)v + a];
        l[a] = fminf(l[a], p);
        h[a] = fmaxf(h[a], p);
      }
    }
    lo[i] = make_float4(l[0], l[1], l[2], 0.0f);
    hi[i] = make_float4(h[0], h[1], h[2], 0.0f);
  }
  warp_centroid_bounds(centroid_bounds, valid, l, h);
}

// Instance world boxes: the BLAS root box's corners through
// world_from_object, widened by a relative margin. The linear BVH's build
// also takes the centroids' bounds (`centroid_bounds`), the SAH builder the
// instances' indices (`idx`); the other is null.
__global__ void k_instance_boxes(const InstanceShading* __restrict__ shade,
    const InstanceTraversal* __restrict__ trav, const BvhNode* __restrict__ blas, uint32_t n,
    float4* __restrict__ lo, float4* __restrict__ hi, uint32_t* __restrict__ centroid_bounds,
    uint32_t* __restrict__ idx) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (idx != nullptr) idx[i] = i;
  float l[3] = {kFloatMax, kFloatMax, kFloatMax}, h[3] = {-kFloatMax, -kFloatMax, -kFloatMax};
  const uint32_t root = trav[i].blas_root;
  if (root != (uint32_t)kEmptyChild) {
    const BvhNode nd = blas[root];
    float bl[3] = {nd.x.x, nd.y.x, nd.z.x}, bh[3] = {nd.x.y, nd.y.y, nd.z.y};
    if (nd.c.y != kEmptyChild) {
      bl[0] = fminf(bl[0], nd.x.z); bl[1] = fminf(bl[1], nd.y.z); bl[2] = fminf(bl[2], nd.z.z);
      bh[0] = fmaxf(bh[0], nd.x.w); bh[1] = fmaxf(bh[1], nd.y.w); bh[2] = fmaxf(bh[2], nd.z.w);
    }
    const InstanceShading s = shade[i];
    for (int corner = 0; corner < 8; ++corner) {
      const F3 c = V((corner & 1) ? bh[0] : bl[0], (corner & 2) ? bh[1] : bl[1],
          (corner & 4) ? bh[2] : bl[2]);
      const F3 w = row_point(s.m, c);
      l[0] = fminf(l[0], w.x); l[1] = fminf(l[1], w.y); l[2] = fminf(l[2], w.z);
      h[0] = fmaxf(h[0], w.x); h[1] = fmaxf(h[1], w.y); h[2] = fmaxf(h[2], w.z);
    }
    for (int a = 0; a < 3; ++a) {
      const float pad = 1e-6f * fmaxf(fabsf(l[a]), fabsf(h[a])) + 1e-7f;
      l[a] -= pad;
      h[a] += pad;
    }
  } else {
    // An empty instance: a point box that no ray enters deeply.
    for (int a = 0; a < 3; ++a) l[a] = h[a] = 0.0f;
  }
  lo[i] = make_float4(l[0], l[1], l[2], 0.0f);
  hi[i] = make_float4(h[0], h[1], h[2], 0.0f);
  if (centroid_bounds == nullptr) return;
  for (int a = 0; a < 3; ++a) {
    const float c = 0.5f * (l[a] + h[a]);
    atomicMin(&centroid_bounds[a], ordered(c));
    atomicMax(&centroid_bounds[3 + a], ordered(c));
  }
}

__device__ __forceinline__ uint64_t spread21(uint64_t x) {
  x &= 0x1FFFFFull;
  x = (x | (x << 32)) & 0x1F00000000FFFFull;
  x = (x | (x << 16)) & 0x1F0000FF0000FFull;
  x = (x | (x << 8)) & 0x100F00F00F00F00Full;
  x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

__global__ void k_morton(const float4* __restrict__ lo, const float4* __restrict__ hi, uint32_t n,
    const uint32_t* __restrict__ cb, uint64_t* __restrict__ keys, uint32_t* __restrict__ values) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float l[3] = {lo[i].x, lo[i].y, lo[i].z}, h[3] = {hi[i].x, hi[i].y, hi[i].z};
  uint64_t q[3];
  for (int a = 0; a < 3; ++a) {
    const float cmin = unordered(cb[a]), cmax = unordered(cb[3 + a]);
    const float c = 0.5f * (l[a] + h[a]);
    const float extent = cmax - cmin;
    float t = extent > 0.0f ? (c - cmin) / extent : 0.5f;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    q[a] = (uint64_t)fminf(t * 2097152.0f, 2097151.0f);
  }
  keys[i] = spread21(q[0]) | (spread21(q[1]) << 1) | (spread21(q[2]) << 2);
  values[i] = i;
}

__device__ __forceinline__ int delta(const uint64_t* __restrict__ keys, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const uint64_t a = keys[i], b = keys[j];
  if (a == b) return 64 + __clz((uint32_t)i ^ (uint32_t)j);
  return __clzll(a ^ b);
}

// Karras's hierarchy: internal node i's children. Leaves are encoded as
// (leaf | kLeafBit).
constexpr uint32_t kLeafBit = 0x80000000u;

__global__ void k_karras(const uint64_t* __restrict__ keys, int n, uint32_t* __restrict__ left,
    uint32_t* __restrict__ right, uint32_t* __restrict__ parent_internal,
    uint32_t* __restrict__ parent_leaf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  const int dmin = delta(keys, n, i, i - d);
  int lmax = 2;
  while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int dnode = delta(keys, n, i, j);
  int s = 0;
  int t = l;
  do {
    t = (t + 1) >> 1;
    if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  const int gamma = i + s * d + min(d, 0);
  const uint32_t lc = (min(i, j) == gamma) ? ((uint32_t)gamma | kLeafBit) : (uint32_t)gamma;
  const uint32_t rc = (max(i, j) == gamma + 1) ? ((uint32_t)(gamma + 1) | kLeafBit) : (uint32_t)(gamma + 1);
  left[i] = lc;
  right[i] = rc;
  if (lc & kLeafBit) parent_leaf[lc & ~kLeafBit] = (uint32_t)i; else parent_internal[lc] = (uint32_t)i;
  if (rc & kLeafBit) parent_leaf[rc & ~kLeafBit] = (uint32_t)i; else parent_internal[rc] = (uint32_t)i;
}

// Bottom-up bounds: the second child to arrive at a node fits it and
// carries on to its parent.
__global__ void k_fit(const uint32_t* __restrict__ values, const float4* __restrict__ plo,
    const float4* __restrict__ phi, int n, const uint32_t* __restrict__ left,
    const uint32_t* __restrict__ right, const uint32_t* __restrict__ parent_internal,
    const uint32_t* __restrict__ parent_leaf, float4* nlo, float4* nhi, uint32_t* flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t node = parent_leaf[i];
  // A tree over n < 2^31 primitives with 63-bit keys and index tie-breaks
  // is at most 96 levels deep; the bound only guards against corrupt input.
  for (int level = 0; level < 256; ++level) {
    __threadfence();
    if (atomicAdd(&flags[node], 1u) == 0) return;
    __threadfence();
    float4 l[2], h[2];
    const uint32_t ch[2] = {left[node], right[node]};
    for (int k = 0; k < 2; ++k) {
      if (ch[k] & kLeafBit) {
        const uint32_t p = values[ch[k] & ~kLeafBit];
        l[k] = plo[p];
        h[k] = phi[p];
      } else {
        l[k] = __ldcg(&nlo[ch[k]]);
        h[k] = __ldcg(&nhi[ch[k]]);
      }
    }
    nlo[node] = make_float4(fminf(l[0].x, l[1].x), fminf(l[0].y, l[1].y), fminf(l[0].z, l[1].z), 0.0f);
    nhi[node] = make_float4(fmaxf(h[0].x, h[1].x), fmaxf(h[0].y, h[1].y), fmaxf(h[0].z, h[1].z), 0.0f);
    if (node == 0) return;
    node = parent_internal[node];
  }
}

// The 64-byte nodes. Child leaves point into the primitive pool at
// `leaf_base` + sorted position (BLAS), or at the sorted value itself (TLAS).
__global__ void k_write_nodes(const uint32_t* __restrict__ values, const float4* __restrict__ plo,
    const float4* __restrict__ phi, int n, const uint32_t* __restrict__ left,
    const uint32_t* __restrict__ right, const float4* __restrict__ nlo,
    const float4* __restrict__ nhi, BvhNode* __restrict__ out, uint32_t node_base,
    uint32_t leaf_base, int leaves_are_values) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const uint32_t ch[2] = {left[i], right[i]};
  float4 l[2], h[2];
  int32_t c[2];
  for (int k = 0; k < 2; ++k) {
    if (ch[k] & kLeafBit) {
      const uint32_t pos = ch[k] & ~kLeafBit;
      const uint32_t p = values[pos];
      l[k] = plo[p];
      h[k] = phi[p];
      c[k] = ~(int32_t)(leaves_are_values ? p : leaf_base + pos);
    } else {
      l[k] = nlo[ch[k]];
      h[k] = nhi[ch[k]];
      c[k] = (int32_t)(node_base + ch[k]);
    }
  }
  BvhNode nd;
  nd.x = make_float4(l[0].x, h[0].x, l[1].x, h[1].x);
  nd.y = make_float4(l[0].y, h[0].y, l[1].y, h[1].y);
  nd.z = make_float4(l[0].z, h[0].z, l[1].z, h[1].z);
  nd.c = make_int4(c[0], c[1], 1, 1);
  out[node_base + i] = nd;
}

// A one-primitive BVH: a root with one leaf child and an empty one.
__global__ void k_single_root(const float4* __restrict__ plo, const float4* __restrict__ phi,
    BvhNode* __restrict__ out, uint32_t node_base, uint32_t leaf_base, int leaves_are_values) {
  BvhNode nd;
  const float4 l = plo[0], h = phi[0];
  nd.x = make_float4(l.x, h.x, 0.0f, 0.0f);
  nd.y = make_float4(l.y, h.y, 0.0f, 0.0f);
  nd.z = make_float4(l.z, h.z, 0.0f, 0.0f);
  nd.c = make_int4(~(int32_t)(leaves_are_values ? 0u : leaf_base), kEmptyChild, 1, 0);
  out[node_base] = nd;
}

// The leaf-ordered triangle pool: three object-space corners, the original
// primitive index in the first corner's w.
__global__ void k_write_triangles(const uint32_t* __restrict__ values,
    const float* __restrict__ positions, const uint32_t* __restrict__ triangles, uint32_t n,
    float4* __restrict__ pool, uint32_t base) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t p = values[i];
  float4* out = pool + kTriStride * (size_t)(base + i);
  for (int k = 0; k < 3; ++k) {
    const uint32_t v = triangles[3 * (size_t)p + k];
    out[k] = make_float4(positions[3 * (size_t)v], positions[3 * (size_t)v + 1],
        positions[3 * (size_t)v + 2], k == 0 ? __uint_as_float(p) : 0.0f);
  }
  out[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}


// ---------------------------------------------------------------------------
// SAH builder of a batch of BVHs (a scene's BLASes, or its TLAS), top-down
// (Wald, "On fast Construction of SAH-based Bounding Volume Hierarchies",
// 2007), each node built by as many threads as its primitives can use:
//   - k_sah_large, one CTA per BVH: nodes of more than kSahMedium primitives;
//   - k_sah_medium, one warp per subtree handed on by it: nodes of more than
//     a warp's primitives. Both bin centroids into 16 bins per axis;
//   - k_sah_small, one warp per subtree of at most 32 primitives: one
//     primitive a lane and all of a level's nodes at once, with every split
//     of the sorted centroids tried instead of bins.
// The subtrees of all BVHs lie in one list per kernel, so that the GPU is
// filled whatever the meshes' sizes. One CTA a BVH for all of its nodes (some
// ten barriers each, five of six nodes over fewer than ten primitives) took
// 45 ms for the sphere field's 320 meshes (1.07M triangles) and its 4,161
// instances; the three take 0.32, 0.43 and 0.34 ms.
//
// A subtree over n primitives takes the n - 1 node slots from its own on:
// its root, then the left child's, then the right child's, so that no
// counter is needed and a subtree is contiguous.

constexpr int kSahBlock = 512;
constexpr int kSahBins = 16;
constexpr int kSahStack = 128;
constexpr uint32_t kSahMedium = 512;
constexpr uint32_t kSahSmall = 32;
constexpr unsigned kAllLanes = 0xFFFFFFFFu;

// A node to build: its primitives [begin, end) of the job's and its slot.
struct SahNode {
  uint32_t job, begin, end, slot;
};

// The lists between the kernels and their counters: nodes appended, nodes
// taken, and errors.
struct SahLists {
  SahNode* medium;
  SahNode* small;
  uint32_t* counters;
};
constexpr int kMediumCount = 0, kMediumTaken = 1, kSmallCount = 2, kSmallTaken = 3, kSahErrors = 4, kSahCounters = 5;

// The threads that build one node together: a block or a warp.
template <int kThreads>
struct SahGroup {
  static constexpr bool kWarp = kThreads == 32;
  static __device__ __forceinline__ uint32_t rank() { return kWarp ? threadIdx.x & 31u : threadIdx.x; }
  static __device__ __forceinline__ void sync() {
    if (kWarp) __syncwarp();
    else __syncthreads();
  }
};

template <int kThreads>
struct SahShared {
  uint32_t count[3][kSahBins];
  uint32_t lo[3][3][kSahBins];  // [binned axis][component][bin], ordered floats
  uint32_t hi[3][3][kSahBins];
  uint32_t bounds[12];          // centroid bounds; the halves' where no axis separates them
  float best_cost[3];
  int split_at[3];
  uint32_t left_count[3];
  float box[3][12];             // the children's boxes of each axis's best split
  uint32_t warp_left[kThreads / 32];
  uint32_t begin, end, slot;
};

__device__ __forceinline__ float sah_half_area(const float* lo, const float* hi) {
  const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
  return dx * dy + dy * dz + dz * dx;
}

// The reference of a child over [begin, end): a leaf, or the node at `slot`.
__device__ __forceinline__ int32_t sah_child(const SahJob& job, const uint32_t* index, uint32_t begin, uint32_t end,
    uint32_t slot, int32_t& count) {
  count = end - begin <= job.leaf_size ? (int32_t)(end - begin) : 0;
  if (count == 0) return (int32_t)(job.node_base + slot);
  return job.leaves_are_values ? ~(int32_t)index[begin] : ~(int32_t)(job.leaf_base + begin);
}

__device__ __forceinline__ void sah_write_node(BvhNode* nodes, const SahJob& job, const uint32_t* index,
    uint32_t begin, uint32_t mid, uint32_t end, uint32_t slot, const float* box) {
  int32_t n0, n1;
  const int32_t c0 = sah_child(job, index, begin, mid, slot + 1, n0);
  const int32_t c1 = sah_child(job, index, mid, end, slot + (mid - begin), n1);
  BvhNode nd;
  nd.x = make_float4(box[0], box[3], box[6], box[9]);
  nd.y = make_float4(box[1], box[4], box[7], box[10]);
  nd.z = make_float4(box[2], box[5], box[8], box[11]);
  nd.c = make_int4(c0, c1, n0, n1);
  nodes[job.node_base + slot] = nd;
}

// The best split of one axis's bins, by the 16 lanes of a half warp (every
// lane of the warp takes part): prefix and suffix boxes by scans. Lane 0 of
// the half writes it down.
template <int kThreads>
__device__ __forceinline__ void sah_sweep(SahShared<kThreads>& sh, int axis, bool separates) {
  const unsigned bin = threadIdx.x & 15u;
  float l[3], h[3], rl[3], rh[3];
  uint32_t left = sh.count[axis][bin], right = left;
  for (int c = 0; c < 3; ++c) {
    l[c] = rl[c] = left ? unordered(sh.lo[axis][c][bin]) : INFINITY;
    h[c] = rh[c] = left ? unordered(sh.hi[axis][c][bin]) : -INFINITY;
  }
#pragma unroll
  for (unsigned off = 1; off < 16; off <<= 1) {
    const uint32_t ln = __shfl_up_sync(kAllLanes, left, off, 16), rn = __shfl_down_sync(kAllLanes, right, off, 16);
    const bool up = bin >= off, down = bin + off < 16;
    left += up ? ln : 0u;
    right += down ? rn : 0u;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float a = __shfl_up_sync(kAllLanes, l[c], off, 16), b = __shfl_up_sync(kAllLanes, h[c], off, 16);
      const float d = __shfl_down_sync(kAllLanes, rl[c], off, 16), e = __shfl_down_sync(kAllLanes, rh[c], off, 16);
      if (up) { l[c] = fminf(l[c], a); h[c] = fmaxf(h[c], b); }
      if (down) { rl[c] = fminf(rl[c], d); rh[c] = fmaxf(rh[c], e); }
    }
  }
  // The right side of a split after this bin begins at the next one.
  right = __shfl_down_sync(kAllLanes, right, 1, 16);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    rl[c] = __shfl_down_sync(kAllLanes, rl[c], 1, 16);
    rh[c] = __shfl_down_sync(kAllLanes, rh[c], 1, 16);
  }
  float cost = INFINITY;
  if (separates && bin < 15 && left != 0 && right != 0)
    cost = sah_half_area(l, h) * (float)left + sah_half_area(rl, rh) * (float)right;
  float best = cost;
  unsigned at = bin;
#pragma unroll
  for (unsigned off = 8; off >= 1; off >>= 1) {
    const float other = __shfl_xor_sync(kAllLanes, best, off, 16);
    const unsigned other_at = __shfl_xor_sync(kAllLanes, at, off, 16);
    if (other < best || (other == best && other_at < at)) { best = other; at = other_at; }
  }
  if (bin == at) {
    sh.best_cost[axis] = best;
    sh.split_at[axis] = best < INFINITY ? (int)bin : -1;
    sh.left_count[axis] = left;
    for (int c = 0; c < 3; ++c) {
      sh.box[axis][c] = l[c];
      sh.box[axis][3 + c] = h[c];
      sh.box[axis][6 + c] = rl[c];
      sh.box[axis][9 + c] = rh[c];
    }
  }
}

// Builds one node: splits [begin, end) of the job's primitives (index, with
// tmp as scratch) at the cheapest plane between bins, the order within each
// side kept, and writes the node. Returns the first primitive of the right
// side. Group-uniform; ends with the group in step.
template <int kThreads>
__device__ __forceinline__ uint32_t sah_split(const SahJob& job, uint32_t begin, uint32_t end, uint32_t slot,
    const float4* __restrict__ plo, const float4* __restrict__ phi, uint32_t* index, uint32_t* tmp, BvhNode* nodes,
    SahShared<kThreads>& sh) {
  using G = SahGroup<kThreads>;
  const uint32_t rank = G::rank();
  const unsigned lane = threadIdx.x & 31u;
  if (rank < 12) sh.bounds[rank] = rank % 6 < 3 ? 0xFFFFFFFFu : 0u;
  for (uint32_t k = rank; k < 3 * kSahBins; k += kThreads) {
    const uint32_t a = k / kSahBins, b = k % kSahBins;
    sh.count[a][b] = 0;
    for (int c = 0; c < 3; ++c) {
      sh.lo[a][c][b] = 0xFFFFFFFFu;
      sh.hi[a][c][b] = 0u;
    }
  }
  G::sync();
  // Centroid bounds: per thread, per warp, then one atomic a warp and bound.
  uint32_t cl[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, ch[3] = {0u, 0u, 0u};
  for (uint32_t i = begin + rank; i < end; i += kThreads) {
    const uint32_t p = job.prim_offset + index[i];
    const float4 l = plo[p], h = phi[p];
    const uint32_t c[3] = {ordered(0.5f * (l.x + h.x)), ordered(0.5f * (l.y + h.y)), ordered(0.5f * (l.z + h.z))};
    for (int a = 0; a < 3; ++a) {
      cl[a] = min(cl[a], c[a]);
      ch[a] = max(ch[a], c[a]);
    }
  }
  for (int a = 0; a < 3; ++a) {
    const uint32_t l = __reduce_min_sync(kAllLanes, cl[a]), h = __reduce_max_sync(kAllLanes, ch[a]);
    if (lane == 0) {
      atomicMin(&sh.bounds[a], l);
      atomicMax(&sh.bounds[3 + a], h);
    }
  }
  G::sync();
  float cmin[3], scale[3];
  for (int a = 0; a < 3; ++a) {
    cmin[a] = unordered(sh.bounds[a]);
    const float extent = unordered(sh.bounds[3 + a]) - cmin[a];
    scale[a] = extent > 0.0f ? float(kSahBins) / extent : 0.0f;
  }
  auto bin_of = [&](float lo, float hi, int a) {
    // Each operation rounded by itself: the partition has to find the very
    // bins that were counted.
    const float c = __fmul_rn(0.5f, __fadd_rn(lo, hi));
    return min(kSahBins - 1, max(0, (int)__fmul_rn(__fsub_rn(c, cmin[a]), scale[a])));
  };
  for (uint32_t i = begin + rank; i < end; i += kThreads) {
    const uint32_t p = job.prim_offset + index[i];
    const float4 l = plo[p], h = phi[p];
    const uint32_t ol[3] = {ordered(l.x), ordered(l.y), ordered(l.z)}, oh[3] = {ordered(h.x), ordered(h.y), ordered(h.z)};
    const int b[3] = {bin_of(l.x, h.x, 0), bin_of(l.y, h.y, 1), bin_of(l.z, h.z, 2)};
    for (int a = 0; a < 3; ++a) {
      atomicAdd(&sh.count[a][b[a]], 1u);
      for (int c = 0; c < 3; ++c) {
        atomicMin(&sh.lo[a][c][b[a]], ol[c]);
        atomicMax(&sh.hi[a][c][b[a]], oh[c]);
      }
    }
  }
  G::sync();
  // Half warps sweep an axis each: a block's first two warps, or a warp twice.
  if (G::kWarp) {
    const int a = (int)(lane >> 4);
    sah_sweep(sh, a, (a ? scale[1] : scale[0]) > 0.0f);
    sah_sweep(sh, 2, scale[2] > 0.0f);
  } else if (threadIdx.x < 64) {
    const int a = min((int)(threadIdx.x >> 4), 2);
    sah_sweep(sh, a, (a == 0 ? scale[0] : a == 1 ? scale[1] : scale[2]) > 0.0f);
  }
  G::sync();
  int axis = -1;
  float best = INFINITY;
  for (int a = 0; a < 3; ++a)
    if (sh.split_at[a] >= 0 && sh.best_cost[a] < best) {
      best = sh.best_cost[a];
      axis = a;
    }
  uint32_t mid;
  if (axis < 0) {
    // Coincident centroids: the list's halves, whose boxes no bins hold.
    mid = begin + (end - begin) / 2;
    for (int side = 0; side < 2; ++side) {
      G::sync();
      if (rank < 6) sh.bounds[rank] = rank < 3 ? 0xFFFFFFFFu : 0u;
      G::sync();
      for (uint32_t i = (side ? mid : begin) + rank; i < (side ? end : mid); i += kThreads) {
        const float4 l = plo[job.prim_offset + index[i]], h = phi[job.prim_offset + index[i]];
        atomicMin(&sh.bounds[0], ordered(l.x)); atomicMin(&sh.bounds[1], ordered(l.y)); atomicMin(&sh.bounds[2], ordered(l.z));
        atomicMax(&sh.bounds[3], ordered(h.x)); atomicMax(&sh.bounds[4], ordered(h.y)); atomicMax(&sh.bounds[5], ordered(h.z));
      }
      G::sync();
      if (rank < 6) sh.box[0][6 * side + rank] = unordered(sh.bounds[rank]);
    }
    axis = 0;
  } else {
    const int split = sh.split_at[axis];
    const uint32_t left_total = sh.left_count[axis];
    mid = begin + left_total;
    uint32_t left_before = 0;  // lefts of the tiles done
    for (uint32_t t0 = begin; t0 < end; t0 += kThreads) {
      const uint32_t i = t0 + rank;
      bool left = false;
      uint32_t v = 0;
      if (i < end) {
        v = index[i];
        const float4 l = plo[job.prim_offset + v], h = phi[job.prim_offset + v];
        left = (axis == 0 ? bin_of(l.x, h.x, 0) : axis == 1 ? bin_of(l.y, h.y, 1) : bin_of(l.z, h.z, 2)) <= split;
      }
      const unsigned mask = __ballot_sync(kAllLanes, left);
      uint32_t before = left_before + (uint32_t)__popc(mask & ((1u << lane) - 1u));
      if (G::kWarp) {
        left_before += (uint32_t)__popc(mask);
      } else {
        G::sync();
        if (lane == 0) sh.warp_left[threadIdx.x >> 5] = (uint32_t)__popc(mask);
        G::sync();
        for (uint32_t w = 0; w < kThreads / 32; ++w) {
          const uint32_t n = sh.warp_left[w];
          if (w < threadIdx.x >> 5) before += n;
          left_before += n;
        }
      }
      if (i < end) tmp[left ? begin + before : mid + (i - begin - before)] = v;
    }
    G::sync();
    for (uint32_t i = begin + rank; i < end; i += kThreads) index[i] = tmp[i];
  }
  G::sync();
  if (rank == 0) sah_write_node(nodes, job, index, begin, mid, end, slot, sh.box[axis]);
  G::sync();
  return mid;
}

// Where a child that is no leaf is built: true when the caller builds it.
__device__ __forceinline__ bool sah_keep(const SahJob& job, uint32_t job_index, uint32_t begin, uint32_t end,
    uint32_t slot, uint32_t above, const SahLists& lists, bool write) {
  const uint32_t n = end - begin;
  if (n <= job.leaf_size) return false;
  if (n > above) return true;
  if (write) {
    const bool small = n <= kSahSmall;
    (small ? lists.small : lists.medium)[atomicAdd(&lists.counters[small ? kSmallCount : kMediumCount], 1u)] =
        SahNode{job_index, begin, end, slot};
  }
  return false;
}

__global__ void __launch_bounds__(kSahBlock) k_sah_large(const SahJob* __restrict__ jobs,
    const float4* __restrict__ plo, const float4* __restrict__ phi, uint32_t* __restrict__ idx,
    uint32_t* __restrict__ scratch, BvhNode* __restrict__ nodes, SahLists lists) {
  __shared__ SahShared<kSahBlock> sh;
  __shared__ uint32_t stack[kSahStack][3];
  const SahJob job = jobs[blockIdx.x];
  uint32_t* index = idx + job.prim_offset;
  if (job.count == 0) return;
  // Small sets: one leaf under the root, its second child empty.
  if (job.count <= job.leaf_size) {
    if (threadIdx.x != 0) return;
    float l[3] = {kFloatMax, kFloatMax, kFloatMax}, h[3] = {-kFloatMax, -kFloatMax, -kFloatMax};
    for (uint32_t i = 0; i < job.count; ++i) {
      const float4 a = plo[job.prim_offset + index[i]], b = phi[job.prim_offset + index[i]];
      l[0] = fminf(l[0], a.x); l[1] = fminf(l[1], a.y); l[2] = fminf(l[2], a.z);
      h[0] = fmaxf(h[0], b.x); h[1] = fmaxf(h[1], b.y); h[2] = fmaxf(h[2], b.z);
    }
    BvhNode nd;
    nd.x = make_float4(l[0], h[0], 0.0f, 0.0f);
    nd.y = make_float4(l[1], h[1], 0.0f, 0.0f);
    nd.z = make_float4(l[2], h[2], 0.0f, 0.0f);
    const int32_t leaf = job.leaves_are_values ? ~(int32_t)index[0] : ~(int32_t)job.leaf_base;
    nd.c = make_int4(leaf, kEmptyChild, (int32_t)job.count, 0);
    nodes[job.node_base] = nd;
    return;
  }
  uint32_t begin = 0, end = job.count, slot = 0;
  if (!sah_keep(job, blockIdx.x, begin, end, slot, kSahMedium, lists, threadIdx.x == 0)) return;
  int sp = 0;
  // Every step splits one node, of at most count - 1. The smaller side is
  // built first, so that the stack holds at most one range per halving.
  for (uint32_t step = 0; step < job.count; ++step) {
    const uint32_t mid = sah_split<kSahBlock>(job, begin, end, slot, plo, phi, index, scratch + job.prim_offset, nodes, sh);
    uint32_t r[2][3] = {{begin, mid, slot + 1}, {mid, end, slot + (mid - begin)}};
    const bool keep[2] = {sah_keep(job, blockIdx.x, r[0][0], r[0][1], r[0][2], kSahMedium, lists, threadIdx.x == 0),
        sah_keep(job, blockIdx.x, r[1][0], r[1][1], r[1][2], kSahMedium, lists, threadIdx.x == 0)};
    int next = keep[0] ? 0 : keep[1] ? 1 : -1;
    if (keep[0] && keep[1]) {
      next = mid - begin <= end - mid ? 0 : 1;
      if (sp >= kSahStack) {
        if (threadIdx.x == 0) atomicAdd(&lists.counters[kSahErrors], 1u);
        return;
      }
      if (threadIdx.x < 3) stack[sp][threadIdx.x] = r[1 - next][threadIdx.x];
      ++sp;
    }
    __syncthreads();
    if (next >= 0) {
      begin = r[next][0];
      end = r[next][1];
      slot = r[next][2];
    } else {
      if (sp == 0) return;
      --sp;
      begin = stack[sp][0];
      end = stack[sp][1];
      slot = stack[sp][2];
    }
    __syncthreads();
  }
}

constexpr int kMediumWarps = 4;
__global__ void __launch_bounds__(32 * kMediumWarps) k_sah_medium(const SahJob* __restrict__ jobs,
    const float4* __restrict__ plo, const float4* __restrict__ phi, uint32_t* __restrict__ idx,
    uint32_t* __restrict__ scratch, BvhNode* __restrict__ nodes, SahLists lists) {
  __shared__ SahShared<32> shared[kMediumWarps];
  __shared__ uint32_t stacks[kMediumWarps][16][3];
  SahShared<32>& sh = shared[threadIdx.x >> 5];
  uint32_t(*stack)[3] = stacks[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t total = lists.counters[kMediumCount];
  for (;;) {
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&lists.counters[kMediumTaken], 1u);
    at = __shfl_sync(kAllLanes, at, 0);
    if (at >= total) return;
    const SahNode root = lists.medium[at];
    const SahJob job = jobs[root.job];
    uint32_t begin = root.begin, end = root.end, slot = root.slot;
    int sp = 0;
    for (uint32_t step = 0; step < kSahMedium; ++step) {
      const uint32_t mid = sah_split<32>(job, begin, end, slot, plo, phi, idx + job.prim_offset,
          scratch + job.prim_offset, nodes, sh);
      uint32_t r[2][3] = {{begin, mid, slot + 1}, {mid, end, slot + (mid - begin)}};
      const bool keep[2] = {sah_keep(job, root.job, r[0][0], r[0][1], r[0][2], kSahSmall, lists, lane == 0),
          sah_keep(job, root.job, r[1][0], r[1][1], r[1][2], kSahSmall, lists, lane == 0)};
      int next = keep[0] ? 0 : keep[1] ? 1 : -1;
      if (keep[0] && keep[1]) {
        // The smaller side first: at most one range per halving of kSahMedium.
        next = mid - begin <= end - mid ? 0 : 1;
        if (lane < 3) stack[sp][lane] = next ? r[0][lane] : r[1][lane];
        ++sp;
      }
      __syncwarp();
      if (next >= 0) {
        begin = next ? r[1][0] : r[0][0];
        end = next ? r[1][1] : r[0][1];
        slot = next ? r[1][2] : r[0][2];
      } else {
        if (sp == 0) break;
        --sp;
        begin = stack[sp][0];
        end = stack[sp][1];
        slot = stack[sp][2];
      }
      __syncwarp();
    }
  }
}

// Subtrees of at most 32 primitives, one primitive a lane, level by level:
// each lane of a node tries the split after its own centroid on each axis
// (ties by lane), the node's cheapest is taken, and the primitives move to
// their side in order. A level takes as many steps as its largest node has
// primitives, whatever the number of nodes.
constexpr int kSmallWarps = 8;
__global__ void __launch_bounds__(32 * kSmallWarps) k_sah_small(const SahJob* __restrict__ jobs,
    const float4* __restrict__ plo, const float4* __restrict__ phi, uint32_t* __restrict__ idx,
    BvhNode* __restrict__ nodes, SahLists lists) {
  __shared__ float4 shared_lo[kSmallWarps][32], shared_hi[kSmallWarps][32];  // w of lo: the primitive
  __shared__ float shared_keys[kSmallWarps][32];
  __shared__ int shared_axes[kSmallWarps][32];
  float4* lo = shared_lo[threadIdx.x >> 5];
  float4* hi = shared_hi[threadIdx.x >> 5];
  float* keys = shared_keys[threadIdx.x >> 5];
  int* axes = shared_axes[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t total = lists.counters[kSmallCount];
  for (;;) {
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&lists.counters[kSmallTaken], 1u);
    at = __shfl_sync(kAllLanes, at, 0);
    if (at >= total) return;
    const SahNode root = lists.small[at];
    const SahJob job = jobs[root.job];
    const uint32_t n = root.end - root.begin;
    uint32_t* index = idx + job.prim_offset + root.begin;
    {
      const uint32_t v = lane < n ? index[lane] : 0u;
      float4 l = lane < n ? plo[job.prim_offset + v] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      l.w = __uint_as_float(v);
      lo[lane] = l;
      hi[lane] = lane < n ? phi[job.prim_offset + v] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncwarp();
    // This lane's node: lanes [begin, end), its slot.
    uint32_t begin = lane < n ? 0u : lane, end = lane < n ? n : lane, slot = root.slot;
    for (int level = 0; level < 32; ++level) {
      const bool inner = end - begin > job.leaf_size;
      if (!__any_sync(kAllLanes, inner)) break;
      float cost = INFINITY, box[12];
      int axis = 0;
      if (inner) {
        const float4 ml = lo[lane], mh = hi[lane];
        const float c[3] = {ml.x + mh.x, ml.y + mh.y, ml.z + mh.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          float b[12];
#pragma unroll
          for (int k = 0; k < 12; ++k) b[k] = (k % 6) < 3 ? INFINITY : -INFINITY;
          uint32_t lefts = 0;
          for (uint32_t j = begin; j < end; ++j) {
            const float4 l = lo[j], h = hi[j];
            const float cj = a == 0 ? l.x + h.x : a == 1 ? l.y + h.y : l.z + h.z;
            if (cj < c[a] || (cj == c[a] && j <= lane)) {
              ++lefts;
              b[0] = fminf(b[0], l.x); b[1] = fminf(b[1], l.y); b[2] = fminf(b[2], l.z);
              b[3] = fmaxf(b[3], h.x); b[4] = fmaxf(b[4], h.y); b[5] = fmaxf(b[5], h.z);
            } else {
              b[6] = fminf(b[6], l.x); b[7] = fminf(b[7], l.y); b[8] = fminf(b[8], l.z);
              b[9] = fmaxf(b[9], h.x); b[10] = fmaxf(b[10], h.y); b[11] = fmaxf(b[11], h.z);
            }
          }
          const uint32_t rights = end - begin - lefts;
          if (rights == 0) continue;
          const float v = sah_half_area(b, b + 3) * (float)lefts + sah_half_area(b + 6, b + 9) * (float)rights;
          if (v < cost) {
            cost = v;
            axis = a;
#pragma unroll
            for (int k = 0; k < 12; ++k) box[k] = b[k];
          }
        }
      }
      keys[lane] = cost;
      axes[lane] = axis;
      __syncwarp();
      // The node's cheapest split (the first of equals); the middle of its
      // lanes where no cost is finite (boxes beyond the floats' range).
      unsigned pivot = lane;
      int by = 3;
      if (inner) {
        float best = INFINITY;
        for (uint32_t j = begin; j < end; ++j)
          if (keys[j] < best) {
            best = keys[j];
            pivot = j;
          }
        if (best < INFINITY) {
          by = axes[pivot];
        } else {
          pivot = begin + (end - begin) / 2 - 1;
          if (lane == pivot) {
#pragma unroll
            for (int k = 0; k < 12; ++k) box[k] = (k % 6) < 3 ? INFINITY : -INFINITY;
            for (uint32_t j = begin; j < end; ++j) {
              const float4 l = lo[j], h = hi[j];
              if (j <= pivot) {
                box[0] = fminf(box[0], l.x); box[1] = fminf(box[1], l.y); box[2] = fminf(box[2], l.z);
                box[3] = fmaxf(box[3], h.x); box[4] = fmaxf(box[4], h.y); box[5] = fmaxf(box[5], h.z);
              } else {
                box[6] = fminf(box[6], l.x); box[7] = fminf(box[7], l.y); box[8] = fminf(box[8], l.z);
                box[9] = fmaxf(box[9], h.x); box[10] = fmaxf(box[10], h.y); box[11] = fmaxf(box[11], h.z);
              }
            }
          }
        }
      }
      const float4 ml = lo[lane], mh = hi[lane], pl = lo[pivot], ph = hi[pivot];
      const float mine = by == 0 ? ml.x + mh.x : by == 1 ? ml.y + mh.y : ml.z + mh.z;
      const float at_pivot = by == 0 ? pl.x + ph.x : by == 1 ? pl.y + ph.y : pl.z + ph.z;
      const bool left = by == 3 ? lane <= pivot : mine < at_pivot || (mine == at_pivot && lane <= pivot);
      const unsigned lefts = __ballot_sync(kAllLanes, left);
      const unsigned in_node = end - begin == 32u ? kAllLanes : ((1u << (end - begin)) - 1u) << (begin & 31u);
      const unsigned below = (1u << lane) - 1u;
      const uint32_t mid = begin + (uint32_t)__popc(lefts & in_node);
      const uint32_t to = !inner ? lane
          : left ? begin + (uint32_t)__popc(lefts & in_node & below) : mid + (uint32_t)__popc(~lefts & in_node & below);
      __syncwarp();
      lo[to] = ml;
      hi[to] = mh;
      __syncwarp();
      if (inner && lane == pivot) {
        auto child = [&](uint32_t first, uint32_t last, uint32_t child_slot, int32_t& count) {
          count = last - first <= job.leaf_size ? (int32_t)(last - first) : 0;
          if (count == 0) return (int32_t)(job.node_base + child_slot);
          return job.leaves_are_values ? ~(int32_t)__float_as_uint(lo[first].w)
                                       : ~(int32_t)(job.leaf_base + root.begin + first);
        };
        int32_t n0, n1;
        const int32_t c0 = child(begin, mid, slot + 1, n0), c1 = child(mid, end, slot + (mid - begin), n1);
        BvhNode nd;
        nd.x = make_float4(box[0], box[3], box[6], box[9]);
        nd.y = make_float4(box[1], box[4], box[7], box[10]);
        nd.z = make_float4(box[2], box[5], box[8], box[11]);
        nd.c = make_int4(c0, c1, n0, n1);
        nodes[job.node_base + slot] = nd;
      }
      // This lane's node from here on is the half it lies in.
      if (inner) {
        if (lane < mid) {
          end = mid;
          slot += 1;
        } else {
          slot += mid - begin;
          begin = mid;
        }
      }
      __syncwarp();
    }
    if (lane < n) index[lane] = __float_as_uint(lo[lane].w);
    __syncwarp();
  }
}

// The job that holds primitive g of the batch (jobs in order of prim_offset).
__device__ __forceinline__ uint32_t sah_job_of(const SahJob* __restrict__ jobs, uint32_t count, uint32_t g) {
  uint32_t lo = 0, hi = count;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].prim_offset <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Triangle boxes of every geometry of a batch: primitive i of job j at
// prim_offset + i, its positions and triangles at the job's offsets.
__global__ void k_batch_triangle_boxes(const float* __restrict__ positions, const uint32_t* __restrict__ triangles,
    const SahJob* __restrict__ jobs, uint32_t job_count, uint32_t total, float4* __restrict__ lo,
    float4* __restrict__ hi, uint32_t* __restrict__ idx) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const SahJob& job = jobs[sah_job_of(jobs, job_count, g)];
  const uint32_t local = g - job.prim_offset;
  const float* P = positions + 3 * job.vertex_offset;
  const uint32_t* T = triangles + 3 * (job.triangle_offset + local);
  float l[3] = {kFloatMax, kFloatMax, kFloatMax}, h[3] = {-kFloatMax, -kFloatMax, -kFloatMax};
  for (int k = 0; k < 3; ++k) {
    const uint32_t v = T[k];
    for (int a = 0; a < 3; ++a) {
      const float p = P[3 * (size_t)v + a];
      l[a] = fminf(l[a], p);
      h[a] = fmaxf(h[a], p);
    }
  }
  lo[g] = make_float4(l[0], l[1], l[2], 0.0f);
  hi[g] = make_float4(h[0], h[1], h[2], 0.0f);
  idx[g] = local;
}

// The leaf-ordered triangle pool of a batch: pool slot leaf_base + i holds
// triangle idx[prim_offset + i] of job j.
__global__ void k_batch_write_triangles(const float* __restrict__ positions, const uint32_t* __restrict__ triangles,
    const SahJob* __restrict__ jobs, uint32_t job_count, const uint32_t* __restrict__ idx, uint32_t total,
    float4* __restrict__ pool) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const SahJob& job = jobs[sah_job_of(jobs, job_count, g)];
  const uint32_t local = g - job.prim_offset;
  const uint32_t p = idx[g];
  const float* P = positions + 3 * job.vertex_offset;
  const uint32_t* T = triangles + 3 * (job.triangle_offset + p);
  float4* out = pool + kTriStride * (size_t)(job.leaf_base + local);
  for (int k = 0; k < 3; ++k) {
    const uint32_t v = T[k];
    out[k] = make_float4(P[3 * (size_t)v], P[3 * (size_t)v + 1], P[3 * (size_t)v + 2],
        k == 0 ? __uint_as_float(p) : 0.0f);
  }
  out[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// The 4-wide nodes: wide node i holds binary node i's subtree cut at four
// children, opening the interior child with the largest surface area until
// there are four (the greedy collapse of Wald et al., "Getting Rid of
// Packets", 2008). Every binary node gets a wide node at its own index, so
// the collapse is one independent thread per node; a wide node whose binary
// node was opened by its parent is never referenced.
__global__ void k_collapse4(const BvhNode* __restrict__ bin, uint32_t first, uint32_t count, uint32_t n,
    Bvh4Node* __restrict__ wide, int leaves_are_instances) {
  const uint32_t offset = blockIdx.x * blockDim.x + threadIdx.x;
  if (offset >= count) return;
  const uint32_t i = first + offset;
  if (i >= n) return;
  float lo[4][3], hi[4][3];
  int32_t ref[4], cnt[4];
  int k = 0;
  auto take = [&](const BvhNode& nd) {
    const float bx[4] = {nd.x.x, nd.x.y, nd.x.z, nd.x.w}, by[4] = {nd.y.x, nd.y.y, nd.y.z, nd.y.w},
                bz[4] = {nd.z.x, nd.z.y, nd.z.z, nd.z.w};
    const int32_t c[2] = {nd.c.x, nd.c.y}, m[2] = {nd.c.z, nd.c.w};
    for (int j = 0; j < 2; ++j) {
      if (c[j] == kEmptyChild || k >= 4) continue;
      lo[k][0] = bx[2 * j]; hi[k][0] = bx[2 * j + 1];
      lo[k][1] = by[2 * j]; hi[k][1] = by[2 * j + 1];
      lo[k][2] = bz[2 * j]; hi[k][2] = bz[2 * j + 1];
      ref[k] = c[j];
      cnt[k] = m[j];
      ++k;
    }
  };
  take(bin[i]);
  for (int round = 0; round < 2 && k < 4; ++round) {
    int open = -1;
    float best = -1.0f;
    for (int j = 0; j < k; ++j) {
      if (ref[j] < 0 || (uint32_t)ref[j] >= n) continue;
      const float dx = hi[j][0] - lo[j][0], dy = hi[j][1] - lo[j][1], dz = hi[j][2] - lo[j][2];
      const float area = dx * dy + dy * dz + dz * dx;
      if (area > best) {
        best = area;
        open = j;
      }
    }
    if (open < 0) break;
    const BvhNode child = bin[ref[open]];
    // Replace the opened child by the last one, then append its children.
    --k;
    for (int a = 0; a < 3; ++a) {
      lo[open][a] = lo[k][a];
      hi[open][a] = hi[k][a];
    }
    ref[open] = ref[k];
    cnt[open] = cnt[k];
    take(child);
  }
  float ox[4], oX[4], oy[4], oY[4], oz[4], oZ[4];
  int32_t oc[4], on[4];
  for (int j = 0; j < 4; ++j) {
    const bool used = j < k;
    // An absent child's box is inside out, so that no ray enters it.
    ox[j] = used ? lo[j][0] : kFloatMax; oX[j] = used ? hi[j][0] : -kFloatMax;
    oy[j] = used ? lo[j][1] : kFloatMax; oY[j] = used ? hi[j][1] : -kFloatMax;
    oz[j] = used ? lo[j][2] : kFloatMax; oZ[j] = used ? hi[j][2] : -kFloatMax;
    oc[j] = used ? ref[j] : kEmptyChild;
    on[j] = used ? cnt[j] : 0;
    if (used && ref[j] < 0 && !leaves_are_instances) {
      // BLAS leaf: the count goes into the reference's low bits.
      const uint32_t first = ~(uint32_t)ref[j];
      const uint32_t count = (uint32_t)min(max(cnt[j], 1), 1 << kLeafCountBits);
      oc[j] = (int32_t)~((first << kLeafCountBits) | (count - 1u));
    }
  }
  float4* rows = reinterpret_cast<float4*>(wide + i);
  rows[node_row(i, 0)] = make_float4(ox[0], ox[1], ox[2], ox[3]);
  rows[node_row(i, 1)] = make_float4(oX[0], oX[1], oX[2], oX[3]);
  rows[node_row(i, 2)] = make_float4(oy[0], oy[1], oy[2], oy[3]);
  rows[node_row(i, 3)] = make_float4(oY[0], oY[1], oY[2], oY[3]);
  rows[node_row(i, 4)] = make_float4(oz[0], oz[1], oz[2], oz[3]);
  rows[node_row(i, 5)] = make_float4(oZ[0], oZ[1], oZ[2], oZ[3]);
  reinterpret_cast<int4*>(rows)[node_row(i, 6)] = make_int4(oc[0], oc[1], oc[2], oc[3]);
  reinterpret_cast<int4*>(rows)[node_row(i, 7)] = make_int4(on[0], on[1], on[2], on[3]);
}

// Refit after a point edit (the reference refits its BLAS there,
// backend/vulkan/gpu_scene.cpp:1899-1950 in hydra-lotus): the topology is
// kept and the boxes follow the new positions. First the leaf-ordered
// triangle pool takes the new corners (the primitive index each record
// keeps in its first corner's w names its triangle).
__global__ void k_refit_triangles(const float* __restrict__ positions, const uint32_t* __restrict__ triangles,
    float4* __restrict__ pool, uint32_t tri_base, uint32_t count) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  float4* rec = pool + kTriStride * (size_t)(tri_base + i);
  const uint32_t p = __float_as_uint(rec[0].w);
  for (int k = 0; k < 3; ++k) {
    const uint32_t v = triangles[3 * (size_t)p + k];
    rec[k] = make_float4(positions[3 * (size_t)v], positions[3 * (size_t)v + 1], positions[3 * (size_t)v + 2],
        k == 0 ? __uint_as_float(p) : 0.0f);
  }
}

// Each binary node's parent (the root, node_base, has none) and a cleared
// arrival count.
__global__ void k_refit_parents(const BvhNode* __restrict__ nodes, uint32_t node_base, uint32_t count,
    uint32_t* __restrict__ parent, uint32_t* __restrict__ arrivals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int4 c = nodes[node_base + i].c;
  // Slots that a tree with larger leaves leaves unused name no node of it.
  if (c.x >= 0 && (uint32_t)c.x - node_base < count) parent[(uint32_t)c.x - node_base] = node_base + i;
  if (c.y >= 0 && (uint32_t)c.y - node_base < count) parent[(uint32_t)c.y - node_base] = node_base + i;
  arrivals[i] = 0;
}

__device__ __forceinline__ void store_child_box(BvhNode* node, int slot, float4 lo, float4 hi) {
  float* x = reinterpret_cast<float*>(&node->x);
  float* y = reinterpret_cast<float*>(&node->y);
  float* z = reinterpret_cast<float*>(&node->z);
  x[2 * slot] = lo.x; x[2 * slot + 1] = hi.x;
  y[2 * slot] = lo.y; y[2 * slot + 1] = hi.y;
  z[2 * slot] = lo.z; z[2 * slot + 1] = hi.z;
}

// Bottom-up boxes: each node's thread boxes its leaf children's triangles
// into the node; a node is complete once all its non-empty children have
// arrived (its leaves, then each interior child as it completes), and the
// last arrival writes its box into its parent's slot and carries on there.
__global__ void k_refit_up(BvhNode* nodes, const float4* __restrict__ pool, uint32_t node_base, uint32_t count,
    const uint32_t* __restrict__ parent, uint32_t* arrivals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  uint32_t node = node_base + i;
  int4 c = nodes[node].c;
  const int32_t ref[2] = {c.x, c.y};
  const int32_t cnt[2] = {c.z, c.w};
  uint32_t leaves = 0;
  for (int k = 0; k < 2; ++k) {
    if (ref[k] >= 0) continue;  // interior or empty
    const uint32_t first = ~(uint32_t)ref[k];
    float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.0f), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.0f);
    for (int t = 0; t < max(cnt[k], 1); ++t)
      for (int v = 0; v < 3; ++v) {
        const float4 p = pool[kTriStride * (size_t)(first + t) + v];
        lo = make_float4(fminf(lo.x, p.x), fminf(lo.y, p.y), fminf(lo.z, p.z), 0.0f);
        hi = make_float4(fmaxf(hi.x, p.x), fmaxf(hi.y, p.y), fmaxf(hi.z, p.z), 0.0f);
      }
    store_child_box(&nodes[node], k, lo, hi);
    ++leaves;
  }
  if (leaves == 0) return;
  uint32_t arrived = leaves;
  // A tree over the scene's triangles is far shallower than 256 levels; the
  // bound only guards against corrupt input.
  for (int level = 0; level < 256; ++level) {
    __threadfence();
    const uint32_t before = atomicAdd(&arrivals[node - node_base], arrived);
    c = __ldcg(&nodes[node].c);
    const uint32_t needed = (c.x != kEmptyChild ? 1u : 0u) + (c.y != kEmptyChild ? 1u : 0u);
    if (before + arrived < needed) return;
    __threadfence();
    if (node == node_base) return;
    const float4 bx = __ldcg(&nodes[node].x), by = __ldcg(&nodes[node].y), bz = __ldcg(&nodes[node].z);
    float4 lo, hi;
    if (c.y == kEmptyChild) {
      lo = make_float4(bx.x, by.x, bz.x, 0.0f);
      hi = make_float4(bx.y, by.y, bz.y, 0.0f);
    } else {
      lo = make_float4(fminf(bx.x, bx.z), fminf(by.x, by.z), fminf(bz.x, bz.z), 0.0f);
      hi = make_float4(fmaxf(bx.y, bx.w), fmaxf(by.y, by.w), fmaxf(bz.y, bz.w), 0.0f);
    }
    const uint32_t up = parent[node - node_base];
    const int4 pc = __ldcg(&nodes[up].c);
    store_child_box(&nodes[up], pc.x == (int32_t)node ? 0 : 1, lo, hi);
    node = up;
    arrived = 1;
  }
}

// Blocks of the SAH list kernels: up to eight on each of a B200's SMs.
constexpr uint32_t kListBlocks = 148 * 8;

inline uint32_t blocks(uint64_t n) { return (uint32_t)((n + kBuildBlock - 1) / kBuildBlock); }

}  // namespace

cudaError_t BvhBuilder::refit_triangles(const float* positions, const uint32_t* triangles, uint32_t n,
    BvhNode* nodes, uint32_t node_base, float4* tri_pool, uint32_t tri_base, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  cudaError_t e = reserve(n, stream);
  if (e != cudaSuccess) return e;
  const uint32_t count = node_count(n);
  k_refit_triangles<<<blocks(n), kBuildBlock, 0, stream>>>(positions, triangles, tri_pool, tri_base, n);
  k_refit_parents<<<blocks(count), kBuildBlock, 0, stream>>>(nodes, node_base, count, parent_internal_, flags_);
  k_refit_up<<<blocks(count), kBuildBlock, 0, stream>>>(nodes, tri_pool, node_base, count, parent_internal_,
      flags_);
  return cudaGetLastError();
}

cudaError_t BvhBuilder::reserve(uint32_t n, cudaStream_t stream) {
  if (n <= capacity_) return cudaSuccess;
  release();
  cudaError_t e;
  const size_t nn = n;
  auto alloc = [&](void** p, size_t bytes) {
    if ((e = cudaMalloc(p, bytes)) != cudaSuccess) return false;
    return true;
  };
  if (!alloc((void**)&keys_, nn * 8) || !alloc((void**)&keys_alt_, nn * 8) ||
      !alloc((void**)&values_, nn * 4) || !alloc((void**)&values_alt_, nn * 4) ||
      !alloc((void**)&plo_, nn * 16) || !alloc((void**)&phi_, nn * 16) ||
      !alloc((void**)&nlo_, nn * 16) || !alloc((void**)&nhi_, nn * 16) ||
      !alloc((void**)&left_, nn * 4) || !alloc((void**)&right_, nn * 4) ||
      !alloc((void**)&parent_internal_, nn * 4) || !alloc((void**)&parent_leaf_, nn * 4) ||
      !alloc((void**)&flags_, nn * 4) || !alloc((void**)&bounds_, (8 + kSahCounters) * 4))
    return e;
  size_t temp = 0;
  cub::DoubleBuffer<uint64_t> k(keys_, keys_alt_);
  cub::DoubleBuffer<uint32_t> v(values_, values_alt_);
  cub::DeviceRadixSort::SortPairs(nullptr, temp, k, v, (int)n, 0, 63, stream);
  if (!alloc(&temp_, temp)) return e;
  temp_bytes_ = temp;
  capacity_ = n;
  return cudaSuccess;
}

void BvhBuilder::release() {
  void* ptrs[] = {keys_, keys_alt_, values_, values_alt_, plo_, phi_, nlo_, nhi_, left_, right_,
      parent_internal_, parent_leaf_, flags_, bounds_, temp_, jobs_};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  keys_ = keys_alt_ = nullptr;
  values_ = values_alt_ = nullptr;
  plo_ = phi_ = nlo_ = nhi_ = nullptr;
  left_ = right_ = parent_internal_ = parent_leaf_ = flags_ = bounds_ = nullptr;
  temp_ = nullptr;
  jobs_ = nullptr;
  job_capacity_ = 0;
  capacity_ = 0;
  temp_bytes_ = 0;
}

cudaError_t BvhBuilder::build_common(uint32_t n, BvhNode* nodes, uint32_t node_base,
    uint32_t leaf_base, bool leaves_are_values, cudaStream_t stream, const uint32_t** sorted) {
  k_morton<<<blocks(n), kBuildBlock, 0, stream>>>(plo_, phi_, n, bounds_, keys_, values_);
  cub::DoubleBuffer<uint64_t> k(keys_, keys_alt_);
  cub::DoubleBuffer<uint32_t> v(values_, values_alt_);
  size_t temp = temp_bytes_;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(temp_, temp, k, v, (int)n, 0, 63, stream);
  if (e != cudaSuccess) return e;
  const uint64_t* skeys = k.Current();
  const uint32_t* svalues = v.Current();
  *sorted = svalues;
  if (n == 1) {
    k_single_root<<<1, 1, 0, stream>>>(plo_, phi_, nodes, node_base, leaf_base, leaves_are_values);
    return cudaGetLastError();
  }
  k_karras<<<blocks(n - 1), kBuildBlock, 0, stream>>>(skeys, (int)n, left_, right_,
      parent_internal_, parent_leaf_);
  cudaMemsetAsync(flags_, 0, sizeof(uint32_t) * n, stream);
  k_fit<<<blocks(n), kBuildBlock, 0, stream>>>(svalues, plo_, phi_, (int)n, left_, right_,
      parent_internal_, parent_leaf_, nlo_, nhi_, flags_);
  k_write_nodes<<<blocks(n - 1), kBuildBlock, 0, stream>>>(svalues, plo_, phi_, (int)n, left_,
      right_, nlo_, nhi_, nodes, node_base, leaf_base, leaves_are_values ? 1 : 0);
  return cudaGetLastError();
}

static void init_bounds(uint32_t* bounds, cudaStream_t stream) {
  const uint32_t init[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
  cudaMemcpyAsync(bounds, init, sizeof(init), cudaMemcpyHostToDevice, stream);
}

cudaError_t BvhBuilder::build_triangles(const float* positions, const uint32_t* triangles,
    uint32_t n, BvhNode* nodes, uint32_t node_base, float4* tri_pool, uint32_t tri_base,
    cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  cudaError_t e = reserve(n, stream);
  if (e != cudaSuccess) return e;
  init_bounds(bounds_, stream);
  k_triangle_boxes<<<blocks(n), kBuildBlock, 0, stream>>>(positions, triangles, n, plo_, phi_, bounds_);
  const uint32_t* sorted = nullptr;
  if ((e = build_common(n, nodes, node_base, tri_base, false, stream, &sorted)) != cudaSuccess) return e;
  k_write_triangles<<<blocks(n), kBuildBlock, 0, stream>>>(sorted, positions, triangles, n, tri_pool, tri_base);
  return cudaGetLastError();
}

// Builds the jobs' trees over the boxes in plo_ / phi_ and the indices in
// values_ (both in batch order). One word of errors is left for the caller
// to read.
cudaError_t BvhBuilder::sah_build(const std::vector<SahJob>& jobs, uint32_t total, BvhNode* nodes,
    cudaStream_t stream) {
  uint32_t largest = 0;
  for (const SahJob& j : jobs) {
    largest = std::max(largest, j.count);
    // Leaves of several triangles leave node slots unused, which the refit
    // and the collapse read: as references to no node.
    if (j.leaf_size > 1) cudaMemsetAsync(nodes + j.node_base, 0x7F, node_count(j.count) * sizeof(BvhNode), stream);
  }
  SahLists lists{reinterpret_cast<SahNode*>(keys_alt_), reinterpret_cast<SahNode*>(keys_), bounds_ + 8};
  cudaMemsetAsync(lists.counters, 0, kSahCounters * sizeof(uint32_t), stream);
  k_sah_large<<<(uint32_t)jobs.size(), kSahBlock, 0, stream>>>(jobs_, plo_, phi_, values_, values_alt_, nodes, lists);
  if (largest > kSahSmall) {
    const uint32_t grid = std::min(kListBlocks, total / (kSahSmall * kMediumWarps) + 1);
    k_sah_medium<<<grid, 32 * kMediumWarps, 0, stream>>>(jobs_, plo_, phi_, values_, values_alt_, nodes, lists);
  }
  if (largest > 1) {
    const uint32_t grid = std::min(kListBlocks, total / (2 * kSmallWarps) + 1);
    k_sah_small<<<grid, 32 * kSmallWarps, 0, stream>>>(jobs_, plo_, phi_, values_, nodes, lists);
  }
  return cudaGetLastError();
}

cudaError_t BvhBuilder::upload_jobs(const std::vector<SahJob>& jobs, cudaStream_t stream) {
  if (jobs.size() > job_capacity_) {
    if (jobs_) cudaFree(jobs_);
    jobs_ = nullptr;
    job_capacity_ = 0;
    const cudaError_t e = cudaMalloc(&jobs_, jobs.size() * sizeof(SahJob));
    if (e != cudaSuccess) return e;
    job_capacity_ = jobs.size();
  }
  return cudaMemcpyAsync(jobs_, jobs.data(), jobs.size() * sizeof(SahJob), cudaMemcpyHostToDevice, stream);
}

cudaError_t BvhBuilder::sah_errors(cudaStream_t stream) {
  uint32_t errors = 0;
  cudaMemcpyAsync(&errors, bounds_ + 8 + kSahErrors, 4, cudaMemcpyDeviceToHost, stream);
  const cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return e;
  return errors ? cudaErrorUnknown : cudaSuccess;
}

cudaError_t BvhBuilder::build_triangle_batch(const float* positions, const uint32_t* triangles,
    const std::vector<BatchGeometry>& geometries, BvhNode* nodes, float4* tri_pool, cudaStream_t stream,
    uint32_t leaf_size) {
  std::vector<SahJob> jobs;
  uint32_t total = 0;
  for (const BatchGeometry& g : geometries) {
    if (g.count == 0) continue;
    jobs.push_back(SahJob{total, g.count, g.node_base, g.tri_base, leaf_size, 0, g.vertex_offset, g.tri_base});
    total += g.count;
  }
  if (jobs.empty()) return cudaSuccess;
  cudaError_t e = reserve(total, stream);
  if (e != cudaSuccess || (e = upload_jobs(jobs, stream)) != cudaSuccess) return e;
  const uint32_t count = (uint32_t)jobs.size();
  k_batch_triangle_boxes<<<blocks(total), kBuildBlock, 0, stream>>>(positions, triangles, jobs_, count, total, plo_,
      phi_, values_);
  if ((e = sah_build(jobs, total, nodes, stream)) != cudaSuccess) return e;
  k_batch_write_triangles<<<blocks(total), kBuildBlock, 0, stream>>>(positions, triangles, jobs_, count, values_,
      total, tri_pool);
  return sah_errors(stream);
}

cudaError_t BvhBuilder::build_instances_sah(const InstanceShading* shade, const InstanceTraversal* trav,
    const BvhNode* blas, uint32_t n, BvhNode* nodes, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const std::vector<SahJob> jobs(1, SahJob{0, n, 0, 0, 1, 1, 0, 0});
  cudaError_t e = reserve(n, stream);
  if (e != cudaSuccess || (e = upload_jobs(jobs, stream)) != cudaSuccess) return e;
  k_instance_boxes<<<blocks(n), kBuildBlock, 0, stream>>>(shade, trav, blas, n, plo_, phi_, nullptr, values_);
  if ((e = sah_build(jobs, n, nodes, stream)) != cudaSuccess) return e;
  return sah_errors(stream);
}

cudaError_t BvhBuilder::collapse(const BvhNode* binary, uint32_t n, Bvh4Node* wide, bool leaves_are_instances,
    cudaStream_t stream) {
  return collapse_range(binary, 0, n, n, wide, leaves_are_instances, stream);
}

cudaError_t BvhBuilder::collapse_range(const BvhNode* binary, uint32_t first, uint32_t count, uint32_t n,
    Bvh4Node* wide, bool leaves_are_instances, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  k_collapse4<<<blocks(count), kBuildBlock, 0, stream>>>(binary, first, count, n, wide,
      leaves_are_instances ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t BvhBuilder::build_instances(const InstanceShading* shade,
    const InstanceTraversal* trav, const BvhNode* blas, uint32_t n, BvhNode* nodes,
    cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  cudaError_t e = reserve(n, stream);
  if (e != cudaSuccess) return e;
  init_bounds(bounds_, stream);
  k_instance_boxes<<<blocks(n), kBuildBlock, 0, stream>>>(shade, trav, blas, n, plo_, phi_, bounds_, nullptr);
  const uint32_t* sorted = nullptr;
  return build_common(n, nodes, 0, 0, true, stream, &sorted);
}

}  // namespace lotus
