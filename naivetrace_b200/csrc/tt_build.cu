// Device BVH construction: PLOC (parallel locally-ordered clustering, Meister and Bittner
// 2018) over Morton-ordered primitives, a bottom-up SAH pass that collapses small subtrees
// into leaves of at most four primitives, and emission in the binary layout of tt_bvh.h.
// Replaces the Embree scene commit (Scene::BuildAccelStructure, scene.cxx:116-141) on the
// GPU: the host sends the mesh once and the tree is built next to it.
//
// Clustering: clusters sit in Morton order; each finds the neighbour within kRadius
// positions whose merged box has the least surface area (ties broken by the pair's
// positions, so the relation is a strict order and the globally best pair is always
// mutual); mutual nearest neighbours merge into a new node at the lower position, and the
// array is compacted.  Node ids grow with the iteration that created them, so children
// always precede parents, and one kernel per iteration range walks the tree bottom-up or
// top-down.
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "tt_build.h"
#include "tt_internal.h"

namespace tt {
namespace {

// PLOC neighbourhood (positions on either side); TT_PLOC_RADIUS overrides.  On the terrain
// workload a small radius gave the lowest SAH cost (radius 2: 35.4, 8: 37.2, 16: 38.1,
// 64: 40.1; the host binned-SAH builder: 33.4).
constexpr int kDefaultRadius = 2;
constexpr int kMaxLeaf = 4;
constexpr int kMaxIterations = 4096;
constexpr int kThreads = 256;

struct Aabb {
  float3 lo, hi;
};

__device__ __forceinline__ float half_area(const Aabb& b) {
  const float dx = b.hi.x - b.lo.x, dy = b.hi.y - b.lo.y, dz = b.hi.z - b.lo.z;
  return dx * dy + dy * dz + dz * dx;
}
__device__ __forceinline__ Aabb merge(const Aabb& a, const Aabb& b) {
  return Aabb{make_float3(fminf(a.lo.x, b.lo.x), fminf(a.lo.y, b.lo.y), fminf(a.lo.z, b.lo.z)),
              make_float3(fmaxf(a.hi.x, b.hi.x), fmaxf(a.hi.y, b.hi.y), fmaxf(a.hi.z, b.hi.z))};
}

// Order-preserving map of floats to unsigned ints (for atomic min / max of floats).
__device__ __forceinline__ unsigned ordered(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ Aabb prim_box(const BuildInput& in, uint32_t global) {
  Aabb b;
  if (global < in.num_triangles) {
    const uint32_t* t = in.indices + 3 * (size_t)global;
    const float* v0 = in.vertices + 3 * (size_t)t[0];
    const float* v1 = in.vertices + 3 * (size_t)t[1];
    const float* v2 = in.vertices + 3 * (size_t)t[2];
    b.lo = make_float3(fminf(v0[0], fminf(v1[0], v2[0])), fminf(v0[1], fminf(v1[1], v2[1])),
                       fminf(v0[2], fminf(v1[2], v2[2])));
    b.hi = make_float3(fmaxf(v0[0], fmaxf(v1[0], v2[0])), fmaxf(v0[1], fmaxf(v1[1], v2[1])),
                       fmaxf(v0[2], fmaxf(v1[2], v2[2])));
  } else {
    // One ulp outside centre -/+ radius (SphereBoundsFunc, embreeaccelerator.cxx:263-281).
    const float* q = in.spheres + 4 * (size_t)(global - in.num_triangles);
    b.lo = make_float3(nextafterf(q[0] - q[3], -INFINITY), nextafterf(q[1] - q[3], -INFINITY),
                       nextafterf(q[2] - q[3], -INFINITY));
    b.hi = make_float3(nextafterf(q[0] + q[3], INFINITY), nextafterf(q[1] + q[3], INFINITY),
                       nextafterf(q[2] + q[3], INFINITY));
  }
  return b;
}

__global__ void k_prim_boxes(BuildInput in, const uint32_t* set, uint32_t n, Aabb* boxes, unsigned* cbounds) {
  unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Aabb b = prim_box(in, set[i]);
    boxes[i] = b;
    const float c[3] = {0.5f * (b.lo.x + b.hi.x), 0.5f * (b.lo.y + b.hi.y), 0.5f * (b.lo.z + b.hi.z)};
    for (int k = 0; k < 3; ++k) {
      lo[k] = min(lo[k], ordered(c[k]));
      hi[k] = max(hi[k], ordered(c[k]));
    }
  }
  // One atomic per bound and block: one per warp serialised on the six addresses (161 us of the
  // build of 2.75 M primitives).
  __shared__ unsigned part[6][kThreads / 32];
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] = min(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
      hi[k] = max(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
    }
    if ((threadIdx.x & 31) == 0) {
      part[k][threadIdx.x >> 5] = lo[k];
      part[3 + k][threadIdx.x >> 5] = hi[k];
    }
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    unsigned v = part[threadIdx.x][0];
    for (int w = 1; w < kThreads / 32; ++w)
      v = threadIdx.x < 3 ? min(v, part[threadIdx.x][w]) : max(v, part[threadIdx.x][w]);
    if (threadIdx.x < 3) atomicMin(&cbounds[threadIdx.x], v);
    else atomicMax(&cbounds[threadIdx.x], v);
  }
}

__device__ __forceinline__ uint64_t spread21(uint64_t x) {
  x &= 0x1fffffull;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}

// 63-bit Morton code of the box centre in the centroid bounds, with one scale for all three
// axes: cubic cells keep the curve's neighbours spatial neighbours in flat scenes.
__global__ void k_morton(const Aabb* boxes, uint32_t n, const unsigned* cbounds, uint64_t* keys, uint32_t* vals) {
  float lo[3], ext[3];
  float e = 0.f;
  for (int k = 0; k < 3; ++k) {
    lo[k] = unordered(cbounds[k]);
    e = fmaxf(e, unordered(cbounds[3 + k]) - lo[k]);
  }
  for (int k = 0; k < 3; ++k) ext[k] = e;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Aabb b = boxes[i];
    const float c[3] = {0.5f * (b.lo.x + b.hi.x), 0.5f * (b.lo.y + b.hi.y), 0.5f * (b.lo.z + b.hi.z)};
    uint64_t code = 0;
    for (int k = 0; k < 3; ++k) {
      const float f = ext[k] > 0.f ? (c[k] - lo[k]) / ext[k] : 0.f;
      const uint64_t q = (uint64_t)fminf(fmaxf(f * 2097152.f, 0.f), 2097151.f);
      code |= spread21(q) << (2 - k);
    }
    keys[i] = code;
    vals[i] = i;
  }
}

// Leaves 0..n-1 in Morton order: node box = primitive box, left = -1 - (set position).
__global__ void k_init_leaves(const Aabb* prim_boxes, const uint32_t* perm, uint32_t n, Aabb* node_box,
                              int* left, int* right, int* clusters) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    node_box[i] = prim_boxes[perm[i]];
    left[i] = -1 - (int)perm[i];
    right[i] = -1;
    clusters[i] = (int)i;
  }
}

// Pair order: merged area, then the pair's lower and higher positions.
__device__ __forceinline__ bool pair_less(float a, int lo, int hi, float b, int blo, int bhi) {
  return a < b || (a == b && (lo < blo || (lo == blo && hi < bhi)));
}

__global__ void k_nearest(const int* clusters, int c, const Aabb* node_box, int radius, int* nn) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < c; i += gridDim.x * blockDim.x) {
    const Aabb bi = node_box[clusters[i]];
    float best = INFINITY;
    int bj = -1;
    const int j0 = max(0, i - radius), j1 = min(c - 1, i + radius);
    for (int j = j0; j <= j1; ++j) {
      if (j == i) continue;
      const float a = half_area(merge(bi, node_box[clusters[j]]));
      if (bj < 0 || pair_less(a, min(i, j), max(i, j), best, min(i, bj), max(i, bj))) {
        best = a;
        bj = j;
      }
    }
    nn[i] = bj;
  }
}

// create[i]: i is the lower end of a mutual pair (it makes the new node); keep[i]: i stays
// a cluster after the merge (everything except the higher end of a mutual pair).
__global__ void k_merge_flags(const int* nn, int c, int* create, int* keep) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < c; i += gridDim.x * blockDim.x) {
    const int j = nn[i];
    const bool mutual = j >= 0 && nn[j] == i;
    create[i] = (mutual && i < j) ? 1 : 0;
    keep[i] = (mutual && i > j) ? 0 : 1;
  }
}

__global__ void k_merge(const int* clusters, int c, const int* nn, const int* create, const int* create_off,
                        const int* keep, const int* keep_off, int next_node, Aabb* node_box, int* left, int* right,
                        int* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < c; i += gridDim.x * blockDim.x) {
    if (!keep[i]) continue;
    int id = clusters[i];
    if (create[i]) {
      const int j = nn[i];
      const int k = next_node + create_off[i];
      const int a = clusters[i], b = clusters[j];
      node_box[k] = merge(node_box[a], node_box[b]);
      left[k] = a;
      right[k] = b;
      id = k;
    }
    out[keep_off[i]] = id;
  }
}

// The clustering iterations from at most kTailClusters clusters down to one, in one block: the
// clusters' boxes, ids and neighbours in shared memory, thread t owning clusters 4t .. 4t + 3 so
// that the scans run in cluster order.  The pairs, node numbers and cluster order are those of the
// kernels above; an iteration costs a few microseconds instead of nine launches, four copies and a
// synchronisation (50-60 us), and about half of a build's 46 iterations (2.75 M primitives) start
// with so few clusters.  ranges[i]: first node and node count of iteration i; info: iterations
// done, next node, the last cluster's node, 1 when an iteration made no progress.
constexpr int kTailThreads = 1024, kTailEach = 4, kTailClusters = kTailThreads * kTailEach;
constexpr int kTailSmem = kTailClusters * (int)(sizeof(Aabb) + 2 * sizeof(int));
__global__ void __launch_bounds__(kTailThreads) k_cluster_tail(const int* clusters, int c, int radius, int next_node,
                                                               int total, int max_iterations, Aabb* node_box,
                                                               int* left, int* right, int2* ranges, int* info) {
  extern __shared__ __align__(16) unsigned char tail_smem[];
  Aabb* box = reinterpret_cast<Aabb*>(tail_smem);
  int* id = reinterpret_cast<int*>(box + kTailClusters);
  int* nn = id + kTailClusters;
  __shared__ int wsum[2][kTailThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int i = t; i < c; i += kTailThreads) {
    id[i] = clusters[i];
    box[i] = node_box[id[i]];
  }
  __syncthreads();
  int it = 0;
  bool stuck = false;
  while (c > 1 && it < max_iterations) {
    for (int i = t; i < c; i += kTailThreads) {
      const Aabb bi = box[i];
      float best = INFINITY;
      int bj = -1;
      const int j0 = max(0, i - radius), j1 = min(c - 1, i + radius);
      for (int j = j0; j <= j1; ++j) {
        if (j == i) continue;
        const float a = half_area(merge(bi, box[j]));
        if (bj < 0 || pair_less(a, min(i, j), max(i, j), best, min(i, bj), max(i, bj))) {
          best = a;
          bj = j;
        }
      }
      nn[i] = bj;
    }
    __syncthreads();
    // This thread's clusters after the merge (in registers), and how many nodes and clusters it makes.
    Aabb nb[kTailEach];
    int nid[kTailEach], partner[kTailEach];
    int made = 0, kept = 0;
#pragma unroll
    for (int e = 0; e < kTailEach; ++e) {
      const int i = kTailEach * t + e;
      nid[e] = -1;
      partner[e] = -1;
      if (i < c) {
        const int j = nn[i];
        const bool mutual = j >= 0 && nn[j] == i;
        if (!(mutual && i > j)) {
          nid[e] = id[i];
          nb[e] = box[i];
          ++kept;
          if (mutual) {
            partner[e] = id[j];
            nb[e] = merge(nb[e], box[j]);
            ++made;
          }
        }
      }
    }
    int smade = made, skept = kept;
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, smade, o), b = __shfl_up_sync(0xffffffffu, skept, o);
      if (lane >= o) {
        smade += a;
        skept += b;
      }
    }
    if (lane == 31) {
      wsum[0][warp] = smade;
      wsum[1][warp] = skept;
    }
    __syncthreads();
    int all_made = 0, all_kept = 0, node = smade - made, out = skept - kept;
    for (int w = 0; w < kTailThreads / 32; ++w) {
      if (w < warp) {
        node += wsum[0][w];
        out += wsum[1][w];
      }
      all_made += wsum[0][w];
      all_kept += wsum[1][w];
    }
    if (all_made == 0 || next_node + all_made > total) {  // uniform
      stuck = true;
      break;
    }
#pragma unroll
    for (int e = 0; e < kTailEach; ++e) {
      if (nid[e] < 0) continue;
      if (partner[e] >= 0) {
        const int k = next_node + node++;
        node_box[k] = nb[e];
        left[k] = nid[e];
        right[k] = partner[e];
        nid[e] = k;
      }
      id[out] = nid[e];
      box[out] = nb[e];
      ++out;
    }
    if (t == 0) ranges[it] = make_int2(next_node, all_made);
    next_node += all_made;
    c = all_kept;
    ++it;
    __syncthreads();
  }
  if (t == 0) {
    info[0] = it;
    info[1] = next_node;
    info[2] = id[0];
    info[3] = stuck || c > 1 ? 1 : 0;
  }
}

// Bottom-up over one creation range: subtree sizes and SAH costs (traversal step 1,
// primitive test 1 per primitive), whether a subtree of at most kMaxLeaf primitives is
// cheaper as one leaf, and the number of inner nodes the subtree emits.
__device__ __forceinline__ void costs_range(int start, int step, int first, int count, uint32_t n, const Aabb* node_box,
                                            const int* left, const int* right, int* size, float* cost,
                                            unsigned char* collapse, int* inner) {
  for (int t = start; t < count; t += step) {
    const int k = first + t;
    const int l = left[k], r = right[k];
    const int sl = l < (int)n ? 1 : size[l], sr = r < (int)n ? 1 : size[r];
    const float cl = l < (int)n ? 1.f : cost[l], cr = r < (int)n ? 1.f : cost[r];
    const float a = half_area(node_box[k]);
    const float split = a > 0.f ? 1.f + (half_area(node_box[l]) * cl + half_area(node_box[r]) * cr) / a
                                : 1.f + cl + cr;
    const int s = sl + sr;
    const float leaf = (float)s;
    const bool as_leaf = s <= kMaxLeaf && leaf <= split;
    size[k] = s;
    cost[k] = as_leaf ? leaf : split;
    collapse[k] = as_leaf ? 1 : 0;
    inner[k] = as_leaf ? 0 : 1 + (l < (int)n ? 0 : inner[l]) + (r < (int)n ? 0 : inner[r]);
  }
}

__global__ void k_costs(int first, int count, uint32_t n, const Aabb* node_box, const int* left, const int* right,
                        int* size, float* cost, unsigned char* collapse, int* inner) {
  costs_range(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, first, count, n, node_box, left, right,
              size, cost, collapse, inner);
}
// The small ranges of the clustering tail one after the other in one block.
__global__ void __launch_bounds__(kTailThreads) k_costs_tail(const int2* ranges, int count, uint32_t n,
                                                             const Aabb* node_box, const int* left, const int* right,
                                                             int* size, float* cost, unsigned char* collapse,
                                                             int* inner) {
  for (int r = 0; r < count; ++r) {
    costs_range(threadIdx.x, blockDim.x, ranges[r].x, ranges[r].y, n, node_box, left, right, size, cost, collapse,
                inner);
    __syncthreads();
  }
}

// Top-down over one creation range: primitive offsets and node indices (both in depth-first
// order: an inner node's first child follows it in memory, its second child follows the
// first child's subtree) and whether the node is emitted as an inner node, lies inside a
// leaf, or is a leaf itself.  state: bit 0 = inside a leaf (set by an ancestor that
// became a leaf).
__device__ __forceinline__ void topdown_range(int start, int step, int first, int count, uint32_t n, const int* left,
                                              const int* right, const int* size, const unsigned char* collapse,
                                              const int* inner, int* offset, int* index, unsigned char* state,
                                              int* depth, unsigned char* emit, unsigned* max_depth) {
  for (int t = start; t < count; t += step) {
    const int k = first + t;
    const bool inside = state[k] & 1u;
    const bool leafnode = inside || collapse[k];
    emit[k] = leafnode ? 0 : 1;
    const int l = left[k], r = right[k];
    const int sl = l < (int)n ? 1 : size[l];
    offset[l] = offset[k];
    offset[r] = offset[k] + sl;
    state[l] = leafnode ? 1 : 0;
    state[r] = leafnode ? 1 : 0;
    if (!leafnode) {
      depth[l] = depth[k] + 1;
      depth[r] = depth[k] + 1;
      index[l] = index[k] + 1;
      index[r] = index[k] + 1 + (l < (int)n ? 0 : inner[l]);
      atomicMax(max_depth, (unsigned)(depth[k] + 1));
    }
  }
}

__global__ void k_topdown(int first, int count, uint32_t n, const int* left, const int* right, const int* size,
                          const unsigned char* collapse, const int* inner, int* offset, int* index,
                          unsigned char* state, int* depth, unsigned char* emit, unsigned* max_depth) {
  topdown_range(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, first, count, n, left, right, size,
                collapse, inner, offset, index, state, depth, emit, max_depth);
}
__global__ void __launch_bounds__(kTailThreads) k_topdown_tail(const int2* ranges, int count, uint32_t n,
                                                               const int* left, const int* right, const int* size,
                                                               const unsigned char* collapse, const int* inner,
                                                               int* offset, int* index, unsigned char* state,
                                                               int* depth, unsigned char* emit, unsigned* max_depth) {
  for (int r = count - 1; r >= 0; --r) {
    topdown_range(threadIdx.x, blockDim.x, ranges[r].x, ranges[r].y, n, left, right, size, collapse, inner, offset,
                  index, state, depth, emit, max_depth);
    __syncthreads();
  }
}

// Primitive slots in depth-first order (layout in tt_bvh.h).
__global__ void k_write_slots(BuildInput in, const uint32_t* set, const int* left, const int* offset, uint32_t n,
                              float4* tris) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t pos = (uint32_t)(-1 - left[i]);
    const uint32_t g = set[pos];
    float4* dst = tris + 3 * (size_t)offset[i];
    if (g < in.num_triangles) {
      const uint32_t* t = in.indices + 3 * (size_t)g;
      const float* v0 = in.vertices + 3 * (size_t)t[0];
      const float* v1 = in.vertices + 3 * (size_t)t[1];
      const float* v2 = in.vertices + 3 * (size_t)t[2];
      dst[0] = make_float4(v0[0], v0[1], v0[2], __int_as_float((int)in.prim_ids[pos]));
      dst[1] = make_float4(v1[0], v1[1], v1[2], __int_as_float((int)in.material_ids[g]));
      dst[2] = make_float4(v2[0], v2[1], v2[2], 0.f);
    } else {
      const uint32_t k = g - in.num_triangles;
      const float* q = in.spheres + 4 * (size_t)k;
      dst[0] = make_float4(q[0], q[1], q[2], __int_as_float((int)in.prim_ids[pos]));
      dst[1] = make_float4(q[3], 0.f, 0.f, __int_as_float((int)in.sphere_material_ids[k]));
      dst[2] = make_float4(0.f, 0.f, 0.f, __int_as_float(1));
    }
  }
}

__device__ __forceinline__ int child_ref(int c, uint32_t n, const int* size, const int* offset,
                                         const unsigned char* emit, const int* index) {
  if (c >= (int)n && emit[c]) return index[c];
  const int cnt = c < (int)n ? 1 : size[c];
  return ~(int)(((unsigned)offset[c] << 3) | (unsigned)(cnt - 1));
}

// Emitted inner node k -> device node index[k] (the root is node 0).
__global__ void k_write_nodes(int first, int count, uint32_t n, const Aabb* node_box, const int* left,
                              const int* right, const int* size, const int* offset, const unsigned char* emit,
                              const int* index, float4* nodes) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
    const int k = first + t;
    if (!emit[k]) continue;
    const int l = left[k], r = right[k];
    const Aabb a = node_box[l], b = node_box[r];
    float4* d = nodes + 4 * (size_t)index[k];
    d[0] = make_float4(a.lo.x, a.hi.x, a.lo.y, a.hi.y);
    d[1] = make_float4(b.lo.x, b.hi.x, b.lo.y, b.hi.y);
    d[2] = make_float4(a.lo.z, a.hi.z, b.lo.z, b.hi.z);
    d[3] = make_float4(__int_as_float(child_ref(l, n, size, offset, emit, index)),
                       __int_as_float(child_ref(r, n, size, offset, emit, index)), 0.f, 0.f);
  }
}

// Scenes of at least this many primitives get byte boxes in their 4-wide nodes: below, the
// nodes and primitives stay in the L1 whatever their format.  Float / byte boxes, us a pass:
//   terrain 1920x1080 x 4   4,482 primitives 5,322 / 5,392, 10,498 5,765 / 5,796, 18,760 5,960 / 6,003,
//                           34,818 6,116 / 6,125, 75,040 6,691 / 6,623, 171,010 7,186 / 7,024,
//                           686,082 8,172 / 7,785
//   bumpy mesh in the Cornell box, 1024x1024 x 4   1,956 9,874 / 9,953, 7,972 11,322 / 10,953,
//                           16,234 11,919 / 11,301, 32,292 12,525 / 11,947, 130,084 13,869 / 12,694
// (rooms of 20-40 triangles: closest and any hit 2-6 % slower with byte boxes).
constexpr uint32_t kNode4BytesMin = 16384;

// Writes a 4-wide node of m children with float boxes (layout in tt_build.h).
__device__ void write_node4_float(float4* d, const Aabb* box, const int* ref, int m) {
  const float inf = INFINITY;
  float v[6][4];
  int rf[4];
  for (int j = 0; j < 4; ++j) {
    const Aabb b = j < m ? box[j] : Aabb{make_float3(inf, inf, inf), make_float3(-inf, -inf, -inf)};
    v[0][j] = b.lo.x;
    v[1][j] = b.hi.x;
    v[2][j] = b.lo.y;
    v[3][j] = b.hi.y;
    v[4][j] = b.lo.z;
    v[5][j] = b.hi.z;
    rf[j] = j < m ? ref[j] : 0x7fffffff;
  }
  for (int k = 0; k < 6; ++k) d[k] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
  d[6] = make_float4(__int_as_float(rf[0]), __int_as_float(rf[1]), __int_as_float(rf[2]), __int_as_float(rf[3]));
  d[7] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Writes a 4-wide node of m children with byte boxes (layout in tt_build.h).  Per axis the grid's step is
// 1/253 of the children's extent (at least 2^-22 of the coordinates, so that a step is never
// lost in the float origin) and its origin one step below the lowest plane; lower planes round
// down and upper planes up with a margin of 1/32 step for the traversal's rounding.  An empty
// slot has an inverted box and the first child's reference.  The box is met only by a ray so far away
// that the widening of its exit distances exceeds 255 steps; the first child is then visited again.
// It is a leaf: a node keeps an empty slot only if none of its children is an inner node (k_collapse4),
// so the stack, counted with four entries above every node, holds that too.
__device__ void write_node4_bytes(float4* d, const Aabb* box, const int* ref, int m) {
  float org[3], step[3];
  unsigned qlo[3], qhi[3];
  for (int k = 0; k < 3; ++k) {
    auto lo = [&](int j) { return (double)(k == 0 ? box[j].lo.x : k == 1 ? box[j].lo.y : box[j].lo.z); };
    auto hi = [&](int j) { return (double)(k == 0 ? box[j].hi.x : k == 1 ? box[j].hi.y : box[j].hi.z); };
    double a = lo(0), b = hi(0);
    for (int j = 1; j < m; ++j) {
      a = fmin(a, lo(j));
      b = fmax(b, hi(j));
    }
    const double s = fmax(fmax((b - a) / 253.0, fmax(fabs(a), fabs(b)) * 2.384185791015625e-07), 1e-30);
    step[k] = __double2float_ru(s);
    org[k] = __double2float_rd(a - (double)step[k]);
    qlo[k] = qhi[k] = 0u;
    for (int j = 0; j < 4; ++j) {
      unsigned l = 255u, h = 0u;
      if (j < m) {
        l = (unsigned)fmin(255.0, fmax(0.0, floor((lo(j) - org[k]) / step[k] - 0.03125)));
        h = (unsigned)fmin(255.0, fmax(0.0, ceil((hi(j) - org[k]) / step[k] + 0.03125)));
      }
      qlo[k] |= l << (8 * j);
      qhi[k] |= h << (8 * j);
    }
  }
  d[0] = make_float4(org[0], org[1], org[2], step[0]);
  d[1] = make_float4(step[1], step[2], __uint_as_float(qlo[0]), __uint_as_float(qlo[1]));
  d[2] = make_float4(__uint_as_float(qlo[2]), __uint_as_float(qhi[0]), __uint_as_float(qhi[1]), __uint_as_float(qhi[2]));
  d[3] = make_float4(__int_as_float(ref[0]), __int_as_float(ref[m > 1 ? 1 : 0]), __int_as_float(ref[m > 2 ? 2 : 0]),
                     __int_as_float(ref[m > 3 ? 3 : 0]));
}

// atomicAdd(counter, 1) of every active lane, one atomic per warp.
__device__ __forceinline__ int count_up(int* counter) {
  const unsigned mask = __activemask();
  const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(counter, __popc(mask));
  return __shfl_sync(mask, base, leader) + __popc(mask & ((1u << lane) - 1u));
}

// 4-wide layout, built top down one level at a time: a 4-wide node starts from a binary
// inner node's two children and, while it has fewer than four, replaces the inner child of
// the largest surface area by that child's two children (the usual collapse of a binary
// tree into a wide one); its remaining inner children become the next level's 4-wide
// nodes, numbered by an atomic counter.  frontier: (binary node,
// 4-wide index, stack entries a traversal may hold when it reaches the node).
__global__ void k_collapse4(const int4* frontier, int nfront, uint32_t n, const Aabb* node_box, const int* left,
                            const int* right, const int* size, const int* offset, const unsigned char* emit,
                            const int* index, int* counter, int4* next, int* nnext, int* stack_need, int bytes,
                            float4* nodes4) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nfront; t += gridDim.x * blockDim.x) {
    const int k = frontier[t].x, i4 = frontier[t].y;
    int slot[4] = {left[k], right[k], -1, -1};
    int m = 2;
    while (m < 4) {
      int best = -1;
      float best_area = -1.f;
      for (int j = 0; j < m; ++j) {
        const int c = slot[j];
        if (c >= (int)n && emit[c]) {
          const float a = half_area(node_box[c]);
          if (a > best_area) {
            best_area = a;
            best = j;
          }
        }
      }
      if (best < 0) break;
      const int c = slot[best];
      slot[best] = left[c];
      slot[m++] = right[c];
    }
    Aabb box[4];
    int ref[4];
    for (int j = 0; j < m; ++j) {
      const int c = slot[j];
      box[j] = node_box[c];
      if (c >= (int)n && emit[c]) {
        const int j4 = count_up(counter);
        next[count_up(nnext)] = make_int4(c, j4, frontier[t].z + m - 1, 0);
        ref[j] = j4;
      } else {
        ref[j] = child_ref(c, n, size, offset, emit, index);
      }
    }
    if (bytes) write_node4_bytes(nodes4 + 4 * (size_t)i4, box, ref, m);
    else write_node4_float(nodes4 + 8 * (size_t)i4, box, ref, m);
    if (frontier[t].z + 4 > *(volatile int*)stack_need) atomicMax(stack_need, frontier[t].z + 4);
  }
}
// 4-wide root of a tree whose root is a leaf: one slot with the leaf.
__global__ void k_leaf_root4(const Aabb* node_box, int root, int count, float4* nodes4) {
  const Aabb box = node_box[root];
  const int ref = ~(int)(unsigned)(count - 1);
  write_node4_float(nodes4, &box, &ref, 1);
}

// Root handling for trees whose root is a leaf: one node with the leaf as child 0 and an
// empty child 1 (inverted box, reference to slot 0 with count 1).
__global__ void k_leaf_root(const Aabb* node_box, int root, int count, float4* nodes) {
  const Aabb a = node_box[root];
  const float inf = INFINITY;
  nodes[0] = make_float4(a.lo.x, a.hi.x, a.lo.y, a.hi.y);
  nodes[1] = make_float4(inf, -inf, inf, -inf);
  nodes[2] = make_float4(a.lo.z, a.hi.z, inf, -inf);
  nodes[3] = make_float4(__int_as_float(~(int)(unsigned)(count - 1)), __int_as_float(~0), 0.f, 0.f);
}

int grid_for(long long n) {
  long long g = (n + kThreads - 1) / kThreads;
  return (int)(g < 1 ? 1 : (g > 4096 ? 4096 : g));
}

// Scratch allocations from the library's memory pool, released on scope exit.
struct Scratch {
  cudaStream_t st;
  std::vector<void*> ptrs;
  explicit Scratch(cudaStream_t s) : st(s) {}
  template <class T>
  T* alloc(size_t count) {
    void* p = nullptr;
    if (pool_malloc(&p, (count ? count : 1) * sizeof(T), st) != cudaSuccess) return nullptr;
    ptrs.push_back(p);
    return static_cast<T*>(p);
  }
  ~Scratch() {
    for (void* p : ptrs) pool_free(p, st);
  }
};

}  // namespace

bool device_build_bvh2(const BuildInput& in, const uint32_t* set, uint32_t n, DeviceBvh* out, cudaStream_t st,
                       std::string* err) {
  auto fail = [&](const std::string& m) {
    *err = "device BVH build: " + m;
    return false;
  };
  auto ok = [&](cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    *err = std::string("device BVH build: ") + what + ": " + cudaGetErrorString(e);
    return false;
  };
  out->num_nodes = 0;
  out->max_depth = 0;
  out->nodes = nullptr;
  out->tris = nullptr;
  out->nodes4 = nullptr;  // none for an empty tree: traversal uses the binary layout
  out->num_nodes4 = 0;
  if (n == 0) {
    // No primitives: a root with two empty children and one degenerate slot (prim -1).
    float host_node[16];
    const float inf = INFINITY;
    const float h[12] = {inf, -inf, inf, -inf, inf, -inf, inf, -inf, inf, -inf, inf, -inf};
    for (int k = 0; k < 12; ++k) host_node[k] = h[k];
    const int32_t r0 = ~0, zero = 0;
    std::memcpy(&host_node[12], &r0, 4);
    std::memcpy(&host_node[13], &r0, 4);
    std::memcpy(&host_node[14], &zero, 4);
    std::memcpy(&host_node[15], &zero, 4);
    float host_tri[12] = {0.f};
    const int32_t none = -1;
    std::memcpy(&host_tri[3], &none, 4);
    if (!ok(pool_malloc((void**)&out->nodes, sizeof(host_node), st), "allocation") ||
        !ok(pool_malloc((void**)&out->tris, sizeof(host_tri), st), "allocation"))
      return false;
    if (!ok(cudaMemcpyAsync(out->nodes, host_node, sizeof(host_node), cudaMemcpyHostToDevice, st), "copy") ||
        !ok(cudaMemcpyAsync(out->tris, host_tri, sizeof(host_tri), cudaMemcpyHostToDevice, st), "copy") ||
        !ok(cudaStreamSynchronize(st), "sync"))
      return false;
    out->num_nodes = 1;
    return true;
  }
  Scratch sc(st);
  // Small values read back (or sent) during the build go through page-locked host memory:
  // a copy into a pageable stack variable would make every one of them a synchronous round
  // trip, four per clustering iteration.  One 256-byte area per host thread that builds,
  // kept for the thread's lifetime.
  thread_local int* hb = nullptr;
  if (!hb && !ok(cudaHostAlloc((void**)&hb, 256, cudaHostAllocPortable), "page-locked read-back area")) return false;
  const uint32_t total = 2 * n - 1;
  // TT_BUILD_VERBOSE=1 prints the phase times and the iteration count to stderr.
  const bool verbose = std::getenv("TT_BUILD_VERBOSE") != nullptr;
  const auto t_start = std::chrono::steady_clock::now();
  auto ms_since = [&](std::chrono::steady_clock::time_point t0) {
    cudaStreamSynchronize(st);
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  };
  Aabb* prim_boxes = sc.alloc<Aabb>(n);
  unsigned* cbounds = sc.alloc<unsigned>(6);
  uint64_t* keys = sc.alloc<uint64_t>(n);
  uint64_t* keys2 = sc.alloc<uint64_t>(n);
  uint32_t* vals = sc.alloc<uint32_t>(n);
  uint32_t* perm = sc.alloc<uint32_t>(n);
  Aabb* node_box = sc.alloc<Aabb>(total);
  int* left = sc.alloc<int>(total);
  int* right = sc.alloc<int>(total);
  int* clusters = sc.alloc<int>(n);
  int* clusters2 = sc.alloc<int>(n);
  int* nn = sc.alloc<int>(n);
  int* create = sc.alloc<int>(n);
  int* create_off = sc.alloc<int>(n);
  int* keep = sc.alloc<int>(n);
  int* keep_off = sc.alloc<int>(n);
  if (!prim_boxes || !cbounds || !keys || !keys2 || !vals || !perm || !node_box || !left || !right || !clusters ||
      !clusters2 || !nn || !create || !create_off || !keep || !keep_off)
    return fail("out of device memory");
  const unsigned init_bounds[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
  if (!ok(cudaMemcpyAsync(cbounds, init_bounds, sizeof(init_bounds), cudaMemcpyHostToDevice, st), "copy")) return false;
  k_prim_boxes<<<grid_for(n), kThreads, 0, st>>>(in, set, n, prim_boxes, cbounds);
  k_morton<<<grid_for(n), kThreads, 0, st>>>(prim_boxes, n, cbounds, keys, vals);
  // Sort primitives by Morton code (CUB radix sort).
  size_t sort_bytes = 0, scan_bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, keys, keys2, vals, perm, (int)n, 0, 63, st);
  cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, create, create_off, (int)n, st);
  void* temp = sc.alloc<unsigned char>(std::max(sort_bytes, scan_bytes));
  if (!temp) return fail("out of device memory");
  if (!ok(cub::DeviceRadixSort::SortPairs(temp, sort_bytes, keys, keys2, vals, perm, (int)n, 0, 63, st), "sort"))
    return false;
  k_init_leaves<<<grid_for(n), kThreads, 0, st>>>(prim_boxes, perm, n, node_box, left, right, clusters);
  const double t_sorted = verbose ? ms_since(t_start) : 0.0;
  // Clustering iterations; ranges[] records the node ids each iteration created.
  std::vector<std::pair<int, int>> ranges;
  int c = (int)n, next_node = (int)n;
  int* cur = clusters;
  int* nxt = clusters2;
  int iterations = 0;
  const char* radius_env = std::getenv("TT_PLOC_RADIUS");
  const int radius = radius_env ? std::max(1, std::min(256, std::atoi(radius_env))) : kDefaultRadius;
  while (c > kTailClusters) {
    if (++iterations > kMaxIterations) return fail("clustering did not converge");
    k_nearest<<<grid_for(c), kThreads, 0, st>>>(cur, c, node_box, radius, nn);
    k_merge_flags<<<grid_for(c), kThreads, 0, st>>>(nn, c, create, keep);
    size_t tb = std::max(sort_bytes, scan_bytes);
    cub::DeviceScan::ExclusiveSum(temp, tb, create, create_off, c, st);
    tb = std::max(sort_bytes, scan_bytes);
    cub::DeviceScan::ExclusiveSum(temp, tb, keep, keep_off, c, st);
    int* tail = hb;
    cudaMemcpyAsync(&tail[0], create_off + c - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&tail[1], create + c - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&tail[2], keep_off + c - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&tail[3], keep + c - 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    k_merge<<<grid_for(c), kThreads, 0, st>>>(cur, c, nn, create, create_off, keep, keep_off, next_node, node_box, left,
                                             right, nxt);
    if (!ok(cudaStreamSynchronize(st), "clustering")) return false;
    const int made = tail[0] + tail[1], kept = tail[2] + tail[3];
    if (made <= 0 || next_node + made > (int)total) return fail("clustering made no progress");
    ranges.push_back({next_node, made});
    next_node += made;
    c = kept;
    std::swap(cur, nxt);
  }
  // The rest in one block.
  int2* tail_ranges = sc.alloc<int2>(kMaxIterations);
  int* tail_info = sc.alloc<int>(4);
  if (!tail_ranges || !tail_info) return fail("out of device memory");
  if (!ok(cudaFuncSetAttribute(k_cluster_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem), "attribute"))
    return false;
  k_cluster_tail<<<1, kTailThreads, kTailSmem, st>>>(cur, c, radius, next_node, (int)total, kMaxIterations - iterations,
                                                     node_box, left, right, tail_ranges, tail_info);
  if (!ok(cudaMemcpyAsync(&hb[20], tail_info, 4 * sizeof(int), cudaMemcpyDeviceToHost, st), "copy") ||
      !ok(cudaStreamSynchronize(st), "clustering"))
    return false;
  const int tail_count = hb[20], root = hb[22];
  if (hb[23] != 0) return fail("clustering made no progress or did not converge");
  iterations += tail_count;
  const double t_clustered = verbose ? ms_since(t_start) : 0.0;
  // Bottom-up costs, top-down offsets and emission.
  int* size = sc.alloc<int>(total);
  float* cost = sc.alloc<float>(total);
  unsigned char* collapse = sc.alloc<unsigned char>(total);
  int* offset = sc.alloc<int>(total);
  unsigned char* state = sc.alloc<unsigned char>(total);
  int* depth = sc.alloc<int>(total);
  unsigned char* emit = sc.alloc<unsigned char>(total);
  int* inner = sc.alloc<int>(total);
  int* index = sc.alloc<int>(total);
  unsigned* max_depth = sc.alloc<unsigned>(1);
  if (!size || !cost || !collapse || !offset || !state || !depth || !emit || !inner || !index || !max_depth)
    return fail("out of device memory");
  cudaMemsetAsync(collapse, 1, n, st);  // primitive leaves
  cudaMemsetAsync(emit, 0, total, st);
  cudaMemsetAsync(max_depth, 0, sizeof(unsigned), st);
  for (const auto& r : ranges)
    k_costs<<<grid_for(r.second), kThreads, 0, st>>>(r.first, r.second, n, node_box, left, right, size, cost, collapse,
                                                      inner);
  k_costs_tail<<<1, kTailThreads, 0, st>>>(tail_ranges, tail_count, n, node_box, left, right, size, cost, collapse, inner);
  cudaMemsetAsync(offset + root, 0, sizeof(int), st);
  cudaMemsetAsync(index + root, 0, sizeof(int), st);
  cudaMemsetAsync(state + root, 0, 1, st);  // no state
  cudaMemsetAsync(depth + root, 0, sizeof(int), st);
  k_topdown_tail<<<1, kTailThreads, 0, st>>>(tail_ranges, tail_count, n, left, right, size, collapse, inner, offset,
                                             index, state, depth, emit, max_depth);
  for (auto it = ranges.rbegin(); it != ranges.rend(); ++it)
    k_topdown<<<grid_for(it->second), kThreads, 0, st>>>(it->first, it->second, n, left, right, size, collapse, inner,
                                                          offset, index, state, depth, emit, max_depth);
  hb[5] = 0;
  hb[6] = 0;
  hb[7] = 0;
  if (root >= (int)n) cudaMemcpyAsync(&hb[5], inner + root, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&hb[6], max_depth, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&hb[7], emit + root, 1, cudaMemcpyDeviceToHost, st);
  if (!ok(cudaStreamSynchronize(st), "emission")) return false;
  const int emitted = hb[5];
  const unsigned depth_host = (unsigned)hb[6];
  const unsigned char root_emit = (unsigned char)(hb[7] & 0xff);
  const int num_nodes = root_emit ? emitted : 1;
  // The 4-wide nodes are at most the emitted binary nodes (each 4-wide node replaces at
  // least one); the actual count comes from the collapse.
  const int cap4 = root_emit ? std::max(1, emitted) : 1;
  out->nodes4_bytes = root_emit && n >= kNode4BytesMin ? 1 : 0;
  const size_t f4 = out->nodes4_bytes ? 4 : 8;  // float4 per 4-wide node
  if (!ok(pool_malloc((void**)&out->nodes, 4 * sizeof(float4) * (size_t)num_nodes, st), "allocation") ||
      !ok(pool_malloc((void**)&out->tris, 3 * sizeof(float4) * (size_t)n, st), "allocation") ||
      !ok(pool_malloc((void**)&out->nodes4, f4 * sizeof(float4) * (size_t)cap4, st), "allocation"))
    return false;
  int num4 = 1, need4 = 0;
  // The root is a leaf when the whole tree collapses (or n == 1): its subtree starts at 0.
  if (!root_emit) {
    cudaMemsetAsync(offset + root, 0, sizeof(int), st);
    k_leaf_root<<<1, 1, 0, st>>>(node_box, root, (int)n, out->nodes);
    k_leaf_root4<<<1, 1, 0, st>>>(node_box, root, (int)n, out->nodes4);
  } else {
    k_write_nodes<<<grid_for(total - n), kThreads, 0, st>>>((int)n, (int)(total - n), n, node_box, left, right, size, offset,
                                                              emit, index, out->nodes);
    int4* front[2] = {sc.alloc<int4>(cap4), sc.alloc<int4>(cap4)};
    int* counts = sc.alloc<int>(3);  // [0] 4-wide nodes numbered, [1] next level's size, [2] stack entries needed
    if (!front[0] || !front[1] || !counts) return fail("out of device memory");
    const int first[7] = {root, 0, 0, 0, 1, 0, 0};  // the first front: (root, 0); counts: {1, 0, 0}
    std::copy(first, first + 7, hb + 8);
    cudaMemcpyAsync(front[0], &hb[8], sizeof(int4), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(counts, &hb[12], 3 * sizeof(int), cudaMemcpyHostToDevice, st);
    int nfront = 1;
    for (int level = 0; nfront > 0 && level < 64; ++level) {
      cudaMemsetAsync(counts + 1, 0, sizeof(int), st);
      k_collapse4<<<grid_for(nfront), kThreads, 0, st>>>(front[level & 1], nfront, n, node_box, left, right, size,
                                                          offset, emit, index, counts, front[(level + 1) & 1],
                                                          counts + 1, counts + 2, out->nodes4_bytes, out->nodes4);
      int* c2 = &hb[16];
      cudaMemcpyAsync(c2, counts, 3 * sizeof(int), cudaMemcpyDeviceToHost, st);
      if (!ok(cudaStreamSynchronize(st), "4-wide collapse")) return false;
      nfront = c2[1];
      num4 = c2[0];
      need4 = c2[2];
    }
    if (nfront > 0) return fail("4-wide collapse deeper than 64 levels");
    if (need4 > BVH_STACK) {
      // A path of the 4-wide tree could push more than the traversal's stack holds: the
      // binary tree, whose depth the caller checks, serves all rays.
      pool_free(out->nodes4, st);
      out->nodes4 = nullptr;
    } else {
      // Keep the nodes in a buffer of their exact size (the collapse wrote into an upper bound).
      float4* exact = nullptr;
      if (!ok(pool_malloc((void**)&exact, f4 * sizeof(float4) * (size_t)num4, st), "allocation")) return false;
      cudaMemcpyAsync(exact, out->nodes4, f4 * sizeof(float4) * (size_t)num4, cudaMemcpyDeviceToDevice, st);
      pool_free(out->nodes4, st);
      out->nodes4 = exact;
    }
  }
  k_write_slots<<<grid_for(n), kThreads, 0, st>>>(in, set, left, offset, n, out->tris);
  if (!ok(cudaStreamSynchronize(st), "emission") || !ok(cudaGetLastError(), "kernels")) return false;
  out->num_nodes = (uint32_t)num_nodes;
  out->num_nodes4 = (uint32_t)num4;
  out->max_depth = root_emit ? depth_host : 0;
  if (verbose) {
    float root_cost = 0.f;
    if (root >= (int)n) cudaMemcpy(&root_cost, cost + root, sizeof(float), cudaMemcpyDeviceToHost);
    std::fprintf(stderr,
                 "device BVH build: %u prims, %d iterations, %d nodes, depth %u, SAH cost %.2f; sorted %.1f ms, "
                 "clustered %.1f ms, done %.1f ms\n",
                 n, iterations, num_nodes, out->max_depth, root_cost, t_sorted, t_clustered, ms_since(t_start));
  }
  return true;
}

}  // namespace tt
