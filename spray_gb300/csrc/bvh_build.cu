// Per-domain BVH build on the GPU: binned SAH over the FP32 triangles,
// collapsed into the 4-wide BvhNode4 layout the traversal kernels read.
//
// SpRay rebuilds an Embree BVH (bvh4.triangle4v) whenever it loads a domain
// (TriMeshBuffer::load -> rtcCommit, src/render/trimesh_buffer.cc:104,222-224).
// Here every domain of a batch is built at once:
//   kPrep      per triangle: exact float box, centroid 0.5 (lo + hi), index
//   kRoots     one CTA per domain: the root's box
//   kSplit     binary binned-SAH splits of the tasks above kSmallTask
//              triangles, one CTA per task, a launch per level of the trees (so
//              that a scene of few domains uses every SM: 27 domains of 17144
//              triangles 0.59 ms, 2.36 with one CTA per domain): 16 bins per axis
//              (count, triangle box, centroid box) in warp-private
//              shared-memory bins, the SAH sweep, then a stable partition
//              (block scan) from one index buffer into the other; the
//              children's boxes and centroid boxes come from the bins.
//   kBuildSmall the tasks of at most kSmallTask triangles, one warp each on a
//              copy of its triangles in shared memory, warps of every SM
//              pulling from one counter: depth first, continuing with the
//              smaller child so a warp's stack stays within log2(kSmallTask)
//              + 1 entries (0.56 ms; 2.09 from global memory, with one lane's
//              sweep repeated by all)
//   kCollapse  4-wide nodes: each node takes its binary node's children and
//              opens the inner child with the largest box until it holds
//              four (the host builder's rule), one CTA per domain
//   kTris      leaf-ordered triangles (3 float4, v0.w = the face index)
// Boxes are exact min/max of the float vertices, so the traversal's
// conservative box test never misses a triangle, and the hit (t, triangle)
// key makes the traced image independent of the tree's shape.  Every stack
// and list is bounded; running out of room sets an error flag that the host
// turns into an error (no kernel waits on anything).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "bvh.h"
#include "tracer_internal.h"

namespace spray {
namespace gbvh {

namespace {

constexpr int kBins = 16;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kSplitThreads = 1024;    // of kSplit: its first levels have one task per domain
constexpr int kCollapseThreads = 1024;
constexpr int kBinCopies = 8;          // bin copies a split's warps share
constexpr int kSmallTask = 128;        // tasks of at most this many triangles go to a warp
constexpr int kWarpStack = 12;         // >= log2(kSmallTask) + 2
constexpr int kLevels = 32;            // split levels launched between two looks at what is left (even)
constexpr int kMaxBatchDomains = 4096; // domains built together (kBuildSmall's shared prefix)
constexpr float kTraversalCost = 1.0f;  // relative to one triangle test, as the host builder

enum : int { kErrStack = 1, kErrSmallList = 2, kErrNodes = 4, kErrQueue = 8, kErrLeaf = 16, kErrPartition = 32 };

struct Dom {
  const float* v;        // vertices (3 floats each), device
  const uint32_t* f;     // faces (3 indices each), device
  uint32_t nf;
  uint64_t tri_base;     // offset of the domain's triangles in the batch arrays
  uint64_t node_base;    // offset of its binary nodes (capacity 2 nf)
  uint64_t small_base;   // offset of its small-task list (capacity nf / 16 + 64)
  uint64_t q_base;       // offset of its collapse queue (capacity 2 nf)
  uint64_t out_base;     // offset of its 4-wide nodes (capacity nf)
};

struct BNode {  // binary node
  float lo[3];
  int32_t left;   // -1: leaf
  float hi[3];
  int32_t right;
  uint32_t first, count;
};

struct Task {
  uint32_t node, first, count, parity;  // parity: which index buffer holds the range
  float clo[3], chi[3];                 // centroid bounds
};

// A task above kSmallTask triangles and its domain.
struct BigTask {
  Task t;
  int32_t dom;
};

struct Batch {
  const Dom* doms;
  float4* tlo;           // triangle box lo (w unused)
  float4* thi;
  float4* cen;           // centroid
  uint32_t* idx[2];      // double-buffered permutation, domain-relative triangle numbers
  uint32_t* order;       // final leaf order
  BNode* nodes;
  Task* small;
  BigTask* big[2];       // the large tasks of the level being split and of the next
  uint32_t* nbig;        // [kLevels + 1] tasks per level
  uint32_t big_cap;
  uint32_t* nnodes;      // binary nodes per domain
  uint32_t* nsmall;      // small tasks per domain
  BvhNode4* out;         // 4-wide nodes
  uint32_t* nout;        // 4-wide nodes per domain
  int32_t* depth;        // 4-wide depth per domain (root = 1)
  int2* queue;           // collapse queue: (binary node, 4-wide node)
  int* error;
};

__device__ __forceinline__ int ordf(float f) {
  const int b = __float_as_int(f);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float unordf(int b) { return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff); }

__device__ __forceinline__ float halfArea(const float lo[3], const float hi[3]) {
  const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
  if (dx < 0.f || dy < 0.f || dz < 0.f) return 0.f;
  return dx * dy + dy * dz + dz * dx;
}

__device__ __forceinline__ int binOf(float c, float lo, float scale) {
  int b = (int)((c - lo) * scale);
  return min(max(b, 0), kBins - 1);
}

// Bin statistics of one axis: count, triangle box (lo, hi), centroid box.
// Min/max as order-preserving ints so shared-memory atomics apply.
struct Bins {
  int cnt[3][kBins];
  int blo[3][kBins][3], bhi[3][kBins][3];
  int clo[3][kBins][3], chi[3][kBins][3];
};

__device__ void clearBins(Bins* b, int lane, int width) {
  int* p = reinterpret_cast<int*>(b);
  constexpr int n = sizeof(Bins) / 4;
  for (int i = lane; i < n; i += width) {
    // counts 0, minima +max, maxima -max (as ordered ints)
    const int off = i;
    int v = 0;
    if (off >= 3 * kBins) {
      const int k = (off - 3 * kBins) / (3 * kBins * 3);  // 0 blo, 1 bhi, 2 clo, 3 chi
      v = (k == 0 || k == 2) ? 0x7fffffff : (int)0x80000000;
    }
    p[i] = v;
  }
}

__device__ __forceinline__ void addToBins(Bins* b, const float l3[3], const float h3[3], const float cc[3],
                                          const float clo[3], const float scale[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (!(scale[a] > 0.f)) continue;
    const int k = binOf(cc[a], clo[a], scale[a]);
    atomicAdd(&b->cnt[a][k], 1);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      atomicMin(&b->blo[a][k][q], ordf(l3[q]));
      atomicMax(&b->bhi[a][k][q], ordf(h3[q]));
      atomicMin(&b->clo[a][k][q], ordf(cc[q]));
      atomicMax(&b->chi[a][k][q], ordf(cc[q]));
    }
  }
}

// The SAH sweeps over the bins of the three axes by one warp: the axis and
// split (left = bins < split) of the least cost, -1 when no axis with a positive
// scale can be split; of equal costs the lower axis, then the larger split.
// Lanes 0..15 scan the bins' boxes from the left, lanes 16..31 from the right,
// the axes side by side (one lane after the other over 3 x 30 bins took most of a
// small task's time).
__device__ __forceinline__ void sweepAxes(const Bins* m, const float scale[3], int lane, float* best_cost, int* axis,
                                          int* split) {
  const int j = lane & 15, b = (lane & 16) ? kBins - 1 - j : j;
  int n[3], lo[3][3], hi[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    n[a] = m->cnt[a][b];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      lo[a][q] = m->blo[a][b][q];  // an empty bin holds the neutral elements
      hi[a][q] = m->bhi[a][b][q];
    }
  }
#pragma unroll
  for (int o = 1; o < kBins; o <<= 1) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int pn = __shfl_up_sync(0xffffffffu, n[a], o, 16);
      if (j >= o) n[a] += pn;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int pl = __shfl_up_sync(0xffffffffu, lo[a][q], o, 16);
        const int ph = __shfl_up_sync(0xffffffffu, hi[a][q], o, 16);
        if (j >= o) {
          lo[a][q] = min(lo[a][q], pl);
          hi[a][q] = max(hi[a][q], ph);
        }
      }
    }
  }
  float cost = INFINITY;
  int best = -1;  // 16 * (2 - axis) + split: larger is preferred among equal costs
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float flo[3] = {unordf(lo[a][0]), unordf(lo[a][1]), unordf(lo[a][2])};
    const float fhi[3] = {unordf(hi[a][0]), unordf(hi[a][1]), unordf(hi[a][2])};
    const float area = n[a] ? halfArea(flo, fhi) : 0.f;
    // split s = lane (1..15): bins [0, s) end at lane s - 1, bins [s, 16) at lane 31 - s
    const float la = __shfl_sync(0xffffffffu, area, (lane - 1) & 31), ra = __shfl_sync(0xffffffffu, area, 31 - lane);
    const int lc = __shfl_sync(0xffffffffu, n[a], (lane - 1) & 31), rc = __shfl_sync(0xffffffffu, n[a], 31 - lane);
    const float c = la * (float)lc + ra * (float)rc;
    if (scale[a] > 0.f && lane >= 1 && lane < kBins && lc > 0 && rc > 0 && c < cost) {
      cost = c;
      best = kBins * (2 - a) + lane;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const float oc = __shfl_xor_sync(0xffffffffu, cost, o);
    const int ob = __shfl_xor_sync(0xffffffffu, best, o);
    if (oc < cost || (oc == cost && ob > best)) {
      cost = oc;
      best = ob;
    }
  }
  *best_cost = cost;
  *axis = best < 0 ? -1 : 2 - best / kBins;
  *split = best < 0 ? -1 : best % kBins;
}

// Boxes of the two children of a split: triangle box and centroid box, lo and
// hi, of bins [0, split) and [split, kBins) of axis a, by one warp; every lane
// gets them.
__device__ __forceinline__ void splitBoxes(const Bins* m, int a, int split, int lane, float blo[2][3], float bhi[2][3],
                                           float clo[2][3], float chi[2][3]) {
  // lane = 12 * child + 3 * kind + axis component
  const int child = lane / 12, kind = lane % 12 / 3, q = lane % 3;
  const int b0 = child == 0 ? 0 : split, b1 = child == 0 ? split : kBins;
  const bool is_min = (kind & 1) == 0;
  int v = is_min ? 0x7fffffff : (int)0x80000000;
  if (lane < 24) {
    const int(*src)[3] = kind == 0 ? m->blo[a] : kind == 1 ? m->bhi[a] : kind == 2 ? m->clo[a] : m->chi[a];
#pragma unroll
    for (int b = 0; b < kBins; ++b) {
      const int x = src[b][q];
      if (b >= b0 && b < b1) v = is_min ? min(v, x) : max(v, x);
    }
  }
  const float f = unordf(v);
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      blo[k][c] = __shfl_sync(0xffffffffu, f, 12 * k + c);
      bhi[k][c] = __shfl_sync(0xffffffffu, f, 12 * k + 3 + c);
      clo[k][c] = __shfl_sync(0xffffffffu, f, 12 * k + 6 + c);
      chi[k][c] = __shfl_sync(0xffffffffu, f, 12 * k + 9 + c);
    }
}

__global__ void kPrep(Batch B, int ndoms) {
  const Dom d = B.doms[blockIdx.y];
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < d.nf; t += gridDim.x * blockDim.x) {
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int c = 0; c < 3; ++c) {
      const float* p = d.v + 3 * (size_t)d.f[3 * (size_t)t + c];
      for (int q = 0; q < 3; ++q) {
        lo[q] = fminf(lo[q], p[q]);
        hi[q] = fmaxf(hi[q], p[q]);
      }
    }
    const uint64_t g = d.tri_base + t;
    B.tlo[g] = make_float4(lo[0], lo[1], lo[2], 0.f);
    B.thi[g] = make_float4(hi[0], hi[1], hi[2], 0.f);
    B.cen[g] = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]), 0.f);
    B.idx[0][g] = t;
  }
  (void)ndoms;
}

// Shared memory of kSplit.
struct Shared {
  Bins bins[kBinCopies];
  int scan[kSplitThreads / 32];
  int axis, split;
  int running_left, running_right;
};

// A warp's shared memory in kBuildSmall: the triangles of its task.
struct SmallTask {
  uint32_t node, first, count, parity;  // first relative to the task
  float blo[3], bhi[3], clo[3], chi[3];
};
struct SmallShared {
  Bins bins;
  float lo[3][kSmallTask], hi[3][kSmallTask], c[3][kSmallTask];
  uint32_t tri[kSmallTask];        // domain-relative triangle numbers
  uint8_t idx[2][kSmallTask];      // double-buffered permutation
  SmallTask stack[kWarpStack];
};

// Writes node `id` and its range into the final order when it is a leaf.
__device__ void writeNode(const Batch& B, const Dom& d, uint32_t id, const float lo[3], const float hi[3],
                          int left, int right, uint32_t first, uint32_t count) {
  BNode n;
  for (int q = 0; q < 3; ++q) {
    n.lo[q] = lo[q];
    n.hi[q] = hi[q];
  }
  n.left = left;
  n.right = right;
  n.first = first;
  n.count = count;
  B.nodes[d.node_base + id] = n;
}

// Stable partition of a task's range into the other buffer, CTA-wide.
// Returns (in shared) the number of left elements.
__device__ void partitionCta(const Batch& B, const Dom& d, Shared& S, const Task& t, int axis, int split,
                             bool by_half) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t* src = B.idx[t.parity] + d.tri_base;
  uint32_t* dst = B.idx[t.parity ^ 1] + d.tri_base;
  const float scale = by_half ? 0.f : kBins / (t.chi[axis] - t.clo[axis]);
  // left count: from the bins (or half)
  uint32_t nleft;
  if (by_half) {
    nleft = t.count / 2;
  } else {
    nleft = 0;
    for (int b = 0; b < split; ++b) nleft += (uint32_t)S.bins[0].cnt[axis][b];
  }
  if (tid == 0) {
    S.running_left = 0;
    S.running_right = 0;
  }
  __syncthreads();
  for (uint32_t base = 0; base < t.count; base += kSplitThreads) {
    const uint32_t i = base + tid;
    bool isl = false;
    uint32_t tri = 0;
    if (i < t.count) {
      tri = src[t.first + i];
      if (by_half) {
        isl = i < nleft;
      } else {
        const float4 c = B.cen[d.tri_base + tri];
        const float cc = axis == 0 ? c.x : axis == 1 ? c.y : c.z;
        isl = binOf(cc, t.clo[axis], scale) < split;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, isl);
    if (lane == 0) S.scan[warp] = __popc(m);
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < kSplitThreads / 32; ++w) {
      if (w < warp) before += S.scan[w];
      total += S.scan[w];
    }
    const int lrank = before + __popc(m & ((1u << lane) - 1u));
    if (i < t.count) {
      // positions stay inside the task's range even if the counts disagreed
      const uint32_t pos = isl ? (uint32_t)(S.running_left + lrank)
                               : nleft + (uint32_t)(S.running_right + (int)(i - base) - lrank);
      if (pos < t.count) dst[t.first + pos] = tri;
    }
    __syncthreads();
    if (tid == 0) {
      S.running_left += total;
      S.running_right += (int)min((uint32_t)kSplitThreads, t.count - base) - total;
    }
    __syncthreads();
  }
  if (tid == 0 && (uint32_t)S.running_left != nleft) atomicOr(B.error, kErrPartition);
}

// Box and centroid box of the range [first, first + count) of buffer `parity`,
// reduced by the CTA.
__device__ void rangeBounds(const Batch& B, const Dom& d, uint32_t parity, uint32_t first, uint32_t count,
                            Bins* scratch, float blo[3], float bhi[3], float clo[3], float chi[3]) {
  // reuse bin 0 of axis 0 of the scratch bins as the accumulator
  if (threadIdx.x < 3) {
    scratch->blo[0][0][threadIdx.x] = 0x7fffffff;
    scratch->bhi[0][0][threadIdx.x] = (int)0x80000000;
    scratch->clo[0][0][threadIdx.x] = 0x7fffffff;
    scratch->chi[0][0][threadIdx.x] = (int)0x80000000;
  }
  __syncthreads();
  float l[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, h[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  float cl[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, ch[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
    const uint64_t g = d.tri_base + B.idx[parity][d.tri_base + first + i];
    const float4 a = B.tlo[g], b = B.thi[g], c = B.cen[g];
    l[0] = fminf(l[0], a.x), l[1] = fminf(l[1], a.y), l[2] = fminf(l[2], a.z);
    h[0] = fmaxf(h[0], b.x), h[1] = fmaxf(h[1], b.y), h[2] = fmaxf(h[2], b.z);
    cl[0] = fminf(cl[0], c.x), cl[1] = fminf(cl[1], c.y), cl[2] = fminf(cl[2], c.z);
    ch[0] = fmaxf(ch[0], c.x), ch[1] = fmaxf(ch[1], c.y), ch[2] = fmaxf(ch[2], c.z);
  }
  for (int q = 0; q < 3; ++q) {
    // one atomic per warp and component
    const int lq = __reduce_min_sync(0xffffffffu, ordf(l[q])), hq = __reduce_max_sync(0xffffffffu, ordf(h[q]));
    const int clq = __reduce_min_sync(0xffffffffu, ordf(cl[q])), chq = __reduce_max_sync(0xffffffffu, ordf(ch[q]));
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&scratch->blo[0][0][q], lq);
      atomicMax(&scratch->bhi[0][0][q], hq);
      atomicMin(&scratch->clo[0][0][q], clq);
      atomicMax(&scratch->chi[0][0][q], chq);
    }
  }
  __syncthreads();
  for (int q = 0; q < 3; ++q) {
    blo[q] = unordf(scratch->blo[0][0][q]);
    bhi[q] = unordf(scratch->bhi[0][0][q]);
    clo[q] = unordf(scratch->clo[0][0][q]);
    chi[q] = unordf(scratch->chi[0][0][q]);
  }
  __syncthreads();
}

// The same of the range [first, first + count) of a small task's buffer, by its warp.
__device__ void smallBounds(const SmallShared& S, uint32_t parity, uint32_t first, uint32_t count, int lane,
                            float blo[3], float bhi[3], float clo[3], float chi[3]) {
  int v[4][3];
  for (int q = 0; q < 3; ++q) {
    v[0][q] = v[2][q] = ordf(FLT_MAX);
    v[1][q] = v[3][q] = ordf(-FLT_MAX);
  }
  for (uint32_t i = lane; i < count; i += 32) {
    const int k = S.idx[parity][first + i];
    for (int q = 0; q < 3; ++q) {
      v[0][q] = min(v[0][q], ordf(S.lo[q][k]));
      v[1][q] = max(v[1][q], ordf(S.hi[q][k]));
      v[2][q] = min(v[2][q], ordf(S.c[q][k]));
      v[3][q] = max(v[3][q], ordf(S.c[q][k]));
    }
  }
  for (int q = 0; q < 3; ++q) {
    blo[q] = unordf(__reduce_min_sync(0xffffffffu, v[0][q]));
    bhi[q] = unordf(__reduce_max_sync(0xffffffffu, v[1][q]));
    clo[q] = unordf(__reduce_min_sync(0xffffffffu, v[2][q]));
    chi[q] = unordf(__reduce_max_sync(0xffffffffu, v[3][q]));
  }
}

// Builds the subtree of a small task with one warp, depth first, on the copy of
// its triangles in shared memory.  Binary node ids: a subtree of n triangles has
// at most 2 n - 2 nodes below its root, reserved at once from the domain's
// counter (2 nf ids in all).
__device__ void buildSmall(const Batch& B, const Dom& d, SmallShared& S, const Task& root, int lane,
                           uint32_t* node_counter) {
  for (uint32_t i = lane; i < root.count; i += 32) {
    const uint32_t tri = B.idx[root.parity][d.tri_base + root.first + i];
    const uint64_t g = d.tri_base + tri;
    const float4 lo = B.tlo[g], hi = B.thi[g], c = B.cen[g];
    S.lo[0][i] = lo.x, S.lo[1][i] = lo.y, S.lo[2][i] = lo.z;
    S.hi[0][i] = hi.x, S.hi[1][i] = hi.y, S.hi[2][i] = hi.z;
    S.c[0][i] = c.x, S.c[1][i] = c.y, S.c[2][i] = c.z;
    S.tri[i] = tri;
    S.idx[0][i] = (uint8_t)i;
  }
  uint32_t ids = 0;
  if (lane == 0) ids = atomicAdd(node_counter, 2 * root.count - 2);
  ids = __shfl_sync(0xffffffffu, ids, 0);
  if (ids + 2 * root.count - 2 > 2 * d.nf) {
    if (lane == 0) atomicOr(B.error, kErrNodes);
    return;
  }
  SmallTask t;
  t.node = root.node;
  t.first = 0;
  t.count = root.count;
  t.parity = 0;
  const BNode& rn = B.nodes[d.node_base + root.node];
  for (int q = 0; q < 3; ++q) {
    t.blo[q] = rn.lo[q];
    t.bhi[q] = rn.hi[q];
    t.clo[q] = root.clo[q];
    t.chi[q] = root.chi[q];
  }
  __syncwarp();
  int sp = 0;
  while (true) {
    // t's node is already written (box); decide leaf or split
    bool leaf = t.count <= 2;
    int axis = -1, split = -1;
    float best = INFINITY;
    if (!leaf) {
      clearBins(&S.bins, lane, 32);
      __syncwarp();
      float scale[3];
      for (int a = 0; a < 3; ++a) {
        const float ext = t.chi[a] - t.clo[a];
        scale[a] = ext > 0.f ? kBins / ext : 0.f;
      }
      const uint32_t seg = (t.count + 31) / 32;
      for (uint32_t i = lane * seg; i < min((lane + 1) * seg, t.count); ++i) {
        const int k = S.idx[t.parity][t.first + i];
        const float l3[3] = {S.lo[0][k], S.lo[1][k], S.lo[2][k]}, h3[3] = {S.hi[0][k], S.hi[1][k], S.hi[2][k]};
        const float c3[3] = {S.c[0][k], S.c[1][k], S.c[2][k]};
        addToBins(&S.bins, l3, h3, c3, t.clo, scale);
      }
      __syncwarp();
      sweepAxes(&S.bins, scale, lane, &best, &axis, &split);
      const float area = halfArea(t.blo, t.bhi);
      const float leaf_cost = area * (float)t.count;
      const float split_cost = kTraversalCost * area + best;
      if (axis < 0) leaf = t.count <= (uint32_t)kMaxLeafTris;
      else leaf = t.count <= (uint32_t)kMaxLeafTris && leaf_cost <= split_cost;
    }
    if (leaf) {
      for (uint32_t i = lane; i < t.count; i += 32)
        B.order[d.tri_base + root.first + t.first + i] = S.tri[S.idx[t.parity][t.first + i]];
    } else {
      // stable warp partition into the other buffer
      const uint8_t* src = S.idx[t.parity] + t.first;
      uint8_t* dst = S.idx[t.parity ^ 1] + t.first;
      const bool by_half = axis < 0;
      uint32_t nleft = 0;
      if (by_half) {
        nleft = t.count / 2;
      } else {
        const int n = lane < split ? S.bins.cnt[axis][lane & (kBins - 1)] : 0;  // split < kBins
        nleft = (uint32_t)__reduce_add_sync(0xffffffffu, n);
      }
      const float scale = by_half ? 0.f : kBins / (t.chi[axis] - t.clo[axis]);
      uint32_t rl = 0, rr = 0;
      for (uint32_t base = 0; base < t.count; base += 32) {
        const uint32_t i = base + lane;
        bool isl = false;
        uint8_t k = 0;
        if (i < t.count) {
          k = src[i];
          isl = by_half ? i < nleft : binOf(S.c[axis][k], t.clo[axis], scale) < split;
        }
        const unsigned m = __ballot_sync(0xffffffffu, isl);
        const uint32_t lr = __popc(m & ((1u << lane) - 1u));
        if (i < t.count) {
          const uint32_t pos = isl ? rl + lr : nleft + rr + (lane - lr);
          if (pos < t.count) dst[pos] = k;
        }
        rl += __popc(m);
        rr += min(32u, t.count - base) - __popc(m);
      }
      __syncwarp();
      if (rl != nleft) {
        if (lane == 0) atomicOr(B.error, kErrPartition);
        return;
      }
      // children's boxes: from the bins, or reduced over the halves
      float blo[2][3], bhi[2][3], clo[2][3], chi[2][3];
      if (!by_half) {
        splitBoxes(&S.bins, axis, split, lane, blo, bhi, clo, chi);
      } else {
        smallBounds(S, t.parity ^ 1, t.first, nleft, lane, blo[0], bhi[0], clo[0], chi[0]);
        smallBounds(S, t.parity ^ 1, t.first + nleft, t.count - nleft, lane, blo[1], bhi[1], clo[1], chi[1]);
      }
      if (lane == 0) {
        BNode* self = &B.nodes[d.node_base + t.node];
        self->left = (int)ids;
        self->right = (int)ids + 1;
      }
      // continue with the smaller child, push the larger
      const int small = nleft <= t.count - nleft ? 0 : 1;
      SmallTask kid[2];
      for (int k = 0; k < 2; ++k) {
        kid[k].node = ids + k;
        kid[k].first = k == 0 ? t.first : t.first + nleft;
        kid[k].count = k == 0 ? nleft : t.count - nleft;
        kid[k].parity = t.parity ^ 1;
        for (int q = 0; q < 3; ++q) {
          kid[k].blo[q] = blo[k][q];
          kid[k].bhi[q] = bhi[k][q];
          kid[k].clo[q] = clo[k][q];
          kid[k].chi[q] = chi[k][q];
        }
        if (lane == 0) writeNode(B, d, kid[k].node, blo[k], bhi[k], -1, -1, root.first + kid[k].first, kid[k].count);
      }
      ids += 2;
      if (sp >= kWarpStack) {
        if (lane == 0) atomicOr(B.error, kErrStack);
        return;
      }
      if (lane == 0) S.stack[sp] = small == 0 ? kid[1] : kid[0];
      ++sp;
      __syncwarp();
      t = small == 0 ? kid[0] : kid[1];
      continue;
    }
    if (sp == 0) break;
    --sp;
    __syncwarp();
    t = S.stack[sp];
    __syncwarp();
  }
  __syncwarp();  // the next task overwrites the shared triangles
}

// Hands a task to the next level's splits, or to the small tasks (one thread).
__device__ void pushTask(const Batch& B, const Dom& d, int dom, const Task& t, int level) {
  if (t.count > (uint32_t)kSmallTask) {
    const uint32_t k = atomicAdd(&B.nbig[level], 1u);
    if (k < B.big_cap) {
      B.big[level & 1][k].t = t;
      B.big[level & 1][k].dom = dom;
    } else {
      atomicOr(B.error, kErrStack);
    }
  } else {
    const uint32_t k = atomicAdd(&B.nsmall[dom], 1u);
    if (k < d.nf / 16 + 64) B.small[d.small_base + k] = t;
    else atomicOr(B.error, kErrSmallList);
  }
}

__global__ void __launch_bounds__(kSplitThreads) kRoots(Batch B) {
  __shared__ Bins scratch;
  const Dom d = B.doms[blockIdx.x];
  const int tid = threadIdx.x;
  float blo[3], bhi[3], clo[3], chi[3];
  rangeBounds(B, d, 0, 0, d.nf, &scratch, blo, bhi, clo, chi);
  if (tid == 0) {
    writeNode(B, d, 0, blo, bhi, -1, -1, 0, d.nf);
    B.nnodes[blockIdx.x] = 1u;
    Task r;
    r.node = 0;
    r.first = 0;
    r.count = d.nf;
    r.parity = 0;
    for (int q = 0; q < 3; ++q) {
      r.clo[q] = clo[q];
      r.chi[q] = chi[q];
    }
    pushTask(B, d, blockIdx.x, r, 0);
  }
}

// The large tasks of one level, one CTA each at a time.
__global__ void __launch_bounds__(kSplitThreads) kSplit(Batch B, int level) {
  extern __shared__ __align__(16) unsigned char smem[];
  Shared& S = *reinterpret_cast<Shared*>(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t ntasks = min(B.nbig[level], B.big_cap);
  for (uint32_t k = blockIdx.x; k < ntasks; k += gridDim.x) {
    const Task t = B.big[level & 1][k].t;
    const int dom = B.big[level & 1][k].dom;
    const Dom d = B.doms[dom];
    for (int w = 0; w < kBinCopies; ++w) clearBins(&S.bins[w], tid, kSplitThreads);
    __syncthreads();
    float scale[3];
    for (int a = 0; a < 3; ++a) {
      const float ext = t.chi[a] - t.clo[a];
      scale[a] = ext > 0.f ? kBins / ext : 0.f;
    }
    // a warp's lanes take triangles a 32nd of the task apart: neighbours in the
    // list are neighbours in space and would meet in the same bins' atomics
    const uint32_t seg = (t.count + 31) / 32;
    for (uint32_t j = warp; j < seg; j += kSplitThreads / 32) {
      const uint32_t i = lane * seg + j;
      if (i >= t.count) continue;
      const uint64_t g = d.tri_base + B.idx[t.parity][d.tri_base + t.first + i];
      const float4 lo = B.tlo[g], hi = B.thi[g], c = B.cen[g];
      const float l3[3] = {lo.x, lo.y, lo.z}, h3[3] = {hi.x, hi.y, hi.z}, c3[3] = {c.x, c.y, c.z};
      addToBins(&S.bins[warp % kBinCopies], l3, h3, c3, t.clo, scale);
    }
    __syncthreads();
    // merge the warps' bins into bins[0]
    {
      constexpr int n = sizeof(Bins) / 4;
      int* m0 = reinterpret_cast<int*>(&S.bins[0]);
      for (int i = tid; i < n; i += kSplitThreads) {
        int v = m0[i];
        const bool is_cnt = i < 3 * kBins;
        const int kind = is_cnt ? -1 : (i - 3 * kBins) / (3 * kBins * 3);
        for (int w = 1; w < kBinCopies; ++w) {
          const int x = reinterpret_cast<const int*>(&S.bins[w])[i];
          if (is_cnt) v += x;
          else if (kind == 0 || kind == 2) v = min(v, x);
          else v = max(v, x);
        }
        m0[i] = v;
      }
    }
    __syncthreads();
    if (warp == 0) {
      float cost;
      int axis, split;
      sweepAxes(&S.bins[0], scale, lane, &cost, &axis, &split);
      if (lane == 0) {
        S.axis = axis;
        S.split = split;
      }
    }
    __syncthreads();
    const int axis = S.axis, split = S.split;
    partitionCta(B, d, S, t, axis, split, axis < 0);
    uint32_t nleft = 0;
    if (axis < 0) nleft = t.count / 2;
    else
      for (int b = 0; b < split; ++b) nleft += (uint32_t)S.bins[0].cnt[axis][b];
    float kb[2][3], kh[2][3], kc[2][3], kx[2][3];
    __syncthreads();
    if (axis < 0) {
      rangeBounds(B, d, t.parity ^ 1, t.first, nleft, &S.bins[1], kb[0], kh[0], kc[0], kx[0]);
      rangeBounds(B, d, t.parity ^ 1, t.first + nleft, t.count - nleft, &S.bins[1], kb[1], kh[1], kc[1], kx[1]);
    } else if (warp == 0) {
      splitBoxes(&S.bins[0], axis, split, lane, kb, kh, kc, kx);
    }
    if (tid == 0) {
      const uint32_t ids = atomicAdd(&B.nnodes[dom], 2u);
      if (ids + 2 > 2 * d.nf) {
        atomicOr(B.error, kErrNodes);
      } else {
        BNode* self = &B.nodes[d.node_base + t.node];
        self->left = (int)ids;
        self->right = (int)ids + 1;
        for (int q = 0; q < 2; ++q) {
          Task kid;
          kid.node = ids + q;
          kid.first = q == 0 ? t.first : t.first + nleft;
          kid.count = q == 0 ? nleft : t.count - nleft;
          kid.parity = t.parity ^ 1;
          for (int c = 0; c < 3; ++c) {
            kid.clo[c] = kc[q][c];
            kid.chi[c] = kx[q][c];
          }
          writeNode(B, d, kid.node, kb[q], kh[q], -1, -1, kid.first, kid.count);
          pushTask(B, d, dom, kid, level + 1);
        }
      }
    }
    __syncthreads();
  }
}

// The counters of a group of levels: the tasks left after the last one are the
// next group's first.
__global__ void kNextLevels(Batch B) {
  const uint32_t left = B.nbig[kLevels];
  __syncthreads();
  if (threadIdx.x <= kLevels) B.nbig[threadIdx.x] = threadIdx.x == 0 ? left : 0u;
}

// The small tasks of every domain of the batch, one warp per task, warps of
// all CTAs pulling from one counter (`next`): a domain's subtrees are built
// in parallel on every SM instead of by its one CTA.
__global__ void __launch_bounds__(kThreads) kBuildSmall(Batch B, int nb, uint32_t* next) {
  extern __shared__ __align__(16) unsigned char smem[];
  SmallShared* S = reinterpret_cast<SmallShared*>(smem);
  uint32_t* prefix = reinterpret_cast<uint32_t*>(smem + kWarps * sizeof(SmallShared));  // [nb + 1]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    uint32_t run = 0;
    for (int d = 0; d < nb; ++d) {
      prefix[d] = run;
      run += B.nsmall[d];
    }
    prefix[nb] = run;
  }
  __syncthreads();
  const uint32_t total = prefix[nb];
  while (true) {
    uint32_t k = 0;
    int stop = 0;
    if (lane == 0) {
      k = atomicAdd(next, 1u);
      stop = *((volatile int*)B.error);
    }
    k = __shfl_sync(0xffffffffu, k, 0);
    stop = __shfl_sync(0xffffffffu, stop, 0);
    if (k >= total || stop) break;
    // the domain of task k: last d with prefix[d] <= k
    int lo = 0, hi = nb - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (prefix[mid] <= k) lo = mid;
      else hi = mid - 1;
    }
    const Dom d = B.doms[lo];
    const Task t = B.small[d.small_base + (k - prefix[lo])];
    buildSmall(B, d, S[warp], t, lane, &B.nnodes[lo]);
  }
}

// 4-wide collapse, one CTA per domain: a queue of (binary node, 4-wide node)
// pairs; each item gathers up to four children by opening the inner child with
// the largest box, allocates 4-wide nodes for the inner ones (numbered in queue
// order) and queues them.  1024 items at a time: 27 domains of 17144 triangles
// 0.13 ms, 0.92 with 32.
__global__ void __launch_bounds__(kCollapseThreads) kCollapse(Batch B) {
  const Dom d = B.doms[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ int wsum[(kCollapseThreads / 32)];
  __shared__ int maxdepth, bad;
  int2* q = B.queue + d.q_base;
  const BNode* bn = B.nodes + d.node_base;
  BvhNode4* out = B.out + d.out_base;
  const uint32_t qcap = 2 * d.nf + 4, ocap = d.nf + 4;
  if (tid == 0) {
    q[0] = make_int2(0, 0);
    out[0].pad[0] = 1;  // the root's depth
    maxdepth = 1;
    bad = 0;
  }
  __syncthreads();
  int head = 0, tail = 1, nout = 1;
  // items carry the 4-wide node id in .y; a node's depth = its parent's + 1,
  // recorded in out[].pad[0]
  while (head < tail) {
    const int take = min(kCollapseThreads, tail - head);
    int kids[4];
    int nk = 0, ninner = 0;
    int2 it = make_int2(0, 0);
    if (tid < take) {
      it = q[head + tid];
      const BNode& root = bn[it.x];
      if (root.left < 0) {
        kids[nk++] = it.x;  // a single leaf root: one child, the leaf itself
      } else {
        kids[nk++] = root.left;
        kids[nk++] = root.right;
        while (nk < 4) {
          int best = -1;
          float best_area = -1.f;
          for (int i = 0; i < nk; ++i) {
            const BNode& k = bn[kids[i]];
            if (k.left >= 0) {
              const float a = halfArea(k.lo, k.hi);
              if (a > best_area) {
                best_area = a;
                best = i;
              }
            }
          }
          if (best < 0) break;
          const int opened = kids[best];
          kids[best] = bn[opened].left;
          kids[nk++] = bn[opened].right;
        }
      }
      for (int c = 0; c < nk; ++c) ninner += bn[kids[c]].left >= 0 ? 1 : 0;
    }
    // the inner children's places, in queue order
    int pre = ninner;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += y;
    }
    if (lane == 31) wsum[warp] = pre;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < (kCollapseThreads / 32); ++w) {
      if (w < warp) before += wsum[w];
      total += wsum[w];
    }
    pre += before - ninner;
    if (tid < take) {
      const int base = nout + pre, qb = tail + pre;
      const int my_depth = out[it.y].pad[0];  // set by the parent (root: 1)
      BvhNode4 node;
      for (int c = 0; c < 4; ++c) {
        node.lox[c] = node.loy[c] = node.loz[c] = INFINITY;
        node.hix[c] = node.hiy[c] = node.hiz[c] = -INFINITY;
        node.child[c] = kEmptyChild;
        node.pad[c] = 0;
      }
      node.pad[0] = my_depth;
      int used = 0;
      bool ok = (uint32_t)(base + ninner) <= ocap && (uint32_t)(qb + ninner) <= qcap;
      for (int c = 0; c < nk && ok; ++c) {
        const BNode& k = bn[kids[c]];
        node.lox[c] = k.lo[0];
        node.loy[c] = k.lo[1];
        node.loz[c] = k.lo[2];
        node.hix[c] = k.hi[0];
        node.hiy[c] = k.hi[1];
        node.hiz[c] = k.hi[2];
        if (k.left < 0) {
          if (k.count > (uint32_t)kMaxLeafTris || k.first >= (1u << 27) || k.count == 0) {
            ok = false;
            break;
          }
          node.child[c] = ~(int32_t)((k.first << 3) | (k.count - 1));
        } else {
          const int id = base + used;
          node.child[c] = id;
          out[id].pad[0] = my_depth + 1;  // read when the child's item is processed
          q[qb + used] = make_int2(kids[c], id);
          ++used;
        }
      }
      if (!ok) {
        bad = 1;
      } else {
        atomicMax(&maxdepth, my_depth);
        // keep the depth in pad[0] until the child items have read theirs;
        // cleared by kFinish
        out[it.y] = node;
      }
    }
    __syncthreads();
    head += take;
    tail += total;
    nout += total;
    if (bad) break;
  }
  if (tid == 0) {
    if (bad) atomicOr(B.error, kErrQueue);
    B.nout[blockIdx.x] = (uint32_t)nout;
    B.depth[blockIdx.x] = maxdepth;
  }
}

// Clears the depth bookkeeping kept in pad[0] of every 4-wide node.
__global__ void kFinish(Batch B) {
  const Dom d = B.doms[blockIdx.y];
  const uint32_t n = B.nout[blockIdx.y];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    B.out[d.out_base + i].pad[0] = 0;
}

// The domains' nodes without the gaps between them (depth bookkeeping cleared).
__global__ void kGatherNodes(Batch B, const uint64_t* __restrict__ to, BvhNode4* __restrict__ nodes) {
  const Dom d = B.doms[blockIdx.y];
  const uint32_t n = B.nout[blockIdx.y];
  const float4* src = reinterpret_cast<const float4*>(B.out + d.out_base);
  float4* dst = reinterpret_cast<float4*>(nodes + to[blockIdx.y]);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 8 * n; i += gridDim.x * blockDim.x) dst[i] = src[i];
}

// Leaf-ordered triangles: 3 float4 per triangle, v0.w = the face index bits.
__global__ void kTris(Batch B, float4* tris) {
  const Dom d = B.doms[blockIdx.y];
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < d.nf; k += gridDim.x * blockDim.x) {
    const uint32_t prim = B.order[d.tri_base + k];
    const uint32_t* fi = d.f + 3 * (size_t)prim;
    for (int c = 0; c < 3; ++c) {
      const float* p = d.v + 3 * (size_t)fi[c];
      tris[3 * (d.tri_base + k) + c] = make_float4(p[0], p[1], p[2], c == 0 ? __uint_as_float(prim) : 0.f);
    }
  }
}

// One device allocation cut into aligned pieces.
struct Slab {
  char* base = nullptr;
  size_t size = 0;
  ~Slab() {
    if (base) cudaFree(base);
  }
  template <class T>
  size_t add(T**, size_t n) {
    const size_t at = size;
    size += (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~(size_t)255;
    return at;
  }
  void alloc() { CK(cudaMalloc((void**)&base, size)); }
  template <class T>
  T* at(size_t off) const { return reinterpret_cast<T*>(base + off); }
};

size_t splitShared() { return sizeof(Shared); }
size_t smallShared(int nb) { return kWarps * sizeof(SmallShared) + (size_t)(nb + 1) * 4; }

// Builds the trees of the domains hd (device meshes, bases of a batch filled in
// here) into B.out and their leaf-ordered triangles into `tris` (domain i's at
// 3 * hd[i].tri_base).  Returns node counts and depths; the slab holds B.
void buildBatch(std::vector<Dom>& hd, float4* tris, cudaStream_t stream, int sms, Slab& slab, Batch& B,
                std::vector<uint32_t>& nout, std::vector<int32_t>& depth) {
  const int nb = (int)hd.size();
  uint64_t fo = 0, so = 0, oo = 0, widest = 1;
  for (int i = 0; i < nb; ++i) {
    hd[i].tri_base = fo;
    hd[i].node_base = 2 * fo + 4 * (uint64_t)i;
    hd[i].small_base = so;
    hd[i].q_base = 2 * fo + 4 * (uint64_t)i;
    hd[i].out_base = oo;
    fo += hd[i].nf;
    so += (uint64_t)hd[i].nf / 16 + 64;
    oo += (uint64_t)hd[i].nf + 4;
    widest = std::max<uint64_t>(widest, hd[i].nf);
  }
  B = Batch{};
  B.big_cap = (uint32_t)(fo / kSmallTask + nb + 1);
  const Dom* cd = nullptr;
  const size_t o_doms = slab.add((Dom**)&cd, nb), o_lo = slab.add(&B.tlo, fo), o_hi = slab.add(&B.thi, fo);
  const size_t o_cen = slab.add(&B.cen, fo), o_i0 = slab.add(&B.idx[0], fo), o_i1 = slab.add(&B.idx[1], fo);
  const size_t o_ord = slab.add(&B.order, fo), o_nodes = slab.add(&B.nodes, 2 * fo + 4 * nb);
  const size_t o_small = slab.add(&B.small, so), o_b0 = slab.add(&B.big[0], B.big_cap);
  const size_t o_b1 = slab.add(&B.big[1], B.big_cap), o_out = slab.add(&B.out, oo);
  const size_t o_q = slab.add(&B.queue, 2 * fo + 4 * nb), o_nn = slab.add(&B.nnodes, nb);
  // read back together: error, node counts, depths; cleared together with the task counters
  const size_t o_err = slab.add(&B.error, 1), o_nout = slab.add(&B.nout, nb), o_depth = slab.add(&B.depth, nb);
  const size_t o_nsmall = slab.add(&B.nsmall, nb), o_nbig = slab.add(&B.nbig, kLevels + 1);
  uint32_t* next = nullptr;
  const size_t o_next = slab.add(&next, 1);
  slab.alloc();
  B.doms = slab.at<Dom>(o_doms);
  B.tlo = slab.at<float4>(o_lo), B.thi = slab.at<float4>(o_hi), B.cen = slab.at<float4>(o_cen);
  B.idx[0] = slab.at<uint32_t>(o_i0), B.idx[1] = slab.at<uint32_t>(o_i1), B.order = slab.at<uint32_t>(o_ord);
  B.nodes = slab.at<BNode>(o_nodes), B.small = slab.at<Task>(o_small);
  B.big[0] = slab.at<BigTask>(o_b0), B.big[1] = slab.at<BigTask>(o_b1);
  B.out = slab.at<BvhNode4>(o_out), B.queue = slab.at<int2>(o_q), B.nnodes = slab.at<uint32_t>(o_nn);
  B.error = slab.at<int>(o_err), B.nout = slab.at<uint32_t>(o_nout), B.depth = slab.at<int32_t>(o_depth);
  B.nsmall = slab.at<uint32_t>(o_nsmall), B.nbig = slab.at<uint32_t>(o_nbig);
  next = slab.at<uint32_t>(o_next);
  CK(cudaFuncSetAttribute(kSplit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)splitShared()));
  CK(cudaFuncSetAttribute(kBuildSmall, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smallShared(kMaxBatchDomains)));
  CK(cudaMemcpyAsync(slab.at<Dom>(o_doms), hd.data(), nb * sizeof(Dom), cudaMemcpyHostToDevice, stream));
  CK(cudaMemsetAsync(slab.base + o_err, 0, slab.size - o_err, stream));
  const int gx = 64;
  kPrep<<<dim3(gx, nb), 256, 0, stream>>>(B, nb);
  kRoots<<<nb, kSplitThreads, 0, stream>>>(B);
  // the first group of levels takes all but lopsided trees
  int levels = 2;
  while (levels < kLevels && ((uint64_t)kSmallTask << (levels / 2)) < widest) levels += 2;
  for (int level = 0; level < kLevels; ++level) {
    if (level == levels) {  // look whether any task is left before the other levels are launched
      uint32_t left = 0;
      CK(cudaMemcpyAsync(&left, B.nbig + level, 4, cudaMemcpyDeviceToHost, stream));
      CK(cudaStreamSynchronize(stream));
      if (left == 0) break;
      levels = std::min(levels + 8, kLevels);
    }
    kSplit<<<2 * sms, kSplitThreads, splitShared(), stream>>>(B, level);
    if (level == kLevels - 1) {
      uint32_t left = 0;
      int bad = 0;
      CK(cudaMemcpyAsync(&left, B.nbig + kLevels, 4, cudaMemcpyDeviceToHost, stream));
      CK(cudaMemcpyAsync(&bad, B.error, 4, cudaMemcpyDeviceToHost, stream));
      CK(cudaStreamSynchronize(stream));
      if (left == 0 || bad) break;
      kNextLevels<<<1, 64, 0, stream>>>(B);  // deeper still: a further group
      level = -1;
      levels = kLevels;
    }
  }
  kBuildSmall<<<3 * sms, kThreads, smallShared(nb), stream>>>(B, nb, next);
  kCollapse<<<nb, kCollapseThreads, 0, stream>>>(B);
  kFinish<<<dim3(gx, nb), 256, 0, stream>>>(B);
  kTris<<<dim3(gx, nb), 256, 0, stream>>>(B, tris);
  CK(cudaGetLastError());
  std::vector<char> back(o_nsmall - o_err);
  CK(cudaMemcpyAsync(back.data(), slab.base + o_err, back.size(), cudaMemcpyDeviceToHost, stream));
  CK(cudaStreamSynchronize(stream));
  int err = 0;
  std::memcpy(&err, back.data(), 4);
  if (err) throw std::runtime_error("device BVH build ran out of room (error flags " + std::to_string(err) + ")");
  nout.resize(nb);
  depth.resize(nb);
  std::memcpy(nout.data(), back.data() + (o_nout - o_err), nb * 4);
  std::memcpy(depth.data(), back.data() + (o_depth - o_err), nb * 4);
}

// Consecutive domains from `k` with at most `batch_tris` triangles together (at
// least one; at most kMaxBatchDomains: kBuildSmall keeps their prefix in shared memory).
template <class F>
size_t batchEnd(size_t k, size_t n, uint64_t batch_tris, F&& faces) {
  uint64_t tris = 0;
  size_t j = k;
  while (j < n && j - k < (size_t)kMaxBatchDomains && (j == k || tris + faces(j) <= batch_tris)) tris += faces(j++);
  return j;
}

int smCount() {
  int dev = 0, sms = 1;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return sms;
}

}  // namespace
}  // namespace gbvh

// Builds the BVHs of `n` domains (vertices and faces in host memory) on the
// current device and returns them in the packs (nodes, leaf-ordered
// triangles, depth).  Domains go in batches of at most `batch_tris`
// triangles to bound the device memory the build holds.
void buildBvhsOnDevice(const spray_gpu_domain* src, const std::vector<int>& which, std::vector<DomainPack>& packs,
                       cudaStream_t stream, uint64_t batch_tris) {
  using namespace gbvh;
  const int sms = smCount();
  size_t k = 0;
  while (k < which.size()) {
    const size_t j = batchEnd(k, which.size(), batch_tris, [&](size_t i) { return (uint64_t)src[which[i]].num_faces; });
    const int nb = (int)(j - k);
    uint64_t tris = 0, verts = 0;
    for (size_t i = k; i < j; ++i) {
      tris += (uint64_t)src[which[i]].num_faces;
      verts += (uint64_t)src[which[i]].num_vertices;
    }
    Slab mesh;
    float* dv = nullptr;
    uint32_t* df = nullptr;
    float4* dtris = nullptr;
    const size_t o_v = mesh.add(&dv, 3 * verts), o_f = mesh.add(&df, 3 * tris), o_t = mesh.add(&dtris, 3 * tris);
    mesh.alloc();
    dv = mesh.at<float>(o_v), df = mesh.at<uint32_t>(o_f), dtris = mesh.at<float4>(o_t);
    std::vector<Dom> hd(nb);
    uint64_t vo = 0, fo = 0;
    for (int i = 0; i < nb; ++i) {
      const spray_gpu_domain& s = src[which[k + i]];
      CK(cudaMemcpyAsync(dv + 3 * vo, s.vertices, (size_t)s.num_vertices * 12, cudaMemcpyHostToDevice, stream));
      CK(cudaMemcpyAsync(df + 3 * fo, s.faces, (size_t)s.num_faces * 12, cudaMemcpyHostToDevice, stream));
      hd[i].v = dv + 3 * vo;
      hd[i].f = df + 3 * fo;
      hd[i].nf = (uint32_t)s.num_faces;
      vo += (uint64_t)s.num_vertices;
      fo += (uint64_t)s.num_faces;
    }
    Slab work;
    Batch B;
    std::vector<uint32_t> nout;
    std::vector<int32_t> depth;
    buildBatch(hd, dtris, stream, sms, work, B, nout, depth);
    for (int i = 0; i < nb; ++i) {
      DomainPack& p = packs[which[k + i]];
      p.nodes.resize(nout[i]);
      p.tris.resize(3 * (size_t)hd[i].nf);
      CK(cudaMemcpyAsync(p.nodes.data(), B.out + hd[i].out_base, nout[i] * sizeof(BvhNode4), cudaMemcpyDeviceToHost,
                         stream));
      CK(cudaMemcpyAsync(p.tris.data(), dtris + 3 * hd[i].tri_base, 3 * (size_t)hd[i].nf * sizeof(float4),
                         cudaMemcpyDeviceToHost, stream));
      p.bvh_depth = depth[i];
    }
    CK(cudaStreamSynchronize(stream));
    k = j;
  }
}

// The same for meshes already on the device, whose results stay there.
void buildBvhsInPlace(const std::vector<DeviceMesh>& meshes, cudaStream_t stream, uint64_t batch_tris, float4* tris,
                      BvhNode4** nodes, std::vector<uint32_t>* counts, int* max_depth) {
  using namespace gbvh;
  const int sms = smCount();
  std::vector<std::pair<BvhNode4*, size_t>> parts;  // a batch's nodes
  size_t total = 0;
  uint64_t tri0 = 0;
  *max_depth = 0;
  counts->clear();
  try {
    size_t k = 0;
    while (k < meshes.size()) {
      const size_t j = batchEnd(k, meshes.size(), batch_tris, [&](size_t i) { return (uint64_t)meshes[i].nf; });
      const int nb = (int)(j - k);
      std::vector<Dom> hd(nb);
      uint64_t n = 0;
      for (int i = 0; i < nb; ++i) {
        hd[i].v = meshes[k + i].v;
        hd[i].f = meshes[k + i].f;
        hd[i].nf = meshes[k + i].nf;
        n += meshes[k + i].nf;
      }
      Slab work;
      Batch B;
      std::vector<uint32_t> nout;
      std::vector<int32_t> depth;
      buildBatch(hd, tris + 3 * tri0, stream, sms, work, B, nout, depth);
      std::vector<uint64_t> to(nb);
      size_t nn = 0;
      for (int i = 0; i < nb; ++i) {
        to[i] = nn;
        nn += nout[i];
        *max_depth = std::max(*max_depth, (int)depth[i]);
      }
      BvhNode4* part = nullptr;
      CK(cudaMalloc(&part, std::max<size_t>(nn, 1) * sizeof(BvhNode4)));
      parts.push_back({part, nn});
      // the queue is free by now
      uint64_t* dto = reinterpret_cast<uint64_t*>(B.queue);
      CK(cudaMemcpyAsync(dto, to.data(), nb * sizeof(uint64_t), cudaMemcpyHostToDevice, stream));
      kGatherNodes<<<dim3(64, nb), 256, 0, stream>>>(B, dto, part);
      CK(cudaGetLastError());
      CK(cudaStreamSynchronize(stream));  // the work slab and the host list end here
      counts->insert(counts->end(), nout.begin(), nout.end());
      total += nn;
      tri0 += n;
      k = j;
    }
    if (parts.size() == 1) {
      *nodes = parts[0].first;
      return;
    }
    CK(cudaMalloc(nodes, std::max<size_t>(total, 1) * sizeof(BvhNode4)));
    size_t at = 0;
    for (auto& p : parts) {
      CK(cudaMemcpyAsync(*nodes + at, p.first, p.second * sizeof(BvhNode4), cudaMemcpyDeviceToDevice, stream));
      at += p.second;
    }
    CK(cudaStreamSynchronize(stream));
    for (auto& p : parts) cudaFree(p.first);
  } catch (...) {
    for (auto& p : parts) cudaFree(p.first);
    throw;
  }
}

}  // namespace spray
