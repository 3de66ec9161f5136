// The domains a ray may enter: the descent of the 4-wide hierarchy over the
// domain boxes (the scheduler, sched.cu, the non-speculative round loop,
// rounds.cu, and scenes of many domains) and the test of their groups of 64, 16
// and 4 with a ray's sorted list (the whole-ray walks, walk_rays.cu, and the
// allocation-free scheduler, noalloc.cu).
#pragma once

#include "kernels.cuh"
#include "spray_math.cuh"
#include "traverse.cuh"

namespace spray {

// Calls consider(d) for every domain d of the 4-wide hierarchy over the domain
// boxes (8 float4 per node, BvhNode4 layout; NN nodes) whose node boxes the ray
// (org, inv = 1 / dir) enters within (1e-3, t1].  The node boxes are enlarged
// outward and the test widened by 2 ulp, so the descent is conservative: the
// caller's exact slab test at the leaf decides.  Children go near to far, so
// domains arrive roughly in entry order.
template <class F>
__device__ __forceinline__ void descendDomains(const float4* nodes, int NN, V3 org, V3 inv, float t1, F&& consider,
                                               Counters* ctr) {
  const int sx = inv.x < 0.0f, sy = inv.y < 0.0f, sz = inv.z < 0.0f;
  const float tfar = t1 * 1.0000004f;
  int stack[32];
  int sp = 0;
  int node = 0;
  for (int steps = 0; steps < NN + 4; ++steps) {
    const float4* nd = nodes + 8 * node;
    const float4 nx = nd[sx], fx = nd[sx ^ 1], ny = nd[2 + sy], fy = nd[3 - sy];
    const float4 nz = nd[4 + sz], fz = nd[5 - sz];
    const int4 ch = *reinterpret_cast<const int4*>(nd + 6);
    const float nxa[4] = {nx.x, nx.y, nx.z, nx.w}, fxa[4] = {fx.x, fx.y, fx.z, fx.w};
    const float nya[4] = {ny.x, ny.y, ny.z, ny.w}, fya[4] = {fy.x, fy.y, fy.z, fy.w};
    const float nza[4] = {nz.x, nz.y, nz.z, nz.w}, fza[4] = {fz.x, fz.y, fz.z, fz.w};
    const int cha[4] = {ch.x, ch.y, ch.z, ch.w};
    uint32_t k[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float t0 = fmaxf(fmaxf((nxa[c] - org.x) * inv.x, (nya[c] - org.y) * inv.y),
                             fmaxf((nza[c] - org.z) * inv.z, kRayEpsilon));
      const float tt = fminf(fminf((fxa[c] - org.x) * inv.x, (fya[c] - org.y) * inv.y),
                             fminf((fza[c] - org.z) * inv.z, tfar)) * 1.0000004f;
      // (entry t with the slot in its two low bits: t > 0 orders like its bits)
      k[c] = (t0 <= tt && cha[c] != kEmptyChild) ? ((__float_as_uint(t0) & ~3u) | (uint32_t)c) : 0xffffffffu;
    }
    auto cswap = [](uint32_t& x, uint32_t& y) {
      const uint32_t lo = min(x, y), hi = max(x, y);
      x = lo;
      y = hi;
    };
    cswap(k[0], k[1]);
    cswap(k[2], k[3]);
    cswap(k[0], k[2]);
    cswap(k[1], k[3]);
    cswap(k[1], k[2]);
    int inner[4], ni = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (k[j] == 0xffffffffu) break;
      const int ref = cha[k[j] & 3u];
      if (ref < 0) consider(~ref);
      else inner[ni++] = ref;
    }
    // the nearest inner child next, the others on the stack far to near
    for (int j = ni - 1; j >= 1; --j) {
      if (sp < 32) stack[sp++] = inner[j];
      else atomicAdd(&ctr->list_overflows, 1ull);  // unreachable: depth <= 8, 3 per level
    }
    if (ni > 0) {
      node = inner[0];
    } else {
      if (sp == 0) break;
      node = stack[--sp];
    }
  }
}

namespace {

// A node of the group table in shared memory takes 9 float4 instead of 8: the
// four boxes of a node are read by all lanes at once, but near and far planes
// differ by lane, and the exact tests read different nodes.
constexpr int kNodeStride = 9;
// Slack of the group test: the exact slab test rounds (plane - org) * inv and
// this one fma(plane, inv, -org * inv); 2e-6 covers both by far.
constexpr float kGroupSlack = 1.000002f;

// Floats as integers that order like them (negative t: the ray starts inside
// the box; -0 was made +0 by the caller).
__device__ __forceinline__ uint32_t orderedBits(float t) {
  const uint32_t u = __float_as_uint(t);
  return u ^ ((u & 0x80000000u) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float orderedFloat(uint32_t k) {
  return __uint_as_float(k ^ ((k & 0x80000000u) ? 0x80000000u : 0xffffffffu));
}

// Per-lane sorted list of (entry t, domain), 64-bit keys in local memory.
struct DomainList {
  uint64_t key[kMaxList];
  int n = 0;
  __device__ __forceinline__ void insert(float t, int d, Counters* ctr) {
    const uint64_t k = ((uint64_t)orderedBits(t + 0.0f) << 32) | (uint32_t)d;
    if (n == kMaxList) {
      atomicAdd(&ctr->list_overflows, 1ull);
      return;  // the frame is refused
    }
    int j = n++;
    while (j > 0 && key[j - 1] > k) {
      key[j] = key[j - 1];
      --j;
    }
    key[j] = k;
  }
};

// The four boxes of a table node against the ray: bit k set when box k may be hit.
__device__ __forceinline__ uint32_t boxMask(const float4* p, const BoxRay& r, float t1) {
  float tn[4];
  bool h[4];
  testBoxes(p[r.sx], p[r.sx ^ 1], p[2 + r.sy], p[3 - r.sy], p[4 + r.sz], p[5 - r.sz], r, kRayEpsilon, t1, kGroupSlack,
            tn, h);
  return (h[0] ? 1u : 0u) | (h[1] ? 2u : 0u) | (h[2] ? 4u : 0u) | (h[3] ? 8u : 0u);
}

// Calls consider(d) for a superset of the domains whose boxes the ray enters
// within (1e-3, t1], 64 at a time: every group of 16 is tested, the four nodes
// of a group some lane may enter are tested by all of the warp's lanes that
// may, at the same addresses, and then each lane goes through its own bits.
// Against the descent of a hierarchy (descendDomains) that is more tests and
// far fewer instructions, for the lanes of a warp stay together.
template <class F>
__device__ __forceinline__ void groupDomains(const float4* table, int n1, int n2, const BoxRay& r, float t1,
                                             F&& consider) {
  const float4* l2 = table + n1 * kNodeStride;
  for (int q = 0; q < n1; ++q) {
    const uint32_t groups = boxMask(table + q * kNodeStride, r, t1);
    uint32_t bits[2] = {0u, 0u};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (!(groups & (1u << c))) continue;
      const int first = 16 * q + 4 * c;
      uint32_t m = 0;
#pragma unroll 1
      for (int j = 0; j < 4 && first + j < n2; ++j)
        m |= boxMask(l2 + (first + j) * kNodeStride, r, t1) << (4 * j);
      bits[c >> 1] |= m << (16 * (c & 1));
    }
#pragma unroll
    for (int w = 0; w < 2; ++w)
      for (uint32_t m = bits[w]; m; m &= m - 1) {
        const int b = 32 * w + __ffs(m) - 1;
        consider(reinterpret_cast<const int*>(l2 + (16 * q + (b >> 2)) * kNodeStride + 6)[b & 3]);
      }
  }
}

__device__ __forceinline__ uint32_t warpScan(uint32_t v, uint32_t* total) {
  const int lane = threadIdx.x & 31;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  *total = __shfl_sync(0xffffffffu, x, 31);
  return x - v;
}

}  // namespace
}  // namespace spray
