// Per-thread BVH walks of one (ray, domain) pair, shared by the queue
// kernels (trace.cu) and the round loop of the non-speculative tracer
// (rounds.cu): the 4-wide node test, the closest-hit walk and the any-hit
// walk.  Scene::intersect / Scene::occluded (src/render/scene.inl:189-209)
// with tnear = 1e-3.
#pragma once

#include "kernels.cuh"
#include "spray_math.cuh"

namespace spray {
namespace {

// Box test slack: (1 + 2*gamma(3)) rounded up (Ize, "Robust BVH Ray
// Traversal", JCGT 2(2), 2013), so rounding never culls a box the ray touches.
constexpr float kBoxSlack = 1.0000004f;
constexpr int kStack = 64;

// A ray as the box tests use it.  The distance of a plane p along an axis is
// fma(p, inv, c): with inv = 1 / dir and c = -org * inv that is (p - org) / dir
// but for relative roundings (the slack's part) and the rounding of org * inv,
// at most 2^-24 of |org * inv| for the product and as much for c.  c is
// therefore kept twice, moved by 2^-22 of |org * inv|: down for near planes, up
// for far ones, so that the interval only ever grows.  |inv| is held within
// [1e-30, 1e18], so that an empty slot (lo = +inf, hi = -inf) is never entered
// and an axis the ray is parallel to gives finite distances of the right sign
// (fma(p, inf, -inf) would be a NaN); its planes count as touched within 1e-6
// of the origin (1e12 / 1e18), as (p - org) * inf = NaN for p = org would.  A NaN
// component of the direction passes the comparisons of the exact slab test, so here
// its axis spans [-1e12, 1e12].
struct BoxRay {
  V3 inv, cnear, cfar;
  int sx, sy, sz;  // 1 when the direction component is negative
};

__device__ __forceinline__ float boxPad(float oi, float inv) {
  return fabsf(oi) * 2.384185791015625e-7f + (fabsf(inv) <= 1e18f ? 0.0f : 1e12f);
}

__device__ __forceinline__ void boxAxis(float org, float inv, float& binv, float& cnear, float& cfar) {
  binv = copysignf(fminf(fmaxf(fabsf(inv), 1e-30f), 1e18f), inv);
  const float oi = org * binv;
  const float pad = boxPad(oi, inv);
  cnear = -oi - pad;
  cfar = pad - oi;
}

// inv = 1 / dir, as IEEE division gives it
__device__ __forceinline__ BoxRay makeBoxRay(V3 org, V3 inv) {
  BoxRay r;
  boxAxis(org.x, inv.x, r.inv.x, r.cnear.x, r.cfar.x);
  boxAxis(org.y, inv.y, r.inv.y, r.cnear.y, r.cfar.y);
  boxAxis(org.z, inv.z, r.inv.z, r.cnear.z, r.cfar.z);
  r.sx = inv.x < 0.0f;
  r.sy = inv.y < 0.0f;
  r.sz = inv.z < 0.0f;
  return r;
}

// A ray as the walks use it.
struct TravRay {
  V3 org;
  BoxRay box;
  RayShear sh;
};

__device__ __forceinline__ TravRay makeTravRay(V3 org, V3 dir) {
  TravRay r;
  r.org = org;
  r.box = makeBoxRay(org, v3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z));
  r.sh = makeShear(dir);
  return r;
}

// max and min of three (one instruction on sm_100 and later; a NaN operand is
// dropped, as by fmaxf and fminf)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Intersects the four boxes of a node: their entry distances tn, and hit.
// Near and far planes are picked by the direction's sign, by address: the
// node stores lo/hi per axis as float4 pairs.  Per box: t0 = max(near x, y, z,
// tnear), t1 = min(far x, y, z, tfar) * slack; boxes (0, 1) and (2, 3) share
// packed multiply-adds, and the maxima take three operands: the walks are
// bound by instruction issue, the min/max/compare pipe first.
__device__ __forceinline__ void testBoxes(float4 nx, float4 fx, float4 ny, float4 fy, float4 nz, float4 fz,
                                          const BoxRay& r, float tnear, float tfar, float slack, float tn[4],
                                          bool hit[4]) {
  const unsigned long long ix = f2pack(r.inv.x, r.inv.x), iy = f2pack(r.inv.y, r.inv.y),
                           iz = f2pack(r.inv.z, r.inv.z);
  const unsigned long long nx2 = f2pack(r.cnear.x, r.cnear.x), ny2 = f2pack(r.cnear.y, r.cnear.y),
                           nz2 = f2pack(r.cnear.z, r.cnear.z);
  const unsigned long long fx2 = f2pack(r.cfar.x, r.cfar.x), fy2 = f2pack(r.cfar.y, r.cfar.y),
                           fz2 = f2pack(r.cfar.z, r.cfar.z);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float2 ax = f2fma(h ? f2pack(nx.z, nx.w) : f2pack(nx.x, nx.y), ix, nx2);
    const float2 ay = f2fma(h ? f2pack(ny.z, ny.w) : f2pack(ny.x, ny.y), iy, ny2);
    const float2 az = f2fma(h ? f2pack(nz.z, nz.w) : f2pack(nz.x, nz.y), iz, nz2);
    const float2 bx = f2fma(h ? f2pack(fx.z, fx.w) : f2pack(fx.x, fx.y), ix, fx2);
    const float2 by = f2fma(h ? f2pack(fy.z, fy.w) : f2pack(fy.x, fy.y), iy, fy2);
    const float2 bz = f2fma(h ? f2pack(fz.z, fz.w) : f2pack(fz.x, fz.y), iz, fz2);
    const float t00 = fmaxf(max3(ax.x, ay.x, az.x), tnear);
    const float t01 = fmaxf(max3(ax.y, ay.y, az.y), tnear);
    const float t10 = fminf(min3(bx.x, by.x, bz.x), tfar) * slack;
    const float t11 = fminf(min3(bx.y, by.y, bz.y), tfar) * slack;
    tn[2 * h] = t00;
    tn[2 * h + 1] = t01;
    hit[2 * h] = t00 <= t10;
    hit[2 * h + 1] = t01 <= t11;
  }
}

__device__ __forceinline__ void testChildren(const BvhNode4* __restrict__ nodes, int node, const TravRay& r,
                                             float tnear, float tfar, float tn[4], bool hit[4]) {
  const float4* p = reinterpret_cast<const float4*>(nodes + node);
  testBoxes(__ldg(p + r.box.sx), __ldg(p + (r.box.sx ^ 1)), __ldg(p + 2 + r.box.sy), __ldg(p + (3 - r.box.sy)),
            __ldg(p + 4 + r.box.sz), __ldg(p + (5 - r.box.sz)), r.box, tnear, tfar, kBoxSlack, tn, hit);
}

__device__ __forceinline__ int4 loadChildren(const BvhNode4* __restrict__ nodes, int node) {
  const int4* p = reinterpret_cast<const int4*>(nodes + node);
  return __ldg(p + 6);
}

__device__ __forceinline__ int childAt(int4 c, int k) {
  return k == 0 ? c.x : (k == 1 ? c.y : (k == 2 ? c.z : c.w));
}

// Upper bound on node visits of one traversal; reaching it means a corrupt
// hierarchy, which is reported through Counters::error_flags.
constexpr int kMaxSteps = 1 << 20;

__device__ __forceinline__ void raise(Counters* ctr, unsigned long long bit) {
  atomicOr(&ctr->error_flags, bit);
}

// Marks the end of a traversal (never a child reference: empty slots are skipped).
constexpr int kDone = (int)kEmptyChild;
// Closest hit in one domain.  best_key enters as the key to beat and leaves as
// the best found; returns true when this domain improved it.
//
// While-while traversal: a thread expands inner nodes until the nearest
// pending entry is a leaf (the loop ends when every active thread holds a
// leaf or has finished), then the threads test their leaves together.  Inner
// nodes and leaves share one near-to-far stack, so a leaf is tested only after
// every nearer subtree, and entries beyond the best hit are dropped on pop.
// The hit does not depend on the order: the packed (t | triangle) key is a
// total order and a subtree is skipped only when its box starts beyond the
// best t found.
__device__ bool traverseClosest(const SceneDev& sc, const DomainDev& dom, const TravRay& r,
                                uint64_t& best_key, float& best_t, uint32_t& best_prim,
                                float& best_u, float& best_v, Counters* ctr,
                                uint32_t& nnodes, uint32_t& ntris) {
  const DomArrays g = domArrays(sc, dom);
  const BvhNode4* nodes = g.nodes;
  const float4* tris = g.tris;
  uint2 stack[kStack];
  int sp = 0;
  bool found = false;
  // node and triangle counts of this walk (32 bits: a walk is bounded by
  // kMaxSteps); the node count is also the step bound's counter
  uint32_t steps = 0, tested = 0;
  auto finish = [&]() {
    nnodes += steps;
    ntris += tested;
    return found;
  };
  auto pop = [&]() -> int {
    while (sp > 0) {
      const uint2 e = stack[--sp];
      if (__uint_as_float(e.y) <= best_t) return (int)e.x;
    }
    return kDone;
  };
  // triangles of one leaf; false on a corrupt leaf reference
  auto testLeaf = [&](int lf) -> bool {
    const uint32_t v = ~(uint32_t)lf;
    const uint32_t first = v >> 3, cnt = (v & 7u) + 1u;
    if (first + cnt > (uint32_t)dom.num_tris) {
      raise(ctr, kErrBadNode);
      return false;
    }
    tested += cnt;
    for (uint32_t q = 0; q < cnt; ++q) {
      const float4* tp = tris + 3 * (size_t)(first + q);
      const float4 a = __ldg(tp), b = __ldg(tp + 1), cc = __ldg(tp + 2);
      float t, u, vv;
      if (intersectTriangle(r.sh, r.org, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(cc.x, cc.y, cc.z),
                            kRayEpsilon, __int_as_float(0x7f800000), &t, &u, &vv)) {
        const uint32_t prim = __float_as_uint(a.w);
        const uint64_t key = packHitKey(t, dom.gprim_base + prim);
        if (key < best_key) {
          best_key = key;
          best_t = t;
          best_prim = prim;
          best_u = u;
          best_v = vv;
          found = true;
        }
      }
    }
    return true;
  };
  int cur = 0;
  while (cur != kDone) {
    // inner nodes until the nearest pending entry is a leaf
    while (cur >= 0) {
      if (++steps > (uint32_t)kMaxSteps) {
        raise(ctr, kErrTraversalBound);
        return finish();
      }
      if ((unsigned)cur >= (unsigned)dom.num_nodes) {
        raise(ctr, kErrBadNode);
        return finish();
      }
      float tn[4];
      bool hit[4];
      testChildren(nodes, cur, r, kRayEpsilon, best_t, tn, hit);
      const int4 ch = loadChildren(nodes, cur);
      // The nearest child continues the walk, the others go on the stack in
      // slot order: a node rarely has more than two children hit (sorting
      // them by a network costs more than the order of a third and fourth
      // saves), and a pushed entry beyond the best hit is dropped on pop.
      // The key is the entry t with its two low bits replaced by the slot:
      // t >= tnear > 0, so the bits order like the value, and the key's t
      // (rounded down by at most 3 ulp) stays a lower bound of the entry.
      uint32_t k[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) k[c] = hit[c] ? (__float_as_uint(tn[c]) & ~3u) | (uint32_t)c : 0xffffffffu;
      const uint32_t kmin = min(__vimin3_u32(k[0], k[1], k[2]), k[3]);
      if (kmin != 0xffffffffu) {
        if (sp > kStack - 3) {
          raise(ctr, kErrTraversalBound);
          return finish();
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (hit[c] && k[c] != kmin) stack[sp++] = make_uint2((uint32_t)childAt(ch, c), k[c] & ~3u);
        cur = childAt(ch, (int)(kmin & 3u));
      } else {
        cur = pop();
      }
    }
    if (cur == kDone) break;
    if (!testLeaf(cur)) return finish();
    cur = pop();
  }
  return finish();
}

// Any hit in (tnear, tfar) in one domain, the whole walk at once: the last
// hit child continues, the others are pushed.  Returns true on a hit.
__device__ bool traverseAny(const SceneDev& sc, const DomainDev& dom, const TravRay& r, float tfar,
                            Counters* ctr, uint32_t& nnodes, uint32_t& ntris) {
  const DomArrays g = domArrays(sc, dom);
  int stack[kStack];
  int sp = 0, cur = 0;
  uint32_t steps = 0;
  while (cur != kDone) {
    while (cur >= 0) {
      if (++steps > (uint32_t)kMaxSteps || (unsigned)cur >= (unsigned)dom.num_nodes) {
        raise(ctr, steps > (uint32_t)kMaxSteps ? kErrTraversalBound : kErrBadNode);
        nnodes += steps;
        return false;
      }
      float tn[4];
      bool hit[4];
      testChildren(g.nodes, cur, r, kRayEpsilon, tfar, tn, hit);
      const int4 ch = loadChildren(g.nodes, cur);
      if (sp > kStack - 3) {
        raise(ctr, kErrTraversalBound);
        nnodes += steps;
        return false;
      }
      int next = kDone;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (!hit[c]) continue;
        if (next != kDone) stack[sp++] = next;
        next = childAt(ch, c);
      }
      cur = next != kDone ? next : (sp > 0 ? stack[--sp] : kDone);
    }
    if (cur == kDone) break;
    const uint32_t v = ~(uint32_t)cur;
    const uint32_t first = v >> 3, cnt = (v & 7u) + 1u;
    if (first + cnt > (uint32_t)dom.num_tris) {
      raise(ctr, kErrBadNode);
      nnodes += steps;
      return false;
    }
    ntris += cnt;
    for (uint32_t q = 0; q < cnt; ++q) {
      const float4* tp = g.tris + 3 * (size_t)(first + q);
      const float4 a = __ldg(tp), b = __ldg(tp + 1), cc = __ldg(tp + 2);
      float t, u, vv;
      if (intersectTriangle(r.sh, r.org, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(cc.x, cc.y, cc.z),
                            kRayEpsilon, tfar, &t, &u, &vv)) {
        nnodes += steps;
        return true;
      }
    }
    cur = sp > 0 ? stack[--sp] : kDone;
  }
  nnodes += steps;
  return false;
}

}  // namespace
}  // namespace spray
