// Closest hits and occlusion of whole rays, in core.
//
// When every domain is resident no domain has to be waited for, so a ray's
// domains need no queues.  kListDomains writes each ray's (t, id)-sorted domain
// list (the list Isector::isect makes, src/ooc/ooc_isector.h:116-174, exact slab
// tests and all); then a thread walks a ray's listed domains front to back.
// Radiance rays stop at the first domain that starts beyond the hit found;
// shadow rays run first in the domain that spawned them (TContext::procShads2)
// and stop at the first occluder.  The closest hit is the smallest packed
// (t | triangle) key over the domains visited, as in the queue kernels
// (trace.cu), so the image does not change; visits plus culled entries still
// add up to the listed (ray, domain) pairs.
//
// The queues' partition (histogram, scan, scatter), the per-entry records and
// the resolve pass fall away, and a ray sets up its walk once instead of once
// per domain.  Path tracing 64 domains at 1920x1080, 16 spp, 5 bounces: lists
// 1.72 -> 0.87 ms a frame (with the partition), closest hits with their colours
// and normals 4.48 + 0.39 -> 3.68 ms, occlusion 1.71 -> 1.37 ms.
#include "domain_walk.cuh"
#include "kernels.cuh"
#include "spray_math.cuh"
#include "traverse.cuh"

namespace spray {

namespace {

constexpr int kWalkThreads = 256;
// The rounds' thresholds, in lanes of 32.  Each was varied by itself; the figures are
// frames of 24 views of up to 2048x2048, 16 spp, ambient occlusion and path tracing.
// Idle lanes a warp gathers before it fetches new rays for them (12, 16, 20 and 24:
// 113.0, 110.4, 109.1 and 110.2 ms).
constexpr int kRefill = 20;
// Lanes at the end of a domain that the warp gathers before it moves them on: closest
// hits (1, 2 and 4: 109.7, 109.1 and 109.8 ms) and occlusion (2, 4, 6 and 8: 108.9,
// 109.1, 109.6 and 110.5 ms).
constexpr int kSwitch = 2, kShadowSwitch = 4;
// Lanes at inner nodes with which a warp takes another node (3, 5, 7, 9 and 12: 111.4,
// 109.5, 109.1, 109.6 and 111.1 ms), lanes at triangles with which it takes another
// triangle (1, 3, 5, 8 and 12: 111.5, 109.4, 109.1, 109.9 and 111.2 ms).
constexpr int kStay = 7, kLeaves = 5;

__device__ __forceinline__ uint32_t lanesBelowMask() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

enum ListKind { kListBounce, kListPrimary, kListShadow };

}  // namespace

// The sorted domain list of every ray, into the arena (one atomic per block of
// 256 rays), the group table in shared memory (kNodeStride).
template <int kKind>
__global__ void __launch_bounds__(kWalkThreads) kListDomains(RayWalkArgs a) {
  extern __shared__ float4 table[];
  __shared__ uint32_t wsum[kWalkThreads / 32];
  __shared__ unsigned long long wbase;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n1 = a.groups.l1, n2 = a.groups.l2, D = a.scene.num_domains;
  if (kKind != kListPrimary) {
    const float4* src = reinterpret_cast<const float4*>(a.groups.nodes);
    for (int k = threadIdx.x; k < 8 * (n1 + n2); k += blockDim.x) table[(k >> 3) * kNodeStride + (k & 7)] = src[k];
    __syncthreads();
  }
  const uint32_t n = *a.count;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = base + threadIdx.x;
    const bool active = i < n;
    DomainList list;
    int origin = -1;
    uint32_t emit = 0;
    if (active) {
      const uint32_t rid = a.list[i];
      V3 org, dir;
      float t1 = INFINITY;
      if (kKind == kListShadow) {
        const float4 hp = a.sh.hitpos[rid / a.slots], d4 = a.sh.dir[rid];
        org = v3(hp.x, hp.y, hp.z);
        origin = __float_as_int(hp.w);
        dir = v3(d4.x, d4.y, d4.z);
        t1 = d4.w;
      } else {
        const float4 o4 = a.rays.org[rid], d4 = a.rays.dir[rid];
        org = v3(o4.x, o4.y, o4.z);
        dir = v3(d4.x, d4.y, d4.z);
        a.ray_key[rid] = kNoHit;
      }
      const V3 inv = v3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
      auto consider = [&](int d) {
        float t;
        if (slabTest(a.dboxes + 6 * d, a.dboxes + 6 * d + 3, org, inv, kRayEpsilon, t1, &t)) list.insert(t, d, a.ctr);
      };
      if (kKind == kListPrimary) {
        // the domains whose projected box covers this pixel's bin
        const int pid = a.rays.pixid[rid];
        const ViewDev& vw = a.views[a.rays.view[rid]];
        const int bx = (pid % vw.image_w) >> a.bin_shift, by = (pid / vw.image_w) >> a.bin_shift;
        const int bin = vw.bin_base + by * vw.bins_x + bx;
        const uint32_t c1 = a.bin_start[bin + 1];
        for (uint32_t c = a.bin_start[bin]; c < c1; ++c) consider((int)a.bin_ids[c]);
      } else if (n1 > 0) {
        groupDomains(table, n1, n2, makeBoxRay(org, inv), t1, consider);
      } else if (a.groups.tree_count > 0) {
        descendDomains(reinterpret_cast<const float4*>(a.groups.tree), a.groups.tree_count, org, inv, t1, consider, a.ctr);
      } else {
        for (int d = 0; d < D; ++d) consider(d);
      }
      emit = (uint32_t)list.n;
      if (kKind == kListShadow) {
        emit += 1u;
        for (int j = 0; j < list.n; ++j)
          if ((int)(uint32_t)list.key[j] == origin) --emit;
      }
    }
    uint32_t total;
    uint32_t pos = warpScan(emit, &total);
    if (lane == 31) wsum[warp] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t run = 0;
      for (int w = 0; w < kWalkThreads / 32; ++w) {
        const uint32_t v = wsum[w];
        wsum[w] = run;
        run += v;
      }
      unsigned long long b = run ? atomicAdd(a.arena_top, (unsigned long long)run) : 0ull;
      if (b + run > a.arena_cap) {
        atomicAdd(&a.ctr->arena_overflows, 1ull);  // the frame is traced again with a larger arena
        b = ~0ull;
      }
      wbase = b;
    }
    __syncthreads();
    const unsigned long long b = wbase;
    pos += wsum[warp];
    __syncthreads();  // wsum and wbase are rewritten by the next round
    if (!active) continue;
    const bool fits = b != ~0ull;
    a.list_ref[i] = make_uint2(fits ? (uint32_t)(b + pos) : 0u, fits ? emit : 0u);
    if (!fits) continue;
    uint2* out = a.arena + b + pos;
    if (kKind == kListShadow) *out++ = make_uint2((uint32_t)origin, 0u);
    for (int j = 0; j < list.n; ++j) {
      const uint64_t k = list.key[j];
      if (kKind == kListShadow && (int)(uint32_t)k == origin) continue;
      *out++ = make_uint2((uint32_t)k, __float_as_uint(orderedFloat((uint32_t)(k >> 32))));
    }
  }
}

namespace {

// A ray in the domain it walks.  Per axis a box spans tc -+ h with tc =
// fma(c, inv, o) and h = fma(e, |inv|, pad), where inv = half * (1 / dir) and o =
// (centre - org) * (1 / dir) take the node's relative coordinates to distances.
// The roundings of inv and o move a plane by at most 2^-22 of |inv| + |o|, which
// pad exceeds (and by 1e12 for an axis the ray is parallel to, see BoxRay); what
// is relative to the plane's own distance is kBoxSlack's part.
struct WalkRay {
  V3 org;
  V3 rinv;            // 1 / dir, held within [1e-30, 1e18]
  V3 inv, o, pad;     // in the current domain
  RayShear sh;
};

__device__ __forceinline__ float walkInverse(float d) {
  const float inv = 1.0f / d;
  return copysignf(fminf(fmaxf(fabsf(inv), 1e-30f), 1e18f), inv);
}

__device__ __forceinline__ WalkRay makeWalkRay(V3 org, V3 dir) {
  WalkRay r;
  r.org = org;
  r.rinv = v3(walkInverse(dir.x), walkInverse(dir.y), walkInverse(dir.z));
  r.inv = r.o = r.pad = v3(0.f, 0.f, 0.f);
  r.sh = makeShear(dir);
  return r;
}

// 32 bytes through the read-only cache in one request: a warp's lanes are at
// different nodes, so the requests of a walk, not its bytes, load L1.
__device__ __forceinline__ void load256(const void* p, uint32_t* v) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "l"(p));
}

// Takes the ray to domain d; returns its root node.
__device__ __forceinline__ int enterDomain(const RayWalkArgs& a, int d, WalkRay& r) {
  uint32_t w[8];
  load256(a.domains + d, w);
  auto axis = [&](int k, float org, float rinv, float& inv, float& o, float& pad) {
    const float c = __uint_as_float(w[k]), h = __uint_as_float(w[3 + k]);
    inv = copysignf(fmaxf(fabsf(h * rinv), 1e-30f), rinv);
    o = (c - org) * rinv;
    pad = (fabsf(inv) + fabsf(o)) * 4.76837158203125e-7f + (fabsf(rinv) == 1e18f ? 1e12f : 0.0f);
  };
  axis(0, r.org.x, r.rinv.x, r.inv.x, r.o.x, r.pad.x);
  axis(1, r.org.y, r.rinv.y, r.inv.y, r.o.y, r.pad.y);
  axis(2, r.org.z, r.rinv.z, r.inv.z, r.o.z, r.pad.z);
  return (int)w[6];
}

__device__ __forceinline__ unsigned long long f2add(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long f2sub(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long f2fmaPacked(unsigned long long a, unsigned long long b,
                                                          unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// two halves of a word as packed floats
__device__ __forceinline__ unsigned long long f2half(uint32_t w) {
  float lo, hi;
  asm("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %2;\n cvt.f32.f16 %0, l;\n cvt.f32.f16 %1, h;\n}\n"
      : "=f"(lo), "=f"(hi)
      : "r"(w));
  return f2pack(lo, hi);
}

// The four children of a walk node: entry distances, hits and references.
// kPacked: multiply-adds two children at a time, fewer instructions but pairs of
// registers for every constant of the ray.  It suits the occlusion walk (1.40
// and 1.42 ms a frame, packed and scalar); the closest-hit walk spills with it
// (4.01 and 3.73 ms).
template <bool kPacked>
__device__ __forceinline__ int4 testNode(const WalkNode* __restrict__ nodes, int node, const WalkRay& r, float tfar,
                                         float tn[4], bool hit[4]) {
  uint32_t w[16];  // cx cx ex ex cy cy ey ey cz cz ez ez child x 4
  load256(nodes + node, w);
  load256(reinterpret_cast<const char*>(nodes + node) + 32, w + 8);
  auto span = [](uint32_t c, uint32_t e, float inv, float o, float pad, float2* near, float2* far) {
    if (kPacked) {
      const unsigned long long tc = f2fmaPacked(f2half(c), f2pack(inv, inv), f2pack(o, o));
      const unsigned long long hw = f2fmaPacked(f2half(e), f2pack(fabsf(inv), fabsf(inv)), f2pack(pad, pad));
      *near = f2unpack(f2sub(tc, hw));
      *far = f2unpack(f2add(tc, hw));
    } else {
      const float2 c2 = f2unpack(f2half(c)), e2 = f2unpack(f2half(e));
      const float ta = fmaf(c2.x, inv, o), tb = fmaf(c2.y, inv, o);
      const float ha = fmaf(e2.x, fabsf(inv), pad), hb = fmaf(e2.y, fabsf(inv), pad);
      *near = make_float2(ta - ha, tb - hb);
      *far = make_float2(ta + ha, tb + hb);
    }
  };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float2 nx, fx, ny, fy, nz, fz;
    span(w[h], w[2 + h], r.inv.x, r.o.x, r.pad.x, &nx, &fx);
    span(w[4 + h], w[6 + h], r.inv.y, r.o.y, r.pad.y, &ny, &fy);
    span(w[8 + h], w[10 + h], r.inv.z, r.o.z, r.pad.z, &nz, &fz);
    const float t00 = fmaxf(max3(nx.x, ny.x, nz.x), kRayEpsilon);
    const float t01 = fmaxf(max3(nx.y, ny.y, nz.y), kRayEpsilon);
    const float t10 = fminf(min3(fx.x, fy.x, fz.x), tfar) * kBoxSlack;
    const float t11 = fminf(min3(fx.y, fy.y, fz.y), tfar) * kBoxSlack;
    tn[2 * h] = t00;
    tn[2 * h + 1] = t01;
    hit[2 * h] = t00 <= t10;
    hit[2 * h + 1] = t01 <= t11;
  }
  return make_int4((int)w[12], (int)w[13], (int)w[14], (int)w[15]);
}

__device__ __forceinline__ void addCounts(unsigned long long* dst, uint32_t v, int lane) {
  unsigned long long s = v;
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0 && s) atomicAdd(dst, s);
}

// Lanes of each warp that take rays.  With fewer rays than half the launch's
// lanes they are spread over its warps, for a warp's rounds serve one step at a
// time: 6144 rays in 192 full warps walk for 51 us, spread over all for 35 us.  Full
// warps keep constants for the lane counts (variable ones cost 4 %).
__device__ __forceinline__ int walkLanes(uint32_t n) {
  const uint32_t warps = gridDim.x * (kWalkThreads / 32);
  const uint32_t lanes = (n + warps - 1) / warps;
  return lanes > 16u ? 32 : (int)lanes;
}

// Work indices for the idle lanes of a warp (mask), one atomic; n when the
// counter has run out.  *exhausted is set once it has.
__device__ __forceinline__ uint32_t fetchWork(unsigned int* work, uint32_t idle, uint32_t n, bool* exhausted) {
  const uint32_t need = __popc(idle);
  uint32_t base = 0;
  if ((threadIdx.x & 31) == 0) base = atomicAdd(work, need);
  base = __shfl_sync(0xffffffffu, base, 0);
  if (base + need >= n) *exhausted = true;
  return base + __popc(idle & lanesBelowMask());
}

}  // namespace

// Closest hits.  The lanes of a warp walk independently: each is at an inner
// node, at a triangle, at the end of a domain, or idle, and a round of the warp
// goes through the four: new rays for the idle lanes once kRefill have gathered,
// domain ends once kSwitch have, then nodes and triangles, each as long as kStay,
// kLeaves lanes are at one.
//
// Rays walk 12 nodes and 4 triangles each, unevenly: lanes that take whole
// leaves and node runs together leave two thirds of a warp idle (7 to 13 of 32
// lanes, 5.8 ms a frame; with refilling but without the rounds 6.8 ms).  In
// rounds 15 to 19 lanes are active; then L1's requests bound the walks (75 % of
// its data pipe with 128-byte nodes in four requests, 4.02 ms; in seven, 4.35),
// so nodes take 64 bytes in two, which leaves instruction issue (70 %) and
// latency: 3.68 ms.  Runs of triangles as well as of nodes took another 3 % off the
// frame (7.05 -> 6.83 ms), rounds that go through the steps in turn instead of
// running the one most lanes are at 3 % more (6.62 ms).
template <bool kFull>
__device__ __forceinline__ void walkClosest(const RayWalkArgs& a, uint32_t n, int spread) {
  const int lane = threadIdx.x & 31;
  uint32_t visits = 0, culled = 0, nnodes = 0, ntris = 0;
  const int lanes = kFull ? 32 : spread;
  const int refill = kFull ? kRefill : (lanes * kRefill + 31) / 32, turn = kFull ? kSwitch : (lanes * kSwitch + 31) / 32;
  const int stay = kFull ? kStay : (lanes * kStay + 31) / 32, leaves = kFull ? kLeaves : (lanes * kLeaves + 31) / 32;
  const uint32_t used = kFull ? 0xffffffffu : (1u << lanes) - 1u;
  bool has = false, exhausted = n == 0;
  uint32_t rid = 0, next = 0, end = 0;
  WalkRay r{};
  uint64_t best_key = kNoHit;
  float best_t = 0.f, best_u = 0.f, best_v = 0.f;
  int best_dom = 0, dom = 0;
  uint2 stack[kStack];
  int sp = 0, cur = kDone;
  uint32_t steps = 0;
  auto pop = [&]() -> int {
    while (sp > 0) {
      const uint2 e = stack[--sp];
      if (__uint_as_float(e.y) <= best_t) return (int)e.x;
    }
    return kDone;
  };
  while (true) {
    const uint32_t idle = __ballot_sync(0xffffffffu, !has) & used;
    const int nd = __popc(idle);
    if (nd == lanes || (nd >= refill && !exhausted)) {
      if (!has && best_key != kNoHit) {
        // the finished ray's hit: TriMeshBuffer::updateIntersection
        // (src/render/trimesh_buffer.cc:328-360)
        const DomainDev* p = a.scene.domains + best_dom;
        const uint32_t* f = a.scene.faces + 3 * ((size_t)p->face_base + ((uint32_t)best_key - p->gprim_base));
        const uint32_t i0 = f[0], i1 = f[1], i2 = f[2];
        const uint32_t* colors = a.scene.colors + p->vert_base;
        const float* nb = a.scene.normals + 3 * (size_t)p->vert_base;
        const uint32_t col = interpolateColor(colors[i0], colors[i1], colors[i2], best_u, best_v);
        const V3 ns = interpolateNormal(
            v3(nb[3 * (size_t)i0], nb[3 * (size_t)i0 + 1], nb[3 * (size_t)i0 + 2]),
            v3(nb[3 * (size_t)i1], nb[3 * (size_t)i1 + 1], nb[3 * (size_t)i1 + 2]),
            v3(nb[3 * (size_t)i2], nb[3 * (size_t)i2 + 1], nb[3 * (size_t)i2 + 2]), best_u, best_v);
        a.ray_key[rid] = best_key;
        a.hit_ns[rid] = make_float4(ns.x, ns.y, ns.z, __uint_as_float(col));
        best_key = kNoHit;
      }
      if (exhausted) break;  // every lane is idle
      __syncwarp();
      const uint32_t i = fetchWork(a.work, idle, n, &exhausted);
      if ((kFull || lane < lanes) && !has && i < n) {
        const uint2 ref = a.list_ref[i];
        if (ref.y > 0) {
          rid = a.list[i];
          next = ref.x;
          end = ref.x + ref.y;
          const float4 o4 = a.rays.org[rid], d4 = a.rays.dir[rid];
          r = makeWalkRay(v3(o4.x, o4.y, o4.z), v3(d4.x, d4.y, d4.z));
          best_t = __int_as_float(0x7f800000);
          steps = 0;
          sp = 0;
          cur = kDone;
          has = true;
        }
      }
    }
    const uint32_t ends = __ballot_sync(0xffffffffu, has && cur == kDone);
    if (__popc(ends) >= turn || !__any_sync(0xffffffffu, cur != kDone)) {
      if (has && cur == kDone) {
        // the next domain of the list; the rest start beyond the hit once one does
        has = next < end;
        if (has) {
          const uint2 e = a.arena[next];
          if (beyondHit(__uint_as_float(e.y), best_t)) {
            culled += end - next;
            has = false;
          } else {
            ++next;
            ++visits;
            dom = (int)e.x;
            cur = enterDomain(a, dom, r);
          }
        }
        if (!has) nnodes += steps;
      }
    }
    if (__any_sync(0xffffffffu, cur >= 0)) {
      do {
        if (cur >= 0) {
          ++steps;
          if (sp > kStack - 3) {
            raise(a.ctr, kErrTraversalBound);
            cur = kDone;
            sp = 0;
            next = end;
          } else {
            float tn[4];
            bool hit[4];
            const int4 ch = testNode<false>(a.nodes, cur, r, best_t, tn, hit);
            // nearest child first, the others in slot order (as in traverseClosest)
            uint32_t k[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) k[c] = hit[c] ? (__float_as_uint(tn[c]) & ~3u) | (uint32_t)c : 0xffffffffu;
            const uint32_t kmin = min(__vimin3_u32(k[0], k[1], k[2]), k[3]);
            if (kmin != 0xffffffffu) {
#pragma unroll
              for (int c = 0; c < 4; ++c)
                if (hit[c] && k[c] != kmin) stack[sp++] = make_uint2((uint32_t)childAt(ch, c), k[c] & ~3u);
              cur = childAt(ch, (int)(kmin & 3u));
            } else {
              cur = pop();
            }
          }
        }
      } while (__popc(__ballot_sync(0xffffffffu, cur >= 0)) >= stay);
    }
    if (__any_sync(0xffffffffu, cur < 0 && cur != kDone)) {
      do {
        if (cur < 0 && cur != kDone) {
          // the leaf's first triangle; the leaf reference moves on to the rest
          const uint32_t v = ~(uint32_t)cur;
          const uint32_t first = v >> 3;
          ++ntris;
          const float4* tp = a.scene.tris + 3 * (size_t)first;
          const float4 ta = __ldg(tp), tb = __ldg(tp + 1), tc = __ldg(tp + 2);
          float t, u, vv;
          if (intersectTriangle(r.sh, r.org, v3(ta.x, ta.y, ta.z), v3(tb.x, tb.y, tb.z), v3(tc.x, tc.y, tc.z),
                                kRayEpsilon, __int_as_float(0x7f800000), &t, &u, &vv)) {
            const uint64_t key = packHitKey(t, a.domains[dom].gprim_base + __float_as_uint(ta.w));
            if (key < best_key) {
              best_key = key;
              best_t = t;
              best_u = u;
              best_v = vv;
              best_dom = dom;
            }
          }
          cur = (v & 7u) ? (int)~(v + 7u) : pop();
        }
      } while (__popc(__ballot_sync(0xffffffffu, cur < 0 && cur != kDone)) >= leaves);
    }
  }
  addCounts(&a.ctr->visits_radiance, visits, lane);
  addCounts(&a.ctr->visits_culled, culled, lane);
  addCounts(&a.ctr->nodes_radiance, nnodes, lane);
  addCounts(&a.ctr->tris_radiance, ntris, lane);
}

// Occlusion, in such rounds, but one that fetches rays or moves lanes on does no more
// (24 views: 109.4 ms; as for closest hits 110.1): a new ray starts in its first
// domain at once.
template <bool kFull>
__device__ __forceinline__ void walkOccluded(const RayWalkArgs& a, uint32_t n, int spread) {
  const int lane = threadIdx.x & 31;
  uint32_t visits = 0, nnodes = 0, ntris = 0;
  const int lanes = kFull ? 32 : spread;
  const int refill = kFull ? kRefill : (lanes * kRefill + 31) / 32;
  const int turn = kFull ? kShadowSwitch : (lanes * kShadowSwitch + 31) / 32;
  const int stay = kFull ? kStay : (lanes * kStay + 31) / 32, leaves = kFull ? kLeaves : (lanes * kLeaves + 31) / 32;
  const uint32_t used = kFull ? 0xffffffffu : (1u << lanes) - 1u;
  bool has = false, exhausted = n == 0;
  uint32_t rid = 0, next = 0, end = 0;
  WalkRay r{};
  float tfar = 0.f;
  int stack[kStack];
  int sp = 0, cur = kDone;
  uint32_t steps = 0;
  while (true) {
    const uint32_t idle = __ballot_sync(0xffffffffu, !has) & used;
    const int nd = __popc(idle);
    if (nd == lanes && exhausted) break;
    if (nd >= refill && !exhausted) {
      const uint32_t i = fetchWork(a.work, idle, n, &exhausted);
      if ((kFull || lane < lanes) && !has && i < n) {
        const uint2 ref = a.list_ref[i];
        if (ref.y > 0) {
          rid = a.list[i];
          next = ref.x;
          end = ref.x + ref.y;
          const float4 hp = a.sh.hitpos[rid / a.slots], d4 = a.sh.dir[rid];
          r = makeWalkRay(v3(hp.x, hp.y, hp.z), v3(d4.x, d4.y, d4.z));
          tfar = d4.w;
          steps = 0;
          sp = 0;
          has = true;
          ++visits;
          cur = enterDomain(a, (int)a.arena[next++].x, r);
        }
      }
    } else if (__popc(__ballot_sync(0xffffffffu, has && cur == kDone)) >= turn ||
               !__any_sync(0xffffffffu, cur != kDone)) {
      if (has && cur == kDone) {
        has = next < end;
        if (has) {
          ++visits;
          cur = enterDomain(a, (int)a.arena[next++].x, r);
        } else {
          nnodes += steps;
          a.sh.occluded[rid] = 0;
        }
      }
    } else {
      if (__any_sync(0xffffffffu, cur >= 0)) {
        do {
          if (cur >= 0) {
            ++steps;
            if (sp > kStack - 3) {
              raise(a.ctr, kErrTraversalBound);
              cur = kDone;
              sp = 0;
              next = end;
            } else {
              float tn[4];
              bool hit[4];
              const int4 ch = testNode<true>(a.nodes, cur, r, tfar, tn, hit);
              int nx = kDone;
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                if (!hit[c]) continue;
                if (nx != kDone) stack[sp++] = nx;
                nx = childAt(ch, c);
              }
              cur = nx != kDone ? nx : (sp > 0 ? stack[--sp] : kDone);
            }
          }
        } while (__popc(__ballot_sync(0xffffffffu, cur >= 0)) >= stay);
      }
      if (__any_sync(0xffffffffu, cur < 0 && cur != kDone)) {
        do {
          if (cur < 0 && cur != kDone) {
            const uint32_t v = ~(uint32_t)cur;
            const uint32_t first = v >> 3;
            ++ntris;
            const float4* tp = a.scene.tris + 3 * (size_t)first;
            const float4 ta = __ldg(tp), tb = __ldg(tp + 1), tc = __ldg(tp + 2);
            float t, u, vv;
            if (intersectTriangle(r.sh, r.org, v3(ta.x, ta.y, ta.z), v3(tb.x, tb.y, tb.z), v3(tc.x, tc.y, tc.z),
                                  kRayEpsilon, tfar, &t, &u, &vv)) {
              nnodes += steps;
              a.sh.occluded[rid] = 1;
              has = false;
              sp = 0;
              cur = kDone;
            } else {
              cur = (v & 7u) ? (int)~(v + 7u) : (sp > 0 ? stack[--sp] : kDone);
            }
          }
        } while (__popc(__ballot_sync(0xffffffffu, cur < 0 && cur != kDone)) >= leaves);
      }
    }
  }
  addCounts(&a.ctr->visits_shadow, visits, lane);
  addCounts(&a.ctr->nodes_shadow, nnodes, lane);
  addCounts(&a.ctr->tris_shadow, ntris, lane);
}

__global__ void __launch_bounds__(kWalkThreads, 4) kWalkClosest(RayWalkArgs a) {
  const uint32_t n = *a.count;
  const int lanes = walkLanes(n);
  if (lanes == 32) walkClosest<true>(a, n, 32);
  else walkClosest<false>(a, n, lanes);
}

__global__ void __launch_bounds__(kWalkThreads, 4) kWalkOccluded(RayWalkArgs a) {
  const uint32_t n = *a.count;
  const int lanes = walkLanes(n);
  if (lanes == 32) walkOccluded<true>(a, n, 32);
  else walkOccluded<false>(a, n, lanes);
}

// One thread per domain: the box of its root's children.
__global__ void kWalkDomains(const BvhNode4* __restrict__ nodes, const DomainDev* __restrict__ domains, int D,
                             WalkDomain* out) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= D) return;
  const BvhNode4& r = nodes[domains[d].node_base];
  const float* planes[6] = {r.lox, r.hix, r.loy, r.hiy, r.loz, r.hiz};
  WalkDomain w;
  for (int k = 0; k < 3; ++k) {
    float lo = INFINITY, hi = -INFINITY;
    for (int q = 0; q < 4; ++q) {
      if (r.child[q] == kEmptyChild) continue;
      lo = fminf(lo, planes[2 * k][q]);
      hi = fmaxf(hi, planes[2 * k + 1][q]);
    }
    const float c = 0.5f * lo + 0.5f * hi, h = 0.5f * hi - 0.5f * lo;
    const bool ok = isfinite(c) && isfinite(h) && h > 0.0f;
    w.centre[k] = isfinite(c) ? c : 0.0f;
    w.half[k] = ok ? h : 1.0f;
  }
  w.root = domains[d].node_base;
  w.gprim_base = domains[d].gprim_base;
  out[d] = w;
}

// The domain of a node: the last one whose first node is <= k.
__device__ __forceinline__ int domainOfNode(const DomainDev* __restrict__ domains, int D, uint32_t k) {
  int lo = 0, hi = D - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((uint32_t)domains[mid].node_base <= k) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Planes lo, hi of a box along an axis, relative to the domain: centre and half
// extent.  The relative planes are within 2^-22 of their true values (a subtraction
// and a product of values of at most 1), which 1e-6 more extent covers; e is rounded
// up to half.  Infinite or NaN planes, or outside the domain: everything along the
// axis (+inf).
__device__ __forceinline__ void relativeBox(float lo, float hi, float centre, float scale, __half* c, __half* e) {
  const float a = (lo - centre) * scale, b = (hi - centre) * scale;
  const __half m = __float2half_rn(0.5f * a + 0.5f * b);
  const float need = fmaxf(b - __half2float(m), __half2float(m) - a) + 1e-6f;
  const bool ok = need >= 0.0f && fabsf(a) <= 1.0001f && fabsf(b) <= 1.0001f;
  *c = ok ? m : __ushort_as_half(0);
  *e = ok ? __float2half_ru(need) : __ushort_as_half(0x7c00);
}

// Children follow their parent in the domain's nodes, leaves lie in its triangles:
// the walks rely on it and check nothing.
__device__ __forceinline__ bool innerChild(int c, uint32_t parent, int num_nodes) {
  return c >= 0 && (uint32_t)c > parent && c < num_nodes;
}

// The areas of a node's children as shares of the node's own, how often a ray that has
// entered the node enters them: by exact boxes (x) and by relative ones (y).
__device__ __forceinline__ void childShares(const BvhNode4& nd, const WalkDomain& wd, float2 share[4]) {
  const float* planes[6] = {nd.lox, nd.hix, nd.loy, nd.hiy, nd.loz, nd.hiz};
  // half extents of the children and of their union, exact [0] and relative [1]
  float ext[2][4][3], lo[2][3], hi[2][3];
  for (int x = 0; x < 3; ++x) lo[0][x] = lo[1][x] = INFINITY, hi[0][x] = hi[1][x] = -INFINITY;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const float l = planes[2 * x][q], h = planes[2 * x + 1][q];
      __half hc, he;
      relativeBox(l, h, wd.centre[x], 1.0f / wd.half[x], &hc, &he);
      // (an axis that spans everything: the domain's size)
      const float c = __half2float(hc) * wd.half[x], e = (__hisinf(he) ? 1.0f : __half2float(he)) * wd.half[x];
      ext[0][q][x] = 0.5f * h - 0.5f * l;
      ext[1][q][x] = e;
      if (nd.child[q] == kEmptyChild) continue;
      lo[0][x] = fminf(lo[0][x], 0.5f * l), hi[0][x] = fmaxf(hi[0][x], 0.5f * h);
      lo[1][x] = fminf(lo[1][x], 0.5f * c - 0.5f * e), hi[1][x] = fmaxf(hi[1][x], 0.5f * c + 0.5f * e);
    }
  }
  auto halfArea = [](float x, float y, float z) { return x * y + y * z + z * x; };
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    // in units of the union's longest side, so that no product leaves the floats
    float all[3];
    for (int x = 0; x < 3; ++x) all[x] = hi[v][x] - lo[v][x];
    const float unit = 1.0f / max3(all[0], all[1], all[2]);
    const float area = 1.0f / halfArea(all[0] * unit, all[1] * unit, all[2] * unit);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float* x = ext[v][q];
      const float s = halfArea(x[0] * unit, x[1] * unit, x[2] * unit) * area;
      (v == 0 ? share[q].x : share[q].y) = s >= 0.0f && s <= 1.0f ? s : 1.0f;  // 1: no area, or no number
    }
  }
}

// Whether half precision relative to the domain holds a node's surroundings too
// loosely.  Boxes far smaller than their domain (a detailed object on a ground plane, a
// stray vertex far out) grow until every child of a node is entered: 582 nodes a visit
// for 3.4, 82 ms a frame for 0.42.  A ray in node k visits it and, as often as their
// areas are of its own, its children and theirs; where the relative boxes make that
// more than 1.5 times the exact ones' and 1.2 nodes, the scene keeps the queues.
// Frames of 1280x960, 4 spp, by walks and by queues, and the most nodes above 1.5
// times: 0.79 and 1.12 ms at -0.5 (even meshes), 1.08 and 1.39 at -0.2, 0.94 and 0.93
// at 0.0, 1.16 and 1.30 at 0.9, 1.31 and 0.93 at 1.4, 1.30 and 1.26 at 3.0.
__device__ __forceinline__ bool looseNode(const BvhNode4* __restrict__ nodes, uint32_t k, const BvhNode4& nd,
                                          const WalkDomain& wd, int num_nodes) {
  const uint32_t root = (uint32_t)wd.root;
  float2 share[4], visits = make_float2(1.0f, 1.0f);
  childShares(nd, wd, share);
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    if (!innerChild(nd.child[q], k - root, num_nodes)) continue;
    const uint32_t c = root + (uint32_t)nd.child[q];
    const BvhNode4 below = nodes[c];
    float2 sub[4], in = make_float2(1.0f, 1.0f);
    childShares(below, wd, sub);
    for (int r = 0; r < 4; ++r)
      if (innerChild(below.child[r], c - root, num_nodes)) {
        in.x += sub[r].x;
        in.y += sub[r].y;
      }
    visits.x += share[q].x * in.x;
    visits.y += share[q].y * in.y;
  }
  return visits.y > 1.5f * visits.x + 1.2f;
}

// One thread per node: the boxes relative to the domain.
__global__ void kWalkNodes(const BvhNode4* __restrict__ nodes, uint32_t num_nodes, const DomainDev* __restrict__ domains,
                           int D, const WalkDomain* __restrict__ wdomains, WalkNode* out, int* bad, int* loose) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= num_nodes) return;
  const int dom = domainOfNode(domains, D, k);
  const WalkDomain wd = wdomains[dom];
  const uint32_t tri_base = (uint32_t)domains[dom].tri_base;
  const BvhNode4 nd = nodes[k];
  if (looseNode(nodes, k, nd, wd, domains[dom].num_nodes)) *loose = 1;
  WalkNode w;
  auto axis = [&](int x, const float* l, const float* h, __half* c, __half* e) {
    const float centre = wd.centre[x], scale = 1.0f / wd.half[x];
    for (int q = 0; q < 4; ++q) {
      c[q] = __ushort_as_half(0);
      e[q] = __ushort_as_half(0xfc00);  // -inf: an unused slot is not entered
      if (nd.child[q] != kEmptyChild) relativeBox(l[q], h[q], centre, scale, &c[q], &e[q]);
    }
  };
  axis(0, nd.lox, nd.hix, w.cx, w.ex);
  axis(1, nd.loy, nd.hiy, w.cy, w.ey);
  axis(2, nd.loz, nd.hiz, w.cz, w.ez);
  for (int q = 0; q < 4; ++q) {
    const int c = nd.child[q];
    const uint32_t leaf = ~(uint32_t)c;
    const bool ok = c == kEmptyChild || (c >= 0 ? innerChild(c, k - (uint32_t)wd.root, domains[dom].num_nodes)
                                                : (leaf >> 3) + (leaf & 7u) < (uint32_t)domains[dom].num_tris);
    if (!ok) *bad = 1;
    // an unused slot holds the domain's first triangle: a ray whose distances in the
    // domain overflow along every axis (extents near the largest float) enters all
    // four slots, and one more test of a triangle changes nothing
    if (!ok || c == kEmptyChild) w.child[q] = (int)~(tri_base << 3);
    else if (c >= 0) w.child[q] = c + wd.root;
    else w.child[q] = (int)~(leaf + (tri_base << 3));
  }
  out[k] = w;
}

void launchWalkNodes(cudaStream_t s, const BvhNode4* nodes, uint32_t num_nodes, const DomainDev* domains, int D,
                     WalkDomain* wdomains, WalkNode* out, int* bad, int* loose) {
  if (num_nodes == 0) return;
  kWalkDomains<<<(D + 127) / 128, 128, 0, s>>>(nodes, domains, D, wdomains);
  kWalkNodes<<<(num_nodes + 127) / 128, 128, 0, s>>>(nodes, num_nodes, domains, D, wdomains, out, bad, loose);
}

template <int kKind>
static void launchLists(cudaStream_t s, const RayWalkArgs& a, int nblocks) {
  // primary rays read their bin's domains instead
  static_assert((kGroupMax / 64 + kGroupMax / 4) * kNodeStride * 16 <= 48 * 1024, "group table in shared memory");
  const size_t bytes = kKind == kListPrimary ? 0 : (size_t)(a.groups.l1 + a.groups.l2) * kNodeStride * sizeof(float4);
  kListDomains<kKind><<<nblocks, kWalkThreads, bytes, s>>>(a);
}

void launchListDomains(cudaStream_t s, const RayWalkArgs& a, int nblocks) {
  if (a.shadow) launchLists<kListShadow>(s, a, nblocks);
  else if (a.bin_start) launchLists<kListPrimary>(s, a, nblocks);
  else launchLists<kListBounce>(s, a, nblocks);
}

void launchWalkClosest(cudaStream_t s, const RayWalkArgs& a, int nblocks) {
  kWalkClosest<<<nblocks, kWalkThreads, 0, s>>>(a);
}

void launchWalkOccluded(cudaStream_t s, const RayWalkArgs& a, int nblocks) {
  kWalkOccluded<<<nblocks, kWalkThreads, 0, s>>>(a);
}

}  // namespace spray
