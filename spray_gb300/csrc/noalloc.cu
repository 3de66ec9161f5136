// Allocation-free scheduling entry point.
//
// Some callers cannot allocate device memory while they run: a renderer that
// owns a fixed device budget carved out at start-up (cudaMalloc could fail or
// push it over its share), or a host runtime whose GPU memory is handed out by
// its own pool (a cudaMalloc behind its back breaks its accounting, and
// cudaFree synchronises the whole device).  spray_gpu_schedule_static lets
// such callers run the speculative scheduler -- slab test of every ray against
// every domain box, (t, id)-sorted domain lists, stable partition into
// per-domain queues -- with no allocation: the scheduler's scratch lives in
// one file-scope device array of fixed size, and the caller passes only inputs
// and outputs.
//
// Limits and sharing:
//  * at most kStaticMaxRays rays, kStaticMaxDomains domains and
//    kStaticMaxEntries queue entries per call; larger requests are rejected
//    with SPRAY_GPU_EINVAL before any GPU work;
//  * the array (about 14 MB) stays allocated on every device that used this
//    library until the process exits;
//  * every call uses the same array and leaves its contents behind; the
//    counters that must start at zero are cleared by each call, so calls that
//    overlap on the GPU (different streams, or different host threads on one
//    device) race and corrupt each other -- serialise them;
//  * the call reads its entry count back and synchronises the caller's
//    stream before it returns, so it must not be made while that stream (or
//    the device) is being captured into a CUDA graph;
//  * the first call on a device looks up the array's device address
//    (cudaGetSymbolAddress) with that device current and keeps it for the
//    life of the process; after a cudaDeviceReset the kept address is stale,
//    so do not call this entry point again in a process that reset a device
//    it used.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <string>

#include "../../include/spray_gpu.h"
#include "domain_walk.cuh"
#include "kernels.cuh"
#include "spray_math.cuh"

namespace spray {

int fail(int code, const std::string& msg);

namespace {

constexpr int kStaticMaxRays = 1 << 18;
constexpr int kStaticMaxDomains = 256;
constexpr int kStaticMaxEntries = 1 << 20;
// Ray chunks, one warp each, with a histogram row of their own: 32 rays a chunk
// up to 65536 rays, 128 at the most.
constexpr int kStaticChunks = 2048;
constexpr int kStaticScanKeys = 4;  // domains per block of the histogram scan

struct StaticScratch {
  uint32_t list[kStaticMaxRays];
  uint2 arena[kStaticMaxEntries];
  uint32_t list_off[kStaticMaxRays];
  uint32_t list_cnt[kStaticMaxRays];
  uint32_t hist[kStaticMaxDomains * kStaticChunks];
  uint32_t key_total[kStaticMaxDomains];
  // cleared by each call
  unsigned long long arena_top;
  uint32_t count;
  uint32_t ticket;
  uint32_t num_entries;
  Counters ctr;
};

// The scheduler's scratch, laid out as a StaticScratch: one per device,
// shared by every call.  Host code must not use this name as an address.
static __device__ __align__(256) unsigned char g_sched_scratch[sizeof(StaticScratch)];

// Host copy of the array's device address, per device.
std::mutex g_mutex;
StaticScratch* g_scratch_addr[64] = {nullptr};

// The sorted domain lists of a chunk of rays per warp, into the arena, and the
// chunk's counts per domain.  Every block makes the boxes' group table in shared
// memory (domains in index order; groupDomains then tests a sixteenth to all of
// them, four at a time).  65521 rays over 125 boxes: 27 us, against 177 with every box
// tested exactly by 512 warps.
constexpr int kStaticThreads = 256;

__global__ void __launch_bounds__(kStaticThreads) kStaticLists(StaticScratch* s, const float* __restrict__ bounds, int D,
                                                               const float4* __restrict__ ray_org,
                                                               const float4* __restrict__ ray_dir, uint32_t n, int nch) {
  __shared__ float4 table[(kStaticMaxDomains / 64 + kStaticMaxDomains / 4) * kNodeStride];
  __shared__ float sbox[6 * kStaticMaxDomains];
  __shared__ uint32_t hist[kStaticThreads / 32][kStaticMaxDomains];
  const int n1 = (D + 63) / 64, n2 = (D + 3) / 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = threadIdx.x; k < 6 * D; k += blockDim.x) sbox[k] = bounds[k];
  for (int k = lane; k < D; k += 32) hist[warp][k] = 0u;
  __syncthreads();
  // slot c of a node: plane p at float 4 * p + c, the domain at int 24 + c; one
  // thread per slot and axis.  An inverted box spans both of its planes, a NaN
  // bound everything, so that nothing the exact test accepts is left out; an unused
  // slot names a domain that exists (a ray of no finite origin meets every slot).
  for (int q = threadIdx.x; q < 12 * (n1 + n2); q += blockDim.x) {
    const int k = q / 3, c = q - 3 * k;
    const bool group = k < 4 * n1;
    const int d0 = group ? 16 * k : k - 4 * n1, d1 = min(group ? d0 + 16 : d0 + 1, D);
    float lo = INFINITY, hi = -INFINITY;
    for (int d = d0; d < d1; ++d) {
      const float a = sbox[6 * d + c], b = sbox[6 * d + 3 + c];
      const bool bad = a != a || b != b;
      lo = fminf(lo, bad ? -INFINITY : fminf(a, b));
      hi = fmaxf(hi, bad ? INFINITY : fmaxf(a, b));
    }
    float* node = reinterpret_cast<float*>(table + (k >> 2) * kNodeStride);
    node[8 * c + (k & 3)] = lo;
    node[8 * c + 4 + (k & 3)] = hi;
    if (c == 0) reinterpret_cast<int*>(node)[24 + (k & 3)] = min(d0, D - 1);
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0) s->count = n;
  const int ch = blockIdx.x * (kStaticThreads / 32) + warp;
  if (ch >= nch) return;
  const uint32_t size = (uint32_t)chunkSize(n, nch);
  const uint32_t r0 = min(n, (uint32_t)ch * size), r1 = min(n, r0 + size);
  uint32_t* h = hist[warp];
  for (uint32_t base = r0; base < r1; base += 32) {
    const uint32_t i = base + lane;
    DomainList list;
    if (i < r1) {
      const float4 o = ray_org[i], d = ray_dir[i];
      const V3 org = v3(o.x, o.y, o.z), inv = v3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
      groupDomains(table, n1, n2, makeBoxRay(org, inv), INFINITY, [&](int dom) {
        float t;
        // the keys order -0 like 0: the sign goes below the domain
        if (slabTest(&sbox[6 * dom], &sbox[6 * dom + 3], org, inv, kRayEpsilon, INFINITY, &t))
          list.insert(t, 2 * dom + (__float_as_uint(t) == 0x80000000u), &s->ctr);
      });
    }
    uint32_t total;
    const uint32_t pos = warpScan((uint32_t)list.n, &total);
    unsigned long long b = 0;
    if (lane == 0 && total) b = atomicAdd(&s->arena_top, (unsigned long long)total);
    b = __shfl_sync(0xffffffffu, b, 0);
    const bool fits = b + total <= kStaticMaxEntries;
    if (!fits && lane == 0) atomicAdd(&s->ctr.arena_overflows, 1ull);
    if (i < r1) {
      s->list[i] = i;
      s->list_off[i] = (uint32_t)(b + pos);
      s->list_cnt[i] = fits ? (uint32_t)list.n : 0u;
      for (int j = 0; fits && j < list.n; ++j) {
        const uint64_t k = list.key[j];
        const uint32_t d = (uint32_t)k >> 1;
        const float t = ((uint32_t)k & 1u) ? -0.0f : orderedFloat((uint32_t)(k >> 32));
        s->arena[b + pos + j] = make_uint2(d | ((uint32_t)j << 16), __float_as_uint(t));
        atomicAdd(&h[d], 1u);
      }
    }
  }
  __syncwarp();
  for (int k = lane; k < D; k += 32) s->hist[(size_t)ch * D + k] = h[k];
}

// Per domain the exclusive scan of its chunks' counts in place, kStaticScanKeys
// domains a block, and in the block that ends last the scan of the totals: the
// queues' starts and the entry count (0 when they exceed the caller's capacity).
// The queue scheduler's three-kernel scan (sched.cu) is made for tables of 30 MB;
// this one is at most 2 MB and its launches cost more than its bytes (a call with
// 65521 rays over 125 boxes 80 -> 63 us).
__global__ void __launch_bounds__(1024) kStaticScan(StaticScratch* s, int D, int nch, unsigned long long entry_cap,
                                                    uint32_t* domain_start) {
  static_assert(kStaticChunks <= 2048, "two chunks per thread");
  __shared__ uint32_t wsum[32][kStaticScanKeys];
  __shared__ int is_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d0 = blockIdx.x * kStaticScanKeys, nd = min(kStaticScanKeys, D - d0);
  const int c0 = 2 * threadIdx.x;
  uint32_t v[2][kStaticScanKeys], pos[kStaticScanKeys];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int k = 0; k < kStaticScanKeys; ++k)
      v[c][k] = c0 + c < nch && k < nd ? s->hist[(size_t)(c0 + c) * D + d0 + k] : 0u;
#pragma unroll
  for (int k = 0; k < kStaticScanKeys; ++k) {
    uint32_t total;
    pos[k] = warpScan(v[0][k] + v[1][k], &total);
    if (lane == 0) wsum[warp][k] = total;
  }
  __syncthreads();
  if (warp < nd) {
    uint32_t total;
    const uint32_t x = warpScan(wsum[lane][warp], &total);
    wsum[lane][warp] = x;
    if (lane == 0) s->key_total[d0 + warp] = total;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kStaticScanKeys; ++k) {
    if (k >= nd) break;
    const uint32_t p = wsum[warp][k] + pos[k];
    if (c0 < nch) s->hist[(size_t)c0 * D + d0 + k] = p;
    if (c0 + 1 < nch) s->hist[(size_t)(c0 + 1) * D + d0 + k] = p + v[0][k];
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(&s->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  static_assert(kStaticMaxDomains <= 1024, "one thread per total");
  const uint32_t t = threadIdx.x < D ? __ldcg(&s->key_total[threadIdx.x]) : 0u;
  uint32_t total;
  const uint32_t x = warpScan(t, &total);
  if (lane == 0) wsum[warp][0] = total;
  __syncthreads();
  uint32_t run = 0;
  for (int w = 0; w < warp; ++w) run += wsum[w][0];
  if (threadIdx.x < D) domain_start[threadIdx.x] = run + x;
  if (threadIdx.x == D - 1) {
    const uint32_t all = run + x + t;
    domain_start[D] = all;
    if (all > entry_cap) atomicAdd(&s->ctr.entry_overflows, 1ull);
    s->num_entries = all > entry_cap ? 0u : all;
  }
}

}  // namespace
}  // namespace spray

extern "C" int spray_gpu_schedule_static(const float* domain_bounds, int32_t num_domains,
                                         const float* ray_org, const float* ray_dir, int32_t num_rays,
                                         int32_t list_size, uint32_t* entries,
                                         int64_t entry_capacity, uint32_t* domain_start,
                                         int64_t* num_entries, void* stream) {
  using namespace spray;
  try {
  if (!domain_bounds || !ray_org || !ray_dir || !entries || !domain_start || !num_entries)
    return fail(SPRAY_GPU_EINVAL, "null argument");
  if (num_domains <= 0 || num_domains > kStaticMaxDomains)
    return fail(SPRAY_GPU_EINVAL, "num_domains must be in [1, " + std::to_string(kStaticMaxDomains) + "]");
  if (num_rays < 0 || num_rays > kStaticMaxRays)
    return fail(SPRAY_GPU_EINVAL, "num_rays must be in [0, " + std::to_string(kStaticMaxRays) + "]");
  if (list_size <= 0 || list_size > kMaxList) return fail(SPRAY_GPU_EINVAL, "list_size must be in [1, 32]");
  if (entry_capacity < 0) return fail(SPRAY_GPU_EINVAL, "negative entry capacity");
  if ((((uintptr_t)ray_org) | ((uintptr_t)ray_dir) | ((uintptr_t)entries)) & 15u)
    return fail(SPRAY_GPU_EINVAL, "ray and entry arrays must be 16-byte aligned");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(SPRAY_GPU_ECUDA, cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return fail(SPRAY_GPU_ECUDA, "device ordinal out of range");
  StaticScratch* s = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_scratch_addr[dev]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_sched_scratch);
      if (e != cudaSuccess) return fail(SPRAY_GPU_ECUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      g_scratch_addr[dev] = static_cast<StaticScratch*>(p);
    }
    s = g_scratch_addr[dev];
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int D = num_domains;
  // one warp per chunk of 32 rays, more rays a chunk once the chunks run out
  const int nch = std::max(1, std::min(kStaticChunks, (num_rays + 31) / 32));
  e = cudaMemsetAsync(&s->arena_top, 0, sizeof(StaticScratch) - offsetof(StaticScratch, arena_top), st);
  if (e != cudaSuccess) return fail(SPRAY_GPU_ECUDA, cudaGetErrorString(e));
  constexpr int wpb = kStaticThreads / 32;
  kStaticLists<<<(nch + wpb - 1) / wpb, kStaticThreads, 0, st>>>(
      s, domain_bounds, D, reinterpret_cast<const float4*>(ray_org), reinterpret_cast<const float4*>(ray_dir),
      (uint32_t)num_rays, nch);
  SchedArgs a{};
  a.shadow = 0;
  a.count = &s->count;
  a.list = s->list;
  a.slots = 1;
  a.order_by_depth = 0;
  a.list_size = list_size;
  a.arena = s->arena;
  a.list_off = s->list_off;
  a.list_cnt = s->list_cnt;
  a.hist = s->hist;
  a.nchunks = nch;
  a.pack_depth = 1;  // ray | position << 26 | origin << 31, as the header documents
  a.entries = reinterpret_cast<uint2*>(entries);
  a.entry_cap = (unsigned long long)entry_capacity;
  a.key_start = domain_start;
  a.num_entries = &s->num_entries;
  a.ctr = &s->ctr;
  a.key_relative = 1;
  kStaticScan<<<(D + kStaticScanKeys - 1) / kStaticScanKeys, 1024, 0, st>>>(s, D, nch, a.entry_cap, domain_start);
  launchSchedScatter(st, a, D, nch);
  // entry count and counters lie together
  constexpr size_t tail = offsetof(StaticScratch, num_entries);
  unsigned char back[sizeof(StaticScratch) - tail];
  e = cudaMemcpyAsync(back, reinterpret_cast<unsigned char*>(s) + tail, sizeof(back), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return fail(SPRAY_GPU_ECUDA, cudaGetErrorString(e));
  uint32_t ne = 0;
  Counters ctr;
  std::memcpy(&ne, back, sizeof(ne));
  std::memcpy(&ctr, back + (offsetof(StaticScratch, ctr) - tail), sizeof(ctr));
  if (ctr.list_overflows) return fail(SPRAY_GPU_EOVERFLOW, "a ray overlapped more than 32 domains");
  if (ctr.arena_overflows) return fail(SPRAY_GPU_EOVERFLOW, "more queue entries than the static scratch holds");
  if (ctr.entry_overflows) return fail(SPRAY_GPU_EOVERFLOW, "entry_capacity too small");
  *num_entries = (int64_t)ne;
  return SPRAY_GPU_OK;
  } catch (const std::exception& ex) {
    // no C++ exception crosses the C boundary (launch configuration errors,
    // allocation failures of the error strings)
    return fail(SPRAY_GPU_ECUDA, ex.what());
  }
}
