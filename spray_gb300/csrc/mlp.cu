// Tensor-core kernels of the learned domain-order proposal (mlp.cuh).
//
// Operands live in shared memory without swizzle: 8-row x 16-byte core matrices,
// those of a row group adjacent (128 bytes), the row groups columns / 8 * 128 bytes
// apart.  Read with K along the row (K-major) that is leading byte offset 128 and
// the row-group pitch as stride byte offset; read transposed (MN-major: K down the
// rows) the two change places, so that one copy of the activations, of dZ and of
// the weights serves the forward and the backward products.  One thread issues tcgen05.mma (M = 128, K = 16 per
// instruction, BF16 inputs, FP32 accumulator in tensor memory) and commits to
// an mbarrier; the four warps read their 32 accumulator lanes back with
// tcgen05.ld.  Every mbarrier wait is bounded (one second); a wait that gives
// up sets Net::error; the kernel then runs to its end without waiting for another
// product, waits once more, as long, for those in flight and frees its tensor memory.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "mlp.cuh"
#include "spray_math.cuh"

namespace spray {
namespace mlp {
namespace {

constexpr int kReduceThreads = 256;          // threads per block of kReduceAdam
constexpr uint64_t kWaitNs = 1000000000ull;  // bound of one mbarrier wait

__device__ __forceinline__ uint32_t smemAddr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t globalTimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void tmemAlloc(uint32_t dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmemDealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void fenceBeforeSync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fenceAfterSync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// generic-proxy stores to shared memory become visible to the tensor cores
__device__ __forceinline__ void fenceProxyAsync() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbarInit(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbarTryWait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ bool mbarWait(uint32_t bar, uint32_t parity) {
  if (mbarTryWait(bar, parity)) return true;
  const uint64_t t0 = globalTimer();
  while (!mbarTryWait(bar, parity))
    if (globalTimer() - t0 > kWaitNs) return false;
  return true;
}

// Shared-memory matrix descriptor: start, leading and stride byte offsets
// (all >> 4), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, transposed
// (MN-major) A at bit 15 and B at bit 16, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idescBf16(int M, int N, bool ta, bool tb) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)ta << 15) | ((uint32_t)tb << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// A converged warp calls mma and commit; the lane with `on` issues.  (In a branch of
// one lane the operands are moved to uniform registers one by one before each
// product: 100 cycles a product.)
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc, uint32_t on) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(on)
      : "memory");
}

// The same with A in tensor memory: lane = row, a column = two elements along K.
__device__ __forceinline__ void mmaTmem(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc, uint32_t on) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(on)
      : "memory");
}

__device__ __forceinline__ void commit(uint32_t bar, uint32_t on) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
      " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
      "r"(on)
      : "memory");
}

// An operand: its address, the pitch of its row groups (columns / 8 * 128 bytes)
// and whether K runs down its rows.
struct Operand {
  uint32_t addr, pitch;
  bool transposed;
  __device__ __forceinline__ uint64_t at(int k) const {  // the k-th 16 of K
    return transposed ? sdesc(addr + 2 * pitch * k, pitch, 128u) : sdesc(addr + 256u * k, 128u, pitch);
  }
};

// D (M = 128 x N) (+)= A (128 x K) * B (N x K)^T, issued by one lane of a warp.  A
// transposed A of fewer than 128 columns reads on into what follows it (row groups
// 16 x 128 bytes long, inside the kernel's shared memory): rows of D nobody reads.
__device__ __forceinline__ void gemm(uint32_t d, Operand a, Operand b, int K, int N, bool accumulate,
                                     uint32_t on) {
  const uint32_t id = idescBf16(128, N, a.transposed, b.transposed);
#pragma unroll
  for (int k = 0; k < K / 16; ++k) mma(d, a.at(k), b.at(k), id, (accumulate || k > 0) ? 1u : 0u, on);
}

__device__ __forceinline__ void gemmTmem(uint32_t d, uint32_t a, Operand b, int K, int N, uint32_t on) {
  const uint32_t id = idescBf16(128, N, false, b.transposed);
#pragma unroll
  for (int k = 0; k < K / 16; ++k) mmaTmem(d, a + 8 * k, b.at(k), id, k > 0 ? 1u : 0u, on);
}

// N consecutive columns of this thread's lane, written.
__device__ __forceinline__ void tmemSt8(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmemStWait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// N consecutive fp32 accumulator columns of this thread's lane.
__device__ __forceinline__ void tmemLd8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmemLd16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
        "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Barrier `id` over `count` threads, by whole warps; barArrive does not wait.
__device__ __forceinline__ void barSync(int id, int count) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void barArrive(int id, int count) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Byte offset of element (r, c) of an operand with kg = columns / 8.
__host__ __device__ __forceinline__ uint32_t opOff(int r, int c, int kg) {
  return (uint32_t)((((r >> 3) * kg + (c >> 3)) << 7) + ((r & 7) << 4) + ((c & 7) << 1));
}

__device__ __forceinline__ uint32_t packBf16(float a, float b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&p);
}

// max(a + ba, 0), max(b + bb, 0) as bfloat16 (rounding is monotonic, so the
// maximum after it is the rounded maximum; a NaN becomes 0 as with fmaxf)
__device__ __forceinline__ uint32_t reluBf16(float a, float b, float ba, float bb) {
  const __nv_bfloat162 p = __hmax2(__floats2bfloat162_rn(a + ba, b + bb), __floats2bfloat162_rn(0.0f, 0.0f));
  return *reinterpret_cast<const uint32_t*>(&p);
}

// Eight accumulators of a hidden layer -> eight activations.
__device__ __forceinline__ uint4 activate8(const float* z, const float* bias) {
  const float4 b0 = *reinterpret_cast<const float4*>(bias), b1 = *reinterpret_cast<const float4*>(bias + 4);
  uint4 q;
  q.x = reluBf16(z[0], z[1], b0.x, b0.y);
  q.y = reluBf16(z[2], z[3], b0.z, b0.w);
  q.z = reluBf16(z[4], z[5], b1.x, b1.y);
  q.w = reluBf16(z[6], z[7], b1.z, b1.w);
  return q;
}

// All bits of each half that is above zero.
__device__ __forceinline__ uint32_t positive(uint32_t v) {
  return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&v), __floats2bfloat162_rn(0.0f, 0.0f));
}

__device__ __forceinline__ uint4 pack8(const float* z) {
  uint4 q;
  q.x = packBf16(z[0], z[1]);
  q.y = packBf16(z[2], z[3]);
  q.z = packBf16(z[4], z[5]);
  q.w = packBf16(z[6], z[7]);
  return q;
}

// All weights [out][64] and biases of the fp32 vector -> shared memory: W1..W3 at
// op (8 KB each), W4 after them, the four bias vectors at bias.  A thread's loads
// are all in flight before it stores (a loop of them took 7 400 cycles, this one
// 2 900).
template <int kThreads>
struct NetStage {
  static constexpr int kPairs = (3 * kHid * kK + kOutPad * kHid) / 2, kEach = (kPairs + kThreads - 1) / kThreads;
  static_assert(kHid * kK == 4096 && kW2 - kW1 == 4096 + 64 && kW4 - kW3 == 4096 + 64, "pair p of layer p / 2048");
  float v[kEach][2], b;
  int tid;
  __device__ __forceinline__ explicit NetStage(int thread) : tid(thread) {}
  __device__ __forceinline__ void load(const float* params) {
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
      const int p = tid + k * kThreads;
      if (p < kPairs) {
        v[k][0] = params[2 * p + 64 * (p >> 11)];
        v[k][1] = params[2 * p + 64 * (p >> 11) + 1];
      }
    }
    if (tid < 3 * kHid + kOutPad)
      b = params[tid < 3 * kHid ? kB1 + tid + (tid >> 6) * 4096 : kB4 + tid - 3 * kHid];
  }
  __device__ __forceinline__ void store(uint8_t* op, float* bias) const {
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
      const int p = tid + k * kThreads;
      if (p < kPairs)
        *reinterpret_cast<uint32_t*>(op + 8192 * (p >> 11) + opOff((p >> 5) & 63, (2 * p) & 63, 8)) =
            packBf16(v[k][0], v[k][1]);
    }
    if (tid < 3 * kHid + kOutPad) bias[tid] = b;
  }
};

// What the features take from a domain's box, in the scene box normalised to
// [-1, 1]: its centre, its half diagonal r and 1 / r (0 for r = 0).
__device__ __forceinline__ void boxRecord(const float* b, const Norm& nm, float4* rec, float* ir) {
  float pc[3], hh[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float lo = (b[c] - nm.centre[c]) * nm.scale;
    const float hi = (b[3 + c] - nm.centre[c]) * nm.scale;
    pc[c] = (lo + hi) * 0.5f;
    hh[c] = (hi - lo) * 0.5f;
  }
  const float r = sqrtf((hh[0] * hh[0] + hh[1] * hh[1]) + hh[2] * hh[2]);
  *rec = make_float4(pc[0], pc[1], pc[2], r);
  *ir = r > 0.0f ? 1.0f / r : 0.0f;
}

// Records of the first kBoxCache domains in shared memory: those the
// caller vouches for when the kernel starts, others as candidates name them (a caller
// of the entry points does not say how many boxes there are).  `ir` doubles as the
// flag: it is written after the record, and 1 / r never has kNoBox's bits.  Every
// thread that misses writes the same values.  Domains beyond the cache are
// computed at each use.
constexpr int kBoxCache = 1024;
constexpr uint32_t kNoBox = 0xffffffffu;
constexpr int kBoxBytes = kBoxCache * 20;
struct BoxCache {
  float4* rec;
  uint32_t* ir;
  __device__ explicit BoxCache(uint8_t* sm)
      : rec(reinterpret_cast<float4*>(sm)), ir(reinterpret_cast<uint32_t*>(sm + kBoxCache * 16)) {}
  // by `threads` threads; four boxes of a thread are read before the first is used
  __device__ __forceinline__ void init(const Net& net, int tid, int threads) {
    const int known = min(net.more_boxes ? (int)*net.more_boxes : net.num_boxes, kBoxCache);
    for (int i0 = tid; i0 < kBoxCache; i0 += 4 * threads) {
      float b[4][6];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int k = 0; k < 6; ++k) b[q][k] = i0 + q * threads < known ? net.boxes[6 * (i0 + q * threads) + k] : 0.0f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = i0 + q * threads;
        if (i >= kBoxCache) break;
        float inv;
        boxRecord(b[q], net.norm, &rec[i], &inv);
        ir[i] = i < known ? __float_as_uint(inv) : 0u + kNoBox;
      }
    }
  }
};

// A row: ray, candidates, label.
struct Row {
  float o[3], d[3];
  uint32_t cand[kCand];
  int ncand, label;
};

// Features of candidates j0 and j0 + 1 of a row whose origin is `on` in the
// normalised box, per candidate j (zeros when absent)
//   along  distance along the ray to the point closest to the box centre
//   miss   distance of the ray from the box centre there
//   r      half diagonal of the box
//   miss / r (at most 4), along / r (within [-4, 4]), 1 (present)
// passed to put(column, value, value of column + 1).  Whether a ray meets a
// domain's surface depends mostly on how close it passes the domain's centre
// relative to its size, which a small ReLU network cannot form from box corners;
// these are the same inputs (origin, direction, boxes) put in that form.  Every
// operation rounds once (-fmad=false; IEEE division and square root), as the numpy
// restatement does.
template <class Put>
__device__ __forceinline__ void candFeatures(const float* on, const float* d, const uint32_t* cand, int j0, int ncand,
                                             const Net& net, const BoxCache& cache, Put&& put) {
  uint32_t u[2];
  bool miss_any = false;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    u[j] = 0u;
    if (j0 + j < ncand) u[j] = cand[j] < kBoxCache ? *(volatile uint32_t*)&cache.ir[cand[j]] : 0u + kNoBox;
    miss_any |= u[j] == kNoBox;
  }
  __threadfence_block();  // the records after their flags
  float4 c[2];
  if (!miss_any) {
#pragma unroll
    for (int j = 0; j < 2; ++j) c[j] = cache.rec[j0 + j < ncand ? cand[j] : 0];
  } else {
    // both boxes are read before either is used
    float b[2][6];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 6; ++k) b[j][k] = j0 + j < ncand ? net.boxes[6 * (size_t)cand[j] + k] : 0.0f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float ir;
      boxRecord(b[j], net.norm, &c[j], &ir);
      u[j] = __float_as_uint(ir);
      if (j0 + j < ncand && cand[j] < kBoxCache) cache.rec[cand[j]] = c[j];
    }
    __threadfence_block();
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (j0 + j < ncand && cand[j] < kBoxCache) *(volatile uint32_t*)&cache.ir[cand[j]] = u[j];
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const bool present = j0 + j < ncand;
    const float ir = __uint_as_float(u[j]), r = c[j].w;
    const float pc[3] = {c[j].x - on[0], c[j].y - on[1], c[j].z - on[2]};
    const float along = (pc[0] * d[0] + pc[1] * d[1]) + pc[2] * d[2];
    const float pp = (pc[0] * pc[0] + pc[1] * pc[1]) + pc[2] * pc[2];
    const float miss = sqrtf(fmaxf(pp - along * along, 0.0f));
    const float mr = fminf(miss * ir, 4.0f), ar = fminf(fmaxf(along * ir, -4.0f), 4.0f);
    const int col = 6 + 6 * (j0 + j);
    put(col, present ? along : 0.0f, present ? miss : 0.0f);
    put(col + 2, present ? r : 0.0f, present ? mr : 0.0f);
    put(col + 4, present ? ar : 0.0f, present ? 1.0f : 0.0f);
  }
}

// The 64 features of a row, in order: put(column, value, value of column + 1).
template <class Put>
__device__ __forceinline__ void rowFeatures(const Row& r, const Net& net, const BoxCache& cache, Put&& put) {
  float on[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) on[c] = (r.o[c] - net.norm.centre[c]) * net.norm.scale;
  put(0, on[0], on[1]);
  put(2, on[2], r.d[0]);
  put(4, r.d[1], r.d[2]);
#pragma unroll
  for (int j = 0; j < kCand; j += 2) candFeatures(on, r.d, r.cand + j, j, r.ncand, net, cache, put);
#pragma unroll
  for (int c = kIn; c < kK; c += 2) put(c, 0.0f, 0.0f);
}

// Row t of the operand x: 16 bytes are stored when complete.
__device__ __forceinline__ void features(const Row& r, int t, const Net& net, const BoxCache& cache, uint8_t* x) {
  uint4 q;
  rowFeatures(r, net, cache, [&](int c, float a, float b) {
    const uint32_t p = packBf16(a, b);
    if ((c & 7) == 0) q.x = p;
    else if ((c & 7) == 2) q.y = p;
    else if ((c & 7) == 4) q.z = p;
    else {
      q.w = p;
      *reinterpret_cast<uint4*>(x + opOff(t, c & ~7, 8)) = q;
    }
  });
}
__device__ __forceinline__ void noFeatures(int t, uint8_t* x) {
#pragma unroll
  for (int c = 0; c < kK; c += 8) *reinterpret_cast<uint4*>(x + opOff(t, c, 8)) = make_uint4(0u, 0u, 0u, 0u);
}

// Samples of a tile -> stage (shared, 48 bytes per row), asynchronously; a row past
// the end is left alone.
__device__ __forceinline__ void stageSamples(const Sample* s, int64_t n, int64_t tile, uint32_t stage, int t,
                                             int threads) {
  const Sample* src = s + tile * kTile;
  const int bytes = (int)min((int64_t)kTile, n - tile * kTile) * (int)sizeof(Sample);
  if ((reinterpret_cast<uintptr_t>(s) & 15) == 0) {  // samples are 48 bytes: all aligned or none
    for (int k = 16 * t; k < bytes; k += 16 * threads)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(stage + k),
                   "l"(reinterpret_cast<const char*>(src) + k)
                   : "memory");
  } else {
    for (int k = 4 * t; k < bytes; k += 4 * threads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(stage + k),
                   "l"(reinterpret_cast<const char*>(src) + k)
                   : "memory");
  }
}
__device__ __forceinline__ void stageWait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
constexpr int kStageBytes = kTile * sizeof(Sample);

__device__ __forceinline__ Row unpackRow(uint4 a, uint4 b, uint4 c) {
  Row r;
  r.o[0] = __uint_as_float(a.x);
  r.o[1] = __uint_as_float(a.y);
  r.o[2] = __uint_as_float(a.z);
  r.d[0] = __uint_as_float(a.w);
  r.d[1] = __uint_as_float(b.x);
  r.d[2] = __uint_as_float(b.y);
  const uint32_t w[4] = {b.z, b.w, c.x, c.y};
#pragma unroll
  for (int j = 0; j < kCand; ++j) r.cand[j] = (w[j >> 1] >> (16 * (j & 1))) & 0xffffu;
  r.ncand = (int)c.z;
  r.label = (int)c.w;
  return r;
}
__device__ __forceinline__ Row stagedRow(const uint8_t* stage, int t) {
  const uint4* p = reinterpret_cast<const uint4*>(stage + t * sizeof(Sample));
  return unpackRow(p[0], p[1], p[2]);
}
__device__ __forceinline__ Row loadRow(const Sample* s) {
  if ((reinterpret_cast<uintptr_t>(s) & 15) == 0) {
    const uint4* p = reinterpret_cast<const uint4*>(s);
    return unpackRow(p[0], p[1], p[2]);
  }
  const uint32_t* p = reinterpret_cast<const uint32_t*>(s);
  return unpackRow(make_uint4(p[0], p[1], p[2], p[3]), make_uint4(p[4], p[5], p[6], p[7]),
                   make_uint4(p[8], p[9], p[10], p[11]));
}

// Sources of rows for the forward kernel.
struct StagedRows {
  const Sample* s;
  int64_t n;
  static constexpr bool kStaged = true;
  __device__ int64_t rows() const { return n; }
  __device__ void stage(int64_t tile, uint32_t to, int t) const { stageSamples(s, n, tile, to, t, kTile); }
  __device__ Row load(int64_t, const uint8_t* st, int t) const { return stagedRow(st, t); }
};

struct SampleRows : StagedRows {
  float* logits;
  int32_t* pred;
  __device__ void store(int64_t i, const float* lg, int ncand, int best) const {
    float* dst = logits + i * kCand;
    if ((reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
      reinterpret_cast<float4*>(dst)[0] = make_float4(lg[0], lg[1], lg[2], lg[3]);
      reinterpret_cast<float4*>(dst)[1] = make_float4(lg[4], lg[5], lg[6], lg[7]);
    } else {
#pragma unroll
      for (int c = 0; c < kCand; ++c) dst[c] = lg[c];
    }
    pred[i] = best;
  }
};

// Held-out evaluation: counts[0] += labelled rows with at least two
// candidates, counts[1] += those whose argmax is the label, counts[2] +=
// those whose label is the nearest candidate (position 0).
struct EvalRows : StagedRows {
  unsigned long long* counts;
  __device__ void store(int64_t i, const float*, int ncand, int best) const {
    const int label = s[i].label;
    if (label < 0 || ncand < 2) return;
    atomicAdd(&counts[0], 1ull);
    if (best == label) atomicAdd(&counts[1], 1ull);
    if (label == 0) atomicAdd(&counts[2], 1ull);
  }
};

struct ArenaRows {
  ArenaSource a;
  uint8_t* pred;
  static constexpr bool kStaged = false;
  __device__ int64_t rows() const { return *a.count; }
  __device__ void stage(int64_t, uint32_t, int) const {}
  __device__ Row load(int64_t i, const uint8_t*, int) const {
    Row r;
    const uint32_t rid = a.list[i];
    const float4 o4 = a.org[rid], d4 = a.dir[rid];
    r.o[0] = o4.x;
    r.o[1] = o4.y;
    r.o[2] = o4.z;
    r.d[0] = d4.x;
    r.d[1] = d4.y;
    r.d[2] = d4.z;
    r.ncand = (int)a.list_cnt[i];
    const uint32_t off = a.list_off[i];
#pragma unroll
    for (int j = 0; j < kCand; ++j) r.cand[j] = j < r.ncand ? a.arena[off + j].x & 0xffffu : 0u;
    return r;
  }
  __device__ void store(int64_t i, const float*, int ncand, int best) const {
    pred[i] = (uint8_t)(ncand >= 2 ? best : 0);
  }
};

// Inference.  A CTA per SM of five groups of 128 threads, each with its own tile of
// rows, 96 tensor-memory columns and barriers; they share the weights and the box
// records.  A tile's own chain (rows, features, four products with a read-back
// each) is serial, so the groups fill each other's waits.  The activations stay in
// tensor memory, written there as the next product's A: through shared memory they
// were half of its traffic, which bound the kernel (80 % of its data pipe), although
// eight groups fitted then.  1048576 rows: 157 us with five CTAs of one group that
// held their own weights and read six scattered words of every candidate's box,
// 81 us with eight groups and the activations in shared memory, now 71 us (four groups 79, three
// 89); issue bounds it, 63 %.
constexpr int kFwdGroups = 5, kFwdThreads = kFwdGroups * kTile;
// Shared memory: W1 W2 W3 (8 KB each), W4 (2 KB), box records, biases, mbarriers,
// (each group's, and one more that a wait which gave up needs), the tensor-memory
// address; per group the staged samples.
constexpr int kFwdW = 0, kFwdBox = 3 * 8192 + 2048, kFwdBias = kFwdBox + kBoxBytes;
constexpr int kFwdBar = kFwdBias + (3 * kHid + kOutPad) * 4, kFwdDrain = kFwdBar + 8 * kFwdGroups;
constexpr int kFwdSlot = kFwdDrain + 8 * kFwdGroups;
constexpr int kFwdStage = (kFwdSlot + 4 + 15) / 16 * 16, kFwdSmem = 116 * 1024;
static_assert(kFwdStage + kFwdGroups * kStageBytes <= kFwdSmem, "forward shared memory");
// (more than half of an SM's, so that one CTA has it and its tensor memory alone)
static_assert(2 * kFwdSmem > 227 * 1024, "one CTA per SM: 512 columns");
// Group g: its accumulators in 64 columns from 96 g (the logits reuse the first 16
// once layer 3's output has been read back; the tcgen05 fences around the barrier
// order the read before the next MMA, as between the hidden layers), its
// activations in the 32 after them.
constexpr uint32_t kFwdCols = 96, kFwdAct = 64;
static_assert(kFwdGroups * kFwdCols <= 512, "tensor memory");

template <class Rows>
__global__ void __launch_bounds__(kFwdThreads, 1) kForward(Net net, Rows rows) {
  extern __shared__ __align__(128) uint8_t sm[];
  const int t = threadIdx.x % kTile;
  // (warp-uniform, and the compiler knows)
  const int g = __shfl_sync(0xffffffffu, (int)threadIdx.x / kTile, 0), warp = __shfl_sync(0xffffffffu, t >> 5, 0);
  float* bias = reinterpret_cast<float*>(sm + kFwdBias);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kFwdSlot);
  uint8_t* stage = sm + kFwdStage + kStageBytes * g;
  BoxCache cache(sm + kFwdBox);
  const uint32_t mbar = smemAddr(sm + kFwdBar + 8 * g), drain = smemAddr(sm + kFwdDrain + 8 * g);
  const uint32_t stage_to = smemAddr(stage);
  const int64_t n = rows.rows();
  // tiles go to the CTAs first, then to their groups
  int64_t tile = blockIdx.x + (int64_t)gridDim.x * g;
  if (tile * kTile < n) rows.stage(tile, stage_to, t);
  NetStage<kFwdThreads> weights(threadIdx.x);
  weights.load(net.params);
  cache.init(net, threadIdx.x, kFwdThreads);
  weights.store(sm + kFwdW, bias);
  if (threadIdx.x < 32) tmemAlloc(smemAddr(tslot), 512);
  if (t == 0) {
    mbarInit(mbar, 1);
    mbarInit(drain, 1);
  }
  fenceProxyAsync();
  fenceBeforeSync();
  __syncthreads();
  fenceAfterSync();
  const uint32_t tm = __shfl_sync(0xffffffffu, *tslot, 0) + kFwdCols * g;
  const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
  const uint32_t b_w = smemAddr(sm + kFwdW);
  uint32_t phase = 0;
  bool ok = true;
  for (; tile * kTile < n; tile += (int64_t)gridDim.x * kFwdGroups) {
    const int64_t i = tile * kTile + t;
    if (Rows::kStaged) {
      stageWait();
      barSync(1 + g, kTile);
    }
    int ncand = 0;
    {
      uint32_t x[kK / 2];
      if (i < n) {
        const Row r = rows.load(i, stage, t);
        ncand = r.ncand;
        rowFeatures(r, net, cache, [&](int c, float a, float b) { x[c / 2] = packBf16(a, b); });
      } else {
#pragma unroll
        for (int c = 0; c < kK / 2; ++c) x[c] = 0u;
      }
      __syncwarp();
#pragma unroll
      for (int c = 0; c < kK / 2; c += 8) tmemSt8(tm + lane_base + kFwdAct + c, x + c);
    }
    tmemStWait();
    fenceBeforeSync();
    barSync(1 + g, kTile);
    const int64_t next = tile + (int64_t)gridDim.x * kFwdGroups;
    if (next * kTile < n) rows.stage(next, stage_to, t);
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
      if (warp == 0) {
        fenceAfterSync();
        const Operand w{b_w + 8192 * l, 1024u, false};
        if (l < 3) gemmTmem(tm, tm + kFwdAct, w, kK, kHid, t == 0);
        else gemmTmem(tm, tm + kFwdAct, w, kHid, kOutPad, t == 0);
        commit(mbar, t == 0);
      }
      ok = ok && mbarWait(mbar, phase);
      __syncwarp();
      phase ^= 1;
      fenceAfterSync();
      if (l < 3) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          float z[16];
          tmemLd16(tm + lane_base + 16 * h, z);
          const uint4 a = activate8(z, bias + l * kHid + 16 * h), b = activate8(z + 8, bias + l * kHid + 16 * h + 8);
          const uint32_t x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
          tmemSt8(tm + lane_base + kFwdAct + 8 * h, x);
        }
        tmemStWait();
        fenceBeforeSync();
        barSync(1 + g, kTile);
      } else {
        float z[8];
        tmemLd8(tm + lane_base, z);
        float lg[kCand], top = 0.0f;
        int best = 0;
#pragma unroll
        for (int c = 0; c < kCand; ++c) {
          lg[c] = c < ncand ? z[c] + bias[3 * kHid + c] : -INFINITY;
          if (c == 0) top = lg[0];
          else if (lg[c] > top) {
            top = lg[c];
            best = c;
          }
        }
        if (i < n) rows.store(i, lg, ncand, best);
        fenceBeforeSync();  // ordered before the next tile's products by its barrier
      }
    }
  }
  if (!ok) atomicExch(net.error, 1);
  fenceBeforeSync();
  if (__syncthreads_or(!ok)) {
    // products may still be in flight: their memory is kept until they end, or for
    // another second
    if (warp == 0) {
      commit(drain, t == 0);
      mbarWait(drain, 0);
    }
    __syncthreads();
  }
  fenceAfterSync();
  if (threadIdx.x < 32) tmemDealloc(*tslot, 512);
}

// Training.  A CTA per SM and 128 rows a tile as the partial sums have it.  The
// chain of a tile (seven products with a read-back each) is serial; its latency is
// what bounds the kernel, and everything else is kept off it.  512 threads take four
// to a row, 16 columns of every layer each.  Four warps make the next tile's
// features meanwhile.  One warp issues the products, each dH before the dW that
// reads the same dZ: the chain waits for dH, and nobody waits for dW (the next
// tile's first wait covers it).  A warp per layer sums dZ down its rows, in row
// order, for the biases.  With 128 threads that did it all in turn and kept
// transposed copies of every activation and dZ: 65536 rows 101 -> 33 us.
constexpr int kGradThreads = 4 * kTile;           // row threads
constexpr int kGThreads = kGradThreads + kTile + 4 * 32 + 32;  // feature threads, bias warps, issuing warp
// Shared memory: W1..W3 (8 KB each), W4 (2 KB); X of this tile and the last, H1, H2,
// H3, dZ1..dZ3 (128 x 64, 16 KB each), dZ4 (128 x 16), exponentials (128 x 8), box
// records, (candidates, label) of both X, biases, mbarrier, tensor-memory address, a
// second mbarrier that a wait which gave up needs.
constexpr int kGW = 0, kGAct = 3 * 8192 + 2048, kGDz = kGAct + 5 * 16384, kGDz4 = kGDz + 3 * 16384;
constexpr int kGExp = kGDz4 + 4096, kGBox = kGExp + 4096, kGRow = kGBox + kBoxBytes, kGBias = kGRow + 2 * kTile * 8;
constexpr int kGBar = kGBias + (3 * kHid + kOutPad) * 4, kGSmem = kGBar + 32;
static_assert(kGSmem <= 227 * 1024, "training shared memory");  // one CTA per SM: 512 columns
// Tensor-memory columns: D0 (64), logits (16), dW1..dW4 (64 each).
constexpr uint32_t kGCols = 512, kColLogit = 64, kColDw = 128;
// Named barriers.  X of a tile is written (feature threads -> issuing warp and row
// threads); the older X may be overwritten (row threads -> feature threads); a later
// operand is written (rows -> issuing warp); dZ of layer l + 1 is (kBarDz + l, rows ->
// its bias warp); the bias warps have read the tile's dZ (-> rows); the rows alone;
// the feature threads alone.
// Two arrivals at one barrier always have a wait for its first between them; the
// two X have a barrier each for that (kBarX, kBarX + 1).
constexpr int kBarOp = 1, kBarDz = 2, kBarFree = 6, kBarXFree = 7, kBarX = 8, kBarRows = 10, kBarBoxes = 11;
constexpr int kXCount = kTile + 32 + kGradThreads, kXFreeCount = kTile + kGradThreads;
constexpr int kBarCount = kGradThreads + 32, kFreeCount = kGradThreads + 4 * 32;
constexpr int kDwPitch = 68;  // floats between the rows of dW on their way out (no bank conflicts)

__global__ void __launch_bounds__(kGThreads, 1) kGrad(Net net, const Sample* batch, int64_t n, float inv_count,
                                                              const uint32_t* labelled_rows, float* partial) {
  extern __shared__ __align__(128) uint8_t sm[];
  const int t = threadIdx.x % kTile, lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);  // (the compiler knows it uniform)
  const int quarter = threadIdx.x / kTile;          // of the row threads
  const int lanes = (t >> 5) * 32;                  // first tensor-memory lane of the warp
  const bool rows = warp < 16, feature_warp = warp >= 16 && warp < 20, bias_warp = warp >= 20 && warp < 24;
  float* bias = reinterpret_cast<float*>(sm + kGBias);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kGBar + 8);
  int2* row_data = reinterpret_cast<int2*>(sm + kGRow);
  BoxCache cache(sm + kGBox);
  const uint32_t mbar = smemAddr(sm + kGBar), drain = mbar + 16;
  const int64_t ntiles = (n + kTile - 1) / kTile;
  const bool any = blockIdx.x < ntiles;
  if (labelled_rows) {
    const uint32_t count = *labelled_rows;
    inv_count = count > 0 ? 1.0f / (float)count : 0.0f;
  }
  // the features of a tile into X number x
  auto makeX = [&](int64_t tile, const Row& r, int x) {
    const int64_t i = tile * kTile + t;
    uint8_t* to = sm + kGAct + 16384 * x;
    int2 rd = make_int2(0, -1);
    if (i < n) {
      features(r, t, net, cache, to);
      rd.x = r.ncand < kCand ? r.ncand : kCand;
      if (r.label >= 0 && r.label < rd.x) rd.y = r.label;
    } else {
      noFeatures(t, to);
    }
    row_data[kTile * x + t] = rd;
    fenceProxyAsync();
    barArrive(kBarX + x, kXCount);
  };
  auto rowOf = [&](int64_t tile) {
    const int64_t i = tile * kTile + t;
    Row r = {};
    if (i < n) r = loadRow(batch + i);
    return r;
  };
  // The feature threads begin with the boxes and the first tile, beside the others'
  // weights.
  if (feature_warp) {
    const Row r = rowOf(blockIdx.x);
    cache.init(net, t, kTile);
    barSync(kBarBoxes, kTile);
    if (any) makeX(blockIdx.x, r, 0);
  } else {
    NetStage<kGThreads - kTile> weights(rows ? threadIdx.x : threadIdx.x - kTile);
    weights.load(net.params);
    weights.store(sm + kGW, bias);
  }
  // columns 8..15 of dZ4 stay zero
  if (quarter == 0) *reinterpret_cast<uint4*>(sm + kGDz4 + opOff(t, 8, 2)) = make_uint4(0u, 0u, 0u, 0u);
  if (warp == 0) tmemAlloc(smemAddr(tslot), kGCols);
  if (threadIdx.x == 0) {
    mbarInit(mbar, 1);
    mbarInit(drain, 1);
  }
  fenceProxyAsync();
  fenceBeforeSync();
  __syncthreads();
  fenceAfterSync();
  const uint32_t tm = __shfl_sync(0xffffffffu, *tslot, 0);
  const uint32_t lane_base = (uint32_t)lanes << 16;
  float* out = partial + (size_t)blockIdx.x * kPartialPitch;
  bool ok = true;
  float loss = 0.0f, labelled = 0.0f;
  if (feature_warp) {
    int x = 1;
    for (int64_t tile = blockIdx.x + (int64_t)gridDim.x; tile < ntiles; tile += gridDim.x) {
      const Row r = rowOf(tile);
      // (the second tile finds its X free)
      if (tile != blockIdx.x + (int64_t)gridDim.x) barSync(kBarXFree, kXFreeCount);
      makeX(tile, r, x);
      x ^= 1;
    }
  } else if (bias_warp) {
    // layer l + 1: lane k has columns 2k, 2k + 1.  The eight groups of four lanes read
    // eight different rows at a time, group g one row behind group g - 1: at the same
    // row their 16-byte pieces would lie 128 bytes apart, in the same banks.
    const int l = warp - 20, kg = l == 3 ? 2 : 8, group = lane >> 2;
    const uint8_t* dz = l == 3 ? sm + kGDz4 : sm + kGDz + 16384 * l;
    const bool mine = l < 3 || lane < kOutPad / 2;
    int at[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      at[j] = group * 128 + ((j - group) >> 3) * (kg * 128) + ((j - group) & 7) * 16 + (lane & 3) * 4;
    float db0 = 0.0f, db1 = 0.0f;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      barSync(kBarDz + l, kBarCount);
      float s0 = 0.0f, s1 = 0.0f;
      auto rows8 = [&](int b, auto&& valid) {  // step 8 b + j: row 8 b + j - group
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t v = 0u;
          if (valid(j)) v = *reinterpret_cast<const uint32_t*>(dz + b * (kg * 128) + at[j]);
          s0 += __uint_as_float(v << 16);
          s1 += __uint_as_float(v & 0xffff0000u);
        }
      };
      if (mine) {
        rows8(0, [&](int j) { return j >= group; });
#pragma unroll 3
        for (int b = 1; b < kTile / 8; ++b) rows8(b, [](int) { return true; });
        rows8(kTile / 8, [&](int j) { return j < group; });
      }
      db0 += s0;
      db1 += s1;
      if (tile + gridDim.x < ntiles) barArrive(kBarFree, kFreeCount);
    }
    if (mine) {
      float* dst = out + (l < 3 ? kB1 + l * (kHid * kK + kHid) : kB4) + 2 * lane;
      dst[0] = db0;
      dst[1] = db1;
    }
  } else if (!rows) {
    // issuing warp: operands as the row threads write them
    const uint32_t w = smemAddr(sm + kGW), acts = smemAddr(sm + kGAct), dzs = smemAddr(sm + kGDz);
    uint32_t x = acts;  // X of this tile, then H1, H2, H3 behind the two X
    auto h = [&](int l) { return l == 0 ? x : acts + 16384 * (l + 1); };
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        if (l == 0) barSync(x == acts ? kBarX : kBarX + 1, kXCount);
        else barSync(kBarOp, kBarCount);
        fenceAfterSync();
        gemm(l < 3 ? tm : tm + kColLogit, Operand{h(l), 1024u, false}, Operand{w + 8192 * l, 1024u, false}, kK,
             l < 3 ? kHid : kOutPad, false, lane == 0);
        commit(mbar, lane == 0);
      }
#pragma unroll
      for (int l = 3; l >= 0; --l) {
        // dH_{l-1} = dZ_l W_l; dW_l += dZ_l^T H_{l-1}
        const uint32_t dz = l == 3 ? smemAddr(sm + kGDz4) : dzs + 16384 * l, pitch = l == 3 ? 256u : 1024u;
        barSync(kBarOp, kBarCount);
        fenceAfterSync();
        if (l > 0) {
          gemm(tm, Operand{dz, pitch, false}, Operand{w + 8192 * l, 1024u, true}, l == 3 ? kOutPad : kHid, kHid, false,
               lane == 0);
          commit(mbar, lane == 0);
        }
        gemm(tm + kColDw + 64 * l, Operand{dz, pitch, true}, Operand{h(l), 1024u, true}, kTile, kHid,
             tile != blockIdx.x, lane == 0);
      }
      x = x == acts ? acts + 16384 : acts;
    }
    if (any) commit(mbar, lane == 0);  // the last dW products
  } else {
    const int c0 = 16 * quarter;  // this thread's columns of a layer
    uint32_t phase = 0;
    uint8_t* x = sm + kGAct;
    auto h = [&](int l) { return l == 0 ? x : sm + kGAct + 16384 * (l + 1); };
    // an operand is written: its product may be issued.  The rows meet the issuing
    // warp here (their wait for the product would, too): an arrival alone could be
    // repeated before the issuing warp has taken the last one, once a wait for a
    // product gave up, and the barrier would be out of step for good.
    auto ready = [&]() {
      fenceProxyAsync();
      fenceBeforeSync();
      barSync(kBarOp, kBarCount);
    };
    auto product = [&]() {
      ok = ok && mbarWait(mbar, phase);
      __syncwarp();
      phase ^= 1;
      fenceAfterSync();
    };
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const int xi = x == sm + kGAct ? 0 : 1;
      barSync(kBarX + xi, kXCount);
      const int2 rd = row_data[kTile * xi + t];
      const int ncand = rd.x, label = rd.y;
      // forward: H1, H2, H3
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        product();
        // (every product of the last tile is done, too)
        if (l == 0 && tile != blockIdx.x && tile + gridDim.x < ntiles) barArrive(kBarXFree, kXFreeCount);
        float z[16];
        tmemLd16(tm + lane_base + c0, z);
#pragma unroll
        for (int c = 0; c < 16; c += 8)
          *reinterpret_cast<uint4*>(h(l + 1) + opOff(t, c0 + c, 8)) = activate8(z + c, bias + l * kHid + c0 + c);
        ready();
      }
      // logits: each of a row's four threads takes two exponentials, and two of the
      // gradients once all eight are there.  The bias warps have to be done with the
      // last tile's dZ.
      product();
      {
        float z[8], m = -INFINITY, zl = 0.0f, mine[2];
        tmemLd8(tm + lane_base + kColLogit, z);
#pragma unroll
        for (int c = 0; c < kCand; ++c) {
          z[c] = z[c] + bias[3 * kHid + c];
          m = c < ncand ? fmaxf(m, z[c]) : m;
          zl = c == label ? z[c] : zl;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
          mine[k] = expf((quarter == 0 ? z[k] : quarter == 1 ? z[2 + k] : quarter == 2 ? z[4 + k] : z[6 + k]) - m);
        float* e = reinterpret_cast<float*>(sm + kGExp) + kCand * t;
        *reinterpret_cast<float2*>(e + 2 * quarter) = make_float2(mine[0], mine[1]);
        if (tile == blockIdx.x) barSync(kBarRows, kGradThreads);
        else barSync(kBarFree, kFreeCount);
        const float4 ea = *reinterpret_cast<const float4*>(e), eb = *reinterpret_cast<const float4*>(e + 4);
        const float ev[8] = {ea.x, ea.y, ea.z, ea.w, eb.x, eb.y, eb.z, eb.w};
        float s = 0.0f;
#pragma unroll
        for (int c = 0; c < kCand; ++c) s = c < ncand ? s + ev[c] : s;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int c = 2 * quarter + k;
          const float p = (mine[k] / s - (c == label ? 1.0f : 0.0f)) * inv_count;
          mine[k] = label >= 0 && c < ncand ? p : 0.0f;
        }
        *reinterpret_cast<uint32_t*>(sm + kGDz4 + opOff(t, 2 * quarter, 2)) = packBf16(mine[0], mine[1]);
        barArrive(kBarDz + 3, kBarCount);
        ready();
        if (quarter == 0 && label >= 0) {
          loss += logf(s) - (zl - m);
          labelled += 1.0f;
        }
      }
      // backward: dZ3, dZ2, dZ1
#pragma unroll
      for (int l = 3; l > 0; --l) {
        // ReLU mask of H_l
        uint4 a[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          a[c] = *reinterpret_cast<const uint4*>(h(l) + opOff(t, c0 + 8 * c, 8));
          a[c] = make_uint4(positive(a[c].x), positive(a[c].y), positive(a[c].z), positive(a[c].w));
        }
        product();
        float z[16];
        tmemLd16(tm + lane_base + c0, z);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint4 p = pack8(z + 8 * c);
          *reinterpret_cast<uint4*>(sm + kGDz + 16384 * (l - 1) + opOff(t, c0 + 8 * c, 8)) =
              make_uint4(p.x & a[c].x, p.y & a[c].y, p.z & a[c].z, p.w & a[c].w);
        }
        barArrive(kBarDz + l - 1, kBarCount);
        ready();
      }
      x = x == sm + kGAct ? sm + kGAct + 16384 : sm + kGAct;
    }
    if (any) {
      product();  // the last dW
      // dW1..dW3: rows 0..63 (warps 0, 1 of a quarter); dW4: rows 0..15 (warp 0);
      // through shared memory (the activations are done with), so that a warp writes
      // whole lines
      float* dw = reinterpret_cast<float*>(sm + kGAct);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const int nrows = l == 3 ? kOutPad : kHid;
        if (lanes >= nrows) continue;
        float v[16];
        tmemLd16(tm + lane_base + kColDw + 64 * l + c0, v);
        if (t < nrows) {
          float* dst = dw + (l * kHid + t) * kDwPitch + c0;
#pragma unroll
          for (int c = 0; c < 16; c += 4)
            *reinterpret_cast<float4*>(dst + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        }
      }
      barSync(kBarRows, kGradThreads);
      for (int k = threadIdx.x; k < (3 * kHid + kOutPad) * 16; k += kGradThreads) {
        const int r = k >> 4, c = (k & 15) * 4;  // row of W1..W4, column
        *reinterpret_cast<float4*>(out + r * kHid + (r >> 6) * kHid + c) =
            *reinterpret_cast<const float4*>(dw + r * kDwPitch + c);
      }
    } else {
      for (int l = 0; l < 4; ++l) {
        const int first = l < 3 ? kW1 + l * (kHid * kK + kHid) : kW4, count = l < 3 ? kHid * kK : kOutPad * kHid;
        for (int k = threadIdx.x; k < count; k += kGradThreads) out[first + k] = 0.0f;
      }
    }
  }
  if (!ok) atomicExch(net.error, 1);
  // loss and labelled rows: block sums in a fixed order
  float* red = reinterpret_cast<float*>(sm + kGExp);
  fenceBeforeSync();
  if (__syncthreads_or(!ok)) {  // as in kForward
    if (!rows && !feature_warp && !bias_warp) {
      commit(drain, lane == 0);
      mbarWait(drain, 0);
    }
    __syncthreads();
  }
  fenceAfterSync();
  if (quarter == 0) {
    red[t] = loss;
    red[kTile + t] = labelled;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    float a = 0.0f;
#pragma unroll 32
    for (int k = 0; k < kTile; ++k) a += red[threadIdx.x * kTile + k];
    out[kParams + threadIdx.x] = a;
  }
  if (warp == 0) tmemDealloc(tm, kGCols);
}
static_assert((3 * kHid + kOutPad) * kDwPitch * 4 <= 5 * 16384, "dW fits the activations");
static_assert(kPartialPitch % 4 == 0 && kW1 == 0 && kW2 == 65 * kHid && kW4 == 195 * kHid, "rows of a partial");

// 32 parameters a block: its warps bring a share of the partials each (19 loads in
// flight, whole lines), the first then adds them in CTA order, a parameter per lane,
// and takes the Adam step.  A thread per parameter that walked the partials took
// 10.9 us for 152 of them, this 6.5.
__global__ void __launch_bounds__(kReduceThreads) kReduceAdam(const float* __restrict__ partial, int nparts,
                                                              float* grad, float* params, float* m, float* v,
                                                              float lr, int step, float* mean_loss) {
  constexpr int kWarps = kReduceThreads / 32, kEach = 19;
  __shared__ float part[kWarps * kEach][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  float g = 0.0f;
  for (int p0 = 0; p0 < nparts; p0 += kWarps * kEach) {
    const int first = p0 + warp * kEach, here = min(nparts - p0, kWarps * kEach);
    float x[kEach];
#pragma unroll
    for (int q = 0; q < kEach; ++q)
      x[q] = i < kPartial && first + q < nparts ? partial[(size_t)(first + q) * kPartialPitch + i] : 0.0f;
#pragma unroll
    for (int q = 0; q < kEach; ++q) part[warp * kEach + q][lane] = x[q];
    __syncthreads();
    if (warp == 0) {
      int p = 0;
#pragma unroll 1
      for (; p + 16 <= here; p += 16)
#pragma unroll
        for (int q = 0; q < 16; ++q) g += part[p + q][lane];
      for (; p < here; ++p) g += part[p][lane];
    }
    __syncthreads();
  }
  if (warp != 0) return;
  if (i < kPartial) grad[i] = g;
  static_assert(kParams / 32 == (kPartial - 1) / 32, "the last block holds the loss and the row count");
  if (mean_loss && blockIdx.x == gridDim.x - 1) {
    const float loss = __shfl_sync(0xffffffffu, g, kParams % 32), n = __shfl_sync(0xffffffffu, g, kParams % 32 + 1);
    if (lane == 0) *mean_loss = n > 0.0f ? loss / n : 0.0f;
  }
  if (lr > 0.0f && i < kParams) {
    const float mi = 0.9f * m[i] + 0.1f * g;
    const float vi = 0.999f * v[i] + 0.001f * (g * g);
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.0f - powf(0.9f, (float)step));
    const float vh = vi / (1.0f - powf(0.999f, (float)step));
    params[i] -= lr * mh / (sqrtf(vh) + 1e-8f);
  }
}

// Block column = step; its threads stride over the batch.
__global__ void kCountLabelled(const Sample* __restrict__ samples, int64_t n, int64_t b, int64_t first,
                               uint32_t* counts, uint32_t* num_boxes) {
  const int64_t start = ((first + blockIdx.y) * b) % n;
  const int64_t len = min(b, n - start);
  uint32_t c = 0, boxes = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x) {
    const Sample& q = samples[start + i];
    c += q.label >= 0 && q.label < min(q.ncand, kCand) ? 1u : 0u;
#pragma unroll
    for (int j = 0; j < kCand; ++j)
      if (j < q.ncand) boxes = max(boxes, q.cand[j] + 1u);
  }
  c = __reduce_add_sync(0xffffffffu, c);
  boxes = __reduce_max_sync(0xffffffffu, boxes);
  if ((threadIdx.x & 31) == 0) {
    if (c) atomicAdd(&counts[blockIdx.y], c);
    if (boxes) atomicMax(num_boxes, boxes);
  }
}

// Per alive ray: the list position of the candidate that holds its hit, when
// the ray has at least two candidates and the hit is among the first eight.
__global__ void kCollectLabel(ArenaSource a, const uint64_t* __restrict__ ray_key,
                              const DomainDev* __restrict__ doms, int8_t* label, uint8_t* flag) {
  const uint32_t n = *a.count;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int lab = -1;
    const uint32_t cnt = a.list_cnt[i];
    if (cnt >= 2) {
      const uint64_t key = ray_key[a.list[i]];
      if (key != kNoHit) {
        const uint32_t prim = (uint32_t)key;
        const uint32_t off = a.list_off[i];
        const int nc = cnt < (uint32_t)kCand ? (int)cnt : kCand;
        for (int j = 0; j < nc; ++j) {
          const DomainDev& d = doms[a.arena[off + j].x & 0xffffu];
          if (prim - d.gprim_base < (uint32_t)d.num_tris) {
            lab = j;
            break;
          }
        }
      }
    }
    label[i] = (int8_t)lab;
    flag[i] = lab >= 0;
  }
}

__global__ void kCollectWrite(ArenaSource a, const int8_t* __restrict__ label, const uint32_t* sel,
                              const uint32_t* nsel, Sample* out, unsigned long long* filled,
                              uint64_t capacity) {
  const uint64_t base = *filled;
  const uint64_t room = capacity > base ? capacity - base : 0;
  const uint64_t n = min((uint64_t)*nsel, room);
  for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n;
       k += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = sel[k];
    const uint32_t rid = a.list[i];
    const float4 o = a.org[rid], d = a.dir[rid];
    Sample s;
    s.org[0] = o.x;
    s.org[1] = o.y;
    s.org[2] = o.z;
    s.dir[0] = d.x;
    s.dir[1] = d.y;
    s.dir[2] = d.z;
    const uint32_t cnt = a.list_cnt[i], off = a.list_off[i];
    s.ncand = cnt < (uint32_t)kCand ? (int)cnt : kCand;
    for (int j = 0; j < kCand; ++j) s.cand[j] = j < s.ncand ? (uint16_t)(a.arena[off + j].x & 0xffffu) : 0;
    s.label = label[i];
    out[base + k] = s;
  }
}

__global__ void kCollectAdvance(const uint32_t* nsel, unsigned long long* filled, uint64_t capacity) {
  const uint64_t base = *filled;
  const uint64_t room = capacity > base ? capacity - base : 0;
  *filled = base + min((uint64_t)*nsel, room);
}

// One atomic per distinct domain of a warp (rays of a warp often agree).
__global__ void kPredCount(ArenaSource a, const uint8_t* __restrict__ pred, uint32_t* counts) {
  const uint32_t n = *a.count;
  const int lane = threadIdx.x & 31;
  for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < n;
       base += gridDim.x * blockDim.x) {
    const uint32_t i = base + lane;
    uint32_t d = 0xffffffffu;
    if (i < n) {
      const uint32_t cnt = a.list_cnt[i];
      if (cnt) d = a.arena[a.list_off[i] + min((uint32_t)pred[i], cnt - 1)].x & 0xffffu;
    }
    const uint32_t m = __match_any_sync(0xffffffffu, d);
    if (d != 0xffffffffu && (__ffs(m) - 1) == lane) atomicAdd(&counts[d], (uint32_t)__popc(m));
  }
}

}  // namespace

void launchPredCount(cudaStream_t s, const ArenaSource& src, const uint8_t* pred, uint32_t* counts,
                     int nblocks) {
  kPredCount<<<nblocks, 256, 0, s>>>(src, pred, counts);
}

void launchPredictArena(cudaStream_t s, const Net& net, const ArenaSource& src, uint8_t* pred, int nblocks) {
  ArenaRows r{src, pred};
  cudaFuncSetAttribute(kForward<ArenaRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
  kForward<ArenaRows><<<nblocks, kFwdThreads, kFwdSmem, s>>>(net, r);
}

void launchPredictSamples(cudaStream_t s, const Net& net, const Sample* samples, int64_t n, float* logits,
                          int32_t* pred, int nblocks) {
  SampleRows r{samples, n, logits, pred};
  cudaFuncSetAttribute(kForward<SampleRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
  kForward<SampleRows><<<nblocks, kFwdThreads, kFwdSmem, s>>>(net, r);
}

void launchEvaluate(cudaStream_t s, const Net& net, const Sample* samples, int64_t n, unsigned long long* counts,
                    int nblocks) {
  EvalRows r{samples, n, counts};
  cudaFuncSetAttribute(kForward<EvalRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
  kForward<EvalRows><<<nblocks, kFwdThreads, kFwdSmem, s>>>(net, r);
}

void launchGrad(cudaStream_t s, const Net& net, const Sample* batch, int64_t n, float inv_count,
                const uint32_t* labelled, float* partial, int nblocks) {
  cudaFuncSetAttribute(kGrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kGSmem);
  kGrad<<<nblocks, kGThreads, kGSmem, s>>>(net, batch, n, inv_count, labelled, partial);
}

void launchCountLabelled(cudaStream_t s, const Sample* samples, int64_t n, int64_t b, int64_t first, int steps,
                         uint32_t* counts, uint32_t* num_boxes) {
  cudaMemsetAsync(counts, 0, steps * sizeof(uint32_t), s);
  cudaMemsetAsync(num_boxes, 0, sizeof(uint32_t), s);
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((b + 1023) / 1024, 256));
  if (n > 0) kCountLabelled<<<dim3((unsigned)blocks, steps), 256, 0, s>>>(samples, n, b, first, counts, num_boxes);
}

void launchReduceAdam(cudaStream_t s, const float* partial, int nparts, float* grad, float* params, float* m,
                      float* v, float lr, int step, float* mean_loss) {
  kReduceAdam<<<(kPartial + 31) / 32, kReduceThreads, 0, s>>>(
      partial, nparts, grad, params, m, v, lr, step, mean_loss);
}

void launchCollect(cudaStream_t s, const ArenaSource& src, const uint64_t* ray_key, const DomainDev* domains,
                   Sample* out, unsigned long long* filled, uint64_t capacity, int8_t* label, uint8_t* flag,
                   uint32_t* sel, uint32_t* nsel, uint32_t* block_tmp, int nblocks) {
  kCollectLabel<<<nblocks, 256, 0, s>>>(src, ray_key, domains, label, flag);
  launchCompact(s, flag, src.count, 1, 0, sel, nsel, nullptr, block_tmp, nblocks);
  kCollectWrite<<<nblocks, 256, 0, s>>>(src, label, sel, nsel, out, filled, capacity);
  kCollectAdvance<<<1, 1, 0, s>>>(nsel, filled, capacity);
}

int gradBlocks(int num_sms) { return num_sms; }

}  // namespace mlp
}  // namespace spray
