// C ABI of the learned proposal's kernels on caller-owned device buffers.
#include <cuda.h>

#include <algorithm>
#include <map>
#include <stdexcept>
#include <string>

#include "../../include/spray_gpu.h"
#include "mlp.cuh"

namespace spray {
int fail(int code, const std::string& msg);
}

namespace {

using spray::fail;
namespace ml = spray::mlp;
static_assert(sizeof(spray_mlp_sample) == sizeof(ml::Sample), "sample layout");

// A calling thread's workspace, kept between its calls (a call used to create a
// stream and allocate and free its buffers, 140 us around a kernel of 20) and
// freed when the thread ends: the per-CTA gradient partials (8 MB), a gradient,
// the labelled rows of up to kCountSteps batches and the boxes they name, and a pinned word that a
// timed-out wait sets.  Work runs on the thread's own default stream, so threads
// do not wait for one another; a call returns when its work is done, so one
// workspace per thread and device is enough.
constexpr int kCountSteps = 1024;

// The driver's number of the allocation that holds `p`, 0 for none.  Numbers are
// never given twice in a process, so a changed one tells that the allocation went
// away (cudaDeviceReset), also when its address is in use again.  30 ns.
unsigned long long allocationId(const void* p) {
  using Query = CUresult (*)(void*, CUpointer_attribute, CUdeviceptr);
  static const Query query = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &found) != cudaSuccess)
      f = nullptr;
    return reinterpret_cast<Query>(f);
  }();
  unsigned long long id = 0;
  if (!query || query(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS) return 0;
  return id;
}

struct Workspace {
  int device = -1, nsms = 0;
  int* err = nullptr;      // pinned, mapped
  int* err_dev = nullptr;  // the same word as the device addresses it
  unsigned long long err_id = 0;
  float* partial = nullptr;
  float* grad = nullptr;
  uint32_t* counts = nullptr;
  // Whether the buffers are still there: a reset of the device takes them all.
  // (Its context is current.)
  bool alive() const { return err && allocationId(err) == err_id; }
  void release() {
    if (err) cudaFreeHost(err);
    if (partial) cudaFree(partial);
    if (grad) cudaFree(grad);
    if (counts) cudaFree(counts);
    *this = Workspace{};
  }
};

struct Workspaces {
  std::map<int, Workspace> of;
  ~Workspaces() {
    for (auto& w : of)
      if (w.second.err && cudaSetDevice(w.first) == cudaSuccess && w.second.alive()) w.second.release();
  }
};
thread_local Workspaces t_workspaces;

// The calling thread's workspace on `device`, with the gradient buffers when
// training; makes the device current.
int setup(Workspace** out, int32_t device, bool training) {
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return fail(SPRAY_GPU_ECUDA, cudaGetErrorString(e));
  Workspace& w = t_workspaces.of[device];
  if (w.err && !w.alive()) w = Workspace{};
  if (!w.err) {
    e = cudaDeviceGetAttribute(&w.nsms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaHostAlloc(&w.err, sizeof(int), cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer(&w.err_dev, w.err, 0);
    if (e == cudaSuccess && (w.err_id = allocationId(w.err)) == 0) e = cudaErrorNotSupported;
    w.device = device;
  }
  if (e == cudaSuccess && training && !w.counts) {
    e = cudaMalloc(&w.partial, (size_t)ml::gradBlocks(w.nsms) * ml::kPartialPitch * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&w.grad, ml::kPartial * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&w.counts, (kCountSteps + 1) * sizeof(uint32_t));
  }
  if (e != cudaSuccess) {
    w.release();
    return fail(SPRAY_GPU_ECUDA, cudaGetErrorString(e));
  }
  *w.err = 0;
  *out = &w;
  return SPRAY_GPU_OK;
}

int finish(const Workspace& w) {
  cudaError_t e = cudaStreamSynchronize(cudaStreamPerThread);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return fail(SPRAY_GPU_ECUDA, cudaGetErrorString(e));
  if (*(volatile int*)w.err) return fail(SPRAY_GPU_ETIMEOUT, "a tensor-core wait gave up");
  return SPRAY_GPU_OK;
}

ml::Net net(const float* params, const float* boxes, const uint32_t* num_boxes, const float norm[4], int* err) {
  ml::Net n;
  n.params = params;
  n.boxes = boxes;
  n.num_boxes = 0;
  n.more_boxes = num_boxes;
  for (int c = 0; c < 3; ++c) n.norm.centre[c] = norm[c];
  n.norm.scale = norm[3];
  n.error = err;
  return n;
}

int gradGrid(int nsms, int64_t n) {
  const int64_t tiles = (n + ml::kTile - 1) / ml::kTile;
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, ml::gradBlocks(nsms)));
}

}  // namespace

extern "C" {

int32_t spray_mlp_param_count(void) { return ml::kParams; }

int spray_mlp_forward_dev(const float* params, const float* boxes, const float norm[4],
                          const spray_mlp_sample* samples, int64_t n, float* logits, int32_t* pred,
                          int32_t device) {
  if (!params || !boxes || !norm || (n > 0 && (!samples || !logits || !pred)))
    return fail(SPRAY_GPU_EINVAL, "null argument");
  if (n < 0) return fail(SPRAY_GPU_EINVAL, "negative sample count");
  try {
    Workspace* w = nullptr;
    if (int r = setup(&w, device, false)) return r;
    if (n == 0) return SPRAY_GPU_OK;
    const int64_t tiles = (n + ml::kTile - 1) / ml::kTile;
    const int grid = (int)std::min<int64_t>(tiles, w->nsms);
    ml::launchPredictSamples(cudaStreamPerThread, net(params, boxes, nullptr, norm, w->err_dev),
                             reinterpret_cast<const ml::Sample*>(samples), n, logits, pred, grid);
    return finish(*w);
  } catch (const std::exception& ex) {
    return fail(SPRAY_GPU_ECUDA, ex.what());
  }
}

int spray_mlp_grad_dev(const float* params, const float* boxes, const float norm[4],
                       const spray_mlp_sample* samples, int64_t n, float* grad, int32_t device) {
  if (!params || !boxes || !norm || !grad || (n > 0 && !samples)) return fail(SPRAY_GPU_EINVAL, "null argument");
  if (n < 0) return fail(SPRAY_GPU_EINVAL, "negative sample count");
  try {
    Workspace* w = nullptr;
    if (int r = setup(&w, device, true)) return r;
    const int g = gradGrid(w->nsms, n);
    const cudaStream_t st = cudaStreamPerThread;
    const ml::Sample* q = reinterpret_cast<const ml::Sample*>(samples);
    ml::launchCountLabelled(st, q, n, std::max<int64_t>(n, 1), 0, 1, w->counts, w->counts + kCountSteps);
    ml::launchGrad(st, net(params, boxes, w->counts + kCountSteps, norm, w->err_dev), q, n, 0.0f, w->counts, w->partial, g);
    ml::launchReduceAdam(st, w->partial, g, grad, nullptr, nullptr, nullptr, 0.0f, 0, nullptr);
    return finish(*w);
  } catch (const std::exception& ex) {
    return fail(SPRAY_GPU_ECUDA, ex.what());
  }
}

int spray_mlp_train_dev(float* params, float* adam_m, float* adam_v, const float* boxes, const float norm[4],
                        const spray_mlp_sample* samples, int64_t n, int32_t batch, float lr, int32_t steps,
                        int32_t first_step, float* losses, int32_t device) {
  if (!params || !adam_m || !adam_v || !boxes || !norm || !samples) return fail(SPRAY_GPU_EINVAL, "null argument");
  if (n <= 0 || batch <= 0 || steps < 0 || first_step < 1 || !(lr > 0.0f))
    return fail(SPRAY_GPU_EINVAL, "need n > 0, batch > 0, steps >= 0, first_step >= 1, lr > 0");
  try {
    Workspace* w = nullptr;
    if (int r = setup(&w, device, true)) return r;
    const int64_t b = std::min<int64_t>(batch, n);
    const int g = gradGrid(w->nsms, b);
    const cudaStream_t st = cudaStreamPerThread;
    const ml::Sample* q = reinterpret_cast<const ml::Sample*>(samples);
    ml::Net nt = net(params, boxes, w->counts + kCountSteps, norm, w->err_dev);
    for (int k = 0; k < steps; ++k) {
      // the labelled rows of the next batches, on the device
      if (k % kCountSteps == 0)
        ml::launchCountLabelled(st, q, n, b, k, std::min(kCountSteps, steps - k), w->counts,
                                w->counts + kCountSteps);
      const int64_t start = ((int64_t)k * b) % n;
      const int64_t len = std::min<int64_t>(b, n - start);
      ml::launchGrad(st, nt, q + start, len, 0.0f, w->counts + k % kCountSteps, w->partial, g);
      ml::launchReduceAdam(st, w->partial, g, w->grad, params, adam_m, adam_v, lr, first_step + k,
                           losses ? losses + k : nullptr);
    }
    return finish(*w);
  } catch (const std::exception& ex) {
    return fail(SPRAY_GPU_ECUDA, ex.what());
  }
}

}  // extern "C"
