// kgb_dissimilarity_inplace_device: the co-label proximity of
// kgb_dissimilarity_inplace, computed in place on buffers the caller already
// holds on the device, without allocating device memory.
//
// Who needs this: callers whose device memory is not theirs to allocate from.
// A PyTorch process whose caching allocator has reserved most of the GPU, a
// serving loop that must not call cudaMalloc/cudaFree once it is warm
// (cudaFree waits for the whole device, and a failed cudaMalloc mid-request
// is an outage), or a host whose device memory budget is fixed up front.
// They hand in device pointers and a stream; everything else this call needs
// lives in one statically sized __device__ array that the CUDA module
// carries.
//
// Scratch layout (kScratchBytes = 16 MiB, 256-byte aligned):
//   [0, 256)           header; int at offset 0 = "bad graph index seen" flag,
//                      cleared at the start of every call
//   [256, 16 MiB)      labels transposed to samples x stride (int32), which
//                      bounds samples * runs to kMaxLabelCells.  The stride is
//                      the runs rounded up to whole 16-byte vectors where that
//                      fits, else the runs themselves.
//
// The scratch is shared by every call on a device.  Two calls that overlap
// in time on one device (two host threads, or work still queued on another
// stream) race on it and give wrong results; callers must serialise them.

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>

#include "graph_ops.cuh"
#include "../../include/kodama_gb300.h"
#include "launch_count.cuh"

namespace kgb {
void set_last_error(const char* msg);
}  // namespace kgb

namespace {

constexpr size_t kScratchBytes = size_t(16) << 20;
constexpr size_t kHeaderBytes = 256;
constexpr size_t kMaxLabelCells = (kScratchBytes - kHeaderBytes) / sizeof(int);
constexpr int kMaxNeighbors = 2048;  // 8 warps x K x 8 bytes of shared memory <= 128 KB

static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];


struct Fail {
  int code;
  std::string msg;
};

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw Fail{KGB_ECUDA, std::string(what) + ": " + cudaGetErrorString(e)};
}

// Device address of g_scratch on the current device.  It is looked up on
// every call (cheap once the module is loaded), so a call after a
// cudaDeviceReset, which reloads the module and may move the array, uses
// the array's new address.  The first lookup on a device may load the
// module onto it, which is why the first call per device must not happen
// while a stream is being captured.
unsigned char* scratch_here() {
  void* p = nullptr;
  ck(cudaGetSymbolAddress(&p, g_scratch), "cudaGetSymbolAddress(scratch)");
  return static_cast<unsigned char*>(p);
}

// Restores the caller's current device when the call ends.
struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int device) {
    ck(cudaGetDevice(&prev), "cudaGetDevice");
    ck(cudaSetDevice(device), "cudaSetDevice");
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

void run(int32_t* gidx, float* gdist, int32_t samples, int32_t gk, const int32_t* res, int32_t runs,
         int32_t device, void* stream) {
  if (gidx == nullptr || gdist == nullptr || res == nullptr) throw Fail{KGB_EINVAL, "null pointer"};
  if (runs <= 0 || samples <= 0 || gk <= 0) {
    throw Fail{KGB_EINVAL, "KODAMADissimilarityInPlace requires a non-empty graph and label matrix."};
  }
  if (static_cast<size_t>(samples) * static_cast<size_t>(runs) > kMaxLabelCells) {
    throw Fail{KGB_EINVAL, "kgb_dissimilarity_inplace_device: samples * runs = " +
                               std::to_string(static_cast<long long>(samples) * runs) + " exceeds the static scratch (" +
                               std::to_string(kMaxLabelCells) + " labels, 16 MiB); use kgb_dissimilarity_inplace"};
  }
  if (gk > kMaxNeighbors) {
    throw Fail{KGB_EINVAL, "kgb_dissimilarity_inplace_device: neighbors = " + std::to_string(gk) +
                               " exceeds the supported maximum of " + std::to_string(kMaxNeighbors)};
  }
  int ndev = 0;
  ck(cudaGetDeviceCount(&ndev), "cudaGetDeviceCount");
  if (device < 0 || device >= ndev) {
    throw Fail{KGB_EINVAL, "kgb_dissimilarity_inplace_device: no CUDA device " + std::to_string(device)};
  }
  DeviceGuard guard(device);
  unsigned char* scratch = scratch_here();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int* bad = reinterpret_cast<int*>(scratch);
  int* lbs = reinterpret_cast<int*>(scratch + kHeaderBytes);
  const size_t total = static_cast<size_t>(samples) * gk;

  ck(cudaMemsetAsync(scratch, 0, kHeaderBytes, st), "clear scratch header");
  const int padded = kgb::label_stride(runs);
  const int stride = static_cast<size_t>(samples) * padded <= kMaxLabelCells ? padded : runs;
  // both launches report their own status, so an error left on the thread by
  // earlier, unrelated work is left alone
  ck(static_cast<cudaError_t>(kgb::transpose_runs(res, runs, samples, stride, lbs, st, gidx, total, bad)),
     "transpose and check indices");
  kgb::DissimArgs a{};
  a.n = samples;
  a.K = gk;
  a.runs = runs;
  a.in_one_based = 1;
  a.out_one_based = 1;
  a.idx = gidx;
  a.dist = gdist;
  a.lbs = lbs;
  a.stride = stride;
  a.out_idx = gidx;
  a.out_dist = gdist;
  a.bad = bad;
  ck(static_cast<cudaError_t>(kgb::dissimilarity(a, st)), "dissimilarity");
  int h_bad = 0;
  ck(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, st), "read index check");
  ck(cudaStreamSynchronize(st), "synchronize");
  if (h_bad != 0) throw Fail{KGB_EINVAL, "KODAMADissimilarityInPlace expects public one-based graph indices."};
}

}  // namespace

extern "C" int kgb_dissimilarity_inplace_device(int32_t* gidx, float* gdist, int32_t samples, int32_t gk,
                                                const int32_t* res, int32_t runs, int32_t device, void* stream) {
  try {
    run(gidx, gdist, samples, gk, res, runs, device, stream);
    return KGB_OK;
  } catch (const Fail& f) {
    kgb::set_last_error(f.msg.c_str());
    return f.code;
  } catch (const std::exception& e) {
    kgb::set_last_error(e.what());
    return KGB_EINTERNAL;
  }
}
