// call.cu — see call.h.
#include "call.h"

#include <mutex>

namespace tgp {
namespace {

constexpr int kKept = 8;                       // idle streams a device
constexpr int kDevices = 64;                   // devices of a higher number keep none
constexpr unsigned long long kKeptBytes = 64ull << 20;

struct Idle {
  cudaStream_t s;
  cudaEvent_t e0, e1;
};
struct PerDevice {
  Idle idle[kKept];
  int count;
  cudaMemPool_t pool;
};
// plain data, so nothing runs at exit, when CUDA may be gone
PerDevice g_devices[kDevices];
std::mutex g_mu;
PerDevice* of(int device) { return device >= 0 && device < kDevices ? g_devices + device : nullptr; }

}  // namespace

Call::Call(int device) : device_(device) {
  if (cudaSetDevice(device) != cudaSuccess) return;
  if (PerDevice* d = of(device)) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (d->count > 0) {
      const Idle& k = d->idle[--d->count];
      stream_ = k.s;
      e0_ = k.e0;
      e1_ = k.e1;
      return;
    }
  }
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return;
  if (cudaEventCreate(&e0_) != cudaSuccess || cudaEventCreate(&e1_) != cudaSuccess) {
    if (e0_) cudaEventDestroy(e0_);
    cudaStreamDestroy(s);
    return;
  }
  stream_ = s;
}

Call::~Call() {
  if (!stream_) return;
  if (base_) {
    cudaFreeAsync(base_, stream_);
    // a pool gives memory back when a stream is waited for, not when it is freed
    unsigned long long held = 0;
    if (!pool_ || cudaMemPoolGetAttribute(pool_, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess ||
        held > kKeptBytes)
      cudaStreamSynchronize(stream_);
  }
  if (PerDevice* d = sound_ ? of(device_) : nullptr) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (d->count < kKept) {
      d->idle[d->count++] = {stream_, e0_, e1_};
      return;
    }
  }
  cudaStreamSynchronize(stream_);
  cudaEventDestroy(e0_);
  cudaEventDestroy(e1_);
  cudaStreamDestroy(stream_);
}

char* Call::memory(size_t bytes) {
  if (PerDevice* d = of(device_)) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!d->pool) {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = device_;
      cudaMemPool_t made = nullptr;
      unsigned long long keep = kKeptBytes;
      if (cudaMemPoolCreate(&made, &props) == cudaSuccess) {
        if (cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess)
          d->pool = made;
        else
          cudaMemPoolDestroy(made);
      }
    }
    pool_ = d->pool;
  }
  void* p = nullptr;
  if (!pool_ || cudaMallocFromPoolAsync(&p, bytes, pool_, stream_) != cudaSuccess) {
    // the device's default pool may hold what this one cannot get
    cudaGetLastError();
    pool_ = nullptr;
    if (cudaMallocAsync(&p, bytes, stream_) != cudaSuccess) {
      sound_ = false;
      return nullptr;
    }
  }
  return base_ = (char*)p;
}

bool Call::finish(float* ms) {
  bool ok = cudaEventRecord(e1_, stream_) == cudaSuccess;
  if (cudaStreamSynchronize(stream_) != cudaSuccess) ok = false;
  *ms = 0.f;
  cudaEventElapsedTime(ms, e0_, e1_);
  if (!ok) sound_ = false;
  return ok;
}

}  // namespace tgp
