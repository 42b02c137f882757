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
  unsigned long long live, held;   // bytes of the pool in use, and the most since it last gave back
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
    bool wait = true;
    if (PerDevice* d = bytes_ ? of(device_) : nullptr) {
      std::lock_guard<std::mutex> lk(g_mu);
      d->live -= bytes_;
      wait = d->held > kKeptBytes;
      if (wait) d->held = d->live;
    }
    if (wait) cudaStreamSynchronize(stream_);
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
  PerDevice* const d = of(device_);
  cudaMemPool_t pool = nullptr;
  if (d) {
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
    pool = d->pool;
  }
  void* p = nullptr;
  if (pool && cudaMallocFromPoolAsync(&p, bytes, pool, stream_) == cudaSuccess) {
    bytes_ = bytes;
    std::lock_guard<std::mutex> lk(g_mu);
    d->live += bytes;
    if (d->held < d->live) d->held = d->live;
  } else {
    // the device's default pool may hold what this one cannot get
    cudaGetLastError();
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
