#include "scratch.hpp"

#include <cstdint>
#include <mutex>

namespace fc {
namespace host {

namespace {

constexpr int DEVICES = 64;
struct Pool {
  cudaMemPool_t pool = nullptr;
  int users = 0;
};
std::mutex pools_lock;
Pool pools[DEVICES];

// With the lock held: what the device's pool may keep, by its users.
void keep(Pool &q) {
  if (!q.pool) return;
  uint64_t most = q.users > 0 ? SCRATCH_KEEP : 0;
  cudaMemPoolSetAttribute(q.pool, cudaMemPoolAttrReleaseThreshold, &most);
  if (q.users == 0) cudaMemPoolTrimTo(q.pool, 0);
}

cudaMemPool_t pool_of(int device) {
  if (device < 0 || device >= DEVICES) return nullptr;
  std::lock_guard<std::mutex> g(pools_lock);
  Pool &q = pools[device];
  if (!q.pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    if (cudaMemPoolCreate(&q.pool, &props) != cudaSuccess) {
      cudaGetLastError();
      q.pool = nullptr;
      return nullptr;
    }
    keep(q);
  }
  return q.pool;
}

}  // namespace

ScratchUser::ScratchUser(int device) : device_(device) {
  if (device_ < 0 || device_ >= DEVICES) return;
  std::lock_guard<std::mutex> g(pools_lock);
  if (++pools[device_].users == 1) keep(pools[device_]);
}

ScratchUser::~ScratchUser() {
  if (device_ < 0 || device_ >= DEVICES) return;
  std::lock_guard<std::mutex> g(pools_lock);
  if (--pools[device_].users == 0) keep(pools[device_]);
}

Scratch::Scratch(size_t bytes, cudaStream_t stream) : stream_(stream) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  int device = 0;
  cudaMemPool_t pool = nullptr;
  if (cudaStreamIsCapturing(stream, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone &&
      cudaGetDevice(&device) == cudaSuccess)
    pool = pool_of(device);
  const cudaError_t e =
      pool ? cudaMallocFromPoolAsync(&p, bytes, pool, stream) : cudaMallocAsync(&p, bytes, stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
  }
}

Scratch::~Scratch() {
  if (p) cudaFreeAsync(p, stream_);
}

}  // namespace host
}  // namespace fc
