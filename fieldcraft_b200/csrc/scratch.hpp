// Stream-ordered device scratch for entry points without a handle of their own (the product's row
// copies, flexible CG's vectors). It comes from one memory pool per device that keeps at most
// SCRATCH_KEEP bytes between calls while any handle of this library is alive on the device, and
// gives everything back when the last one is destroyed. Without handles, and inside a stream
// capture, nothing is kept.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace fc {
namespace host {

// A synchronisation returns what the default pool has free to the system, so a scratch taken from it
// on every call is mapped anew every time: 0.45 ms beside a 0.06 ms product of 7 vectors with 24 624
// rows, 5.5 ms beside a 0.9 ms one of 64 with 345 744 (354 MB).
constexpr size_t SCRATCH_KEEP = (size_t)512 << 20;

// A handle's life on a device.
class ScratchUser {
 public:
  explicit ScratchUser(int device);
  ~ScratchUser();
  ScratchUser(const ScratchUser &) = delete;
  ScratchUser &operator=(const ScratchUser &) = delete;

 private:
  int device_;
};

// `bytes` on the current device, usable on `stream` from here to the destructor, which releases it
// on the stream. p is null when there was none to be had.
class Scratch {
 public:
  Scratch(size_t bytes, cudaStream_t stream);
  ~Scratch();
  Scratch(const Scratch &) = delete;
  Scratch &operator=(const Scratch &) = delete;
  void *p = nullptr;

 private:
  cudaStream_t stream_;
};

}  // namespace host
}  // namespace fc
