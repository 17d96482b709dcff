// The sums of device_share.hpp: one cache line per device, page-locked and mapped
// for all devices, allocated at the first use and kept for the process.
#include "device_share.hpp"

#include <cuda_runtime.h>

#include <new>

#include "plfbs_internal.hpp"

namespace plfbs {
namespace {

struct alignas(128) Line {
  std::atomic<int> sms{0};
};
static_assert(sizeof(std::atomic<int>) == sizeof(int) && std::atomic<int>::is_always_lock_free,
              "read as an int by kernels");

struct Sums {
  Line* line;
  bool pinned;
};

Sums sums() {
  static const Sums s = [] {
    static Line host[kMaxDevices];
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(Line) * kMaxDevices,
                      cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      return Sums{host, false};
    }
    Line* line = static_cast<Line*>(p);
    for (int d = 0; d < kMaxDevices; d++) new (&line[d]) Line();
    return Sums{line, true};
  }();
  return s;
}

}  // namespace

std::atomic<int>* sms_wanted(int device) {
  return device >= 0 && device < kMaxDevices ? &sums().line[device].sms : nullptr;
}

const int* sms_wanted_on_device(int device) {
  if (device < 0 || device >= kMaxDevices || !sums().pinned) return nullptr;
  void* p = nullptr;
  if (cudaHostGetDevicePointer(&p, &sums().line[device].sms, 0) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return static_cast<const int*>(p);
}

}  // namespace plfbs
