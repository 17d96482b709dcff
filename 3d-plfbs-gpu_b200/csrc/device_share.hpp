// What this process's calls want of each device at the moment, in SMs, so that a
// march (march.cu), which holds its SMs step after step, gives way to them: a call
// that enqueues kernels holds a DeviceShare while it runs, and a march goes on only
// while it is alone or all of it fits on the SMs. The sums sit in page-locked
// memory where the march kernel reads them every few steps, so that it stops well
// within a millisecond of another call's beginning.
#ifndef PLFBS_DEVICE_SHARE_HPP
#define PLFBS_DEVICE_SHARE_HPP

#include <atomic>

namespace plfbs {

constexpr int kWholeDevice = 1 << 12;  // more than any device has

// The device's sum, or null past kMaxDevices. With the device current: the first
// call allocates page-locked memory.
std::atomic<int>* sms_wanted(int device);
// Where kernels read it (null: not page-locked, host only).
const int* sms_wanted_on_device(int device);

// Whether a march of n tiles goes on while w SMs are wanted in all.
#if defined(__CUDACC__)
__host__ __device__
#endif
inline bool march_fits(int w, int n, int sms) { return w == n || w <= sms; }

class DeviceShare {
 public:
  DeviceShare() = default;
  DeviceShare(int device, int sms) { take(device, sms); }
  ~DeviceShare() { drop(); }
  DeviceShare(const DeviceShare&) = delete;
  DeviceShare& operator=(const DeviceShare&) = delete;
  void take(int device, int sms) {
    drop();
    wanted_ = sms_wanted(device);
    n_ = sms;
    if (wanted_) *wanted_ += n_;
  }
  void drop() {
    if (wanted_) *wanted_ -= n_;
    wanted_ = nullptr;
    n_ = 0;
  }
  // What a march of n tiles, n in this share, sees.
  bool march_fits(int sms) const {
    return !wanted_ || plfbs::march_fits(wanted_->load(), n_, sms);
  }

 private:
  std::atomic<int>* wanted_ = nullptr;
  int n_ = 0;
};

}  // namespace plfbs

#endif
