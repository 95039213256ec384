// Rules of the launches that need no CUDA (host only).
#pragma once

namespace eb {

constexpr int kGmresMaxThreads = 512;

// CTA size of k_gmres for the caller's threads_per_sim: whole warps, because a warp owns whole chunks of
// the vectors (fewer than 32 threads would own none and never finish, a partial warp would share
// chunks with another), and at least two of them (the band sweeps' near and far rows).  The results
// do not depend on it.  0: the library's choice; -1: refused.
inline int gmres_cta_threads(int asked) {
  if (asked <= 0) return 0;
  if (asked > kGmresMaxThreads) return -1;
  const int whole = (asked + 31) / 32 * 32;
  return whole < 64 ? 64 : whole;
}

// Makes `device` the thread's current one for a scope, for entry points that launch on a handle's
// stream where the caller may have another device current (copies need no such thing).
template <typename Api>
class OnDevice {
 public:
  explicit OnDevice(int device) : back_(Api::get()), changed_(back_ != device) {
    if (changed_) Api::set(device);
  }
  ~OnDevice() {
    if (changed_) Api::set(back_);
  }
  OnDevice(const OnDevice&) = delete;
  OnDevice& operator=(const OnDevice&) = delete;

 private:
  int back_;
  bool changed_;
};

}  // namespace eb
