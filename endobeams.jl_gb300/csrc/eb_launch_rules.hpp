// Rules of the launches that need no CUDA (host only).
#pragma once
#include <algorithm>
#include <cstdint>
#include <numeric>
#include <vector>

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

// Element launches of more than twenty elements per SM start with thirty elements a CTA, others with ten.
inline bool wide_elements(int64_t n_elem, int sms) { return n_elem > 20 * (int64_t)sms; }

// Element launches that run a thread per element instead of thirty elements a CTA: 168 registers let an SM hold
// 384 threads, whose dependent chains then fill the FP64 pipe better than a CTA's phases with their barriers and
// unequal warps (element passes of a step, ms: 76,000 elements 5.8 -> 5.2, 389,000 31.8 -> 25.4, 642,000 53.2 ->
// 40.8).  A second wave must be worth its chain: 60,800 elements, just over one wave, took 5.1, where thirty a CTA
// at 76 ns an element would take 4.6; hence the line at one wave and a sixth.
inline bool many_elements(int64_t n_elem, int sms) { return n_elem > 448 * (int64_t)sms; }

// Whether the element and the contact pass, which do not depend on each other, run side by side (152 SMs, 64-element
// ring: a step 1.66 -> 1.43 ms, 9,600 elements 16.6 -> 15.8 ms).  Not where both have thirty elements a CTA (three
// groups) and fewer than two CTAs per SM: two such CTAs on an SM compete for its L1, through which the elements'
// temporaries go, while other SMs idle (3,600 elements: 5.14 -> 5.93 ms).  The limit was not measured more closely
// than between these two sizes.
inline bool side_by_side(int beam_groups, int contact_groups, int64_t n_elem, int sms) {
  return !(beam_groups == 3 && contact_groups == 3 && n_elem < 2 * 30 * (int64_t)sms);
}

// What a simulation's preconditioner is, and the device bytes each choice takes.
enum PrecondKind { kPrecondJacobi = 0, kPrecondBand = 1, kPrecondInverse = 2 };
struct PrecondBytes {
  int64_t shared = 0;   // condensation: blocks and lists, whichever of the two follows
  int64_t band = 0;     // 0: too wide for the band LU
  int64_t inverse = 0;
};

// Fits the simulations' choices into `room` bytes: inverses that take more than the band of the same kept
// nodes become bands, the largest gain first; where that is not enough, all become block-Jacobi.
inline void fit_precond(const std::vector<PrecondBytes>& b, int64_t room, std::vector<int>& kind) {
  int64_t need = 0;
  std::vector<int> swap;
  for (size_t s = 0; s < b.size(); ++s) {
    if (kind[s] == kPrecondJacobi) continue;
    need += b[s].shared + (kind[s] == kPrecondInverse ? b[s].inverse : b[s].band);
    if (kind[s] == kPrecondInverse && b[s].band > 0 && b[s].band < b[s].inverse) swap.push_back((int)s);
  }
  std::stable_sort(swap.begin(), swap.end(), [&](int x, int y) { return b[x].inverse - b[x].band > b[y].inverse - b[y].band; });
  for (int s : swap) {
    if (need <= room) return;
    kind[s] = kPrecondBand;
    need -= b[s].inverse - b[s].band;
  }
  if (need > room) std::fill(kind.begin(), kind.end(), (int)kPrecondJacobi);
}

// Blocks [0, dense_reach) of 64 rows and columns that pivot block k of an in-place Gauss-Jordan can change, for a
// matrix of half bandwidth b: what the pivots before it have filled ends b entries past them, and beyond
// the reach the pivot block's column and row are still zero.
#if defined(__CUDACC__)
__host__ __device__
#endif
inline int dense_reach(int k, int b) { return k + 1 + (63 + b) / 64; }

// Per pivot block, the most blocks a side that it can change in any simulation (nb: blocks of 64 a side, b:
// half bandwidths): the grids of a step.  With grids of the largest matrix whole, half of a step's CTAs on
// average had nothing to do but to find that out.
inline std::vector<int> dense_grids(const std::vector<int>& nb, const std::vector<int>& b) {
  std::vector<int> side(nb.empty() ? 0 : *std::max_element(nb.begin(), nb.end()), 0);
  for (size_t s = 0; s < nb.size(); ++s)
    for (int k = 0; k < nb[s]; ++k) side[k] = std::max(side[k], std::min(nb[s], dense_reach(k, b[s])));
  return side;
}

// Steps of an inversion (64 x 64 tiles in all) that run 64 threads a tile: with fewer tiles an SM the
// 256-thread kernel's shorter chain wins (a factorisation in ms, 256 and 64 threads: 8 nets of 33 x 33, 33 tiles an SM, 2.4 and
// 2.5; 16, 66 an SM, 3.9 and 4.0; 64 of 20 x 20, 95 an SM, 3.2 and 3.2; 304 of 33 x 33 62 and 55).
inline bool dense_many(int64_t tiles, int sms) { return tiles > 80 * (int64_t)sms; }

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
