// Host build of the launch rules (csrc/eb_launch_rules.hpp).
#include "../../endobeams.jl_gb300/csrc/eb_launch_rules.hpp"

extern "C" int host_gmres_cta_threads(int asked) { return eb::gmres_cta_threads(asked); }
extern "C" int host_wide_elements(int64_t n_elem, int sms) { return eb::wide_elements(n_elem, sms); }
extern "C" int host_dense_reach(int k, int b) { return eb::dense_reach(k, b); }
extern "C" int host_dense_grids(int n, const int* nb, const int* b, int* side) {
  const std::vector<int> g = eb::dense_grids(std::vector<int>(nb, nb + n), std::vector<int>(b, b + n));
  std::copy(g.begin(), g.end(), side);
  return (int)g.size();
}
extern "C" int host_dense_many(int64_t tiles, int sms) { return eb::dense_many(tiles, sms); }
extern "C" int host_many_elements(int64_t n_elem, int sms) { return eb::many_elements(n_elem, sms); }
extern "C" int host_side_by_side(int beam_groups, int contact_groups, int64_t n_elem, int sms) {
  return eb::side_by_side(beam_groups, contact_groups, n_elem, sms);
}

// n simulations of (shared, band, inverse) bytes each; kind: wanted in, fitted out.
extern "C" void host_fit_precond(int n, const int64_t* bytes, int64_t room, int32_t* kind) {
  std::vector<eb::PrecondBytes> b(n);
  for (int s = 0; s < n; ++s) b[s] = {bytes[3 * s], bytes[3 * s + 1], bytes[3 * s + 2]};
  std::vector<int> k(kind, kind + n);
  eb::fit_precond(b, room, k);
  std::copy(k.begin(), k.end(), kind);
}

// A fake of the two device calls: the current device and how often it was set.
namespace {
int current = 0, sets = 0;
struct FakeDevice {
  static int get() { return current; }
  static void set(int d) { current = d; ++sets; }
};
}  // namespace

// The device during a scope for `device` entered with `caller` current; out: the device after it, set calls.
extern "C" int host_on_device(int caller, int device, int* out) {
  current = caller;
  sets = 0;
  int inside;
  {
    eb::OnDevice<FakeDevice> on(device);
    inside = current;
  }
  out[0] = current;
  out[1] = sets;
  return inside;
}
