// Test infrastructure: what the condensation plan (endobeams.jl_gb300/csrc/eb_cond_plan.hpp) costs by its own
// prices, against no condensation at all.
#include <algorithm>

#include "../../endobeams.jl_gb300/csrc/eb_cond_plan.hpp"

using namespace eb;

// a x b grid of nodes; out: kept DOFs, half bandwidth, levels; cost: of the plan, of the whole band.
extern "C" void host_grid_plan(int a, int b, int max_w, int max_dense, int stage_b, int* out, double* cost) {
  std::vector<std::vector<int>> adj(a * b);
  for (int i = 0; i < a; ++i)
    for (int j = 0; j < b; ++j) {
      const int v = i * b + j;
      if (i) adj[v].push_back(v - b);
      if (j) adj[v].push_back(v - 1);
      if (j + 1 < b) adj[v].push_back(v + 1);
      if (i + 1 < a) adj[v].push_back(v + b);
    }
  CondPlan P;
  cond_plan(adj, max_w, max_dense, P, stage_b);
  const int kept = P.n - P.ne;
  out[0] = 6 * kept;
  out[1] = 6 * P.w + 5;
  out[2] = (int)P.lev_ptr.size() - 1;
  std::vector<int> pos;
  const int w = rcm_order(adj, pos);
  cost[0] = level_cost(a * b) * out[2] + 144e-6 * P.red0 +
            cond_cost(kept, P.w, 6 * kept <= max_dense ? max_dense : 0, stage_b);
  cost[1] = cond_cost(a * b, w, 0, stage_b);
}
