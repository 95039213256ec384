// Host build of the launch rules (csrc/eb_launch_rules.hpp).
#include "../../endobeams.jl_gb300/csrc/eb_launch_rules.hpp"

extern "C" int host_gmres_cta_threads(int asked) { return eb::gmres_cta_threads(asked); }
