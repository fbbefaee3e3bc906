// Internal declarations shared between the library's translation units.
#pragma once

#include <string>

#include "ns3d_gpu.h"
#include "ns3d_launch.cuh"

namespace ns3d {

// Validate `p` as ns3d_create does and fill the kernels' launch configuration
// (DevParams, scheme selection, segment lengths); the stream is left null.
ns3d_status build_launch_cfg(const ns3d_params* p, LaunchCfg* L, std::string* msg);

// ---- discrete adjoint launchers (ns3d_adjoint.cu), FP64 ----
// Number of n-sized scratch blocks adj_rhs_vjp needs in G, and its launches.
int adj_scratch_blocks(const LaunchCfg& L);
int adj_rhs_vjp_launches(const LaunchCfg& L);
// lamW += (dR/dW)^T lamR at state W, then what follows it pointwise in the
// reverse sweep (see k_adj_reduce): finish: lamW += (dU0/dW)^T lamU0; next > 0:
// that stage reversed, W its output and Wp its input state (lamR, lamU0 and lamW
// become that stage's). G: adj_scratch_blocks(L) x n, lg: 16 x n.
cudaError_t adj_rhs_vjp(const LaunchCfg& L, StateView W, double* G, double* lg, double* lamW, int finish, int next,
                        StateView Wp, double* lamU0, double* lamR, double dt);
// One stage reversed (see adj_stage_cell); lamWk and lamWp may be the same array.
cudaError_t adj_stage(const LaunchCfg& L, int stage, StateView Wk, StateView Wp,
                      const double* lamWk, double* lamU0, double* lamR, double* lamWp, double dt);
cudaError_t adj_seed_ke(const LaunchCfg& L, StateView W, double* lamW, double dV);

}  // namespace ns3d
