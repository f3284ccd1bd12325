// Host interface of the tile trajectory kernel (internal to the library).
#pragma once
#include <cuda_runtime.h>
#include <mutex>
#include "trajectory.h"

namespace rcmps {

cudaError_t tile_trajectory_init();       // constant tables on the current device
std::mutex& tile_trajectory_mutex(int device);   // held while a launch of several teams is in flight
size_t tile_sync_bytes();                 // device bytes per state for the teams' flags and records
// Teams (clusters of (dp/16)^2 CTAs up to dp = 64, (dp/32)^2 above) per state for a launch of nstates
// states: 7 (one per channel; a few states at a time) or 1. 0: no cluster fits.
int tile_trajectory_teams(int dp, int nstates);
int tile_trajectory_ctas(int dp, int nstates);   // CTAs it keeps busy
// The quartic trajectories of the states with herm set. zero_samples: also clear the structurally
// zero sample tiles of packed Z2 states, which the kernel does not write.
cudaError_t tile_trajectory_launch(int dp, const TrajState* d_states, int nstates, const double* d_points, int npoints,
                                   const TrajControls& ctl, void* sync, int teams, bool zero_samples,
                                   cudaStream_t stream);

}  // namespace rcmps
