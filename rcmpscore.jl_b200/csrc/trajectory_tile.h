// Host interface of the tile trajectory kernel (internal to the library).
#pragma once
#include <cuda_runtime.h>
#include "trajectory.h"

namespace rcmps {

class Admission;   // capacity.h

cudaError_t tile_trajectory_init();       // constant tables on the current device
size_t tile_sync_bytes();                 // device bytes per state for the teams' flags and records
// Teams (clusters of (dp/16)^2 CTAs up to dp = 64, (dp/32)^2 above) per state for a launch of nstates
// states: 7 (one per channel; a few states at a time) or 1. 0: no cluster fits.
int tile_trajectory_teams(int dp, int nstates);
int tile_trajectory_ctas(int dp, int nstates);   // CTAs it keeps busy
// Admission of launches of several teams per state to their device. Teams of one state wait for one
// another, so every cluster of the launches in flight must be resident: two launches that share the SMs
// could each hold part of them and wait for the rest. Launches of one padded dimension have the same
// clusters and share the device up to the states it holds; another dimension waits until it is empty
// (Admission). Launches of one team per state need none.
class TilePass {
 public:
  void enter(int device, int dp, int nstates, cudaStream_t stream);
  void leave(cudaEvent_t done);   // waits for `done`, recorded behind the launches
  ~TilePass();                    // of a call that failed: waits for the stream
 private:
  Admission* admission_ = nullptr;
  int states_ = 0;
  cudaStream_t stream_ = nullptr;
};
// The quartic trajectories of the states with herm set. zero_samples: also clear the structurally
// zero sample tiles of packed Z2 states, which the kernel does not write.
cudaError_t tile_trajectory_launch(int dp, const TrajState* d_states, int nstates, const double* d_points, int npoints,
                                   const TrajControls& ctl, void* sync, int teams, bool zero_samples,
                                   cudaStream_t stream);

}  // namespace rcmps
