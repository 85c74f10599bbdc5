// The slot DTW kernels (dtw_slots.cuh) with 32 lanes per pair.
#include "dtw_slots.cuh"

namespace dtwj {

void launch_dtw_slots32(int cells, const DevSeries& S, const DevSearch& Q, const int2* pairs,
                      const unsigned int* npairs, int num_sms, int warps, cudaStream_t st) {
  slots::launch_c<32, 2>(cells, S, Q, pairs, npairs, num_sms, st, warps);
}

}  // namespace dtwj
