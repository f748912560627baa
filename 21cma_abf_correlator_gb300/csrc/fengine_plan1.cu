// fengine_plan1.cu -- F-engine FFT plan 1 of n_freq 16384 (fengine_impl.cuh),
// compiled apart so that the groups of lengths build in parallel.

#include "fengine_impl.cuh"

namespace corrgb {

corr_status fengine_launch_plan1(const TwiddleTables &tw, const FengineArgs &a, int num_sms,
                                 cudaStream_t stream) {
    return launch_plan<16384, 1>(a, tw, num_sms, stream);
}

} // namespace corrgb
