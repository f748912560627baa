// fengine_rows_b.cu -- F-engine kernels of n_freq 10240, 12288 (fengine_rows.cuh),
// compiled apart so that the groups of lengths build in parallel.

#include "fengine_rows.cuh"

namespace corrgb {

corr_status fengine_launch_rows_b(int n_freq, const TwiddleTables &tw, const FengineArgs &a,
                                  int num_sms, cudaStream_t stream) {
    switch (n_freq) {
    case 10240: return launch_rows<10240>(a, tw, num_sms, stream);
    case 12288: return launch_rows<12288>(a, tw, num_sms, stream);
    default: return failf(CORR_ERR_INTERNAL, "fengine_launch_rows_b: n_freq=%d", n_freq);
    }
}

} // namespace corrgb
