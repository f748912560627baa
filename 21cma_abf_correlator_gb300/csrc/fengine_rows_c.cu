// fengine_rows_c.cu -- F-engine kernels of n_freq 4096, 6144, 8192 (fengine_rows.cuh),
// compiled apart so that the groups of lengths build in parallel.

#include "fengine_rows.cuh"

namespace corrgb {

corr_status fengine_launch_rows_c(int n_freq, const TwiddleTables &tw, const FengineArgs &a,
                                  int num_sms, cudaStream_t stream) {
    switch (n_freq) {
    case 4096: return launch_rows<4096>(a, tw, num_sms, stream);
    case 6144: return launch_rows<6144>(a, tw, num_sms, stream);
    case 8192: return launch_rows<8192>(a, tw, num_sms, stream);
    default: return failf(CORR_ERR_INTERNAL, "fengine_launch_rows_c: n_freq=%d", n_freq);
    }
}

} // namespace corrgb
