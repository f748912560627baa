// fengine_rows_a.cu -- F-engine kernels of n_freq 14336, 16384 (fengine_rows.cuh),
// compiled apart so that the groups of lengths build in parallel.

#include "fengine_rows.cuh"

namespace corrgb {

corr_status fengine_launch_rows_a(int n_freq, const TwiddleTables &tw, const FengineArgs &a,
                                  int num_sms, cudaStream_t stream) {
    switch (n_freq) {
    case 14336: return launch_rows<14336>(a, tw, num_sms, stream);
    case 16384: return launch_rows<16384>(a, tw, num_sms, stream);
    default: return failf(CORR_ERR_INTERNAL, "fengine_launch_rows_a: n_freq=%d", n_freq);
    }
}

} // namespace corrgb
