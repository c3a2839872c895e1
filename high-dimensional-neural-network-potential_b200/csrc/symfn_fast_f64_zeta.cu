// symfn_fast_f64_zeta.cu -- FP64 kernels of the grid shapes whose zetas are read from
// the model.
#include "symfn_fast.cuh"

namespace hdnnp {

int run_sf_f64_zeta(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask) {
    switch (m.fast) {
        case 1: return run_spec<double, Spec<2, 2, 1>>(b, m, grad, st, ask);
        case 2: return run_spec<double, Spec<2, 4, 2>>(b, m, grad, st, ask);
        case 3: return run_spec<double, Spec<2, 4, 4>>(b, m, grad, st, ask);
        case 4: return run_spec<double, Spec<2, 8, 2>>(b, m, grad, st, ask);
        default: return 0;
    }
}

}  // namespace hdnnp
