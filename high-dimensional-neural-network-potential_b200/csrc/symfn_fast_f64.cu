// symfn_fast_f64.cu -- FP64 kernels of the grid shapes with compiled zetas.
#include "symfn_fast.cuh"

namespace hdnnp {

int run_sf_f64(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask) {
    switch (m.fast) {
        case 5: return run_spec<double, Spec<2, 2, 1, 1, 4>>(b, m, grad, st, ask);
        case 6: return run_spec<double, Spec<2, 4, 2, 1, 2, 4, 16>>(b, m, grad, st, ask);
        default: return 0;
    }
}

}  // namespace hdnnp
