// symfn_fast.cu -- launches of the product-space symmetry-function kernels
// (symfn_fast.cuh) and the limit on their neighbour count.
#include "engine.h"

namespace hdnnp {

// symfn_fast_*.cu: the kernels by precision and kind of shape
int run_sf_f64(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask);
int run_sf_f32(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask);
int run_sf_f64_zeta(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask);
int run_sf_f32_zeta(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask);

static int run(const Batch& b, const DevModel& m, bool fp32, bool grad, cudaStream_t st, SfAsk ask = SfAsk::kNothing) {
    if (m.fast >= 5) return fp32 ? run_sf_f32(b, m, grad, st, ask) : run_sf_f64(b, m, grad, st, ask);
    return fp32 ? run_sf_f32_zeta(b, m, grad, st, ask) : run_sf_f64_zeta(b, m, grad, st, ask);
}

bool sf_fast_lists_atoms(const Batch& b, const DevModel& m, bool fp32) {
    return run(b, m, fp32, false, nullptr, SfAsk::kLists) || run(b, m, fp32, true, nullptr, SfAsk::kLists);
}

// The accepted neighbour counts: those for which two records of four values,
// three accumulators, an entry and an element byte per neighbour and the
// weights (two tensors) of a warp stay within 55 KB, a limit older than the
// kernels' present layout and kept so that the same batches run; and, of
// those, the ones whose warp of either pass fits into a block.
bool sf_fast_takes(const Batch& b, const DevModel& m, bool fp32) {
    const size_t mm = b.mmax > 0 ? ((b.mmax + 31) / 32) * 32 : 32, w = fp32 ? 4 : 8;
    auto a16 = [](size_t x) { return (x + 15) & ~size_t(15); };
    const size_t n = 2 * a16(4 * w * mm) + a16(mm) + 64 * sizeof(unsigned) + a16(sizeof(int) * (kMaxEl + 1)) +
                     a16(sizeof(int) * kMaxEl) + 3 * a16(w * mm) + a16(sizeof(int) * mm) + a16(w * m.g2max) +
                     2 * a16(w * m.nblk * fast_shape_p(m.fast));
    return 4 * n <= 220 * 1024 && run(b, m, fp32, false, nullptr, SfAsk::kFits) &&
           run(b, m, fp32, true, nullptr, SfAsk::kFits);
}

int launch_sf_values_fast(const Batch& b, const DevModel& m, bool fp32, cudaStream_t st) {
    return run(b, m, fp32, false, st);
}

int launch_sf_gradients_fast(const Batch& b, const DevModel& m, bool fp32, cudaStream_t st) {
    return run(b, m, fp32, true, st);
}

}  // namespace hdnnp
