// symfn_fast.cu -- launches of the product-space symmetry-function kernels
// (symfn_fast.cuh) and the limit on their neighbour count.
#include "engine.h"

namespace hdnnp {

static size_t a16(size_t x) { return (x + 15) & ~size_t(15); }

// The bytes per warp by which the pipeline limits the neighbour count (times
// 4 against 220 KB): vectors and factors of 4 values, three accumulators, the
// entry and the element of each neighbour, and the weight tensors.
size_t sf_fast_smem_per_warp(int mmax, int g2max, int nblk, int P, bool grad, bool fp32) {
    const size_t mm = mmax > 0 ? ((mmax + 31) / 32) * 32 : 32, w = fp32 ? 4 : 8;
    size_t n = 2 * a16(4 * w * mm) + a16(mm) + 64 * sizeof(unsigned) + a16(sizeof(int) * (kMaxEl + 1)) + a16(sizeof(int) * kMaxEl);
    if (grad) n += 3 * a16(w * mm) + a16(sizeof(int) * mm) + a16(w * g2max) + 2 * a16(w * nblk * P);
    else n += a16(w * 32 * (P + 1)) + (fp32 ? a16(sizeof(double4) * mm) : 0);
    return n;
}

// symfn_fast_*.cu: the kernels by precision and kind of shape
int run_sf_f64(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, bool query);
int run_sf_f32(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, bool query);
int run_sf_f64_zeta(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, bool query);
int run_sf_f32_zeta(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, bool query);

static int run(const Batch& b, const DevModel& m, bool fp32, bool grad, cudaStream_t st, bool query = false) {
    if (m.fast >= 5) return fp32 ? run_sf_f32(b, m, grad, st, query) : run_sf_f64(b, m, grad, st, query);
    return fp32 ? run_sf_f32_zeta(b, m, grad, st, query) : run_sf_f64_zeta(b, m, grad, st, query);
}

bool sf_fast_lists_atoms(const Batch& b, const DevModel& m, bool fp32) {
    return run(b, m, fp32, false, nullptr, true) || run(b, m, fp32, true, nullptr, true);
}

int launch_sf_values_fast(const Batch& b, const DevModel& m, bool fp32, cudaStream_t st) {
    return run(b, m, fp32, false, st);
}

int launch_sf_gradients_fast(const Batch& b, const DevModel& m, bool fp32, cudaStream_t st) {
    return run(b, m, fp32, true, st);
}

}  // namespace hdnnp
