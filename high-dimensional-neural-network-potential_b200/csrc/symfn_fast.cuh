// symfn_fast.cuh -- K4/K6 symmetry-function kernels on the potential's
// lambda x zeta x eta grid ("product space"), FP64 or FP32.
//
// Same mathematics as symfn.cu (calcAllSymmetryFunctions,
// symmetryFunctions.f90:158-308; scaling hdnnps.f90:471-481), organised so
// that the per-(pair, SF) work is one fused multiply-add:
//   * per neighbour (staging): everything that depends on it alone, 1/r and
//     P_e = fc exp(-eta_e r^2) for every distinct eta;
//   * per pair: cos from the three squared distances, X_l = 1 + lambda_l cos,
//     one square chain X, X^2, X^4, ... shared by every zeta, T_lz =
//     X_l^zeta_z (and X_l^(zeta_z - 1) for the gradient), fc(r_jk) and one
//     exp(-eta_e r_jk^2) per eta;
//   * pass 1 adds acc[l,z,e] += T_lz Y_e, Y_e = P_je P_ke exp(-eta_e r_jk^2)
//     fc(r_jk), on the FP64 tensor cores and maps the product entries to SF
//     indices (G_s = 2^(1-zeta) acc[l,z,e]);
//   * pass 2 stages per element-pair block the weight tensor WA[l,z,e] = w_s
//     2^(1-zeta) (w_s = dE/dG_s / (max_s - min_s)), contracts it with the
//     powers and their derivatives, and takes dE/dr_j and dE/dr_k from the
//     derivatives with respect to r_ij^2, r_ik^2 and r_jk^2.
// A warp per centre atom; neighbours staged in shared memory sorted by
// element; the contributing pairs (r_jk < rc) compacted into lists of which a
// chunk of 32 is evaluated at a time, one pair per lane.
//
// The kernels of a precision and a group of grid shapes are compiled in a
// source file of their own (symfn_fast_f64.cu and the others): a process
// loads the code of those that it runs (1.0-3.6 ms before its first
// evaluation; all of them in one file 13.7).
#pragma once
#include <algorithm>

#include "engine.h"
#include "fastmath.cuh"

namespace hdnnp {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = 4;
// parts of a pass: one launch for all atoms, or one for those with few
// neighbours and one for the listed others
constexpr int kPartAll = 0, kPartFirst = 1, kPartWide = 2;
// Resident blocks per SM that the kernels are compiled for (registers) and
// the default split of a pass is sized for (shared memory): value pass 5 FP64
// (96 registers) and 6 FP32; gradient pass 4 FP64 (122 registers, no spills;
// at 5 its four accumulator copies leave 44 neighbours and the pass takes
// 5.4 ms instead of 3.6 on 1024 structures) and 6 FP32 (2.31 ms, 2.44 at 7
// with spills).
template <typename T>
constexpr int kBlocksV = sizeof(T) == 4 ? 6 : 5;
template <typename T>
constexpr int kBlocksG = sizeof(T) == 4 ? 6 : 4;

template <typename T>
struct alignas(4 * sizeof(T)) V4 {
    T x, y, z, w;
};

__host__ __device__ inline size_t a16(size_t x) { return (x + 15) & ~size_t(15); }

// ---------------------------------------------------------------- grid specs
// Spec<NL, NZ, NE, Z0..Z3>: compiled shape of the lambda x zeta x eta grid.
// With Z0 > 0 the zeta values are compile-time constants (the power chain and
// every product are straight-line code); with Z0 == 0 they are read from the
// model (uniform branches).
template <int NL_, int NZ_, int NE_, int Z0 = 0, int Z1 = 0, int Z2 = 0, int Z3 = 0>
struct Spec {
    static constexpr int NL = NL_, NZ = NZ_, NE = NE_, P = NL_ * NZ_ * NE_;
    static constexpr bool kFixed = Z0 > 0;
    __host__ __device__ static constexpr int zeta(int z) { return z == 0 ? Z0 : z == 1 ? Z1 : z == 2 ? Z2 : Z3; }
    __host__ __device__ static constexpr int maxbit() {
        int mz = 1;
        for (int z = 0; z < NZ_; ++z) mz = zeta(z) > mz ? zeta(z) : mz;
        int b = 0;
        while ((1 << (b + 1)) <= mz) ++b;
        return b;
    }
};

template <class S>
__device__ __forceinline__ double zeta_of(const DevModel& m, int z) {
    return S::kFixed ? (double)S::zeta(z) : m.zet[z];
}

template <class S>
__device__ __forceinline__ int n_eta(const DevModel& m) {
    return S::kFixed ? S::NE : m.fe;
}

// values per neighbour in FSmem::ax: 1/r, rank of the element (value pass,
// an integer in the low bits) or rho (gradient pass) and P_e = fc exp(-eta_e r^2) of every eta, padded to whole vectors
template <class S>
constexpr int kAx = (S::NE + 3) & ~1;
// rows and row stride of the value pass's term buffer (tensor-core A rows)
template <class S>
constexpr int kTRows = ((S::NL * S::NZ + 7) / 8) * 8;
constexpr int kTs = 36;
// row stride of the gradient pass's weight tensors: rows of different blocks
// on different banks (lanes of a chunk read several)
template <class S>
constexpr int kWp = S::P + 4;

// copies of the gradient accumulators, one per group of 32 / kCopies lanes
constexpr int kCopies = 4;

template <typename T>
struct FSmem {
    V4<T>* nb;      // dx, dy, dz, r^2      (centre - neighbour)
    double4* dd;    // FP32 value pass: the FP64 relative vector (x, y, z, -) for the pair cutoff
    float4* sp;     // FP64 value pass: FP32 copy of the relative vector for the candidate test
    T* rf;          // value pass: r and fc for the radial functions; sp takes the place afterwards
    T* ax;          // [mm][kAx] per-neighbour factors
    T* gx;          // gradient accumulators (pass 2): kCopies copies of an array
    int gst;        // per component, gst values apart (a slot's x, y, z in one
                    // 16- or 32-byte record put random slots on 4 (FP64) or 8
                    // (FP32) bank groups only)
    int* ent;       // entry index of a slot (pass 2)
    unsigned* queue;  // contributing pairs j | k << 10 (pass 1: kListCap or more; pass 2: ring of 64 with the block)
    unsigned* mask;   // [mm/32][32] contributing neighbours k > j of the rows j of a batch (pass 1)
    unsigned char* tm;  // [nel][nel] element-pair block of two ranks, 255: no functions (pass 1)
    int* est;         // first slot of an element
    int* cnt;         // its slots
    int* rst;         // first slot of a rank, [nel + 1]
    int* ord;         // element of a rank
    T* w2;          // dE/dG / width of the centre's radial SFs (pass 2)
    T* WA;          // [nblk][P] (pass 2)
    T* tb;          // [kTRows][kTs] powers of a chunk's pairs (pass 1)
    T* yb;          // [8 columns][kTs] their exponential and cutoff factors, zero between uses (pass 1)
};

__host__ __device__ inline int mask_words(int mm) { return (mm + 31) / 32 * 32; }
// pairs the value pass lists at a time: a row (one neighbour's pairs) and a
// chunk's remainder always fit
// (1024 structures, value pass in ms: FP64 3.50, 3.43, 3.47 at 160, 192, 224;
// FP32 2.86, 2.71, 2.93 at 160, 320, 640: fewer refills against fewer
// neighbours per warp)
template <typename T>
constexpr int kListCap = sizeof(T) == 4 ? 320 : 192;
template <typename T>
__host__ __device__ inline int list_cap(int mm) { return mm + 32 > kListCap<T> ? mm + 32 : kListCap<T>; }

template <typename T, class S>
__host__ __device__ inline size_t fast_warp_bytes(int mm, int nel, int g2max, int nblk, bool grad) {
    size_t b = a16(sizeof(V4<T>) * mm) + a16(sizeof(T) * kAx<S> * mm);
    if (grad) b += kCopies * 3 * a16(sizeof(T) * mm) + a16(sizeof(int) * mm) + a16(sizeof(T) * g2max) + a16(sizeof(T) * nblk * kWp<S>);
    else b += (sizeof(T) == 4 ? a16(sizeof(double4) * mm) : 0) + a16(2 * sizeof(T) * mm) +
              (kTRows<S> + 8) * kTs * sizeof(T) + a16(sizeof(unsigned) * mask_words(mm)) + a16(nel * nel);
    b += a16(sizeof(unsigned) * (grad ? 64 : list_cap<T>(mm))) + 3 * a16(sizeof(int) * kMaxEl) + a16(sizeof(int) * (kMaxEl + 1));
    return b;
}

template <typename T, class S>
__device__ inline FSmem<T> fcarve(unsigned char* p, int mm, int nel, int g2max, int nblk, bool grad) {
    FSmem<T> s{};
    auto take = [&](size_t bytes) {
        unsigned char* q = p;
        p += a16(bytes);
        return q;
    };
    s.nb = (V4<T>*)take(sizeof(V4<T>) * mm);
    s.ax = (T*)take(sizeof(T) * kAx<S> * mm);
    if (grad) {
        s.gx = (T*)take(kCopies * 3 * a16(sizeof(T) * mm));
        s.gst = (int)(a16(sizeof(T) * mm) / sizeof(T));
        s.ent = (int*)take(sizeof(int) * mm);
        s.w2 = (T*)take(sizeof(T) * g2max);
        s.WA = (T*)take(sizeof(T) * nblk * kWp<S>);
    } else {
        if (sizeof(T) == 4) s.dd = (double4*)take(sizeof(double4) * mm);
        s.rf = (T*)take(2 * sizeof(T) * mm);
        s.sp = (float4*)s.rf;
        s.tb = (T*)take(kTRows<S> * kTs * sizeof(T));
        s.yb = (T*)take(8 * kTs * sizeof(T));
        s.mask = (unsigned*)take(sizeof(unsigned) * mask_words(mm));
        s.tm = (unsigned char*)take(nel * nel);
    }
    s.queue = (unsigned*)take(sizeof(unsigned) * (grad ? 64 : list_cap<T>(mm)));
    s.est = (int*)take(sizeof(int) * kMaxEl);
    s.cnt = (int*)take(sizeof(int) * kMaxEl);
    s.rst = (int*)take(sizeof(int) * (kMaxEl + 1));
    s.ord = (int*)take(sizeof(int) * kMaxEl);
    return s;
}

// one neighbour's factors (kAx of them) in 16- or 8-byte loads
template <int A, typename T>
__device__ __forceinline__ void ldax(const T* ax, int slot, T (&v)[A]) {
    if constexpr (A % 4 == 0 && sizeof(T) == 4) {
#pragma unroll
        for (int q = 0; q < A / 4; ++q) {
            const float4 x = reinterpret_cast<const float4*>(ax + slot * A)[q];
            v[4 * q] = x.x;
            v[4 * q + 1] = x.y;
            v[4 * q + 2] = x.z;
            v[4 * q + 3] = x.w;
        }
    } else {
        struct alignas(2 * sizeof(T)) V2 { T x, y; };
#pragma unroll
        for (int q = 0; q < A / 2; ++q) {
            const V2 x = reinterpret_cast<const V2*>(ax + slot * A)[q];
            v[2 * q] = x.x;
            v[2 * q + 1] = x.y;
        }
    }
}

// P consecutive weights of one block from shared memory in 16-byte loads
// (P is a multiple of 4; each block's tensor starts on a 16-byte boundary).
template <int P>
__device__ __forceinline__ void ldvec(const float* p, float (&w)[P]) {
#pragma unroll
    for (int q = 0; q < P / 4; ++q) {
        const float4 v = reinterpret_cast<const float4*>(p)[q];
        w[4 * q] = v.x;
        w[4 * q + 1] = v.y;
        w[4 * q + 2] = v.z;
        w[4 * q + 3] = v.w;
    }
}
template <int P>
__device__ __forceinline__ void ldvec(const double* p, double (&w)[P]) {
#pragma unroll
    for (int q = 0; q < P / 2; ++q) {
        const double2 v = reinterpret_cast<const double2*>(p)[q];
        w[2 * q] = v.x;
        w[2 * q + 1] = v.y;
    }
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// precision-dispatched math.  FP64: the branch-free forms of fastmath.cuh
// for the bounded arguments of these kernels (exp of -eta r^2, tanh of
// u = 1 - r/rc in [0, 1], square roots of squared distances).
__device__ __forceinline__ double xsqrt(double x) {
    double r, ir;
    sqrt_rsqrt(x, r, ir);
    return r;
}
__device__ __forceinline__ float xsqrt(float x) { return sqrtf(x); }
// r and 1/r from r^2 > 0: FP64 by the refined reciprocal square root of
// fastmath.cuh, FP32 by rsqrtf (2 ulp) and a product
__device__ __forceinline__ void dist_inv(double r2, double& r, double& ir) { sqrt_rsqrt(r2, r, ir); }
__device__ __forceinline__ void dist_inv(float r2, float& r, float& ir) {
    ir = rsqrtf(r2);
    r = r2 * ir;
}
// a / b: FP64 by division; FP32 by the fast reciprocal-based form (2 ulp,
// b between 2^-126 and 2^126)
__device__ __forceinline__ double xdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float xdiv(float a, float b) { return __fdividef(a, b); }
// FP32 form: the exp2-based intrinsic (max error 2 + floor(1.173 |x|) ulp;
// the angular arguments stay below ~5, where it is within 8 ulp)
__device__ __forceinline__ float xexp(float x) { return __expf(x); }
// tanh of a cutoff argument u = 1 - r/rc in [0, 1]
__device__ __forceinline__ double xtanh(double x) { return tanh01(x); }
__device__ __forceinline__ float xtanh(float x) { return tanhf(x); }

// exp of an angular -eta r^2 and of a radial -eta (r - rs)^2.  kB: every
// argument of the potential's functions is in the range of the functions
// without range tests (DevModel::exp_bounded); a template parameter, so that
// only one form is in a kernel's code.
template <bool kB>
__device__ __forceinline__ double ang_exp(double x) { return kB ? exp_small(x) : exp_clamped(x); }
template <bool kB>
__device__ __forceinline__ float ang_exp(float x) { return xexp(x); }
template <bool kB>
__device__ __forceinline__ double rad_exp(double x) { return kB ? exp_neg(x) : exp_clamped(x); }
template <bool kB>
__device__ __forceinline__ float rad_exp(float x) { return xexp(x); }

// E[e] = exp(-eta_e s) of a pair's r_jk^2 = s for the distinct etas of the
// grid (zero beyond ne).  kB (DevModel::exp_bounded): FP64 without range
// reduction.
template <int NE, bool kB, typename T>
__device__ __forceinline__ void eta_exps(const DevModel& m, int ne, T s, T (&E)[NE]) {
#pragma unroll
    for (int e = 0; e < NE; ++e) E[e] = e < ne ? ang_exp<kB>(-(T)m.eta4[e] * s) : (T)0;
}

template <typename T> struct Buf;
template <> struct Buf<double> {
    static __device__ double* G(const Batch& b) { return b.G; }
    static __device__ const double* dEdG(const Batch& b) { return b.dEdG; }
    static __device__ double* gent(const Batch& b) { return b.gent; }
    static __device__ double* gself(const Batch& b) { return b.gself; }
    static __device__ double* vir(const Batch& b) { return b.vir; }
};
template <> struct Buf<float> {
    static __device__ float* G(const Batch& b) { return b.Gf; }
    static __device__ const float* dEdG(const Batch& b) { return b.dEdGf; }
    static __device__ float* gent(const Batch& b) { return b.gentf; }
    static __device__ float* gself(const Batch& b) { return b.gselff; }
    static __device__ float* vir(const Batch& b) { return b.virf; }
};

// Relative vector centre - image of neighbour entry (j, packed shift), FP64.
__device__ __forceinline__ void entry_vec(const Batch& b, const StructInfo& S, double xi, double yi, double zi, int j,
                                          int sh, double& dx, double& dy, double& dz) {
    int sx, sy, sz;
    unpack_shift(sh, sx, sy, sz);
    const double* h = S.h;
    double lx = 0, ly = 0, lz = 0;
    if (sz) { lx += h[6] * sz; ly += h[7] * sz; lz += h[8] * sz; }
    if (sy) { lx += h[3] * sy; ly += h[4] * sy; lz += h[5] * sy; }
    if (sx) { lx += h[0] * sx; ly += h[1] * sx; lz += h[2] * sx; }
    dx = xi - (b.wpos[3 * j] + lx);
    dy = yi - (b.wpos[3 * j + 1] + ly);
    dz = zi - (b.wpos[3 * j + 2] + lz);
}

// a rank carried in a T
template <typename T>
__device__ __forceinline__ T rank_bits(int r) {
    if constexpr (sizeof(T) == 8) return __hiloint2double(0, r);
    else return __int_as_float(r);
}
__device__ __forceinline__ int rank_of(double x) { return __double2loint(x); }
__device__ __forceinline__ int rank_of(float x) { return __float_as_int(x); }

// Stage the neighbour entries of atom i sorted by element (stable).  The
// relative vectors are formed in FP64 from the wrapped positions and image
// shifts and then rounded to T.  With a Verlet-skin list (list cutoff above
// rc) only entries with r < rc are staged; the gradient pass writes zero
// gradients for the others.  Returns the number of staged entries.
//
// Per neighbour, every factor of the angular terms that depends on it alone
// is formed here, so that a pair evaluates only functions of r_jk:
//   exp(-eta (r_ij^2 + r_ik^2 + r_jk^2)) fc_ij fc_ik fc_jk
//     = P_j P_k exp(-eta r_jk^2) fc_jk,       P = fc exp(-eta r^2),
//   rho = d ln fc / d(r^2) = -3 (1 - t^2) / (2 rc r t), t = tanh(1 - r/rc).
template <typename T, class S, bool kGrad, bool kB>
__device__ int fstage(const Batch& b, const DevModel& m, int i, int c, FSmem<T>& s, int lane, int M) {
    const int e0 = b.nei_off[i];
    const int nel = m.nel;
    const double xi = b.wpos[3 * i], yi = b.wpos[3 * i + 1], zi = b.wpos[3 * i + 2];
    const StructInfo& si = b.info[b.sid[i]];
    const double rc = m.rc[c], irc = 1.0 / rc;
    const bool filt = b.rc_list > rc;
    const double rc2 = rc * rc;
    if (lane < nel) s.cnt[lane] = 0;
    __syncwarp();
    for (int base = 0; base < M; base += 32) {
        const int q = base + lane;
        bool keep = q < M;
        int el = 0;
        if (keep) {
            const int j = b.nei_j[e0 + q];
            el = b.elem[j];
            if (filt) {
                double dx, dy, dz;
                entry_vec(b, si, xi, yi, zi, j, b.nei_s[e0 + q], dx, dy, dz);
                keep = dx * dx + dy * dy + dz * dz < rc2;
            }
        }
        const unsigned act = __ballot_sync(kFull, keep);
        if (keep) {
            const unsigned peers = __match_any_sync(act, el);
            if ((peers & lanemask_lt()) == 0) s.cnt[el] += __popc(peers);
        }
        __syncwarp();
    }
    // elements in ascending order of their counts: the first rows of the
    // angular pass, which meet every element, are few
    int total;
    {
        const int n = lane < nel ? s.cnt[lane] : 0;
        int rank = 0, start = 0;
        total = 0;
        for (int x = 0; x < nel; ++x) {
            const int nx = __shfl_sync(kFull, n, x);
            total += nx;
            if (nx < n || (nx == n && x < lane)) {
                ++rank;
                start += nx;
            }
        }
        if (lane < nel) {
            s.est[lane] = start;
            s.rst[rank] = start;
            s.ord[rank] = lane;
        }
        if (lane == 0) s.rst[nel] = total;
        __syncwarp();
        if (!kGrad) {
            const int mine = lane < nel ? s.ord[lane] : 0;
            for (int q = 0; q < nel; ++q) {
                const int other = __shfl_sync(kFull, mine, q);
                if (lane < nel) {
                    const int lo = min(mine, other), hi = max(mine, other);
                    const int t = lo * nel - lo * (lo - 1) / 2 + hi - lo;
                    const bool has = m.g4_full || m.g4_off[c * m.nblk + t + 1] > m.g4_off[c * m.nblk + t];
                    s.tm[lane * nel + q] = has ? (unsigned char)t : (unsigned char)255;
                }
            }
        }
    }
    // est moves while slots are handed out and is set back below
    __syncwarp();
    for (int base = 0; base < M; base += 32) {
        const int q = base + lane;
        int slot = 0, el = 0, j = 0, sh = 0;
        double dx = 0, dy = 0, dz = 0;
        bool keep = q < M;
        if (keep) {
            j = b.nei_j[e0 + q];
            sh = b.nei_s[e0 + q];
            el = b.elem[j];
            entry_vec(b, si, xi, yi, zi, j, sh, dx, dy, dz);
            if (filt && !(dx * dx + dy * dy + dz * dz < rc2)) {
                keep = false;
                if (kGrad) {
                    T* gent = Buf<T>::gent(b);
                    const size_t e = (size_t)(e0 + q);
                    gent[3 * e] = (T)0;
                    gent[3 * e + 1] = (T)0;
                    gent[3 * e + 2] = (T)0;
                }
            }
        }
        const unsigned act = __ballot_sync(kFull, keep);
        if (keep) {
            const unsigned peers = __match_any_sync(act, el);
            slot = s.est[el] + __popc(peers & lanemask_lt());
            __syncwarp(act);
            if ((peers & lanemask_lt()) == 0) s.est[el] += __popc(peers);
        }
        __syncwarp();
        if (keep) {
            // distance, cutoff and exponentials in FP64
            const double r2 = dx * dx + dy * dy + dz * dz;
            double r, ir;
            sqrt_rsqrt(r2, r, ir);
            double fc = 0.0, rho = 0.0;
            if (r < rc) {
                const double t = tanh01(1.0 - r * irc), tt = t * t;
                fc = tt * t;
                if (kGrad && t > 0.0) rho = -1.5 * irc * ir * (1.0 - tt) / t;
            }
            s.nb[slot] = V4<T>{(T)dx, (T)dy, (T)dz, (T)r2};
            T* ax = s.ax + slot * kAx<S>;
            ax[0] = (T)ir;
            if (kGrad) ax[1] = (T)rho;
#pragma unroll
            for (int e = 0; e < S::NE; ++e)
                ax[2 + e] = e < n_eta<S>(m)
                                ? (T)(fc * ang_exp<kB>(-m.eta4[e] * r2))
                                : (T)0;
            if (kGrad) {
                // r, fc and the element wait in the accumulators for the
                // radial pass, which starts the sums
                s.gx[slot] = (T)r;
                s.gx[s.gst + slot] = (T)fc;
                s.gx[2 * s.gst + slot] = (T)el;
                s.ent[slot] = e0 + q;
            } else {
                if (sizeof(T) == 4) s.dd[slot] = make_double4(dx, dy, dz, 0.0);
                s.rf[2 * slot] = (T)r;
                s.rf[2 * slot + 1] = (T)fc;
            }
        }
    }
    __syncwarp();
    if (lane < nel) s.est[lane] -= s.cnt[lane];
    __syncwarp();
    if (!kGrad) {
        for (int q = lane; q < total; q += 32) {
            int rank = 0;
            for (int x = 1; x < nel; ++x) rank += q >= s.rst[x];
            s.ax[q * kAx<S> + 1] = rank_bits<T>(rank);
        }
        __syncwarp();
    }
    return total;
}

// Candidate pairs of one element-pair block, 32 at a time: lane L holds the
// candidates L, L + 32, ... of na rows (neighbours of element a) times W
// columns.  Different elements: every neighbour of b.  Equal elements: row x
// pairs with the next W = na/2 neighbours in cyclic order, which meets every
// unordered pair once (for even na the last column holds each of its pairs
// twice, and its second half of rows is left out).  Stepping needs no
// division and no square root per candidate.
struct PairRows {
    int sa, sb, na, W, ncand;
    int row, col, qs, rs;
    bool same, even;
    __device__ __forceinline__ void start(int sa_, int na_, int sb_, int nb_, bool same_, bool has, int lane) {
        sa = sa_;
        sb = sb_;
        na = na_;
        same = same_;
        even = same && !(na & 1);
        W = has ? (same ? na >> 1 : nb_) : 0;
        ncand = na * W;
        const float inv = ncand > 0 ? 1.0f / (float)W : 0.0f;
        row = (int)(((float)lane + 0.5f) * inv);
        col = lane - row * W;
        qs = (int)(32.5f * inv);
        rs = 32 - qs * W;
    }
    // the lane's candidate, if it has one in this chunk
    __device__ __forceinline__ bool get(int& j, int& k) const {
        j = sa + row;
        int kk = sb + col;
        bool ok = row < na && ncand > 0;
        if (same) {
            kk = row + 1 + col;
            kk = sa + (kk >= na ? kk - na : kk);
            ok = ok && !(even && col == W - 1 && row >= W);
        }
        k = kk;
        return ok;
    }
    __device__ __forceinline__ void next() {
        row += qs;
        col += rs;
        if (col >= W) {
            col -= W;
            ++row;
        }
    }
};

// u = 1 - r_jk/rc for the pair cutoff.  In the FP32 form the difference
// cancels near rc; it is formed as (rc^2 - r_jk^2) / (rc (rc + r_jk)) with
// rc^2 - r_jk^2 taken in FP64.  The value pass takes it from the FP64
// relative vectors, so G stays accurate to FP32 rounding even for pairs just
// inside rc (whose SFs can have tiny scaling ranges and therefore large
// weights).  The gradient pass takes it from the FP32 vectors: its terms of
// such pairs scale with u^2, so the absolute error stays at FP32 rounding,
// and the FP64 vectors stay out of its shared memory.
template <typename T>
__device__ __forceinline__ T pair_u(const FSmem<T>& s, int j, int k, double rc2d, T rc, T inv_rc, T rjk) {
    if (sizeof(T) == 8) {
        // FP64: 1 - r_jk / rc directly (r_jk < rc by the candidate test); its
        // absolute error is a few ulp, which near rc only touches terms of
        // order u^3
        const T u = (T)1 - rjk * inv_rc;
        return u > (T)0 ? u : (T)0;
    }
    double cx, cy, cz;
    if (sizeof(T) == 4 && s.dd) {
        // the FP64 relative vectors staged beside the FP32 ones (value pass)
        const double4 a = s.dd[j], b = s.dd[k];
        cx = b.x - a.x;
        cy = b.y - a.y;
        cz = b.z - a.z;
    } else {
        const V4<T> a = s.nb[j], b = s.nb[k];
        cx = (double)b.x - (double)a.x;
        cy = (double)b.y - (double)a.y;
        cz = (double)b.z - (double)a.z;
    }
    const double D = rc2d - (cx * cx + cy * cy + cz * cz);
    return D > 0.0 ? xdiv((T)D, rc * (rc + rjk)) : (T)0;
}

// ---------------------------------------------------------------- powers
// X^e from the square chain ch[b] = X^(2^b)
template <typename T>
__device__ __forceinline__ T rpow(const T (&ch)[5], int e) {
    T r = (T)1;
#pragma unroll
    for (int bit = 0; bit < 5; ++bit)
        if ((e >> bit) & 1) r *= ch[bit];
    return r;
}

// Tz[z] = X^zeta_z and (kDeriv) Tp[z] = X^(zeta_z - 1) for one lambda.
template <class S, bool kDeriv, typename T>
__device__ __forceinline__ void powers(const DevModel& m, T X, T (&Tz)[S::NZ], T (&Tp)[S::NZ]) {
    T ch[5];
    ch[0] = X;
    if constexpr (S::kFixed) {
        constexpr int mb = S::maxbit();
#pragma unroll
        for (int b = 1; b < 5; ++b) ch[b] = b <= mb ? ch[b - 1] * ch[b - 1] : (T)0;
#pragma unroll
        for (int z = 0; z < S::NZ; ++z) {
            if constexpr (kDeriv) {
                // X^(zeta-1) from the chain, X^zeta = X^(zeta-1) * X
                T p = (T)1;
#pragma unroll
                for (int bit = 0; bit < 5; ++bit)
                    if (((S::zeta(z) - 1) >> bit) & 1) p = p * ch[bit];
                Tp[z] = p;
                Tz[z] = p * X;
            } else {
                T p = (T)1;
#pragma unroll
                for (int bit = 0; bit < 5; ++bit)
                    if ((S::zeta(z) >> bit) & 1) p = p * ch[bit];
                Tz[z] = p;
            }
        }
    } else {
#pragma unroll
        for (int b = 1; b < 5; ++b) ch[b] = b <= m.zmaxbit ? ch[b - 1] * ch[b - 1] : (T)0;
#pragma unroll
        for (int z = 0; z < S::NZ; ++z) {
            T p = (T)0, q = (T)0;
            if (z < m.fz) {
                const int ez = m.zint[z];
                if (kDeriv) {
                    p = ez >= 0 ? rpow(ch, ez) : base_pow(X, (T)m.zet[z] - (T)1);
                    q = p * X;
                } else {
                    q = ez >= 0 ? rpow(ch, ez + 1) : base_pow(X, (T)m.zet[z]);
                }
            }
            Tz[z] = q;
            if (kDeriv) Tp[z] = p;
        }
    }
}

// Packed FP32 form of powers() for NL == 2: both lambdas of a pair in one
// float2, X = (1 + lambda_0 cos, 1 + lambda_1 cos), squared and multiplied by
// the paired f32x2 instructions of sm_100 (fma.rn.f32x2 / mul.rn.f32x2; each
// half rounds exactly like the scalar instruction, so the results are those
// of powers<S, kDeriv, float>).
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

template <class S, bool kDeriv>
__device__ __forceinline__ void powers2(const DevModel& m, float2 X, float2 (&Tz)[S::NZ], float2 (&Tp)[S::NZ]) {
    float2 ch[5];
    ch[0] = X;
    if constexpr (S::kFixed) {
        constexpr int mb = S::maxbit();
#pragma unroll
        for (int b = 1; b < 5; ++b) ch[b] = b <= mb ? __fmul2_rn(ch[b - 1], ch[b - 1]) : f2(0.0f);
#pragma unroll
        for (int z = 0; z < S::NZ; ++z) {
            const int e = kDeriv ? S::zeta(z) - 1 : S::zeta(z);
            float2 p = f2(1.0f);
            bool first = true;
#pragma unroll
            for (int bit = 0; bit < 5; ++bit)
                if ((e >> bit) & 1) {
                    p = first ? ch[bit] : __fmul2_rn(p, ch[bit]);
                    first = false;
                }
            if constexpr (kDeriv) {
                Tp[z] = p;
                Tz[z] = __fmul2_rn(p, X);
            } else {
                Tz[z] = p;
            }
        }
    } else {
#pragma unroll
        for (int b = 1; b < 5; ++b) ch[b] = b <= m.zmaxbit ? __fmul2_rn(ch[b - 1], ch[b - 1]) : f2(0.0f);
#pragma unroll
        for (int z = 0; z < S::NZ; ++z) {
            float2 p = f2(0.0f), q = f2(0.0f);
            if (z < m.fz) {
                const int ez = m.zint[z];
                const int e = kDeriv ? ez : ez + 1;
                if (ez >= 0) {
                    float2 r = f2(1.0f);
#pragma unroll
                    for (int bit = 0; bit < 5; ++bit)
                        if ((e >> bit) & 1) r = __fmul2_rn(r, ch[bit]);
                    if (kDeriv) {
                        p = r;
                        q = __fmul2_rn(r, X);
                    } else {
                        q = r;
                    }
                } else if (kDeriv) {
                    const float zm = (float)m.zet[z] - 1.0f;
                    p = make_float2(base_pow(X.x, zm), base_pow(X.y, zm));
                    q = __fmul2_rn(p, X);
                } else {
                    const float zz = (float)m.zet[z];
                    q = make_float2(base_pow(X.x, zz), base_pow(X.y, zz));
                }
            }
            Tz[z] = q;
            if (kDeriv) Tp[z] = p;
        }
    }
}


// ---------------------------------------------------------------- pass 1
// One k-step (4 pairs) of the FP64 tensor cores (mma.sync m8n8k4, thread t:
// A[t/4][t%4], B[t%4][t/4], C[t/4][2 (t%4) + v]).
__device__ __forceinline__ void dmma(double (&c)[2], double a, double bb) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(bb));
}

// candidate-test vector of a slot: the FP32 copy (FP64 form) or the FP32
// relative vector itself
__device__ __forceinline__ void cvec(const FSmem<double>& s, int k, float& x, float& y, float& z) {
    const float4 v = s.sp[k];
    x = v.x;
    y = v.y;
    z = v.z;
}
__device__ __forceinline__ void cvec(const FSmem<float>& s, int k, float& x, float& y, float& z) {
    const V4<float> v = s.nb[k];
    x = v.x;
    y = v.y;
    z = v.z;
}

// Bits of word w (slots 32 w ..) that a row of rank ra may pair with: ranks
// ra + d0 .. ra + d0 + nd - 1 whose block has functions.
template <typename T>
__device__ __forceinline__ unsigned allowed(const FSmem<T>& s, int nel, int ra, int d0, int nd, int w) {
    unsigned m = 0;
#pragma unroll 1
    for (int rb = ra + d0; rb < nel && rb < ra + d0 + nd; ++rb) {
        if (s.tm[ra * nel + rb] == 255) continue;
        const int lo = max(s.rst[rb] - 32 * w, 0), hi = min(s.rst[rb + 1] - 32 * w, 32);
        if (lo < hi) m |= (hi == 32 ? ~0u : (1u << hi) - 1u) & ~((1u << lo) - 1u);
    }
    return m;
}

// Bound by instruction issue.  The neighbours are staged by element, rarest
// element first.  Contributing pairs (r_jk < rc) come row by row: for 32 rows
// at a time, each neighbour in turn is tested against 32 others (a ballot per
// row and word, 10 instructions for 32 candidates), the bits are counted and
// each lane writes its row's pairs to its place in the list.  A chunk of 32
// pairs, one per lane, is evaluated up to its powers
// T[l, z] = (1 + lambda_l cos)^zeta_z and factors Y[e]; the sums over pairs
//   acc[(l, z), (block, e)] += T[l, z] Y[e]
// are a matrix product of the FP64 tensor cores over the chunk (8 k-steps of
// 4 pairs): rows (l, z), columns (partner element of the row's element, e), a
// pair's Y entering the columns of its own block.  So a chunk may hold pairs
// of several blocks, the sums are spread over the lanes (2 per lane and tile,
// no reduction across lanes) and G is written once per element of the rows.
// The FP32 form feeds the same product (sums in FP64).
template <typename T, class S, bool kB>
__global__ void __launch_bounds__(32 * kWarps, kBlocksV<T>) k_sfv_fast(Batch b, DevModel m, int mm, int part) {
    constexpr int NL = S::NL, NZ = S::NZ, NE = S::NE, P = S::P, A = kAx<S>;
    // row tiles, blocks per accumulator tile, accumulator tiles
    constexpr int MT = kTRows<S> / 8, SL = 8 / NE, GA = 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
    FSmem<T> s = fcarve<T, S>(smem_raw + wib * fast_warp_bytes<T, S>(mm, m.nel, m.g2max, m.nblk, false), mm, m.nel, m.g2max, m.nblk, false);
    const int nel = m.nel, nblk = m.nblk;
    T* Gout = Buf<T>::G(b);
    const int ne = n_eta<S>(m);
    // fragment rows and columns of this lane
    const T* ta = s.tb + (lane >> 2) * kTs + (lane & 3);
    const T* ya = s.yb + (lane >> 2) * kTs + (lane & 3);
    const int cap = list_cap<T>(mm);
    for (int q = lane; q < 8 * kTs; q += 32) s.yb[q] = (T)0;
    __syncwarp();
    // work counters of this warp's atoms (profiling), added to b.stats once at the end
    unsigned long long st_ent = 0, st_cand = 0, st_pairs = 0, st_g2 = 0;
    const int total_atoms = part == kPartWide ? b.wide[0] : b.natoms;
    for (int q = blockIdx.x * nw + wib; q < total_atoms; q += gridDim.x * nw) {
        const int i = part == kPartWide ? b.wide[1 + q] : q;
        const int c = b.elem[i];
        if (c < 0) continue;
        const int M = b.nei_off[i + 1] - b.nei_off[i];
        // more neighbours than this launch's shared memory takes: listed for
        // the launch beside it (see run_form)
        if (M > mm) {
            if (lane == 0) {
                if (part != kPartFirst) atomicOr(&b.status[0], 4);
            }
            continue;
        }
        const int Ms = fstage<T, S, false, kB>(b, m, i, c, s, lane, M);
        const T rc = (T)m.rc[c], inv_rc = (T)(1.0 / m.rc[c]), rc2 = rc * rc;
        const double rc2d = m.rc[c] * m.rc[c];
        // The FP64 form tests candidates on FP32 copies of the relative
        // vectors.  Their rounding moves d^2 by less than 8e-7 rc^2 (vectors
        // within rc, components to 2^-24), so with this margin no pair within
        // rc is missed; one let in beyond rc has u = 0 and adds zeros.
        const float rc2s = sizeof(T) == 8 ? (float)rc2d * (1.0f + 2e-6f) : (float)rc2;
        T* Gi = Gout + (size_t)i * m.nsf_max;
        const double* mean = m.smean + (size_t)c * m.nsf_max;
        const double* iwidth = m.sinvw + (size_t)c * m.nsf_max;

        // radial SFs: lane = neighbour, its element's functions eight at a time
        // (rows); the sums over neighbours are products with fc in the column
        // of the neighbour's rank
        for (int fb = 0; fb < m.g2el_max; fb += 8)
            for (int x0 = 0; x0 < nel; x0 += 8) {
                double racc[2] = {0.0, 0.0};
                for (int t0 = 0; t0 < Ms; t0 += 32) {
                    const int t = t0 + lane;
                    const bool live = t < Ms;
                    const int rank = live ? rank_of(s.ax[t * A + 1]) : 0;
                    const int g = c * nel + s.ord[rank];
                    const int f0 = m.g2_off[g] + fb, nf = live ? m.g2_off[g + 1] - f0 : 0;
                    const T r = live ? s.rf[2 * t] : (T)0;
                    const bool mine = live && rank >= x0 && rank < x0 + 8;
                    if (mine) s.yb[(rank - x0) * kTs + lane] = s.rf[2 * t + 1];
#pragma unroll (sizeof(T) == 8 ? 1 : 2)  // FP64: the smaller code is the faster one (3.49, 3.57, 3.69 ms at 1, 4, 8)
                    for (int f = 0; f < 8; ++f) {
                        T e = (T)0;
                        if (f < nf) {
                            const SF2 q = m.g2[f0 + f];
                            const T x = r - (T)q.rs;
                            e = rad_exp<kB>(-(T)q.eta * x * x);
                        }
                        s.tb[f * kTs + lane] = e;
                    }
                    __syncwarp();
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) dmma(racc, (double)ta[4 * ks], (double)ya[4 * ks]);
                    __syncwarp();
                    if (mine) s.yb[(rank - x0) * kTs + lane] = (T)0;
                    __syncwarp();
                }
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int rank = x0 + 2 * (lane & 3) + v;
                    if (rank < nel) {
                        const int g = c * nel + s.ord[rank], f = m.g2_off[g] + fb + (lane >> 2);
                        if (f < m.g2_off[g + 1]) {
                            const int sf = m.g2[f].sf;
                            Gi[sf] = (T)((racc[v] - mean[sf]) * iwidth[sf]);
                        }
                    }
                }
            }

        if constexpr (sizeof(T) == 8) {
            // the radial distances give way to the candidate test's vectors
            for (int t = lane; t < Ms; t += 32) {
                const V4<T> d = s.nb[t];
                s.sp[t] = make_float4((float)d.x, (float)d.y, (float)d.z, 0.0f);
            }
            __syncwarp();
        }

        int n_pairs = 0;
        double acc[GA][MT][2];
#pragma unroll
        for (int g = 0; g < GA; ++g)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) acc[g][mt][0] = acc[g][mt][1] = 0.0;
        // potentials with more elements than the accumulators hold blocks for:
        // several passes over the rows, each with the partners of one range of
        // ranks
        for (int d0 = 0; d0 < nel; d0 += GA * SL) {
            int cur = 0;  // rank whose blocks the accumulators hold
            int qn = 0;  // listed pairs
            for (int j0 = 0; j0 < Ms || j0 == 0; j0 += 32) {
                // rows j0 .. j0 + 31: lane = row, the bits of its partners k > j
                const int nrow = min(32, Ms - j0);
                int cnt = 0;
                for (int w = j0 >> 5; 32 * w < Ms; ++w) {
                    const int k = 32 * w + lane;
                    float kx = 1e18f, ky = 0.0f, kz = 0.0f;
                    if (k < Ms) cvec(s, k, kx, ky, kz);
                    unsigned mw = 0;
                    // (rows up to a multiple of 8 lie inside the staging arrays)
                    for (int jj = 0; jj < nrow; jj += 8)
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            float jx, jy, jz;
                            cvec(s, j0 + jj + u, jx, jy, jz);
                            const float ex = kx - jx, ey = ky - jy, ez = kz - jz;
                            const unsigned bal = __ballot_sync(kFull, ex * ex + ey * ey + ez * ez < rc2s);
                            mw = lane == jj + u ? bal : mw;
                        }
                    if (32 * w == j0) mw &= ~((2u << lane) - 1u);
                    if (lane >= nrow) mw = 0;
                    if (!m.g4_full || nel > GA * SL) mw &= lane < nrow ? allowed(s, nel, rank_of(s.ax[(j0 + lane) * A + 1]), d0, GA * SL, w) : 0u;
                    s.mask[32 * w + lane] = mw;
                    cnt += __popc(mw);
                }
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += v;
                }
                const int off = incl - cnt, total = __shfl_sync(kFull, incl, 31);
                int start = 0;
                bool more;
                do {
                    // the rows that fit into the list, in order
                    const bool fits = off >= start && incl - start <= cap - qn;
                    const unsigned who = __ballot_sync(kFull, fits);
                    if (fits && cnt > 0) {
                        unsigned* dst = s.queue + qn + off - start;
                        for (int w = j0 >> 5; 32 * w < Ms; ++w) {
                            unsigned mw = s.mask[32 * w + lane];
                            const unsigned row = (unsigned)(j0 + lane) | ((unsigned)(32 * w) << 10);
                            while (mw) {
                                *dst++ = row + ((unsigned)(__ffs(mw) - 1) << 10);
                                mw &= mw - 1;
                            }
                        }
                    }
                    const int end = __shfl_sync(kFull, incl, 31 - __clz(who));
                    qn += end - start;
                    start = end;
                    more = start < total;
                    const bool fin = !more && j0 + 32 >= Ms;
                    __syncwarp();
                    int pos = 0;
                    // (the last one of a pass also when it is empty: it writes
                    // the sums of the ranks that are left)
                    while (qn - pos >= 32 || (fin && cur < nel)) {
                        // a chunk of 32 pairs, one per lane
                        const int n = min(32, qn - pos);
                        int rj = -1, dr = 0;
                        T cth = (T)0, Y[NE];
#pragma unroll
                        for (int e = 0; e < NE; ++e) Y[e] = (T)0;
                        if (lane < n) {
                            const unsigned pk = s.queue[pos + lane];
                            const int pj = pk & 0x3ff, pq = pk >> 10;
                            const V4<T> a = s.nb[pj], bq = s.nb[pq];
                            T xa[A], xb[A];
                            ldax<A>(s.ax, pj, xa);
                            ldax<A>(s.ax, pq, xb);
                            rj = rank_of(xa[1]);
                            const int rq = rank_of(xb[1]);
                            dr = rq - rj - d0;
                            // contributing-pair list for the gradient pass
                            if (b.pairs && n_pairs + lane < b.pcap)
                                b.pairs[(size_t)i * b.pcap + n_pairs + lane] = pk | ((unsigned)s.tm[rj * nel + rq] << 20);
                            const T cx = bq.x - a.x, cy = bq.y - a.y, cz = bq.z - a.z;
                            const T rjk2 = cx * cx + cy * cy + cz * cz;
                            T E[NE];
                            eta_exps<NE, kB>(m, ne, rjk2, E);
                            const T tj = xtanh(pair_u(s, pj, pq, rc2d, rc, inv_rc, xsqrt(rjk2)));
                            const T fjk = tj * tj * tj;
                            cth = (T)0.5 * (a.w + bq.w - rjk2) * (xa[0] * xb[0]);
#pragma unroll
                            for (int e = 0; e < NE; ++e) Y[e] = xa[2 + e] * xb[2 + e] * (E[e] * fjk);
                        }
                        if constexpr (sizeof(T) == 4 && NL == 2) {
                            const float2 X = __ffma2_rn(make_float2((float)m.lam[0], (float)m.lam[1]), f2((float)cth), f2(1.0f));
                            float2 Tz[NZ], Tp[NZ];
                            powers2<S, false>(m, X, Tz, Tp);
#pragma unroll
                            for (int z = 0; z < NZ; ++z) {
                                s.tb[z * kTs + lane] = Tz[z].x;
                                s.tb[(NZ + z) * kTs + lane] = Tz[z].y;
                            }
                        } else {
#pragma unroll
                            for (int l = 0; l < NL; ++l) {
                                T Tz[NZ], Tp[NZ];
                                powers<S, false>(m, (T)1 + (T)m.lam[l] * cth, Tz, Tp);
#pragma unroll
                                for (int z = 0; z < NZ; ++z) s.tb[(l * NZ + z) * kTs + lane] = Tz[z];
                            }
                        }
                        __syncwarp();
                        const int rlast = fin && pos + n == qn ? nel : __shfl_sync(kFull, rj, n - 1);
                        for (;;) {
#pragma unroll
                            for (int g = 0; g < GA; ++g) {
                                // the pairs of these blocks put their factors into
                                // the columns of their block
                                const bool in = rj == cur && dr >= g * SL && dr < (g + 1) * SL;
                                if (!__any_sync(kFull, in)) continue;
                                T* yc = s.yb + (dr - g * SL) * NE * kTs + lane;
                                if (in)
#pragma unroll
                                    for (int e = 0; e < NE; ++e) yc[e * kTs] = Y[e];
                                __syncwarp();
#pragma unroll
                                for (int ks = 0; ks < 8; ++ks)
#pragma unroll
                                    for (int mt = 0; mt < MT; ++mt) dmma(acc[g][mt], (double)ta[mt * 8 * kTs + 4 * ks], (double)ya[4 * ks]);
                                __syncwarp();
                                if (in)
#pragma unroll
                                    for (int e = 0; e < NE; ++e) yc[e * kTs] = (T)0;
                                __syncwarp();
                            }
                            if (rlast == cur) break;
                            // rank cur is complete: its sums -> G
#pragma unroll
                            for (int g = 0; g < GA; ++g) {
                                if (cur + d0 + g * SL >= nel) break;  // uniform
#pragma unroll
                                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                                    for (int v = 0; v < 2; ++v) {
                                        const int row = mt * 8 + (lane >> 2), col = 2 * (lane & 3) + v;
                                        const int rb = cur + d0 + g * SL + col / NE;
                                        const int t = row < NL * NZ && rb < nel ? s.tm[cur * nel + rb] : 255;
                                        if (t < 255) {
                                            const size_t at = ((size_t)c * nblk + t) * P + row * NE + col % NE;
                                            const int sf = m.pmap[at];
                                            const double2 q = m.pscale[at];
                                            // the difference to the mean before the division by the width
                                            if (sf >= 0) Gi[sf] = (T)(fma(m.pfz[row % NZ], acc[g][mt][v], q.x) * q.y);
                                        }
                                        acc[g][mt][v] = 0.0;
                                    }
                            }
                            if (++cur == nel) break;
                        }
                        __syncwarp();
                        pos += n;
                        n_pairs += n;
                    }
                    // the remainder moves to the front
                    const unsigned v = pos + lane < qn ? s.queue[pos + lane] : 0u;
                    __syncwarp();
                    s.queue[lane] = v;
                    qn -= pos;
                    __syncwarp();
                } while (more);
            }
        }
        if (b.pairs && lane == 0) b.npairs[i] = n_pairs;
        if (b.stats) {
            // per lane: radial terms (staged neighbours of an element x the
            // centre's radial SFs for it) and candidates of an element pair
            for (int el = lane; el < nel; el += 32)
                st_g2 += (unsigned long long)s.cnt[el] *
                         (unsigned long long)(m.g2_off[c * nel + el + 1] - m.g2_off[c * nel + el]);
            for (int t = lane; t < nblk; t += 32)
                if (m.g4_off[c * nblk + t + 1] > m.g4_off[c * nblk + t]) {
                    const int na = s.cnt[m.blk_a[t]], nb = s.cnt[m.blk_b[t]];
                    st_cand += m.blk_a[t] == m.blk_b[t] ? na * (na - 1) / 2 : na * nb;
                }
            st_ent += (unsigned long long)M;
            st_pairs += n_pairs;
        }
        __syncwarp();
    }
    if (b.stats)
        for (int o = 16; o > 0; o >>= 1) {
            st_cand += __shfl_xor_sync(kFull, st_cand, o);
            st_g2 += __shfl_xor_sync(kFull, st_g2, o);
        }
    if (b.stats && lane == 0 && st_ent) {
        atomicAdd(&b.stats[2], st_ent);
        atomicAdd(&b.stats[3], st_cand);
        atomicAdd(&b.stats[4], st_pairs);
        atomicAdd(&b.stats[5], st_pairs * (unsigned long long)P);
        atomicAdd(&b.stats[6], st_g2);
    }
}

// ---------------------------------------------------------------- pass 2
// Gradient contributions of up to 32 contributing pairs (one per lane; pk =
// j | k << 10 | block << 20, live for lane < n).  Runs of equal j are
// contiguous lanes with distinct k, so within a run dE/dr_k needs no care for
// conflicts; dE/dr_j is summed over the run.  Each group of 32 / kCopies lanes
// has accumulators of its own, so runs are cut at the groups' borders, the
// groups work side by side, and a group with several runs takes them one
// after the other: no two lanes ever update one value at a time, and the
// sums do not depend on timing.  (Shared-memory FP64 atomics measured 5.6 of
// the 21 ms FP64 gradient pass on the 4096-structure batch.)  Called by all
// lanes.
template <typename T, class S, bool kB>
__device__ __forceinline__ void grad_pairs(const FSmem<T>& s, const DevModel& m, int ne, T rc, T inv_rc, double rc2d,
                                           unsigned pk_in, int n, int lane) {
    constexpr int NL = S::NL, NZ = S::NZ, NE = S::NE, P = S::P, A = kAx<S>;
        // dE/dr_j of this lane's pair (summed over runs of equal j below) and
        // dE/dr_k
        int pj = -1 - lane, pq = -1 - lane;
        T gjx = (T)0, gjy = (T)0, gjz = (T)0, gkx = (T)0, gky = (T)0, gkz = (T)0;
        if (lane < n) {
            const unsigned pk = pk_in;
            pj = pk & 0x3ff;
            pq = (pk >> 10) & 0x3ff;
            const int pt = pk >> 20;
            const V4<T> a = s.nb[pj], bq = s.nb[pq];
            T xa[A], xb[A];
            ldax<A>(s.ax, pj, xa);
            ldax<A>(s.ax, pq, xb);
            const T cx = bq.x - a.x, cy = bq.y - a.y, cz = bq.z - a.z;  // djk = r_j - r_k
            const T rjk2 = cx * cx + cy * cy + cz * cz;
            T E[NE];
            eta_exps<NE, kB>(m, ne, rjk2, E);
            T rjk, irjk;
            dist_inv(rjk2, rjk, irjk);
            const T tj = xtanh(pair_u(s, pj, pq, rc2d, rc, inv_rc, rjk)), tt = tj * tj;
            const T fjk = tt * tj;
            const T dfjk = (T)(-3) * inv_rc * irjk * (tt - tt * tt);  // 2 d fc / d(r_jk^2)
            const T h = xa[0] * xb[0];  // 1 / (r_ij r_ik)
            const T cth = (T)0.5 * (a.w + bq.w - rjk2) * h;
            T SA[NE], SC[NE];
#pragma unroll
            for (int e = 0; e < NE; ++e) SA[e] = SC[e] = (T)0;
            // weights of the block; those of d/d cos are lambda zeta times
            // them, and the factor goes to the powers (shared by the etas)
            T wa[P];
            ldvec<P>(s.WA + pt * kWp<S>, wa);
            if constexpr (sizeof(T) == 4 && NL == 2) {
                // packed over lambda: the weights are staged as (l = 0, l = 1)
                // pairs, wa[2 (z NE + e) + l] (see the staging in k_sfg_fast)
                const float2 X = __ffma2_rn(make_float2((float)m.lam[0], (float)m.lam[1]), f2((float)cth), f2(1.0f));
                float2 Tz[NZ], Tp[NZ];
                powers2<S, true>(m, X, Tz, Tp);
                const float2 lam = make_float2((float)m.lam[0], (float)m.lam[1]);
#pragma unroll
                for (int z = 0; z < NZ; ++z) Tp[z] = __fmul2_rn(Tp[z], __fmul2_rn(lam, f2((float)zeta_of<S>(m, z))));
                float2 SA2[NE], SC2[NE];
#pragma unroll
                for (int e = 0; e < NE; ++e) SA2[e] = SC2[e] = f2(0.0f);
#pragma unroll
                for (int z = 0; z < NZ; ++z)
#pragma unroll
                    for (int e = 0; e < NE; ++e) {
                        const int q = 2 * (z * NE + e);
                        SA2[e] = __ffma2_rn(make_float2(wa[q], wa[q + 1]), Tz[z], SA2[e]);
                        SC2[e] = __ffma2_rn(make_float2(wa[q], wa[q + 1]), Tp[z], SC2[e]);
                    }
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    SA[e] = SA2[e].x + SA2[e].y;
                    SC[e] = SC2[e].x + SC2[e].y;
                }
            } else {
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    T Tz[NZ], Tp[NZ];
                    powers<S, true>(m, (T)1 + (T)m.lam[l] * cth, Tz, Tp);
#pragma unroll
                    for (int z = 0; z < NZ; ++z) Tp[z] *= (T)m.lam[l] * zeta_of<S>(m, z);
#pragma unroll
                    for (int z = 0; z < NZ; ++z)
#pragma unroll
                        for (int e = 0; e < NE; ++e) {
                            SA[e] += wa[(l * NZ + z) * NE + e] * Tz[z];
                            SC[e] += wa[(l * NZ + z) * NE + e] * Tp[z];
                        }
                }
            }
            // sums over the grid without fc_jk: value, eta-weighted value and
            // d/d cos; then twice the derivatives of the pair's sum with
            // respect to r_ij^2, r_ik^2 and r_jk^2
            T V = (T)0, B = (T)0, C = (T)0;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const T Y = xa[2 + e] * xb[2 + e] * E[e];
                const T y = Y * SA[e];
                V += y;
                B += (T)m.eta4[e] * y;
                C += Y * SC[e];
            }
            const T V2 = (T)2 * fjk * V, B2 = (T)2 * fjk * B, Cf = fjk * C;
            const T q3 = dfjk * V - B2 - Cf * h;
            const T q1 = V2 * xa[1] - B2 + Cf * (h - cth * xa[0] * xa[0]);
            const T q2 = V2 * xb[1] - B2 + Cf * (h - cth * xb[0] * xb[0]);
            gjx = q3 * cx - q1 * a.x;
            gjy = q3 * cy - q1 * a.y;
            gjz = q3 * cz - q1 * a.z;
            gkx = -q3 * cx - q2 * bq.x;
            gky = -q3 * cy - q2 * bq.y;
            gkz = -q3 * cz - q2 * bq.z;
        }
        constexpr int GL = 32 / kCopies;  // lanes of a group
        const int prev_j = __shfl_up_sync(kFull, pj, 1);
        const bool head = lane < n && ((lane & (GL - 1)) == 0 || prev_j != pj);
        const unsigned heads = __ballot_sync(kFull, head);
        const unsigned group = (kCopies == 1 ? kFull : (1u << (GL & 31)) - 1u) << (lane & ~(GL - 1));
        const int run = __popc(heads & group & ~(~1u << lane)) - 1;   // this lane's run in its group
        const int phases = __reduce_max_sync(kFull, __popc(heads & group));
        {
            // a segmented suffix sum over each run (fixed shuffle order)
            // leaves dE/dr_j of the run in its first lane
            const unsigned after = heads & group & (~1u << lane);  // heads above this lane
            const int end = min(n, (lane | (GL - 1)) + 1);
            const int last = after ? __ffs(after) - 2 : end - 1;   // last lane of my run
#pragma unroll
            for (int d = 1; d < GL; d <<= 1) {
                const T ox = __shfl_down_sync(kFull, gjx, d);
                const T oy = __shfl_down_sync(kFull, gjy, d);
                const T oz = __shfl_down_sync(kFull, gjz, d);
                if (lane + d <= last) {
                    gjx += ox;
                    gjy += oy;
                    gjz += oz;
                }
            }
        }
        T* g = s.gx + (lane / GL) * 3 * s.gst;
        for (int r = 0; r < phases; ++r) {
            if (run == r && lane < n) {
                g[pq] += gkx;
                g[s.gst + pq] += gky;
                g[2 * s.gst + pq] += gkz;
                if (head) {
                    g[pj] += gjx;
                    g[s.gst + pj] += gjy;
                    g[2 * s.gst + pj] += gjz;
                }
            }
            __syncwarp();
        }
}

// Bound by instruction issue and shared-memory latency: per pair two dozen
// 16-byte shared loads, the geometry, cutoff, exponentials and powers again,
// the contraction with dE/dG, and the update of two slots.
template <typename T, class S, bool kB>
__global__ void __launch_bounds__(32 * kWarps, kBlocksG<T>) k_sfg_fast(Batch b, DevModel m, int mm, int part) {
    constexpr int NL = S::NL, NZ = S::NZ, NE = S::NE, P = S::P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
    FSmem<T> s = fcarve<T, S>(smem_raw + wib * fast_warp_bytes<T, S>(mm, m.nel, m.g2max, m.nblk, true), mm, m.nel, m.g2max, m.nblk, true);
    const int nel = m.nel;
    const T* dEdG = Buf<T>::dEdG(b);
    const int ne = n_eta<S>(m);
    const int total_atoms = part == kPartWide ? b.wide[0] : b.natoms;
    for (int q = blockIdx.x * nw + wib; q < total_atoms; q += gridDim.x * nw) {
        const int i = part == kPartWide ? b.wide[1 + q] : q;
        const int c = b.elem[i];
        if (c < 0) continue;
        const int M = b.nei_off[i + 1] - b.nei_off[i];
        // more neighbours than this launch's shared memory takes: listed for
        // the launch beside it (see run_form)
        if (M > mm) {
            if (lane == 0) {
                if (part != kPartFirst) atomicOr(&b.status[0], 4);
            }
            continue;
        }
        const int Ms = fstage<T, S, true, kB>(b, m, i, c, s, lane, M);
        const T rc = (T)m.rc[c], inv_rc = (T)(1.0 / m.rc[c]), rc2 = rc * rc;
        const double rc2d = m.rc[c] * m.rc[c];
        // w_s = dE/dG_s / width_s: radial SFs staged per slot of g2, angular
        // ones folded into the product-space weight tensors of each block
        const T* dEdGi = dEdG + (size_t)i * m.nsf_max;
        const double* iwc = m.sinvw + (size_t)c * m.nsf_max;
        const int r0 = m.g2_off[c * nel], r1 = m.g2_off[c * nel + nel];
        for (int f = r0 + lane; f < r1; f += 32) {
            const int sf = m.g2[f].sf;
            s.w2[f - r0] = (T)((double)dEdGi[sf] * iwc[sf]);
        }
        for (int q = lane; q < m.nblk * P; q += 32) {
            const int t = q / P, p = q % P;
            const int sf = m.pmap[((size_t)c * m.nblk + t) * P + p];
            T wa = (T)0;
            const int l = p / (NZ * NE), z = (p / NE) % NZ;
            if (sf >= 0) wa = (T)((double)dEdGi[sf] * iwc[sf]) * (T)m.pfz[z];
            // FP32 with two lambdas: (l = 0, l = 1) pairs for the packed contraction
            s.WA[t * kWp<S> + ((sizeof(T) == 4 && NL == 2) ? 2 * (p % (NZ * NE)) + l : p)] = wa;
        }
        __syncwarp();

        // radial: lane = neighbour slot
        for (int t = lane; t < Ms; t += 32) {
            const T r = s.gx[t], fc = s.gx[s.gst + t];
            const int el = (int)s.gx[2 * s.gst + t];
            const int f0 = m.g2_off[c * nel + el], f1 = m.g2_off[c * nel + el + 1];
            const V4<T> d = s.nb[t];
            const T ir = s.ax[t * kAx<S>], rho = s.ax[t * kAx<S> + 1];
            T coef = (T)0;
            for (int f = f0; f < f1; ++f) {
                const SF2 q = m.g2[f];
                const T eta = (T)q.eta, xr = r - (T)q.rs;
                coef += s.w2[f - r0] * rad_exp<kB>(-eta * xr * xr) * (eta * xr * ir - rho);
            }
            coef *= (T)2 * fc;
            s.gx[t] = coef * d.x;
            s.gx[s.gst + t] = coef * d.y;
            s.gx[2 * s.gst + t] = coef * d.z;
#pragma unroll
            for (int q = 3; q < 3 * kCopies; ++q) s.gx[q * s.gst + t] = (T)0;
        }
        __syncwarp();

        // angular: the contributing pairs listed by the value pass, or (list
        // missing or over capacity) screened again; the queue spans element-pair
        // blocks (entries carry the block)
        const int np = b.pairs ? b.npairs[i] : -1;
        if (np >= 0 && np <= b.pcap) {
            const unsigned* pl = b.pairs + (size_t)i * b.pcap;
            // the next chunk's entries are loaded while this chunk computes
            unsigned nxt = lane < np ? __ldg(pl + lane) : 0u;
            for (int base = 0; base < np; base += 32) {
                const int n = np - base < 32 ? np - base : 32;
                const unsigned pk = nxt;
                if (base + 32 < np) nxt = base + 32 + lane < np ? __ldg(pl + base + 32 + lane) : 0u;
                grad_pairs<T, S, kB>(s, m, ne, rc, inv_rc, rc2d, lane < n ? pk : 0u, n, lane);
                __syncwarp();
            }
        } else {
            unsigned qh = 0;
            int qn = 0;
            PairRows pr;
            for (int t = 0; t <= m.nblk; ++t) {
                const bool fin = t == m.nblk;
                {
                    const int ea = fin ? 0 : m.blk_a[t], eb = fin ? 0 : m.blk_b[t];
                    const bool has = !fin && m.g4_off[c * m.nblk + t + 1] > m.g4_off[c * m.nblk + t];
                    pr.start(s.est[ea], s.cnt[ea], s.est[eb], s.cnt[eb], ea == eb, has, lane);
                }
                for (int cb = 0; cb < pr.ncand || (fin && cb == 0); cb += 32) {
                    int j, k;
                    bool ok = pr.get(j, k);
                    if (ok) {
                        const V4<T> a = s.nb[j], bb = s.nb[k];
                        const T ex = bb.x - a.x, ey = bb.y - a.y, ez = bb.z - a.z;
                        ok = ex * ex + ey * ey + ez * ez < rc2;
                    }
                    pr.next();
                    const unsigned bal = __ballot_sync(kFull, ok);
                    if (ok)
                        s.queue[(qh + qn + __popc(bal & lanemask_lt())) & 63] =
                            (unsigned)j | ((unsigned)k << 10) | ((unsigned)t << 20);
                    qn += __popc(bal);
                    __syncwarp();
                    if (qn >= 32 || (fin && qn > 0)) {
                        const int n = qn < 32 ? qn : 32;
                        grad_pairs<T, S, kB>(s, m, ne, rc, inv_rc, rc2d, lane < n ? s.queue[(qh + lane) & 63] : 0u, n, lane);
                        __syncwarp();
                        qh += n;
                        qn -= n;
                    }
                }
            }
        }
        __syncwarp();
        T* gent = Buf<T>::gent(b);
        T sx = 0, sy = 0, sz = 0;
        T v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int t = lane; t < Ms; t += 32) {
            V4<T> g{s.gx[t], s.gx[s.gst + t], s.gx[2 * s.gst + t], (T)0};
#pragma unroll
            for (int q = 1; q < kCopies; ++q) {
                g.x += s.gx[3 * q * s.gst + t];
                g.y += s.gx[(3 * q + 1) * s.gst + t];
                g.z += s.gx[(3 * q + 2) * s.gst + t];
            }
            const V4<T> d = s.nb[t];
            const size_t e = (size_t)s.ent[t];
            gent[3 * e] = g.x;
            gent[3 * e + 1] = g.y;
            gent[3 * e + 2] = g.z;
            sx -= g.x;
            sy -= g.y;
            sz -= g.z;
            v[0] -= g.x * d.x; v[1] -= g.y * d.x; v[2] -= g.z * d.x;
            v[3] -= g.x * d.y; v[4] -= g.y * d.y; v[5] -= g.z * d.y;
            v[6] -= g.x * d.z; v[7] -= g.y * d.z; v[8] -= g.z * d.z;
        }
        for (int o = 16; o > 0; o >>= 1) {
            sx += __shfl_xor_sync(kFull, sx, o);
            sy += __shfl_xor_sync(kFull, sy, o);
            sz += __shfl_xor_sync(kFull, sz, o);
#pragma unroll
            for (int u = 0; u < 9; ++u) v[u] += __shfl_xor_sync(kFull, v[u], o);
        }
        if (lane == 0) {
            T* gs = Buf<T>::gself(b);
            T* vr = Buf<T>::vir(b);
            gs[3 * (size_t)i] = sx;
            gs[3 * (size_t)i + 1] = sy;
            gs[3 * (size_t)i + 2] = sz;
#pragma unroll
            for (int u = 0; u < 9; ++u) vr[9 * (size_t)i + u] = v[u];
        }
        __syncwarp();
    }
}

// atoms with more than mm neighbours: their number in b.wide[0], then the list
// (in no particular order; every atom's result is its own)
__global__ void k_list_wide(Batch b, int mm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool w = i < b.natoms && b.nei_off[i + 1] - b.nei_off[i] > mm;
    const unsigned bal = __ballot_sync(kFull, w);
    int base = 0;
    if (lane == 0 && bal) base = atomicAdd(&b.wide[0], __popc(bal));
    base = __shfl_sync(kFull, base, 0);
    if (w) b.wide[1 + base + __popc(bal & lanemask_lt())] = i;
}

int nsm() { return device_sm_count(); }

// Shared memory per warp grows with the largest neighbour count of the
// batch, and it sets how many warps an SM holds.  Atoms with at most `split`
// neighbours run in a launch sized for that count; the others are listed and
// run in a launch sized for the batch maximum, beside the first one on the
// context's side stream (after it, the few listed atoms took 80 of the 440 us
// of each pass for 96 structures, one atom's latency on a nearly idle GPU).
// Each atom is evaluated once, by the same code.
// Both launches have the same grid: in a dense batch nearly every atom is
// listed (19,200 atoms with 95-111 neighbours, 5 elements, values / gradients
// in ms: 1.57 / 2.90 FP64 and 1.21 / 1.58 mixed; with two blocks per SM of
// the listed atoms 2.23 / 4.59 and 1.87 / 2.48).
// The split and the persistent grid (blocks per SM) are the knobs of the
// plans' autotuner (Batch::sf_split, Batch::sf_blocks_per_sm).
constexpr int kBlocksPerSm = 32;
constexpr size_t kSmemSm = 228 * 1024;  // shared memory of an SM; 1 KB of every block is the system's

//
// ask: only an answer (1 or 0), no launch.  Without a list (b.wide null) the
// pass runs as one launch.
template <typename T, class S, bool kB>
int run_form(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask) {
    const int mfull = b.mmax > 0 ? ((b.mmax + 31) / 32) * 32 : 32;
    auto warp_bytes = [&](int mm) { return fast_warp_bytes<T, S>(mm, m.nel, m.g2max, m.nblk, grad); };
    // (slots are 10 bits in the pair lists)
    if (ask == SfAsk::kFits) return mfull <= 1024 && warp_bytes(mfull) <= (size_t)kSmemLimit;
    // default split: the largest count at which the blocks the registers
    // allow still fit (1 KB of every block is the system's)
    const int resident = grad ? kBlocksG<T> : kBlocksV<T>;
    // Warps per block at neighbour count mm and the warps that an SM then
    // holds: four, or fewer where a block of four leaves more than an eighth
    // of that number unused (160 neighbours, FP64 gradients: 4 warps an SM in
    // one block, 7 in blocks of one; the dense batch above 4.62 -> 2.90 ms).
    // For one warp more the smaller blocks do not pay: they take the places
    // of the other launch's blocks (758,676 atoms, 12 -> 13 and 8 -> 9 warps:
    // 31.8 -> 32.5 ms per step).
    auto warps_per_block = [&](int mm, int& on_sm) {
        int best = 1;
        on_sm = 0;
        for (int nw = kWarps; nw >= 1; nw >>= 1) {
            const size_t block = warp_bytes(mm) * nw;
            if (block > (size_t)kSmemLimit) continue;
            const int n = nw * (int)std::min<size_t>(resident * kWarps / nw, kSmemSm / (block + 1024));
            if (8 * n > 9 * on_sm) {
                best = nw;
                on_sm = n;
            }
        }
        return best;
    };
    int fitting = 32;
    while (fitting + 8 <= 1024 && (warp_bytes(fitting + 8) * kWarps + 1024) * resident <= kSmemSm) fitting += 8;
    int split = b.sf_split > 0 ? (b.sf_split + 7) / 8 * 8 : b.sf_split < 0 ? mfull : fitting;
    const int per_sm = b.sf_blocks_per_sm > 0 ? b.sf_blocks_per_sm : kBlocksPerSm;
    if (b.sf_split == 0 && mfull > split) {
        // a batch whose warps all fit on the GPU at the full size needs no
        // second launch (same code per atom: same results)
        int fit;
        warps_per_block(mfull, fit);
        if ((long long)b.natoms <= (long long)nsm() * fit) split = mfull;
    }
    if (ask == SfAsk::kLists) return mfull > split;
    if (!b.wide) split = mfull;
    int L = 0;
    auto go = [&](int mm, int part, cudaStream_t on) {
        int fit;
        const int nw = warps_per_block(mm, fit);
        const size_t smem = warp_bytes(mm) * nw;
        int blocks = (b.natoms + nw - 1) / nw;
        const int cap = nsm() * per_sm * kWarps / nw;
        if (blocks > cap) blocks = cap;
        if (blocks < 1) blocks = 1;
        if (grad) {
            raise_smem_limit(k_sfg_fast<T, S, kB>, smem);
            k_sfg_fast<T, S, kB><<<blocks, 32 * nw, smem, on>>>(b, m, mm, part);
        } else {
            raise_smem_limit(k_sfv_fast<T, S, kB>, smem);
            k_sfv_fast<T, S, kB><<<blocks, 32 * nw, smem, on>>>(b, m, mm, part);
        }
        ++L;
    };
    if (mfull > split) {
        cudaMemsetAsync(b.wide, 0, sizeof(int), st);
        k_list_wide<<<(b.natoms + 255) / 256, 256, 0, st>>>(b, split);
        ++L;
        cudaEventRecord(b.fork, st);
        cudaStreamWaitEvent(b.side, b.fork, 0);
        go(mfull, kPartWide, b.side);
        go(split, kPartFirst, st);
        cudaEventRecord(b.join, b.side);
        cudaStreamWaitEvent(st, b.join, 0);
    } else {
        go(mfull, kPartAll, st);
    }
    return L;
}

// FP64: the form without exponential range tests where the potential allows it
template <typename T, class S>
int run_spec(const Batch& b, const DevModel& m, bool grad, cudaStream_t st, SfAsk ask) {
    if constexpr (sizeof(T) == 8)
        if (m.exp_bounded) return run_form<T, S, true>(b, m, grad, st, ask);
    return run_form<T, S, false>(b, m, grad, st, ask);
}

}  // namespace

}  // namespace hdnnp
