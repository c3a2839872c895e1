// mlp.cu -- K5: per-element atomic networks, forward pass and dE/dG (FP64
// on the FP64 tensor cores, FP32 on the CUDA cores).
//
// Same arithmetic as nn_forward / nn_backward(gradOut = 1) per atom
// (neuralNetworks.f90:94-158, 220-313; called from hdnnps.f90:523-531):
//   c_l = W_l y_{l-1} + b_l,  y_l = act_l(c_l);   E_atom = y_L + atom_energy
//   delta_L = act'(c_L);  delta_{l-1} = (W_l^T delta_l) * act'(c_{l-1});
//   dE/dG = W_1^T delta_1
// Atoms are grouped by element (a grouped GEMM: one weight set per element);
// one CTA evaluates a tile of 32 atoms of one element with the activations
// kept in shared memory and the weights read through L1 (W^T for the forward
// pass so that consecutive threads read consecutive outputs, W for dE/dG).
#include "engine.h"
#include "mlp_tile.cuh"

namespace hdnnp {

namespace {

// Counts and slots per element with warp-aggregated atomics: the lanes of
// one element in a warp add their number once (a handful of counters would
// otherwise take one atomic per atom).  The order inside an element group is
// that of the atomics; each atom's network output does not depend on it.
__global__ void k_count_elements(Batch b, int nel) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int e = i < b.natoms ? b.elem[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    if (e >= 0 && (peers & ((1u << (threadIdx.x & 31)) - 1u)) == 0) atomicAdd(&b.el_count[e], __popc(peers));
}

__global__ void k_element_starts(Batch b, int nel) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        int acc = 0;
        for (int e = 0; e < nel; ++e) {
            b.el_start[e] = acc;
            acc += b.el_count[e];
            b.el_count[e] = 0;  // reused as the fill cursor
        }
        b.el_start[nel] = acc;
    }
}

__global__ void k_fill_elements(Batch b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int e = i < b.natoms ? b.elem[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (e >= 0 && lane == leader) base = atomicAdd(&b.el_count[e], __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (e >= 0) b.el_atoms[b.el_start[e] + base + __popc(peers & ((1u << lane) - 1u))] = i;
}

// The three steps in one block for batches of at most kSmallGroup atoms (the
// launches cost more than the work: 10 us in three launches and a clear at 768
// atoms, 4 in one): counts per element and warp, starts, slots in the order
// of the atom indices.
constexpr int kSmallGroup = 2048;
__global__ void __launch_bounds__(1024) k_group_small(Batch b, int nel) {
    __shared__ int cnt[2 * 32 * kMaxEl];  // [chunk of 32 atoms][element], then its first slot
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int q = tid; q < 2 * 32 * kMaxEl; q += 1024) cnt[q] = 0;
    __syncthreads();
    int e[2], rank[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = u * 1024 + tid;
        e[u] = i < b.natoms ? b.elem[i] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, e[u]);
        rank[u] = __popc(peers & ((1u << lane) - 1u));
        if (e[u] >= 0 && rank[u] == 0) cnt[(u * 32 + w) * kMaxEl + e[u]] = __popc(peers);
    }
    __syncthreads();
    if (w == 0) {  // lane = element: its chunks one after the other
        int n = 0;
        if (lane < nel)
            for (int q = 0; q < 64; ++q) n += cnt[q * kMaxEl + lane];
        int at = n;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += y;
        }
        if (lane < nel) {
            b.el_count[lane] = n;
            b.el_start[lane] = at - n;
            if (lane == nel - 1) b.el_start[nel] = at;
            int p = at - n;
            for (int q = 0; q < 64; ++q) {
                const int v = cnt[q * kMaxEl + lane];
                cnt[q * kMaxEl + lane] = p;
                p += v;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u)
        if (e[u] >= 0) b.el_atoms[cnt[(u * 32 + w) * kMaxEl + e[u]] + rank[u]] = u * 1024 + tid;
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_mlp(Batch b, DevModel m, int maxw) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    // locate (element, tile) of this block
    int tile = blockIdx.x, e = -1, t0 = 0, cnt = 0;
    for (int x = 0; x < m.nel; ++x) {
        int n = b.el_start[x + 1] - b.el_start[x];
        int nt = (n + kTile - 1) / kTile;
        if (tile < nt) {
            e = x;
            t0 = b.el_start[x] + tile * kTile;
            cnt = min(kTile, n - tile * kTile);
            break;
        }
        tile -= nt;
    }
    if (e < 0) return;
    mlp_tile<T>(b, m, maxw, e, t0, cnt, sm_raw);
}

// ---------------------------------------------------------------- FP64 tensor cores
// The FP64 networks on the FP64 tensor cores: mma.sync m8n8k4 f64 (tcgen05
// has no FP64 kind), tiles of 8 atoms of one element.  Layer 1 is the GEMM
// (8 x nin) x (nin x 32), dE/dG = delta_1 W_1 the GEMM (8 x 32) x (32 x nin).
// Same formulas as mlp_tile (neuralNetworks.f90:94-158).
//   fragments (thread t): A[t/4][t%4], B[k = t%4][n = t/4],
//   C[t/4][2 (t%4) + v], v = 0, 1
// Two kernels share the work by batch size (launch_mlp):
//   k_mlp_split     a block of 8 warps per tile: the warps split layer 1's
//                   inputs and the columns of dE/dG, so that one tile's chain
//                   of loads is short.
//   k_mlp_resident  a block per SM keeps the weights of one element in shared
//                   memory and its warps take a tile each.
__device__ __forceinline__ void dmma(double (&c)[2], double a, double bb) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(bb));
}

constexpr int kDW = 8;   // warps per block of k_mlp_split, one per atom of the tile
constexpr int kRW = 10;  // most warps per block of k_mlp_resident
constexpr int kDH = 32;  // widest layer the kernels take
constexpr int kDR = 8;   // atoms per tile
// row stride of the activation rows: four rows of four doubles (the A
// fragment's half-warp) fall on distinct banks
constexpr int kDS = 36;

// tiles of 8 atoms of element x
__device__ __forceinline__ int el_tiles(const Batch& b, int x) {
    return (b.el_start[x + 1] - b.el_start[x] + kDR - 1) / kDR;
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The later layers' weights in shared memory, layer by layer the fragments
// [ks][nt][32] of the forward product (B[k][n] = W[n][k]), zero-padded to
// whole tiles of 8 inputs; doubles they take.  The backward product reads the
// same fragments transposed.
__host__ __device__ inline int layer_doubles(const DevModel& m, int l) {
    return 2 * ((m.width[l] + 7) >> 3) * ((m.width[l + 1] + 7) >> 3) * 32;
}
__host__ __device__ inline int hidden_doubles(const DevModel& m) {
    int h = 0;
    for (int l = 1; l < m.nlayers; ++l) h += layer_doubles(m, l);
    return h;
}
__device__ __forceinline__ void stage_hidden(const DevModel& m, int e, double* h, int tid, int nthreads) {
    const int L = m.nlayers;
    for (int l = 1; l < L; ++l) {
        const int wi = m.width[l], wo = m.width[l + 1], NT = (wo + 7) >> 3, nf = layer_doubles(m, l);
        const double* W = m.w + m.w_off[e * L + l];  // [wo][wi]
        for (int idx = tid; idx < nf; idx += nthreads) {
            const int t = idx & 31, f = idx >> 5, n = (f % NT) * 8 + (t >> 2), k = 4 * (f / NT) + (t & 3);
            if (n < wo && k < wi) cp_async8(h + idx, W + (size_t)n * wi + k);
            else h[idx] = 0.0;
        }
        h += nf;
    }
}

// C[8 x 8 NT] = A[8 x k] B: NC n-tiles from n0 on, the A fragments read from
// the rows at `rows` (columns beyond k as zero), the B fragments [ks][nt][32]
// at `B`, both in shared memory.
template <int NC>
__device__ __forceinline__ void rows_gemm(double (&acc)[NC][2], const double* rows, int k, const double* B, int NT, int n0,
                                          int r, int q, int lane) {
#pragma unroll
    for (int nt = 0; nt < NC; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
    const int KS = (k + 3) >> 2;
#pragma unroll 2
    for (int ks = 0; ks < KS; ++ks) {
        const double a = 4 * ks + q < k ? rows[r * kDS + 4 * ks + q] : 0.0;
#pragma unroll
        for (int nt = 0; nt < NC; ++nt)
            if (n0 + nt < NT) dmma(acc[nt], a, B[(ks * NT + n0 + nt) * 32 + lane]);
    }
}

// The same with the transposed product B[k][n] = W[k][n]: element (k, n) lies
// at thread 4 (k % 8) + n % 4 of the fragment [n / 4][k / 8], so a half-warp's
// 16 elements are consecutive.  NTF: n-tiles of the stored (forward) product.
template <int NC>
__device__ __forceinline__ void rows_gemm_t(double (&acc)[NC][2], const double* rows, int k, const double* B, int NTF, int NT,
                                            int n0, int r, int q, int lane) {
#pragma unroll
    for (int nt = 0; nt < NC; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
    const int KS = (k + 3) >> 2;
    B += (lane >> 4) * NTF * 32 + (lane & 3) * 4 + ((lane >> 2) & 3);
#pragma unroll 2
    for (int ks = 0; ks < KS; ++ks) {
        const double a = 4 * ks + q < k ? rows[r * kDS + 4 * ks + q] : 0.0;
#pragma unroll
        for (int nt = 0; nt < NC; ++nt)
            if (n0 + nt < NT) dmma(acc[nt], a, B[(2 * (n0 + nt) * NTF + (ks >> 1)) * 32 + (ks & 1) * 16]);
    }
}

// Pairs of k-steps (8 consecutive inputs; step v of pair p takes 8 p + 2 q + v
// in fragment column q) whose products are summed on their own: both kernels
// add layer 1 in kDW such segments, in order, so that an atom's result does
// not depend on which of them evaluates its batch.
__device__ __forceinline__ int segment_pairs(int nin) { return (((nin + 7) >> 3) + kDW - 1) / kDW; }

// shared memory of k_mlp_split in doubles: later layers, activations or
// deltas [8][kDS], act'(c_l) [L][8][kDS], layer-1 segments [8][8][kDS]
__host__ __device__ inline int split_doubles(const DevModel& m) {
    return hidden_doubles(m) + (1 + m.nlayers + kDW) * kDR * kDS;
}

// Bound by the latency of one tile's chain: element and atom lookup, G and
// W1 loads, the layers, dE/dG.  Each of the 8 warps takes a segment of layer
// 1, an n-tile of the later layers (four warps; their weights arrive in shared
// memory while layer 1 multiplies) and every 8th pair of dE/dG columns.  Cold,
// a warp per tile with all of it in one chain took 113 us for the 768-atom
// cell (96 tiles).
__global__ void __launch_bounds__(32 * kDW) k_mlp_split(Batch b, DevModel m) {
    extern __shared__ __align__(16) double dsm[];
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const int L = m.nlayers;
    int tile = blockIdx.x, e = -1, t0 = 0, cnt = 0;
    for (int x = 0; x < m.nel; ++x) {
        const int nt = el_tiles(b, x);
        if (tile < nt) {
            e = x;
            t0 = b.el_start[x] + tile * kDR;
            cnt = min(kDR, b.el_start[x + 1] - t0);
            break;
        }
        tile -= nt;
    }
    if (e < 0) return;  // uniform per block
    double* h = dsm;
    double* yrow = h + hidden_doubles(m);
    double* da = yrow + kDR * kDS;
    double* part = da + L * kDR * kDS;
    stage_hidden(m, e, h, tid, 32 * kDW);
    const int r = lane >> 2, q = lane & 3;
    const int atom = r < cnt ? b.el_atoms[t0 + r] : -1;
    const int nin = m.nin_el[e], nsf = m.nsf_max, H1 = m.width[1];
    {
        double acc[4][2];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
        const double* grow = atom >= 0 ? b.G + (size_t)atom * nsf : nullptr;
        const int KS = (nin + 3) >> 2, KP = (nin + 7) >> 3, per = segment_pairs(nin);
        // [ks][nt][32]: this lane's inputs 2 q, 2 q + 1 of a pair lie in k-step
        // 2 p + q/2
        const double* F = m.dm_fwd + m.dm_off_f[e] + (lane & ~3) + ((2 * q) & 3);
        const int p0 = wib * per, p1 = min(KP, p0 + per);
#pragma unroll 5
        for (int p = p0; p < p1; ++p) {
            const int k = 8 * p + 2 * q, ks = 2 * p + (q >> 1);
            double a[2], bf[4][2];
#pragma unroll
            for (int v = 0; v < 2; ++v) a[v] = (grow && k + v < nin) ? __ldg(grow + k + v) : 0.0;
            const double* f = F + (size_t)ks * 128;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int v = 0; v < 2; ++v) bf[nt][v] = ks < KS ? __ldg(f + nt * 32 + v) : 0.0;
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) dmma(acc[nt], a[v], bf[nt][v]);
        }
        double* pw = part + wib * kDR * kDS + r * kDS + 2 * q;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) *reinterpret_cast<double2*>(pw + 8 * nt) = make_double2(acc[nt][0], acc[nt][1]);
    }
    cp_async_wait();
    __syncthreads();
    {
        const int row = wib * kDS + lane;  // (atom, neuron)
        if (lane < H1) {
            double c = part[row];
#pragma unroll
            for (int w = 1; w < kDW; ++w) c += part[w * kDR * kDS + row];
            c += m.b[m.b_off[e * L] + lane];
            const double y = act_f(m.act[0], c);
            const double d = act_d(m.act[0], c, y);
            yrow[row] = L > 1 ? y : d;
            da[row] = d;
            if (L == 1 && lane == 0 && wib < cnt) b.atE[b.el_atoms[t0 + wib]] = y + m.atom_energy[e];
        }
    }
    __syncthreads();
    // later layers and the deltas back to layer 1: a warp per n-tile
    for (int l = 1; l < L; ++l) {
        const int wi = m.width[l], wo = m.width[l + 1], NT = (wo + 7) >> 3;
        double acc[1][2];
        if (wib < NT) rows_gemm(acc, yrow, wi, h, NT, wib, r, q, lane);
        h += layer_doubles(m, l);
        __syncthreads();
        if (wib < NT)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int col = wib * 8 + 2 * q + v;
                if (col < wo) {
                    const double c = acc[0][v] + m.b[m.b_off[e * L + l] + col];
                    const double y = act_f(m.act[l], c);
                    const double d = act_d(m.act[l], c, y);
                    yrow[r * kDS + col] = l + 1 < L ? y : d;  // gradOut = 1
                    da[(l * kDR + r) * kDS + col] = d;
                    if (l + 1 == L && atom >= 0 && col == 0) b.atE[atom] = y + m.atom_energy[e];
                }
            }
        __syncthreads();
    }
    const double* dl = da + (L - 1) * kDR * kDS;
    for (int l = L - 1; l >= 1; --l) {
        const int wi = m.width[l], wo = m.width[l + 1], NT = (wi + 7) >> 3;
        dl -= kDR * kDS;
        double acc[1][2];
        h -= layer_doubles(m, l);
        if (wib < NT) rows_gemm_t(acc, yrow, wo, h, (wo + 7) >> 3, NT, wib, r, q, lane);
        __syncthreads();
        if (wib < NT)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int col = wib * 8 + 2 * q + v;
                if (col < wi) yrow[r * kDS + col] = acc[0][v] * dl[r * kDS + col];
            }
        __syncthreads();
    }
    double afr[kDH / 4];
#pragma unroll
    for (int ks = 0; ks < kDH / 4; ++ks) afr[ks] = (4 * ks + q < H1) ? yrow[r * kDS + 4 * ks + q] : 0.0;
    const double* Bw = m.dm_bwd + m.dm_off_b[e] + lane;  // [nb][ks][32]
    const int KB = (H1 + 3) >> 2, NB = (nin + 7) >> 3;
    for (int nb = 2 * wib; nb < NB; nb += 2 * kDW) {
        const bool two = nb + 1 < NB;  // uniform
        const double* b0 = Bw + (size_t)nb * KB * 32;
        const double* b1 = b0 + KB * 32;
        double c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
#pragma unroll
        for (int ks = 0; ks < kDH / 4; ++ks) {
            if (ks < KB) {
                dmma(c0, afr[ks], __ldg(b0 + ks * 32));
                if (two) dmma(c1, afr[ks], __ldg(b1 + ks * 32));
            }
        }
        if (atom >= 0) {
            double* drow = b.dEdG + (size_t)atom * nsf;
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int col = nb * 8 + 2 * q + v;
                if (col < nin) drow[col] = c0[v];
                if (two && col + 8 < nin) drow[col + 8] = c1[v];
            }
        }
    }
}

// Shared memory of k_mlp_resident in doubles: W1 in the fragment orders of
// layer 1 and of dE/dG, the later layers' weights, biases, and for each of nw
// warps one activation/delta row set and act'(c_l) of the layers but the last.
struct DmmaLayout {
    int f1, b1, hid, bias, warps, total;
};
__host__ __device__ inline DmmaLayout dmma_layout(const DevModel& m, int nin, int nw) {
    DmmaLayout o;
    const int H1 = m.width[1], L = m.nlayers;
    o.f1 = 0;
    o.b1 = o.f1 + ((nin + 7) >> 3) * 8 * 32;
    o.hid = o.b1 + ((nin + 7) >> 3) * ((H1 + 3) >> 2) * 32;
    o.bias = o.hid + hidden_doubles(m);
    o.warps = o.bias + L * kDH;
    o.total = o.warps + nw * L * kDR * kDS;
    return o;
}

// Bound by the FP64 tensor cores (about 590 m8n8k4 per tile of a
// 280-25-25-1 network; 0.7 ms for the 758,676 atoms of the 4096-structure
// batch at the FP64 GEMM rate) and by G in, dE/dG out (0.5 ms of HBM).  Both
// orders of W1 (134 KB) and the later layers stay in shared memory, a block
// per SM over a contiguous share of the tiles, so every B fragment is a
// conflict-free shared load; every layer is a tensor-core product.  A
// fragments come straight from the G rows, 12 pairs of k-steps (two
// consecutive inputs per 16-byte load) ahead, across tiles too.  With the
// weights from L2 and a warp per tile this pass took 2.92 ms; this form takes
// 1.95.
// kVec: G and dE/dG rows start on 16-byte boundaries (nsf_max even).
template <bool kVec>
__global__ void __launch_bounds__(32 * kRW, 1) k_mlp_resident(Batch b, DevModel m, int nin_max) {
    extern __shared__ __align__(16) double dsm[];
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5, nw = blockDim.x >> 5;
    const int L = m.nlayers, H1 = m.width[1], nsf = m.nsf_max;
    const DmmaLayout lo = dmma_layout(m, nin_max, nw);
    double* yrow = dsm + lo.warps + wib * L * kDR * kDS;
    double* da = yrow + kDR * kDS;
    const int r = lane >> 2, q = lane & 3;
    const int KB = (H1 + 3) >> 2;
    long long T = 0;
    for (int x = 0; x < m.nel; ++x) T += el_tiles(b, x);
    const int first = (int)(T * blockIdx.x / gridDim.x), end = (int)(T * (blockIdx.x + 1) / gridDim.x);
    constexpr int kCh = 12;  // pairs of k-steps in flight
    int base = 0;
    for (int e = 0; e < m.nel; ++e) {
        const int nte = el_tiles(b, e);
        const int s0 = max(first, base) - base, s1 = min(end, base + nte) - base;
        base += nte;
        if (s0 >= s1) continue;  // uniform per block
        const int nin = m.nin_el[e], KP = (nin + 7) >> 3, NB = KP, per = segment_pairs(nin);
        __syncthreads();  // the previous element's weights are no longer read
        {
            // [2 p + v][nt][t] = W1[8 nt + t/4][8 p + 2 (t%4) + v], from the
            // packed k-steps of four consecutive inputs (coalesced reads; the
            // steps beyond the last one of an odd count are zero)
            const double* src = m.dm_fwd + m.dm_off_f[e];
            const int nf1 = ((nin + 3) >> 2) * 128;
            for (int idx = tid; idx < KP * 256; idx += 32 * nw) {
                const int t = idx & 31, nt = (idx >> 5) & 3, ks = idx >> 7;
                const int kk = 4 * (ks & 1) + (t & 3);
                double* dst = dsm + lo.f1 + ((((ks & ~1) | (kk & 1)) * 4 + nt) << 5) + ((t & ~3) | (kk >> 1));
                if (idx < nf1) cp_async8(dst, src + idx);
                else *dst = 0.0;
            }
            for (int idx = tid; idx < NB * KB * 32; idx += 32 * nw)
                cp_async8(dsm + lo.b1 + idx, m.dm_bwd + m.dm_off_b[e] + idx);
            stage_hidden(m, e, dsm + lo.hid, tid, 32 * nw);
            for (int idx = tid; idx < L * kDH; idx += 32 * nw) {
                const int l = idx / kDH, n = idx % kDH;
                dsm[lo.bias + idx] = n < m.width[l + 1] ? m.b[m.b_off[e * L + l] + n] : 0.0;
            }
        }
        cp_async_wait();
        __syncthreads();
        const double* F = dsm + lo.f1 + lane;
        const double* Bw = dsm + lo.b1 + lane;
        const int a0 = b.el_start[e], a1 = b.el_start[e + 1];
        auto atom_of = [&](int tile) {
            const int at = a0 + tile * kDR + r;
            return (tile < s1 && at < a1) ? b.el_atoms[at] : -1;
        };
        // inputs 8 p + 2 q and the next of an atom's row, zero beyond nin
        auto load = [&](int atom, int p, double2& v) {
            v = make_double2(0.0, 0.0);
            const int k = 8 * p + 2 * q;
            if (atom >= 0 && p < KP && k < nin) {
                const double* g = b.G + (size_t)atom * nsf + k;
                if (kVec) v = __ldcs(reinterpret_cast<const double2*>(g));
                else {
                    v.x = __ldcs(g);
                    if (k + 1 < nin) v.y = __ldcs(g + 1);
                }
                if (k + 1 >= nin) v.y = 0.0;
            }
        };
        // the ring holds kCh pairs of k-steps ahead: a slot is loaded again as
        // soon as it has been multiplied, at the end of a row with the next
        // tile's first inputs
        double2 an[kCh];
        int atom_n = atom_of(s0 + wib);
#pragma unroll
        for (int i = 0; i < kCh; ++i) load(atom_n, i, an[i]);
        for (int tile = s0 + wib; tile < s1; tile += nw) {
            const int atom = atom_n;
            atom_n = atom_of(tile + nw);
            double acc[4][2], sum[4][2];  // a segment's products, the segments before it
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = sum[nt][0] = sum[nt][1] = 0.0;
            int left = per;
            for (int p0 = 0; p0 < KP; p0 += kCh) {
                const bool more = p0 + kCh < KP;
                const int an_atom = more ? atom : atom_n, an_p = more ? p0 + kCh : 0;
#pragma unroll
                for (int i = 0; i < kCh; ++i) {
                    if (p0 + i < KP) {
                        const double* f = F + (size_t)(p0 + i) * 256;
#pragma unroll
                        for (int nt = 0; nt < 4; ++nt) dmma(acc[nt], an[i].x, f[nt * 32]);
#pragma unroll
                        for (int nt = 0; nt < 4; ++nt) dmma(acc[nt], an[i].y, f[128 + nt * 32]);
                        if (--left == 0) {
                            left = per;
#pragma unroll
                            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                                for (int v = 0; v < 2; ++v) {
                                    sum[nt][v] += acc[nt][v];
                                    acc[nt][v] = 0.0;
                                }
                        }
                    }
                    load(an_atom, an_p + i, an[i]);
                }
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int v = 0; v < 2; ++v) acc[nt][v] = sum[nt][v] + acc[nt][v];
            const double* h = dsm + lo.hid;
            for (int l = 0; l < L; ++l) {
                const int wo = m.width[l + 1], NT = (wo + 7) >> 3;
                if (l > 0) {
                    const int wi = m.width[l];
                    rows_gemm(acc, yrow, wi, h, NT, 0, r, q, lane);
                    h += layer_doubles(m, l);
                    __syncwarp();
                }
                const char act = m.act[l];
#pragma unroll
                for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const int col = nt * 8 + 2 * q + v;
                        if (col < wo) {
                            const double c = acc[nt][v] + dsm[lo.bias + l * kDH + col];
                            const double y = act_f(act, c);
                            const double d = act_d(act, c, y);
                            if (l + 1 < L) {
                                yrow[r * kDS + col] = y;
                                da[(l * kDR + r) * kDS + col] = d;
                            } else {
                                yrow[r * kDS + col] = d;  // gradOut = 1
                                if (atom >= 0 && col == 0) b.atE[atom] = y + m.atom_energy[e];
                            }
                        }
                    }
                __syncwarp();
            }
            for (int l = L - 1; l >= 1; --l) {
                const int wi = m.width[l], wo = m.width[l + 1], NT = (wi + 7) >> 3;
                h -= layer_doubles(m, l);
                rows_gemm_t(acc, yrow, wo, h, (wo + 7) >> 3, NT, 0, r, q, lane);
                __syncwarp();
#pragma unroll
                for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const int col = nt * 8 + 2 * q + v;
                        if (col < wi) yrow[r * kDS + col] = acc[nt][v] * da[((l - 1) * kDR + r) * kDS + col];
                    }
                __syncwarp();
            }
            // dE/dG = delta_1 W1, four column tiles (independent chains) at a time
            double afr[kDH / 4];
#pragma unroll
            for (int ks = 0; ks < kDH / 4; ++ks) afr[ks] = (4 * ks + q < H1) ? yrow[r * kDS + 4 * ks + q] : 0.0;
            __syncwarp();
            double* drow = b.dEdG + (size_t)(atom >= 0 ? atom : 0) * nsf;
            for (int nb = 0; nb < NB; nb += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[u][0] = acc[u][1] = 0.0;
#pragma unroll
                for (int ks = 0; ks < kDH / 4; ++ks)
                    if (ks < KB)
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (nb + u < NB) dmma(acc[u], afr[ks], Bw[((nb + u) * KB + ks) * 32]);
                if (atom >= 0)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int col = (nb + u) * 8 + 2 * q;
                        if (kVec && col + 1 < nin) {
                            *reinterpret_cast<double2*>(drow + col) = make_double2(acc[u][0], acc[u][1]);
                        } else {
                            if (col < nin) drow[col] = acc[u][0];
                            if (col + 1 < nin) drow[col + 1] = acc[u][1];
                        }
                    }
            }
        }
    }
}

}  // namespace

int launch_element_groups(const Batch& b, const DevModel& m, cudaStream_t s) {
    if (b.natoms <= kSmallGroup) {
        k_group_small<<<1, 1024, 0, s>>>(b, m.nel);
        return 1;
    }
    const int g = (b.natoms + 255) / 256;
    cudaMemsetAsync(b.el_count, 0, sizeof(int) * (m.nel + 1), s);
    k_count_elements<<<g, 256, 0, s>>>(b, m.nel);
    k_element_starts<<<1, 32, 0, s>>>(b, m.nel);
    k_fill_elements<<<g, 256, 0, s>>>(b);
    return 3;
}

size_t mlp_smem_bytes(const DevModel& m, size_t elem) {
    int nin = 0, maxw = 1;
    for (int e = 0; e < m.nel; ++e) nin = nin > m.nin_el[e] ? nin : m.nin_el[e];
    size_t n = (size_t)kTile * nin;
    for (int l = 0; l < m.nlayers; ++l) {
        n += 2 * (size_t)kTile * m.width[l + 1];
        if (m.width[l + 1] > maxw) maxw = m.width[l + 1];
    }
    n += 2 * (size_t)kTile * maxw;  // deltas of the hidden/output layers
    return n * elem;
}

template <typename T>
void run_mlp(const Batch& b, const DevModel& m, cudaStream_t s) {
    int nin = 0, maxw = 1;
    for (int e = 0; e < m.nel; ++e) nin = nin > m.nin_el[e] ? nin : m.nin_el[e];
    for (int l = 0; l < m.nlayers; ++l)
        if (m.width[l + 1] > maxw) maxw = m.width[l + 1];
    size_t smem = mlp_smem_bytes(m, sizeof(T));
    raise_smem_limit(k_mlp<T>, smem);
    int tiles = b.natoms / kTile + m.nel + 1;
    k_mlp<T><<<tiles, kThreads, smem, s>>>(b, m, maxw);
}

// The tensor-core forms take networks whose layers are at most kDH wide,
// with one output and at most 8 layers (dm_ok, set with the fragments at
// model upload).  The resident form needs an element's weights and the rows of
// at least kRWLeast warps in shared memory, and enough tiles to keep its warps
// busy: its time for one tile is long (53 us from 4,500 atoms down, against
// 18-35 us of the split form).  Measured for 280-25-25-1 networks, split /
// resident: 93 / 88 us at 18,000 atoms, 156 / 145 at 36,000.  With fewer than
// ten warps, 316,116 atoms, split / resident in ms: 280-25-25-25-1 (8 warps)
// 1.24 / 0.98, 280-32-32-32-1 (7) 1.31 / 1.18, 280-25-25-25-25-1 (6) 1.79 /
// 1.44; 280-30-30-30-30-1 (5) 1.85 / 1.79, but 0.286 / 0.296 at 40,272 atoms.
// Both give an atom the same bits.
constexpr int kRWLeast = 6;
constexpr int kResidentTilesPerSm = 16;

int launch_mlp(const Batch& b, const DevModel& m, cudaStream_t s) {
    if (!m.dm_ok) {
        run_mlp<double>(b, m, s);
        return 1;
    }
    int nin = 0;
    for (int e = 0; e < m.nel; ++e) nin = nin > m.nin_el[e] ? nin : m.nin_el[e];
    // as many warps as fit beside the weights
    int nw = kRW;
    auto bytes = [&](int w) { return (size_t)dmma_layout(m, nin, w).total * sizeof(double); };
    while (nw > kRWLeast && bytes(nw) > (size_t)kSmemLimit) --nw;
    const size_t rsm = bytes(nw);
    const int nsm = device_sm_count();
    if (rsm <= (size_t)kSmemLimit && b.natoms >= nsm * kResidentTilesPerSm * kDR) {
        auto k = (m.nsf_max & 1) ? k_mlp_resident<false> : k_mlp_resident<true>;
        raise_smem_limit(k, rsm);
        k<<<nsm, 32 * nw, rsm, s>>>(b, m, nin);
        return 1;
    }
    const size_t smem = (size_t)split_doubles(m) * sizeof(double);
    raise_smem_limit(k_mlp_split, smem);
    k_mlp_split<<<b.natoms / kDR + m.nel + 1, 32 * kDW, smem, s>>>(b, m);
    return 1;
}

int launch_mlp_fp32(const Batch& b, const DevModel& m, cudaStream_t s) {
    run_mlp<float>(b, m, s);
    return 1;
}

}  // namespace hdnnp
