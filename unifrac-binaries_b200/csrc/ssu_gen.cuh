// Generalized UniFrac over the pairs of samples that share a node (sm_100a).
//
// With s = u(k) + u(l), a node adds L s^alpha |u(k) - u(l)| / s to the numerator
// and L s^alpha to the denominator.  Where only one sample has it, both are
// L u^alpha: a sum over that sample's own nodes, r = sum L u^alpha.  So
//   num = r_k + r_l - sum_both [L u(k)^alpha + L u(l)^alpha - L s^alpha |u(k) - u(l)| / s]
//   den = r_k + r_l - sum_both [L u(k)^alpha + L u(l)^alpha - L s^alpha],
// and only the nodes that both samples have are evaluated pair by pair (a
// sample has 5% of the nodes: 1 node in 400 against 1 in 10 for those either
// has).  The bracketed terms of nodes that few samples have are summed through
// the sample lists as whole numbers of a fixed-point unit, the one-sided parts
// by the same rounding, so both differences are exact (modulo 2^64: the brackets may be
// negative for alpha > 1); the other nodes are summed for every pair by
// the dense kernel.  Pairs whose numerator is below tau of r_k + r_l, and those
// whose r_k + r_l is few units, are summed again over their own nodes.  Terms are fp64 for both precisions.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ssu_close.cuh"
#include "ssu_kernels.cuh"
#include "ssu_lists.cuh"
#include "ssu_pairs.cuh"

namespace ssu {
namespace dev {

// 1 / sqrt(s) for s in [1e-37, 4] without a branch, so that a thread's terms
// overlap (with rsqrt, whose special cases are a branch each, the dense rows of
// eight uneven tables took 4.45 ms, with this 1.89 ms): the single-precision
// approximation y, and one step of Householder's third-order iteration for
// y^-2 = s,  y (1 + e / 2 + 3 e^2 / 8) with e = 1 - s y^2.  e is at most 2^-21, the
// step's own error 5 e^3 / 16 below 2^-64; the roundings leave at most 0.99 and on
// average 0.28 units in the last place on a million values (rsqrt: up to 1).  With
// y^2 first, which is exact, 0.50 and 0.25, but the dense rows take 3% longer and the distances' error stays.
__device__ __forceinline__ double rsqrt_step(double s) {
    float f;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(static_cast<float>(s)));
    const double y = static_cast<double>(f), e = fma(-s * y, y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// d / s for 0 <= d <= s <= 2, without a branch; 0 for s = 0.  Both are scaled
// by the power of two that takes s to [1, 2) (a denormal s to 2^-51 or more), as
// s may be far below the range of a single, and 1 / s is its single-precision
// approximation (relative error e below 2^-22) and Newton's iteration to third order,
// y (1 + e + e^2): error e^3 < 2^-66; at most 1.44 and on average 0.34 units in the
// last place on a million pairs.  (The remainder in one more step takes that to 0.50
// and 0.25, and 5% longer; the distances' error stays.)
__device__ __forceinline__ double ratio_step(double d, double s) {
    const double up = __hiloint2double(0x7fe00000 - (__double2hiint(s) & 0x7ff00000), 0);
    const double ss = fma(s, up, 1e-37);
    float f;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(static_cast<float>(ss)));
    const double y = static_cast<double>(f), e = fma(-ss, y, 1.0);
    return d * up * fma(y, fma(e, e, e), y);
}

// The generalized operator's term without branches.  Alpha 0.5: a pair with
// s = 0 takes s = 1e-37 in its place, and adds 0 as |a - b| and s are 0; to a
// node of 1e-21 or more the 1e-37 adds nothing, and what it changes in a smaller
// one is below 2e-19 of its length.  Alpha 0: every s counts alike, so the
// quotient is exact over the whole range, and the denominator's L is by a select.
template <int AK>
struct OpGenRows {
    static constexpr int NACC = 2;
    static constexpr bool COUNTS = false;
    __device__ static void term(double *acc, double a, double b, double ca, double cb, double m, double L, double alpha) {
        if constexpr (AK == 1 || AK == 3) {
            const double s = a + b;
            if constexpr (AK == 1) {
                const double t = L * rsqrt_step(s + 1e-37);
                acc[0] = fma(t, fabs(a - b), acc[0]);
                acc[1] = fma(t, s, acc[1]);
            } else {
                acc[0] = fma(L, ratio_step(fabs(a - b), s), acc[0]);
                acc[1] += s > 0.0 ? L : 0.0;
            }
        } else {
            OpGeneralized<double, AK>::term(acc, a, b, ca, cb, m, L, alpha);
        }
    }
    __device__ static double value(const double *acc, double, double) { return acc[0] / acc[1]; }
};

// s^alpha L |a - b| / s and s^alpha L of a node that both samples have.
template <int AK>
__device__ __forceinline__ void gen_both(double a, double b, double L, double alpha, double &n, double &d) {
    double acc[2] = {0.0, 0.0};
    OpGenRows<AK>::term(acc, a, b, 0.0, 0.0, 0.0, L, alpha);
    n = acc[0];
    d = acc[1];
}
template <int AK>
__device__ __forceinline__ double gen_power(double u, double alpha) {
    return AK == 1 ? sqrt(u) : AK == 2 ? u : AK == 3 ? 1.0 : pow(u, alpha);
}

struct GenSums {
    unsigned long long *num, *den;  // per pair, at out_off + k n + l
};

// As shared_sums_kernel, with the two brackets in place of q.  Bound: the fp64
// pipe and the shared-memory atomics, about half of each.  Eight lanes a list
// and two entries a lane and step (eight uneven tables on 50,000 tips, the same
// nodes: 1.51 ms, before this split 2.39).
template <typename IDX, int AK>
__global__ void __launch_bounds__(512)
    gen_sums_kernel(const ListArgs la, const GenSums out, const double *__restrict__ len, double alpha, double scale,
                    uint32_t cols, uint32_t chunk) {
    extern __shared__ uint32_t acc_s[];  // lo, hi of the numerator, lo, hi of the denominator: [cols] each
    const uint32_t j = blockIdx.x;
    const uint32_t t = la.block_table[j >> 7];
    const TableDesc td = la.tables[t];
    const uint32_t k = j - td.base;
    if (k + 1 >= td.n) return;
    const uint32_t part_rows = list_part_rows(td.n, la.parts);
    const uint32_t part0 = blockIdx.y * chunk;  // the chunk's parts
    const uint64_t cbeg = static_cast<uint64_t>(part0) * part_rows, cend = cbeg + static_cast<uint64_t>(chunk) * part_rows;
    if (cbeg >= td.n || cend <= k + 1) return;
    const uint32_t c0 = max(k + 1, static_cast<uint32_t>(cbeg));
    const uint32_t nc = static_cast<uint32_t>(min(static_cast<uint64_t>(td.n), cend)) - c0;
    const uint64_t slot0 = static_cast<uint64_t>(t - la.t0) * la.n_nodes;
    const uint32_t n_ids = la.node_cnt[j];
    const uint64_t own = la.node_ptr[j];
    constexpr uint32_t GL = 8, QE = 2;  // lanes per list, entries per lane and step
    const uint32_t groups = blockDim.x / GL, grp = threadIdx.x / GL, gl = threadIdx.x % GL;
    const uint32_t first = c0 / part_rows, last = part0 + chunk;
    const uint32_t *before = first ? la.part_count + (first - 1) * la.slots + slot0 : nullptr;
    const uint32_t *upto = (last < la.parts ? la.part_count + (last - 1) * la.slots : la.count) + slot0;
    const uint32_t base = smem_u32(acc_s), row_bytes = cols * sizeof(uint32_t);
    for (uint32_t i = threadIdx.x; i < 4 * cols; i += blockDim.x) acc_s[i] = 0;
    __syncthreads();
    for (uint32_t i = grp; i < n_ids; i += groups) {
        const uint32_t e = la.node[own + i];
        const double a = la.node_u[own + i], L = len[e];
        const unsigned long long qa = la.node_q[own + i];
        const uint32_t m = upto[e], p0 = before ? before[e] & ~(LIST_ALIGN - 1) : 0u;
        const uint64_t at0 = static_cast<uint64_t>(la.off[slot0 + e]) * LIST_ALIGN;
        for (uint32_t p = p0 + gl * QE; p < m; p += GL * QE) {
            uint32_t l[QE];
            if constexpr (sizeof(IDX) == 2) {
                const uint32_t v = *reinterpret_cast<const uint32_t *>(static_cast<const uint16_t *>(la.idx) + at0 + p);
                l[0] = v & 0xFFFFu;
                l[1] = v >> 16;
            } else {
                const uint2 v = *reinterpret_cast<const uint2 *>(static_cast<const uint32_t *>(la.idx) + at0 + p);
                l[0] = v.x;
                l[1] = v.y;
            }
            // (entries past the list's end are 0, never > k; those of other
            // parts are outside the chunk)
            const bool any = l[0] - c0 < nc || l[1] - c0 < nc;
            if (!any) continue;
            const double2 ub = *reinterpret_cast<const double2 *>(la.idx_u + at0 + p);
            const ulonglong2 qb = *reinterpret_cast<const ulonglong2 *>(la.idx_q + at0 + p);
            const double b[QE] = {ub.x, ub.y};
            const unsigned long long q[QE] = {qb.x, qb.y};
#pragma unroll
            for (uint32_t x = 0; x < QE; x++) {
                const uint32_t c = l[x] - c0;
                double n, d;
                gen_both<AK>(a, b[x], L, alpha, n, d);
                const unsigned long long sum = qa + q[x];
                const unsigned long long vn = sum - static_cast<unsigned long long>(__double2ll_rn(n * scale));
                const unsigned long long vd = sum - static_cast<unsigned long long>(__double2ll_rn(d * scale));
                const uint32_t at = base + c * static_cast<uint32_t>(sizeof(uint32_t));
                const uint32_t nl = static_cast<uint32_t>(vn), dl = static_cast<uint32_t>(vd);
                const uint32_t on = shared_add_below(at, nl, c, nc);
                const uint32_t od = shared_add_below(at + 2 * row_bytes, dl, c, nc);
                shared_carry_below(at + row_bytes, static_cast<uint32_t>(vn >> 32) + (on > ~nl ? 1u : 0u), c, nc);
                shared_carry_below(at + 3 * row_bytes, static_cast<uint32_t>(vd >> 32) + (od > ~dl ? 1u : 0u), c, nc);
            }
        }
    }
    __syncthreads();
    const uint64_t row = td.out_off + static_cast<uint64_t>(k) * td.n + c0;
    for (uint32_t i = threadIdx.x; i < nc; i += blockDim.x) {
        out.num[row + i] = (static_cast<unsigned long long>(acc_s[cols + i]) << 32) | acc_s[i];
        out.den[row + i] = (static_cast<unsigned long long>(acc_s[3 * cols + i]) << 32) | acc_s[2 * cols + i];
    }
}

struct GenFinish {
    const uint4 *tiles;
    uint32_t n_tiles, n_splits;
    const TableDesc *tables;
    const double *partial;     // the dense kernel's sums (store_partial)
    const unsigned long long *num, *den;  // nullptr: no list nodes
    const unsigned long long *rs;
    const double *W;           // r over every node, per column
    double unit, tau;
    int *tile_flags;
    uint32_t *close;           // per tile a bit for each pair (zero before the launch)
    OutSpec out;
};

// The dense kernel's split sums of a tile, the lists' sums, and the distance.
template <typename T, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gen_finalize_kernel(const GenFinish a) {
    constexpr int NT = (BM / TM) * (BN / TN), TX = BN / TN, NV = TM * TN * 2;
    const uint32_t ti = blockIdx.x;
    const uint4 tile = a.tiles[ti];
    const TableDesc td = a.tables[tile.z];
    OutSpec o = a.out;
    if (o.mode == 0) o.ptr = static_cast<T *>(o.ptr) + td.out_off;
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    for (int i = 0; i < TM; i++) {
        const int row = tile_row<BM, TM>(ty, i);
        const uint32_t k = tile.x * BM + row - td.base;
        if (k >= td.n) continue;
        const unsigned long long rk = a.rs[td.base + k];
        const double wk = a.W[td.base + k];
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int col = tile_row<BN, TN>(tx, j);
            const uint32_t l = tile.y * BN + col - td.base;
            if (!(k < l && l < td.n)) continue;
            double n = 0.0, d = 0.0;
            for (uint32_t s = 0; s < a.n_splits; s++) {
                const double *p = a.partial + (static_cast<uint64_t>(s) * a.n_tiles + ti) * NV * NT +
                                  static_cast<uint64_t>((i * TN + j) * 2) * NT + threadIdx.x;
                n += p[0];
                d += p[NT];
            }
            if (a.num) {
                const uint64_t at = td.out_off + static_cast<uint64_t>(k) * td.n + l;
                const unsigned long long own = rk + a.rs[td.base + l];
                n += static_cast<double>(static_cast<long long>(own - a.num[at])) * a.unit;
                d += static_cast<double>(static_cast<long long>(own - a.den[at])) * a.unit;
            }
            const double w = wk + a.W[td.base + l];
            if (n < a.tau * w || (a.num && w < kSharedLeast * a.unit)) {
                const uint32_t e = static_cast<uint32_t>(row * BN + col);
                atomicOr(a.close + static_cast<uint64_t>(ti) * (BM * BN / 32) + e / 32, 1u << (e & 31));
                a.tile_flags[ti] = 1;
            }
            emit_pair<T>(o, td.n, k, l, static_cast<T>(n / d));
        }
    }
}

// The operator's terms, the pairs that the finalize pass marked close (close_strips_kernel).
template <int AK>
struct OpCloseGen {
    static constexpr int NACC = 2;
    __device__ static void term(double *acc, double a, double b, double L, double alpha) {
        OpGenRows<AK>::term(acc, a, b, 0.0, 0.0, 0.0, L, alpha);
    }
    template <typename T>
    __device__ static T value(const double *acc, const T *, uint32_t, uint32_t) {
        return static_cast<T>(acc[0] / acc[1]);
    }
};

// Method dispatch (ssu_gen.cu).
struct GenLaunch {
    int ak;
    double alpha, scale;
    const double *len;  // per sparse node, then the dense nodes
    uint32_t n_words;   // 32-bit words of a bitmap over them
    int n_sms;
};
cudaError_t gen_configure();
cudaError_t gen_sums_launch(const GenLaunch &g, const ListArgs &la, const GenSums &out, uint32_t columns, uint32_t cols,
                            uint32_t chunk, uint32_t chunks, cudaStream_t s);
template <typename T>
cudaError_t gen_finish_launch(const GenLaunch &g, const ListArgs &la, const GenFinish &f, bool small, cudaStream_t s);
std::vector<PairKernel<double>> gen_rows_candidates(int ak);  // 128 x 64, 64 x 64 tiles
constexpr uint32_t kGenCols = 6144;  // columns of a row of sums held at once (16 bytes each)

}  // namespace dev
}  // namespace ssu
