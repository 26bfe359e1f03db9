// Weighted pair sums over the nodes that many samples have (sm_100a).
//
// The walk over each sample's tips (weighted_walk_kernel) leaves those nodes as
// rows of L u, one column per sample; a pair's part of the distance is
// sum |a - b| over the rows: two additions a pair and row (the absolute value
// is a source modifier), where L |a - b| over rows of u takes three
// instructions.  The other nodes' part comes from the sample lists' exact
// shared sums (ssu_lists.cuh).  Bound: the fp64 (or fp32) pipe's issue rate.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ssu_close.cuh"
#include "ssu_kernels.cuh"
#include "ssu_lists.cuh"

namespace ssu {
namespace dev {

constexpr int RB = 128;        // tile edge
constexpr int RTHREADS = 512;  // 16 (l) x 32 (k) threads, 4 x 8 pairs each
constexpr int RWARPS = RTHREADS / 32;
constexpr int RSTAGES = 4;
constexpr int RLD = RB + 1;    // row stride of the epilogue's shared tile (conflict-free both ways)
// rows per stage: 16 KB
template <typename T>
constexpr int rows_per_stage() {
    return sizeof(T) == 8 ? 8 : 16;
}
template <typename T>
constexpr size_t rows_smem() {
    constexpr size_t ring = RSTAGES * sizeof(T) * rows_per_stage<T>() * 2 * RB, tile = sizeof(double) * RB * RLD;
    return ring > tile ? ring : tile;
}

template <typename T>
struct RowsArgs {
    const uint4 *tiles;  // 128 x 128 tiles: x, y blocks of 128 columns, z table
    uint32_t n_tiles, n_splits;
    const TableDesc *tables;
    const T *U;          // [n_rows][ld], L u
    uint32_t n_rows;
    uint64_t ld;
    const T *W;          // one-sided sums over every node
    // sample lists: sums of min(q(k), q(l)) at out_off + k n + l (the fp64
    // result itself: read before it is written), sums of q per column, 2^-s
    const unsigned long long *S;
    const unsigned long long *rs;
    double unit;
    double tau;
    int *tile_flags;     // tiles with a close pair
    uint32_t *close;     // per tile a bit for each pair, row-major
    double *partial;     // per (split, tile) 128 x 128 raw sums; nullptr: no splits
    OutSpec out;
};

// The tile's distances from its raw sums in shared memory, by the whole block.
// A pair is close when its distance is below tau of its samples' one-sided sums,
// or these are few units, where the rounding of L u (to fp64, and to half a unit in the lists) could
// show; close_strips_kernel sums it again.
template <typename T, bool NORM>
__device__ __forceinline__ void rows_epilogue(const RowsArgs<T> &a, uint32_t ti, double *Mt) {
    const uint4 tile = a.tiles[ti];
    const TableDesc td = a.tables[tile.z];
    const uint32_t k0 = tile.x * RB - td.base, l0 = tile.y * RB - td.base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    OutSpec o = a.out;
    if (o.mode == 0) o.ptr = static_cast<T *>(o.ptr) + td.out_off;
    unsigned long long rl[4];
    T wl[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t l = l0 + lane + 32 * i;
        rl[i] = l < td.n ? a.rs[td.base + l] : 0ull;
        wl[i] = l < td.n ? a.W[td.base + l] : T(0);
    }
    bool any = false;
    const double least = (sizeof(T) == 8 ? kSharedLeast : 0x1p30) * a.unit;
    constexpr int G = 4;  // rows of a warp whose shared sums are in flight together
    for (int r0 = warp; r0 < RB; r0 += RWARPS * G) {
        unsigned long long sh[G][4], rk[G];
        T wk[G];
#pragma unroll
        for (int u = 0; u < G; u++) {
            const uint32_t k = k0 + r0 + u * RWARPS;
            rk[u] = k < td.n ? a.rs[td.base + k] : 0ull;
            wk[u] = k < td.n ? a.W[td.base + k] : T(0);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t l = l0 + lane + 32 * i;
                sh[u][i] = k < l && l < td.n ? a.S[td.out_off + static_cast<uint64_t>(k) * td.n + l] : 0ull;
            }
        }
#pragma unroll
        for (int u = 0; u < G; u++) {
            const int row = r0 + u * RWARPS;
            const uint32_t k = k0 + row;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t l = l0 + lane + 32 * i;
                const bool on = k < l && l < td.n;
                const double x = Mt[row * RLD + lane + 32 * i];
                const unsigned long long own = rk[u] + rl[i];
                const double d = x + static_cast<double>(own - 2 * sh[u][i]) * a.unit;
                const T w = wk[u] + wl[i];
                const bool close = on && (d < a.tau * static_cast<double>(w) || static_cast<double>(w) < least);
                const T v = NORM ? static_cast<T>(d) / w : static_cast<T>(d);
                if (on && o.mode == 0) {
                    static_cast<T *>(o.ptr)[static_cast<uint64_t>(k) * td.n + l] = v;
                    Mt[row * RLD + lane + 32 * i] = static_cast<double>(v);
                } else if (on) {
                    emit_pair<T>(o, td.n, k, l, v);
                }
                const uint32_t b = __ballot_sync(0xffffffffu, close);
                any = any || b;
                if (lane == 0) a.close[static_cast<uint64_t>(ti) * (RB * RB / 32) + row * (RB / 32) + i] = b;
            }
        }
    }
    if (any && lane == 0) atomicOr(a.tile_flags + ti, 1);
    if (o.mode == 0) {  // the mirror images, along rows too
        __syncthreads();
        for (int c = warp; c < RB; c += RWARPS) {
            const uint32_t l = l0 + c;
            if (l >= td.n) break;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t k = k0 + lane + 32 * i;
                if (k < l)
                    static_cast<T *>(o.ptr)[static_cast<uint64_t>(l) * td.n + k] =
                        static_cast<T>(Mt[(lane + 32 * i) * RLD + c]);
            }
        }
    }
}

// Persistent grid over work items (tile, row split).  Rows stream through a
// cp.async ring; fp64 sums in registers, fp32 rows summed in fp32 over a stage
// (16 rows) and folded into fp64 (a conversion costs eight additions' issue
// slots: 1,537 samples 689 us, folded every 32 rows 664 us; but the error, 2-norm
// against long double, was then up to 1.06 times that of the embedding's form,
// and is 0.89 to 0.97 times so).
template <typename T, bool NORM>
__global__ void __launch_bounds__(RTHREADS, 1) pair_rows_kernel(const RowsArgs<T> a) {
    constexpr int TM = 4, TN = 8, R = rows_per_stage<T>();
    constexpr int VEC = 16 / sizeof(T), CPR = 2 * RB / VEC;  // 16-byte pieces per staged row (k block, then l block)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *Vs = reinterpret_cast<T *>(smem_raw);            // [RSTAGES][R][2 RB]
    double *Mt = reinterpret_cast<double *>(smem_raw);  // [RB][RLD], once the ring has drained
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const uint32_t n_work = a.n_tiles * a.n_splits;
    for (uint32_t w = blockIdx.x; w < n_work; w += gridDim.x) {
        const uint32_t split = w / a.n_tiles, ti = w - split * a.n_tiles;
        const uint4 tile = a.tiles[ti];
        const uint32_t k0 = tile.x * RB, l0 = tile.y * RB;
        const uint32_t per = ((a.n_rows + a.n_splits - 1) / a.n_splits + R - 1) / R * R;
        const uint32_t begin = min(a.n_rows, split * per), end = min(a.n_rows, begin + per);
        const uint32_t n_chunks = (end - begin + R - 1) / R;
        auto load = [&](uint32_t chunk) {
            T *dst = Vs + (chunk % RSTAGES) * R * 2 * RB;
#pragma unroll
            for (int c = tid; c < R * CPR; c += RTHREADS) {
                const int r = c / CPR, q = c % CPR;
                const uint32_t e = begin + chunk * R + r;
                const uint32_t cl = q < CPR / 2 ? k0 + q * VEC : l0 + (q - CPR / 2) * VEC;
                const bool ok = e < end;
                cp_async16(dst + r * 2 * RB + q * VEC, a.U + static_cast<uint64_t>(ok ? e : 0) * a.ld + cl, ok ? 16 : 0);
            }
        };
        double acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) acc[i][j] = 0.0;
        float part[TM][TN];
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) part[i][j] = 0.0f;
        }
        for (uint32_t c = 0; c + 1 < RSTAGES; c++) {
            if (c < n_chunks) load(c);
            cp_async_commit();
        }
        for (uint32_t ch = 0; ch < n_chunks; ch++) {
            cp_async_wait<RSTAGES - 2>();
            __syncthreads();  // chunk ch has landed, and every thread is done with chunk ch - 1
            if (ch + RSTAGES - 1 < n_chunks) load(ch + RSTAGES - 1);
            cp_async_commit();
            const T *vs = Vs + (ch % RSTAGES) * R * 2 * RB;
#pragma unroll 2
            for (int c = 0; c < R; c++) {
                T av[TM], bv[TN];
                load_half<T, TM / 2>(av, vs + c * 2 * RB + ty * (TM / 2));
                load_half<T, TM / 2>(av + TM / 2, vs + c * 2 * RB + RB / 2 + ty * (TM / 2));
                load_half<T, TN / 2>(bv, vs + c * 2 * RB + RB + tx * (TN / 2));
                load_half<T, TN / 2>(bv + TN / 2, vs + c * 2 * RB + RB + RB / 2 + tx * (TN / 2));
#pragma unroll
                for (int i = 0; i < TM; i++)
#pragma unroll
                    for (int j = 0; j < TN; j++) {
                        if constexpr (sizeof(T) == 8)
                            acc[i][j] += fabs(av[i] - bv[j]);
                        else
                            part[i][j] += fabsf(av[i] - bv[j]);
                    }
            }
            if constexpr (sizeof(T) == 4) {
#pragma unroll
                for (int i = 0; i < TM; i++)
#pragma unroll
                    for (int j = 0; j < TN; j++) {
                        acc[i][j] += static_cast<double>(part[i][j]);
                        part[i][j] = 0.0f;
                    }
            }
        }
        cp_async_wait<0>();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) Mt[tile_row<RB, TM>(ty, i) * RLD + tile_row<RB, TN>(tx, j)] = acc[i][j];
        __syncthreads();
        if (a.partial) {
            double *dst = a.partial + (static_cast<uint64_t>(split) * a.n_tiles + ti) * RB * RB;
            for (int e = tid; e < RB * RB; e += RTHREADS) dst[e] = Mt[e / RB * RLD + e % RB];
        } else {
            rows_epilogue<T, NORM>(a, ti, Mt);
        }
        __syncthreads();  // the next item's ring lies over the tile
    }
}

// Split partials of each tile summed in split order, then the epilogue.
template <typename T, bool NORM>
__global__ void __launch_bounds__(RTHREADS) rows_finalize_kernel(const RowsArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *Mt = reinterpret_cast<double *>(smem_raw);
    const uint32_t ti = blockIdx.x;
    for (int e = threadIdx.x; e < RB * RB; e += RTHREADS) {
        double x = 0.0;
        for (uint32_t s = 0; s < a.n_splits; s++) x += a.partial[(static_cast<uint64_t>(s) * a.n_tiles + ti) * RB * RB + e];
        Mt[e / RB * RLD + e % RB] = x;
    }
    __syncthreads();
    rows_epilogue<T, NORM>(a, ti, Mt);
}

// L |u(k) - u(l)|, the pairs that the epilogue marked close (close_strips_kernel).
template <bool NORM>
struct OpCloseWeighted {
    static constexpr int NACC = 1;
    __device__ static void term(double *acc, double a, double b, double L, double) { acc[0] = fma(fabs(a - b), L, acc[0]); }
    template <typename T>
    __device__ static T value(const double *acc, const T *W, uint32_t kc, uint32_t lc) {
        return NORM ? static_cast<T>(acc[0]) / (W[kc] + W[lc]) : static_cast<T>(acc[0]);
    }
};

}  // namespace dev
}  // namespace ssu
