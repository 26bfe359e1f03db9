// Close pairs summed again (sm_100a).
//
// Where a pair's distance is a small share of its samples' one-sided sums, the
// roundings of L u and of the lists' unit could show, and the pair is summed
// again directly over its samples' own nodes, in fp64.  A block takes a strip of
// 32 x 64 pairs of a flagged tile: it marks the nodes that the strip's samples
// with a close pair have in a bitmap, and walks the marked nodes 128 at a time:
// their values (0 where a sample has not the node) are laid out in shared
// memory, a row a node, and every thread adds the rows' terms of its pairs in
// registers.  Near duplicates share their nodes, so the marked ones are little
// more than one sample's, and each node's value is read once for 32 or 64 pairs of its
// sample.  Blocks share the strips out in turn; strips of other tiles cost a flag.
// Bound: the latency of the chunk's steps (its values' loads, then the pairs'
// terms), then the fp64 pipe (weighted: two operations a pair and node).  (700 near
// duplicates on 5,000 tips, every pair close: weighted 395 us, generalized 950 us;
// a thread a pair merging the two samples' lists 46 and 13 ms.  Strips of 16 x 128,
// their rows' stride a multiple of the banks, 678 us; of 32 x 32 485 and 820 us.)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ssu_kernels.cuh"
#include "ssu_lists.cuh"

namespace ssu {
namespace dev {

constexpr int CK = 32, CL = 64;      // samples k and l of a strip
constexpr int CROWS = 128;           // nodes laid out at once
constexpr int CLD = CK + CL + 1;     // row stride (a column of rows spreads over the banks)
constexpr int CTHREADS = 256;
constexpr uint32_t CWORDS = 256;     // bitmap words of them, at most

struct CloseArgs {
    const uint4 *tiles;
    uint32_t n_tiles;
    const TableDesc *tables;
    const int *tile_flags;   // tiles with a close pair
    const uint32_t *close;   // per tile a bit for each pair, row-major
    const void *W;           // one-sided sums per column, in T (weighted)
    const double *len;       // per node id (sparse nodes, then dense ones)
    uint32_t n_words;        // 32-bit words of a bitmap over the ids
    double alpha;
    OutSpec out;
};

constexpr size_t close_smem(uint32_t n_words) {
    return sizeof(double) * CROWS * CLD + sizeof(uint32_t) * n_words;
}
template <int BM, int BN>
constexpr uint32_t close_strips() {
    return (BM / CK) * (BN / CL);  // per tile
}

// Op: NACC sums a pair; term(acc, a, b, L, alpha); value<T>(acc, W_k, W_l).
template <typename T, class Op, int BM, int BN>
__global__ void __launch_bounds__(CTHREADS, 2) close_strips_kernel(const CloseArgs a, const ListArgs la) {
    constexpr int LD = CLD, ALL = CK + CL, WPR = CL / 32, WARPS = CTHREADS / 32, TM = CK / WARPS, TN = CL / 32;
    constexpr uint32_t STRIPS = close_strips<BM, BN>();
    static_assert(BM % CK == 0 && BN % CL == 0 && TM * WARPS == CK && ALL <= 256, "whole strips, places in a byte");
    extern __shared__ __align__(16) unsigned char close_raw[];
    double *V = reinterpret_cast<double *>(close_raw);             // [CROWS][LD]
    uint32_t *bits = reinterpret_cast<uint32_t *>(V + CROWS * LD);  // [n_words]
    __shared__ double row_len[CROWS];
    __shared__ unsigned long long first_s[ALL];  // per involved sample: its first node, how many, how many laid out
    __shared__ uint32_t count_s[ALL], at_s[ALL];
    __shared__ uint8_t slot_s[ALL];              // and its place in a row
    __shared__ uint32_t base_s[CWORDS];         // rows before each word of the chunk
    __shared__ uint32_t mask_s[CK * WPR], any_s[1 + WPR];
    __shared__ uint32_t found_s[CTHREADS];
    __shared__ uint32_t n_found, n_who, chunk_words, chunk_rows;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n_strips = a.n_tiles * STRIPS;
    for (uint64_t s0 = blockIdx.x; s0 < n_strips; s0 += static_cast<uint64_t>(gridDim.x) * CTHREADS) {
        // the block's flagged strips among the next CTHREADS
        if (tid == 0) n_found = 0;
        __syncthreads();
        {
            const uint64_t s = s0 + static_cast<uint64_t>(tid) * gridDim.x;
            if (s < n_strips && a.tile_flags[s / STRIPS]) found_s[atomicAdd(&n_found, 1u)] = static_cast<uint32_t>(s);
        }
        __syncthreads();
        const uint32_t n_mine = n_found;
        for (uint32_t f = 0; f < n_mine; f++) {
            const uint32_t strip = found_s[f], ti = strip / STRIPS;
            const uint32_t row0 = strip % STRIPS / (BN / CL) * CK, col0 = strip % (BN / CL) * CL;
            const uint4 tile = a.tiles[ti];
            const TableDesc td = a.tables[tile.z];
            const uint32_t kc0 = tile.x * BM + row0, lc0 = tile.y * BN + col0;
            // close pairs and the samples that have one
            if (tid < 1 + WPR) any_s[tid] = 0;
            if (tid == 0) n_who = 0;
            __syncthreads();
            if (tid < CK * WPR) {
                const uint32_t m = a.close[static_cast<uint64_t>(ti) * (BM * BN / 32) + (row0 + tid / WPR) * (BN / 32) + col0 / 32 + tid % WPR];
                mask_s[tid] = m;
                if (m) {
                    atomicOr(&any_s[0], 1u << (tid / WPR));
                    atomicOr(&any_s[1 + tid % WPR], m);
                }
            }
            __syncthreads();
            if (!any_s[0]) continue;  // uniform over the block
            for (uint32_t w = tid; w < a.n_words; w += CTHREADS) bits[w] = 0u;
            if (tid < ALL) {
                const bool on = tid < CK ? (any_s[0] >> tid) & 1u : (any_s[1 + (tid - CK) / 32] >> ((tid - CK) & 31)) & 1u;
                if (on) {
                    const uint32_t c = tid < CK ? kc0 + tid : lc0 + tid - CK;
                    const uint32_t i = atomicAdd(&n_who, 1u);
                    first_s[i] = la.node_ptr[c];
                    count_s[i] = la.node_all[c];
                    at_s[i] = 0;
                    slot_s[i] = static_cast<uint8_t>(tid);
                }
            }
            __syncthreads();
            const uint32_t who = n_who;
            for (uint32_t i = warp; i < who; i += WARPS) {
                const uint32_t *ids = la.node + first_s[i];
                // (most nodes are marked already)
                for (uint32_t p = lane; p < count_s[i]; p += 32) {
                    const uint32_t id = ids[p], m = 1u << (id & 31);
                    if (!(reinterpret_cast<volatile uint32_t *>(bits)[id >> 5] & m)) atomicOr(&bits[id >> 5], m);
                }
            }
            uint32_t mine[TM];  // words of the warp's rows, a bit for each lane's column
            double acc[TM][TN][Op::NACC];
            bool busy = false;
#pragma unroll
            for (int i = 0; i < TM; i++) {
                mine[i] = 0;
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    const uint32_t m = mask_s[(warp + WARPS * i) * WPR + j];
                    busy = busy || m;
                    mine[i] |= ((m >> lane) & 1u) << j;
#pragma unroll
                    for (int c = 0; c < Op::NACC; c++) acc[i][j][c] = 0.0;
                }
            }
            __syncthreads();
            for (uint32_t w = 0; w < a.n_words;) {
                // the next words with up to CROWS marked nodes, by the first warp; the others clear the rows
                if (warp == 0) {
                    uint32_t n = 0, nw = 0;
                    for (bool more = true; more;) {
                        const uint32_t x = w + nw + lane;
                        const uint32_t c = x < a.n_words ? __popc(bits[x]) : 0u;
                        uint32_t incl = c;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                            if (lane >= o) incl += y;
                        }
                        const bool fits = n + incl <= CROWS;  // (monotone over the lanes)
                        const uint32_t fit = __popc(__ballot_sync(0xffffffffu, fits));
                        if (fits) base_s[nw + lane] = n + incl - c;
                        if (fit) n += __shfl_sync(0xffffffffu, incl, fit - 1);
                        nw += fit;
                        more = fit == 32 && nw + 32 <= CWORDS && w + nw < a.n_words;
                    }
                    if (lane == 0) {
                        chunk_words = nw;
                        chunk_rows = n;
                    }
                } else {
                    for (int x = tid - 32; x < CROWS * LD; x += CTHREADS - 32) V[x] = 0.0;
                }
                __syncthreads();
                const uint32_t nw = chunk_words, n = chunk_rows;  // (nw >= 2: a word has 32 nodes at most)
                for (uint32_t x = tid; x < nw * 32; x += CTHREADS) {
                    const uint32_t m = w + x / 32 < a.n_words ? bits[w + x / 32] : 0u, b = x & 31;
                    if ((m >> b) & 1u) row_len[base_s[x / 32] + __popc(m & ((1u << b) - 1u))] = a.len[w * 32 + x];
                }
                const uint32_t end = (w + nw) * 32;
                constexpr int U = 6;  // samples of a warp with loads in flight
                for (uint32_t i0 = warp; i0 < who; i0 += WARPS * U) {
                    uint32_t p[U], left[U], slot[U];
                    uint64_t from[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const uint32_t i = i0 + u * WARPS;
                        const bool on = i < who;
                        p[u] = on ? at_s[i] : 0u;
                        left[u] = on ? count_s[i] : 0u;
                        from[u] = on ? first_s[i] : 0ull;
                        slot[u] = on ? slot_s[i] : 0u;
                    }
                    for (bool more = true; more;) {
                        more = false;
                        uint32_t id[U];
                        double v[U];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const bool on = p[u] + lane < left[u];
                            id[u] = on ? la.node[from[u] + p[u] + lane] : 0xFFFFFFFFu;
                            v[u] = on ? la.node_u[from[u] + p[u] + lane] : 0.0;
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const bool in = id[u] < end;  // (ids ascend)
                            if (in) {
                                const uint32_t x = id[u] >> 5, m = bits[x] & ((1u << (id[u] & 31)) - 1u);
                                V[(base_s[x - w] + __popc(m)) * LD + slot[u]] = v[u];
                            }
                            const uint32_t took = __popc(__ballot_sync(0xffffffffu, in));
                            p[u] += took;
                            if (took == 32)
                                more = true;
                            else
                                left[u] = 0;
                        }
                    }
                    if (lane == 0) {
#pragma unroll
                        for (int u = 0; u < U; u++)
                            if (i0 + u * WARPS < who) at_s[i0 + u * WARPS] = p[u];
                    }
                }
                __syncthreads();
                if (busy) {
                    // (the chunk's terms apart, so that no sum runs over more than CROWS)
                    double part[TM][TN][Op::NACC] = {};
                    const double *row = V;
                    for (uint32_t r = 0; r < n; r++, row += LD) {
                        const double L = row_len[r];
                        double ak[TM], bl[TN];
#pragma unroll
                        for (int i = 0; i < TM; i++) ak[i] = row[warp + WARPS * i];
#pragma unroll
                        for (int j = 0; j < TN; j++) bl[j] = row[CK + lane + 32 * j];
#pragma unroll
                        for (int i = 0; i < TM; i++)
#pragma unroll
                            for (int j = 0; j < TN; j++) Op::term(part[i][j], ak[i], bl[j], L, a.alpha);
                    }
#pragma unroll
                    for (int i = 0; i < TM; i++)
#pragma unroll
                        for (int j = 0; j < TN; j++)
#pragma unroll
                            for (int c = 0; c < Op::NACC; c++) acc[i][j][c] += part[i][j][c];
                }
                w += nw;
                __syncthreads();  // the next chunk's words and rows lie over these
            }
            OutSpec o = a.out;
            if (o.mode == 0) o.ptr = static_cast<T *>(o.ptr) + td.out_off;
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    if (!((mine[i] >> j) & 1u)) continue;
                    const uint32_t kc = kc0 + warp + WARPS * i, lc = lc0 + lane + 32 * j;
                    emit_pair<T>(o, td.n, kc - td.base, lc - td.base,
                                 Op::template value<T>(acc[i][j], static_cast<const T *>(a.W), kc, lc));
                }
        }
        __syncthreads();
    }
}

}  // namespace dev
}  // namespace ssu
