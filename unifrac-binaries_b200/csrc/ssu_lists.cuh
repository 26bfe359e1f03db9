// Sums over nodes that few samples have, through sample lists.
//
// Unweighted.  For a set S of sparse nodes and a pair (k, l),
//   sum_{n in S, k has n and l not} L_n = rs_k - shared_kl,
//   rs_k = sum_{n in S, k has n} L_n,  shared_kl = sum_{n in S, both have n} L_n,
// and shared_kl only needs, for sample k, the lists of the samples of k's own
// nodes: m^2 / 2 additions for a node that m samples have, against n^2 / 2
// terms in a dense form.  The lengths are 64-bit fixed point,
// q = round(L 2^s) with sum_S L 2^s < 2^62 (fp64 results, where every node's length
// is one: with every sample's sum below 2^63), and every sum of them is exact,
// so the differences above are exact sums of the q: no cancellation (two
// samples with the same nodes differ by exactly 0), and no dependence on the
// order of the additions.
//
// Weighted.  With q_n(k) = round(L_n u_n(k) 2^s), u the node's proportion in
// the sample (or its counts),
//   sum_{n in S} L |u(k) - u(l)| 2^s = rs_k + rs_l - 2 sum min(q_n(k), q_n(l)),
// rs_k = sum q_n(k): the same sums with min(q(k), q(l)) in place of q, exact in
// the same way (rounding keeps the order, so the smaller q is the smaller
// value's).  A sample's rs never exceeds its total times the largest sum of sparse
// lengths on a path from the root to a tip, which sets the scale.
//
// Lists (built by the walk over each sample's tips, per execute):
//   node side:   per (table, node) the table's samples that have it, 16 or 32
//                bits each, at a 16-byte offset laid out once from the tips'
//                entry counts (an upper bound of the length); a table's
//                samples are walked in up to LIST_PARTS launches (twice as
//                many while a part's columns do not fit a block) of consecutive samples, so a list is in order from part to
//                part (in any order within one), and where each part starts
//                is kept: a sample reads its own part and the later ones;
//   sample side: per sample its sparse nodes, in node order, in one array.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ssu_kernels.cuh"
#include "ssu_walk_size.hpp"

namespace ssu {
namespace dev {

constexpr uint32_t LIST_ALIGN = 8;  // entries; node lists start on a multiple (16 bytes of 16-bit entries)
constexpr uint32_t LIST_PARTS = 8;  // launches of the walk, unless a part's columns do not fit a block then

// Lists of one group of tables.  Node e of table t (from the group's first)
// is slot t * n_nodes + e.
struct ListArgs {
    uint32_t n_nodes = 0;                // sparse nodes
    const uint32_t *off = nullptr;       // per slot: first entry, in units of LIST_ALIGN
    uint32_t *count = nullptr;           // per slot: entries so far (zero at the walk's start)
    void *idx = nullptr;                 // entries: table-local sample positions
    int wide = 0;                        // entries of 32 bits (a table of more than 65,536 samples)
    uint32_t *node = nullptr;            // sample side: node ids
    unsigned long long *node_ptr = nullptr;  // per column: first id
    uint32_t *node_cnt = nullptr;        // per column: ids
    unsigned long long *cursor = nullptr;    // ids handed out (zero at the walk's start)
    const unsigned long long *q = nullptr;   // per node: round(L 2^s)
    unsigned long long *rs = nullptr;    // per column: sum of q over its nodes
    const uint32_t *block_table = nullptr;   // per 128 columns: the table
    const TableDesc *tables = nullptr;
    uint32_t t0 = 0;                     // the group's first table
    uint32_t parts = 1;                  // parts of a table's samples, each list_part_rows long
    uint32_t *part_count = nullptr;      // [parts - 1][slots]: entries before part 1, 2, ...
    uint64_t slots = 0;
    // weighted: q of each entry, node side and sample side; on the sample side
    // u too, and the dense nodes behind the sparse ones (node_all of both)
    unsigned long long *idx_q = nullptr, *node_q = nullptr;
    double *node_u = nullptr;
    uint32_t *node_all = nullptr;
    double *idx_u = nullptr;  // generalized: u of each entry
};

// Samples per part of a table of n samples.
__host__ __device__ __forceinline__ uint32_t list_part_rows(uint32_t n, uint32_t parts) {
    return (n + parts - 1) / parts;
}

// top = the largest sum, over a sample's tips, of the sparse length above the
// tip (path); it bounds every sample's sum over its sparse nodes (shared ones
// count more than once here).  A warp per sample; positive doubles order as
// whole numbers.
static __global__ void __launch_bounds__(256)
    list_bound_kernel(const uint32_t *__restrict__ sample_ptr, const int32_t *__restrict__ start, uint32_t n,
                      const double *__restrict__ path, unsigned long long *__restrict__ top) {
    const uint32_t j = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (j >= n) return;
    double s = 0.0;
    for (uint32_t e = sample_ptr[j] + lane; e < sample_ptr[j + 1]; e += 32)
        if (start[e] >= 0) s += path[start[e]];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) atomicMax(top, static_cast<unsigned long long>(__double_as_longlong(s)));
}

// q = round(L 2^s), unit = 2^-s (and 1 behind it, zero before the launch, where a
// positive length has no units).  The scale is `least`, at which the sum of
// every sparse length stays below 2^62 units, or (top != nullptr: every column
// is summed as q) the finest at which no sample's sum reaches 2^63: it is at
// most *top, and at most `all`, the sum of every length.  (`least` counts the
// sparse lengths alone, and would wrap the sums of samples that are mostly dense nodes.)
static __global__ void fixed_lengths_kernel(const double *__restrict__ len, uint32_t n,
                                            const unsigned long long *__restrict__ top, double all, double least,
                                            unsigned long long *__restrict__ q, double *__restrict__ unit) {
    double scale = least;
    if (top) {
        const double m = fmin(__longlong_as_double(static_cast<long long>(*top)), all);
        int x = 0;
        frexp(m * (1.0 + 1e-9), &x);  // m < 2^x, by more than the roundings add
        scale = m > 0.0 ? ldexp(1.0, min(63 - x, 1000)) : 1.0;
    }
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) unit[0] = 1.0 / scale;
    if (i < n) {
        q[i] = static_cast<unsigned long long>(__double2ll_rn(len[i] * scale));
        if (len[i] > 0.0 && q[i] == 0) unit[1] = 1.0;
    }
}

// Walks up from a sample's tips: marks every node on their paths in the
// shared bitmap `bits`, stopping at nodes already marked.  A step waits for
// the parent's load, so each thread keeps WALKS paths in flight (2,000 tips,
// a path at a time: about 100 us for the one sample, with idle SMs beside it).
constexpr int WALKS = 4;
static __device__ __forceinline__ void mark_paths(const int32_t *__restrict__ start, uint32_t n,
                                                  const int32_t *__restrict__ parent, uint32_t *bits) {
    if (n <= blockDim.x) {  // one path a thread: nothing beside it in a step
        int32_t c = threadIdx.x < n ? start[threadIdx.x] : -1;
        while (c >= 0) {
            const uint32_t m = 1u << (c & 31);
            const int32_t up = parent[c];
            c = atomicOr(&bits[c >> 5], m) & m ? -1 : up;
        }
        return;
    }
    for (uint32_t e = threadIdx.x; e < n; e += WALKS * blockDim.x) {
        int32_t c[WALKS];
#pragma unroll
        for (int u = 0; u < WALKS; u++) {
            const uint32_t i = e + u * blockDim.x;
            c[u] = i < n ? start[i] : -1;
        }
        for (bool any = true; any;) {
            any = false;
#pragma unroll
            for (int u = 0; u < WALKS; u++)
                if (c[u] >= 0) {
                    const uint32_t m = 1u << (c[u] & 31);
                    const int32_t up = parent[c[u]];
                    c[u] = atomicOr(&bits[c[u] >> 5], m) & m ? -1 : up;
                    any = any || c[u] >= 0;
                }
        }
    }
}

// Faith PD by the walk: one block per sample marks its tips' paths in a bitmap
// over the tree's rows (columns are rows here), then a warp per bitmap word
// adds the lengths of its nodes, coalesced.  Bound: the walk's loads of
// parents.  (2,048 samples with 5% of 20,000 tips: 54 us and 64 us for the samples'
// tips; embedding every row for every sample and summing the rows, 655 MB
// written and read, 690 us.)
static __global__ void __launch_bounds__(256)
    faith_walk_kernel(const uint32_t *__restrict__ sample_ptr, const int32_t *__restrict__ start,
                      const int32_t *__restrict__ parent, const double *__restrict__ len, uint32_t n_rows,
                      double *__restrict__ out) {
    extern __shared__ uint32_t faith_bits[];
    __shared__ double warp_sum[8];
    const uint32_t j = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n_words = (n_rows + 31) / 32;
    for (uint32_t w = tid; w < n_words; w += 256) faith_bits[w] = 0u;
    __syncthreads();
    const uint32_t e0 = sample_ptr[j];
    mark_paths(start + e0, sample_ptr[j + 1] - e0, parent, faith_bits);
    __syncthreads();
    double sum = 0.0;
    constexpr uint32_t UN = 4;
    for (uint32_t w = warp; w < n_words; w += 8 * UN) {
        double v[UN];
#pragma unroll
        for (uint32_t u = 0; u < UN; u++) {
            const uint32_t x = w + 8 * u;
            // (bits past the last row are never set)
            v[u] = x < n_words && (faith_bits[x] >> lane) & 1u ? len[x * 32 + lane] : 0.0;
        }
        sum += (v[0] + v[1]) + (v[2] + v[3]);
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) warp_sum[warp] = sum;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < 8; w++) sum += warp_sum[w];
        out[j] = sum;
    }
}

// Both sides of the lists for column j, from its presence bitmap over the
// sparse nodes (words 32-bit words in shared memory), by the whole block of
// 256 threads; writes rs[j], the threads' `sum` included, and adds their
// shares of the nodes' fp64 lengths to `part`.  Thread t takes consecutive words, so the sample side
// comes out in node order; the positions on the node side come from one
// atomic per entry.
static __device__ __forceinline__ void write_lists(const ListArgs &la, uint32_t j, const uint32_t *bits, uint32_t words,
                                                   const double *__restrict__ len, unsigned long long sum,
                                                   double &part) {
    __shared__ uint32_t warp_tot[8];
    __shared__ unsigned long long warp_q[8];
    __shared__ unsigned long long first;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t per = (words + 255) / 256;
    const uint32_t w0 = min(words, threadIdx.x * per), w1 = min(words, w0 + per);
    uint32_t c = 0;
    for (uint32_t w = w0; w < w1; w++) c += __popc(bits[w]);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8; w++) {
        if (w < warp) before += warp_tot[w];
        total += warp_tot[w];
    }
    if (threadIdx.x == 0) {
        first = total ? atomicAdd(la.cursor, static_cast<unsigned long long>(total)) : 0ull;
        la.node_ptr[j] = first;
        la.node_cnt[j] = total;
    }
    __syncthreads();
    uint32_t *ids = la.node + first;
    uint32_t at = before + incl - c;
    for (uint32_t w = w0; w < w1; w++) {
        uint32_t m = bits[w];
        while (m) {
            ids[at++] = w * 32 + __ffs(m) - 1;
            m &= m - 1;
        }
    }
    __syncthreads();
    const uint32_t t = la.block_table[j >> 7];
    const uint32_t pos = j - la.tables[t].base;
    const uint64_t slot0 = static_cast<uint64_t>(t - la.t0) * la.n_nodes;
    constexpr int U = 4;  // entries of a thread in flight
    for (uint32_t i0 = threadIdx.x; i0 < total; i0 += U * 256) {
        uint32_t e[U], rank[U], off[U];
        unsigned long long q[U];
        double L[U];
#pragma unroll
        for (int u = 0; u < U; u++) e[u] = i0 + u * 256 < total ? ids[i0 + u * 256] : 0xFFFFFFFFu;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool on = e[u] != 0xFFFFFFFFu;
            rank[u] = on ? atomicAdd(la.count + slot0 + e[u], 1u) : 0u;
            off[u] = on ? la.off[slot0 + e[u]] : 0u;
            q[u] = on ? la.q[e[u]] : 0ull;
            L[u] = on ? len[e[u]] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            sum += q[u];
            part += L[u];
            const uint64_t to = static_cast<uint64_t>(off[u]) * LIST_ALIGN + rank[u];
            if (e[u] == 0xFFFFFFFFu) continue;
            if (la.wide)
                static_cast<uint32_t *>(la.idx)[to] = pos;
            else
                static_cast<uint16_t *>(la.idx)[to] = static_cast<uint16_t>(pos);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) warp_q[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long s = 0;
        for (int w = 0; w < 8; w++) s += warp_q[w];
        la.rs[j] = s;
    }
}

// 32-bit shared-memory additions where c < n, without a branch: the first
// returns the old value (0 where nothing is added).
__device__ __forceinline__ uint32_t shared_add_below(uint32_t addr, uint32_t v, uint32_t c, uint32_t n) {
    uint32_t old;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.lt.u32 p, %3, %4;\n\t"
        "mov.u32 %0, 0;\n\t"
        "@p atom.shared.add.u32 %0, [%1], %2;\n\t}"
        : "=&r"(old)
        : "r"(addr), "r"(v), "r"(c), "r"(n)
        : "memory");
    return old;
}
__device__ __forceinline__ void shared_carry_below(uint32_t addr, uint32_t v, uint32_t c, uint32_t n) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.lt.u32 p, %2, %3;\n\t"
        "setp.ne.and.u32 p, %1, 0, p;\n\t"
        "@p red.shared.add.u32 [%0], %1;\n\t}" ::"r"(addr),
        "r"(v), "r"(c), "r"(n)
        : "memory");
}

// shared_kl for one sample k (blockIdx.x) and the l > k of one chunk of
// columns (blockIdx.y: `chunk` whole parts) per block: the lists of k's nodes
// are read eight lanes to a list (four entries a lane), and each entry l > k
// adds the node's q to a row of 64-bit sums in shared memory, kept as two
// 32-bit halves.  Two native 32-bit shared atomics with the carry taken from
// the first one's old value add 64 bits at about 1e12 entries/s over the
// chip, a 64-bit shared atomic at 4.4e11/s.  A block reads only the parts of
// its chunk, from k's own on.
template <typename IDX, bool WEIGHTED>
__global__ void __launch_bounds__(768, 2)
    shared_sums_kernel(const ListArgs la, const SharedOut out, uint32_t col0, uint32_t cols, uint32_t chunk) {
    extern __shared__ uint32_t acc_s[];  // lo[cols], hi[cols]
    const uint32_t j = col0 + blockIdx.x;
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
    uint32_t *lo = acc_s, *hi = acc_s + cols;
    const uint32_t n_ids = la.node_cnt[j];
    const uint32_t *ids = la.node + la.node_ptr[j];
    const uint64_t slot0 = static_cast<uint64_t>(t - la.t0) * la.n_nodes;
    const IDX *idx = static_cast<const IDX *>(la.idx);
    unsigned long long *row = shared_row(out, td, t - la.t0, k);
    constexpr uint32_t GL = 8, QE = 4;  // lanes per list, entries per lane and step
    const uint32_t groups = blockDim.x / GL, grp = threadIdx.x / GL, gl = threadIdx.x % GL;
    // entries before the first part read, and before the part after the chunk
    const uint32_t first = c0 / part_rows, last = part0 + chunk;
    const uint32_t *before = first ? la.part_count + (first - 1) * la.slots + slot0 : nullptr;
    const uint32_t *upto = (last < la.parts ? la.part_count + (last - 1) * la.slots : la.count) + slot0;
    const uint32_t lo_s = smem_u32(lo), hi_off = cols * sizeof(uint32_t);
    for (uint32_t i = threadIdx.x; i < nc; i += blockDim.x) {
        lo[i] = 0;
        hi[i] = 0;
    }
    __syncthreads();
    {
        // A node takes three dependent loads (id, list bounds, entries): the
        // next node's bounds and the id after it are in flight meanwhile.
        struct Node {
            uint32_t m, p0, off;
            unsigned long long q;
        };
        auto bounds = [&](uint32_t e) {
            Node v;
            v.m = upto[e];
            // down to a whole step's boundary (entries of other parts are not in the chunk)
            v.p0 = before ? before[e] & ~(LIST_ALIGN - 1) : 0u;
            v.off = la.off[slot0 + e];
            if (!WEIGHTED) v.q = la.q[e];
            return v;
        };
        const unsigned long long *own = WEIGHTED ? la.node_q + la.node_ptr[j] : nullptr;
        uint32_t i = grp;
        Node next{};
        uint32_t id = 0;
        if (i < n_ids) {
            next = bounds(ids[i]);
            if (WEIGHTED) next.q = own[i];
        }
        if (i + groups < n_ids) id = ids[i + groups];
        for (; i < n_ids; i += groups) {
            const Node cur = next;
            if (i + groups < n_ids) {
                next = bounds(id);
                if (WEIGHTED) next.q = own[i + groups];
            }
            if (i + 2 * groups < n_ids) id = ids[i + 2 * groups];
            const uint32_t m = cur.m, p0 = cur.p0;
            const IDX *list = idx + static_cast<uint64_t>(cur.off) * LIST_ALIGN;
            const unsigned long long *list_q = WEIGHTED ? la.idx_q + static_cast<uint64_t>(cur.off) * LIST_ALIGN : nullptr;
            const uint32_t ql = static_cast<uint32_t>(cur.q), qh = static_cast<uint32_t>(cur.q >> 32);
            for (uint32_t p = p0 + gl * QE; p < m; p += GL * QE) {
                uint32_t l[QE];
                if constexpr (sizeof(IDX) == 2) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(list + p);
                    l[0] = v.x & 0xFFFFu;
                    l[1] = v.x >> 16;
                    l[2] = v.y & 0xFFFFu;
                    l[3] = v.y >> 16;
                } else {
                    const uint4 v = *reinterpret_cast<const uint4 *>(list + p);
                    l[0] = v.x;
                    l[1] = v.y;
                    l[2] = v.z;
                    l[3] = v.w;
                }
                // (entries past the list's end are 0, never > k; those of other
                // parts are outside the chunk)
                uint32_t at[QE], old[QE];
                uint32_t vl[QE], vh[QE];  // what each entry adds
                if constexpr (WEIGHTED) {
                    const ulonglong2 *qp = reinterpret_cast<const ulonglong2 *>(list_q + p);
                    const ulonglong2 q01 = qp[0], q23 = qp[1];
                    const unsigned long long qe[QE] = {q01.x, q01.y, q23.x, q23.y};
#pragma unroll
                    for (uint32_t x = 0; x < QE; x++) {
                        const unsigned long long v = qe[x] < cur.q ? qe[x] : cur.q;
                        vl[x] = static_cast<uint32_t>(v);
                        vh[x] = static_cast<uint32_t>(v >> 32);
                    }
                } else {
#pragma unroll
                    for (uint32_t x = 0; x < QE; x++) {
                        vl[x] = ql;
                        vh[x] = qh;
                    }
                }
#pragma unroll
                for (uint32_t x = 0; x < QE; x++) {
                    l[x] -= c0;
                    at[x] = lo_s + l[x] * static_cast<uint32_t>(sizeof(uint32_t));
                    old[x] = shared_add_below(at[x], vl[x], l[x], nc);
                }
#pragma unroll
                for (uint32_t x = 0; x < QE; x++)
                    shared_carry_below(at[x] + hi_off, vh[x] + (old[x] > ~vl[x] ? 1u : 0u), l[x], nc);
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nc; i += blockDim.x)
        row[c0 + i] = (static_cast<unsigned long long>(hi[i]) << 32) | lo[i];
}

// Presence words of the unweighted forms, one block of 256 threads per
// sample: bit b of P[w][j] is node column 64 w + b of sample j, for the dense
// nodes' words and then the sparse nodes'; and the sample's entries of the
// sparse nodes' lists.  Walking up from the sample's own tips replaces the
// embedding (proportions of every node for every sample, 95% of them zero).
static __global__ void __launch_bounds__(256)
    presence_words_kernel(const uint32_t *__restrict__ sample_ptr, const int32_t *__restrict__ start,
                          const int32_t *__restrict__ parent, const double *__restrict__ len,
                          const unsigned long long *__restrict__ q, uint32_t dense_words, uint32_t n_words, uint64_t ld,
                          unsigned long long *__restrict__ P, const uint32_t *__restrict__ column, const ListArgs la) {
    extern __shared__ uint32_t bits[];  // 2 n_words
    const uint32_t j = column ? column[blockIdx.x] : blockIdx.x;
    for (uint32_t w = threadIdx.x; w < 2 * n_words; w += 256) bits[w] = 0u;
    __syncthreads();
    mark_paths(start + sample_ptr[j], sample_ptr[j + 1] - sample_ptr[j], parent, bits);
    __syncthreads();
    for (uint32_t w = threadIdx.x; w < n_words; w += 256)
        P[static_cast<uint64_t>(w) * ld + j] =
            (static_cast<unsigned long long>(bits[2 * w + 1]) << 32) | bits[2 * w];
    unsigned long long sum = 0;
    for (uint32_t w = threadIdx.x; w < 2 * dense_words; w += 256) {
        uint32_t m = bits[w];
        while (m) {
            sum += q[w * 32 + __ffs(m) - 1];
            m &= m - 1;
        }
    }
    double unused = 0.0;
    write_lists(la, j, bits + 2 * dense_words, 2 * (n_words - dense_words), len + 64ull * dense_words, sum, unused);
}

// Node values of one sample per block of 256 threads (weighted methods), in
// place of an embedding of every node for every sample: the sample's tips,
// then level by level the sums of a node's children that the sample has, left
// child first as the reference sums them (src/unifrac_internal.cpp:240-257).
// Node columns: value-only tips (bypassed), sparse nodes, dense nodes, each
// section from a multiple of 32 and by height, so every child's column comes
// before its parent's.  Written: the sparse nodes' lists, the dense nodes' rows
// of L u (U), the one-sided sums W (every embedded node) and rs (sparse nodes).
struct WalkArgs {
    const uint32_t *sample_ptr;  // per column j: its entries
    const int32_t *start;        // per entry: the tip's node column
    const double *start_val;     // and count
    const int32_t *parent;       // per node column
    const int2 *child;           // per node column: children, -1 none; y == -2: a list at kids + x (count, columns)
    const int32_t *kids;
    const uint32_t *level;       // node columns where a level of internal nodes starts; n_levels pairs (start, end)
    uint32_t n_levels;
    const double *len;           // per node column
    const double *totals;        // per column j
    int normalize;
    uint32_t n_words;            // 32-bit words of the bitmap
    uint32_t sparse0, dense0;    // section starts
    double scale;                // 2^s
    int gen;                     // generalized: q = round(L u^alpha 2^s), rows of u, W = sum L u^alpha
    double alpha;
    uint32_t cap;                // nodes held in shared memory
    double *spill;               // values (and ids) of samples with more
    uint32_t *spill_id;
    unsigned long long *spill_cursor;
    uint64_t ld;
};

template <typename T>
__global__ void __launch_bounds__(256, walk::kBlocks)
    weighted_walk_kernel(const WalkArgs a, T *__restrict__ U, T *__restrict__ W, const uint32_t *__restrict__ column,
                         const ListArgs la) {
    extern __shared__ double walk_s[];
    double *vals = walk_s;                                         // [cap]
    uint32_t *ids = reinterpret_cast<uint32_t *>(vals + a.cap);    // [cap]
    uint32_t *bits = ids + a.cap;                                  // [n_words]
    uint32_t *pre = bits + a.n_words;                              // [n_words + 1] nodes before each word
    uint32_t *level_s = pre + a.n_words + 1;                       // [2 n_levels + 4] ranks where levels start and end
    __shared__ uint32_t warp_tot[8];
    __shared__ double warp_w[8];
    __shared__ unsigned long long warp_q[8];
    __shared__ unsigned long long first[2];
    const uint32_t j = column[blockIdx.x], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t w = tid; w < a.n_words; w += 256) bits[w] = 0u;
    __syncthreads();
    const uint32_t e0 = a.sample_ptr[j], n_e = a.sample_ptr[j + 1] - e0;
    // (the thread's first tip, for the values below)
    const int32_t tip = tid < n_e ? a.start[e0 + tid] : 0;
    const double count = tid < n_e ? a.start_val[e0 + tid] : 0.0, total_count = a.totals[j];
    mark_paths(a.start + e0, n_e, a.parent, bits);
    __syncthreads();
    // ranks
    const uint32_t per = (a.n_words + 255) / 256;
    const uint32_t w0 = min(a.n_words, tid * per), w1 = min(a.n_words, w0 + per);
    uint32_t c = 0;
    for (uint32_t w = w0; w < w1; w++) c += __popc(bits[w]);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8; w++) {
        if (w < warp) before += warp_tot[w];
        total += warp_tot[w];
    }
    before += incl - c;
    if (total > a.cap) {  // uniform over the block
        if (tid == 0) first[0] = atomicAdd(a.spill_cursor, static_cast<unsigned long long>(total));
        __syncthreads();
        vals = a.spill + first[0];
        ids = a.spill_id + first[0];
    }
    {
        uint32_t at = before;
        for (uint32_t w = w0; w < w1; w++) {
            pre[w] = at;
            uint32_t m = bits[w];
            while (m) {
                ids[at++] = w * 32 + __ffs(m) - 1;
                m &= m - 1;
            }
        }
        if (tid == 255) pre[a.n_words] = total;
    }
    __syncthreads();
    auto rank = [&](uint32_t col) { return pre[col >> 5] + __popc(bits[col >> 5] & ((1u << (col & 31)) - 1u)); };
    auto value = [&](int32_t col) {
        return (bits[col >> 5] >> (col & 31)) & 1u ? vals[rank(static_cast<uint32_t>(col))] : 0.0;
    };
    for (uint32_t i = tid; i < 2 * a.n_levels + 4; i += 256) level_s[i] = i < 2 * a.n_levels ? rank(a.level[i]) : total;
    for (uint32_t e = tid; e < n_e; e += 256) {
        const double v = e == tid ? count : a.start_val[e0 + e];
        vals[rank(static_cast<uint32_t>(e == tid ? tip : a.start[e0 + e]))] = a.normalize ? v / total_count : v;
    }
    __syncthreads();
    // (a thread's first nodes of the next two levels have their children on
    // their way while the current level is summed)
    auto children = [&](uint32_t lv) {
        const uint32_t r = level_s[2 * lv] + tid;
        return r < level_s[2 * lv + 1] ? a.child[ids[r]] : make_int2(-1, -1);
    };
    int2 ch = children(0), next = children(1);
    for (uint32_t lv = 0; lv < a.n_levels; lv++) {
        const int2 after = lv + 2 < a.n_levels ? children(lv + 2) : make_int2(-1, -1);
        const uint32_t r0 = level_s[2 * lv], r1 = level_s[2 * lv + 1];
        if (r0 != r1) {  // uniform over the block
            for (uint32_t r = r0 + tid; r < r1; r += 256) {
                if (r >= r0 + 256) ch = a.child[ids[r]];
                double s = 0.0;
                if (ch.y != -2) {
                    if (ch.x >= 0) s += value(ch.x);
                    if (ch.y >= 0) s += value(ch.y);
                } else {
                    const int32_t *k = a.kids + ch.x;
                    for (int32_t q = 1; q <= k[0]; q++) s += value(k[q]);
                }
                vals[r] = s;
            }
            __syncthreads();
        }
        ch = next;
        next = after;
    }
    const uint32_t rs0 = rank(a.sparse0), rd0 = rank(a.dense0);
    const uint32_t n_sp = rd0 - rs0;
    if (tid == 0) {
        first[1] = total > rs0 ? atomicAdd(la.cursor, static_cast<unsigned long long>(total - rs0)) : 0ull;
        la.node_ptr[j] = first[1];
        la.node_cnt[j] = n_sp;
        la.node_all[j] = total - rs0;
    }
    __syncthreads();
    auto power = [&](double u) {
        return !a.gen || a.alpha == 1.0 ? u : a.alpha == 0.5 ? sqrt(u) : a.alpha == 0.0 ? 1.0 : pow(u, a.alpha);
    };
    // dense rows
    double wsum = 0.0;
    for (uint32_t r = rd0 + tid; r < total; r += 256) {
        const uint32_t c = ids[r];
        const double u = vals[r], lu = a.len[c] * power(u);
        wsum += lu;
        U[static_cast<uint64_t>(c - a.dense0) * a.ld + j] = static_cast<T>(a.gen ? u : lu);
        la.node[first[1] + r - rs0] = c - a.sparse0;
        la.node_u[first[1] + r - rs0] = u;
    }
    // lists
    const uint32_t t = la.block_table[j >> 7];
    const uint32_t pos = j - la.tables[t].base;
    const uint64_t slot0 = static_cast<uint64_t>(t - la.t0) * la.n_nodes;
    unsigned long long qsum = 0;
    constexpr int UN = 4;  // entries of a thread in flight
    for (uint32_t i0 = tid; i0 < n_sp; i0 += UN * 256) {
        uint32_t e[UN], at[UN], off[UN];
        double v[UN], lu[UN];
#pragma unroll
        for (int u = 0; u < UN; u++) {
            const uint32_t i = i0 + u * 256;
            const bool on = i < n_sp;
            e[u] = on ? ids[rs0 + i] - a.sparse0 : 0xFFFFFFFFu;
            at[u] = on ? atomicAdd(la.count + slot0 + e[u], 1u) : 0u;
            off[u] = on ? la.off[slot0 + e[u]] : 0u;
            v[u] = on ? vals[rs0 + i] : 0.0;
            lu[u] = on ? a.len[a.sparse0 + e[u]] * power(v[u]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < UN; u++) {
            if (e[u] == 0xFFFFFFFFu) continue;
            wsum += lu[u];
            const unsigned long long q = static_cast<unsigned long long>(__double2ll_rn(lu[u] * a.scale));
            qsum += q;
            const uint64_t to = static_cast<uint64_t>(off[u]) * LIST_ALIGN + at[u];
            if (la.wide)
                static_cast<uint32_t *>(la.idx)[to] = pos;
            else
                static_cast<uint16_t *>(la.idx)[to] = static_cast<uint16_t>(pos);
            la.idx_q[to] = q;
            if (a.gen) la.idx_u[to] = v[u];
            la.node[first[1] + i0 + u * 256] = e[u];
            la.node_q[first[1] + i0 + u * 256] = q;
            la.node_u[first[1] + i0 + u * 256] = v[u];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
        qsum += __shfl_xor_sync(0xffffffffu, qsum, o);
    }
    if (lane == 0) {
        warp_w[warp] = wsum;
        warp_q[warp] = qsum;
    }
    __syncthreads();
    if (tid == 0) {
        double w = 0.0;
        unsigned long long q = 0;
        for (int i = 0; i < 8; i++) {
            w += warp_w[i];
            q += warp_q[i];
        }
        if (W) W[j] = static_cast<T>(w);
        la.rs[j] = q;
    }
}

}  // namespace dev
}  // namespace ssu
