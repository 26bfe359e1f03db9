// Unweighted sums over nodes that few samples have, through sample lists.
//
// For a set S of sparse nodes and a pair (k, l),
//   sum_{n in S, k has n and l not} L_n = rs_k - shared_kl,
//   rs_k = sum_{n in S, k has n} L_n,  shared_kl = sum_{n in S, both have n} L_n,
// and shared_kl only needs, for sample k, the lists of the samples of k's own
// nodes: m^2 / 2 additions for a node that m samples have, against n^2 / 2
// terms in a dense form.  The lengths are 64-bit fixed point,
// q = round(L 2^s) with sum_S L 2^s < 2^62, and every sum of them is exact,
// so the differences above are exact sums of the q: no cancellation (two
// samples with the same nodes differ by exactly 0), and no dependence on the
// order of the additions.
//
// Lists (built by the walk over each sample's tips, per execute):
//   node side:   per (table, node) the table's samples that have it, 16 or 32
//                bits each, at a 16-byte offset laid out once from the tips'
//                entry counts (an upper bound of the length); a table's
//                samples are walked in up to LIST_PARTS launches of
//                consecutive samples, so a list is in order from part to
//                part (in any order within one), and where each part starts
//                is kept: a sample reads its own part and the later ones;
//   sample side: per sample its sparse nodes, in node order, in one array.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ssu_kernels.cuh"

namespace ssu {
namespace dev {

constexpr uint32_t LIST_ALIGN = 8;  // entries; node lists start on a multiple (16 bytes of 16-bit entries)
constexpr uint32_t LIST_PARTS = 8;  // launches of the walk, at most

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

// q = round(L 2^s), unit = 2^-s.  The scale is `least`, at which the sum of
// every sparse length stays below 2^62 units, or (top != nullptr) the finest
// at which the largest sample's does.
static __global__ void fixed_lengths_kernel(const double *__restrict__ len, uint32_t n,
                                            const unsigned long long *__restrict__ top, double least,
                                            unsigned long long *__restrict__ q, double *__restrict__ unit) {
    double scale = least;
    if (top) {
        const double m = __longlong_as_double(static_cast<long long>(*top));
        int x = 0;
        frexp(m * (1.0 + 1e-9), &x);  // m < 2^x
        if (m > 0.0) scale = fmax(ldexp(1.0, min(62 - x, 1000)), least);
    }
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *unit = 1.0 / scale;
    if (i < n) q[i] = static_cast<unsigned long long>(__double2ll_rn(len[i] * scale));
}

// Walks up from a sample's tips: marks every node on their paths in the
// shared bitmap `bits`, stopping at nodes already marked.  A step waits for
// the parent's load, so each thread keeps WALKS paths in flight (2,000 tips,
// a path at a time: about 100 us for the one sample, with idle SMs beside it).
constexpr int WALKS = 4;
static __device__ __forceinline__ void mark_paths(const int32_t *__restrict__ start, uint32_t n,
                                                  const int32_t *__restrict__ parent, uint32_t *bits) {
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
template <typename IDX>
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
            v.q = la.q[e];
            return v;
        };
        uint32_t i = grp;
        Node next{};
        uint32_t id = 0;
        if (i < n_ids) next = bounds(ids[i]);
        if (i + groups < n_ids) id = ids[i + groups];
        for (; i < n_ids; i += groups) {
            const Node cur = next;
            if (i + groups < n_ids) next = bounds(id);
            if (i + 2 * groups < n_ids) id = ids[i + 2 * groups];
            const uint32_t m = cur.m, p0 = cur.p0;
            const IDX *list = idx + static_cast<uint64_t>(cur.off) * LIST_ALIGN;
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
#pragma unroll
                for (uint32_t x = 0; x < QE; x++) {
                    l[x] -= c0;
                    at[x] = lo_s + l[x] * static_cast<uint32_t>(sizeof(uint32_t));
                    old[x] = shared_add_below(at[x], ql, l[x], nc);
                }
#pragma unroll
                for (uint32_t x = 0; x < QE; x++)
                    shared_carry_below(at[x] + hi_off, qh + (old[x] > ~ql ? 1u : 0u), l[x], nc);
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

}  // namespace dev
}  // namespace ssu
