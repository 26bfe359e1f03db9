// Shared memory of the weighted walk (weighted_walk_kernel): a bit and a rank
// per node column, the ranks where each level of each section starts and
// ends, and the values (and columns) of up to `cap` nodes; a sample with more
// keeps them in memory.  Plain C++ (no CUDA), so that the choice of a plan's
// form and its setup go by the same sizes, and the host tests can check them.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace ssu {
namespace walk {

constexpr int kBlocks = 6;                     // blocks an SM: the walk waits on loads and barriers, so samples in flight set its pace
constexpr size_t kSharedMost = 200 * 1024;     // the kernel's limit
constexpr size_t kValuesLeast = 8 * 1024;      // bytes of values held at least
constexpr size_t kPerNode = sizeof(double) + sizeof(uint32_t);

// Words of n_cols columns and n_levels (start, end) pairs.
constexpr size_t fixed_bytes(uint64_t n_cols, uint64_t n_levels) {
    return sizeof(uint32_t) * (2 * (n_cols / 32) + 1 + 2 * n_levels + 4) + 8;
}

// Nodes held in shared memory: what leaves kBlocks to an SM, or the least.
// (eight tables on 50,000 tips, 4,500 nodes a sample: the walk takes the same
// with fewer blocks and all of them in shared memory)
inline uint32_t capacity(uint32_t n_cols, uint64_t n_levels) {
    const size_t fixed = fixed_bytes(n_cols, n_levels);
    constexpr size_t block = 227 * 1024 / kBlocks - 1536;  // (1 KB of it the system's)
    const size_t room = fixed + kValuesLeast < block ? block - fixed : kValuesLeast;
    return static_cast<uint32_t>(std::min<size_t>(n_cols, room / kPerNode));
}

inline size_t shared_bytes(uint32_t n_cols, uint64_t n_levels) {
    return capacity(n_cols, n_levels) * kPerNode + fixed_bytes(n_cols, n_levels);
}

// Whether a tree of n_nodes nodes and `heights` levels of internal nodes fits,
// however its nodes fall into the three sections (each a multiple of 32
// columns; both sparse and dense nodes may have every level).
inline bool fits(uint32_t n_nodes, uint64_t heights) {
    return fixed_bytes(static_cast<uint64_t>(n_nodes) + 3 * 32, 2 * heights) + kValuesLeast <= kSharedMost;
}

}  // namespace walk
}  // namespace ssu
