// Unweighted presence-word pair-kernel instances
// (src/unifrac_task_impl.hpp:1424-1753).
#include "ssu_pairs.cuh"

namespace ssu {

template <typename T>
std::vector<PairKernel<T>> bits_candidates(bool normalized) {
    constexpr int KW = sizeof(T) == 8 ? 2 : 4;
    if (normalized)
        return {bits_kernel<T, true, 128, 64, 8, 4, KW>("pair_bits<unweighted>", "128x64/8x4"),
                bits_kernel<T, true, 64, 64, 4, 4, KW>("pair_bits<unweighted>", "64x64/4x4")};
    return {bits_kernel<T, false, 128, 64, 8, 4, KW>("pair_bits<unweighted_unnormalized>", "128x64/8x4"),
            bits_kernel<T, false, 64, 64, 4, 4, KW>("pair_bits<unweighted_unnormalized>", "64x64/4x4")};
}

template <bool NORM, int BM, int BN>
static void xor_pairs(const dev::PairArgs<double> &a, const double *len, uint32_t ctas, cudaStream_t s) {
    dev::xor_pairs_kernel<NORM, BM, BN><<<ctas, 256, 0, s>>>(a, len);
}

template <bool NORM>
static SharedBits shared_bits_of(const char *name, bool small) {
    if (small) return {shared_bits_kernel<NORM, 32, 32, 2, 2, 4>(name, "32x32/2x2"), xor_pairs<NORM, 32, 32>};
    return {shared_bits_kernel<NORM, 128, 64, 8, 4, 4>(name, "128x64/8x4"), xor_pairs<NORM, 128, 64>};
}

SharedBits shared_bits(bool normalized, bool small) {
    return normalized ? shared_bits_of<true>("pair_shared_bits<unweighted>", small)
                      : shared_bits_of<false>("pair_shared_bits<unweighted_unnormalized>", small);
}

template std::vector<PairKernel<double>> bits_candidates<double>(bool);
template std::vector<PairKernel<float>> bits_candidates<float>(bool);

}  // namespace ssu
