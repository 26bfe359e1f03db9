// Generalized UniFrac by sample lists: instances and launches.
#include "ssu_gen.cuh"

namespace ssu {
namespace dev {

namespace {

template <typename IDX>
void (*sums_of(int ak))(const ListArgs, const GenSums, const double *, double, double, uint32_t, uint32_t) {
    switch (ak) {
    case 1: return gen_sums_kernel<IDX, 1>;
    case 2: return gen_sums_kernel<IDX, 2>;
    case 3: return gen_sums_kernel<IDX, 3>;
    default: return gen_sums_kernel<IDX, 0>;
    }
}

template <typename T, int BM, int BN>
void (*close_of(int ak))(const GenFinish, const ListArgs, const double *, double) {
    switch (ak) {
    case 1: return gen_close_kernel<T, 1, BM, BN>;
    case 2: return gen_close_kernel<T, 2, BM, BN>;
    case 3: return gen_close_kernel<T, 3, BM, BN>;
    default: return gen_close_kernel<T, 0, BM, BN>;
    }
}

template <int AK>
std::vector<PairKernel<double>> rows_family() {
    using Op = OpGenRows<AK>;
    return {values_kernel<double, Op, 128, 64, 8, 4, 16>("pair_union_lists<generalized>", "128x64/8x4"),
            values_kernel<double, Op, 64, 64, 4, 4, 16>("pair_union_lists<generalized>", "64x64/4x4")};
}

}  // namespace

std::vector<PairKernel<double>> gen_rows_candidates(int ak) {
    switch (ak) {
    case 1: return rows_family<1>();
    case 2: return rows_family<2>();
    case 3: return rows_family<3>();
    default: return rows_family<0>();
    }
}

cudaError_t gen_configure() {
    for (int ak = 0; ak < 4; ak++)
        for (int wide = 0; wide < 2; wide++) {
            const cudaError_t e =
                cudaFuncSetAttribute(wide ? sums_of<uint32_t>(ak) : sums_of<uint16_t>(ak),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(16 * kGenCols));
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

cudaError_t gen_sums_launch(const GenLaunch &g, const ListArgs &la, const GenSums &out, uint32_t columns, uint32_t cols,
                            uint32_t chunk, uint32_t chunks, cudaStream_t s) {
    const auto kernel = la.wide ? sums_of<uint32_t>(g.ak) : sums_of<uint16_t>(g.ak);
    kernel<<<dim3(columns, chunks), cols > 1024 ? 512 : 256, 16 * cols, s>>>(la, out, g.len, g.alpha, g.scale, cols, chunk);
    return cudaGetLastError();
}

template <typename T>
cudaError_t gen_finish_launch(const GenLaunch &g, const ListArgs &la, const GenFinish &f, bool small, cudaStream_t s) {
    if (small) {
        gen_finalize_kernel<T, 64, 64, 4, 4><<<f.n_tiles, 256, 0, s>>>(f);
        close_of<T, 64, 64>(g.ak)<<<f.n_tiles, 256, 0, s>>>(f, la, g.len, g.alpha);
    } else {
        gen_finalize_kernel<T, 128, 64, 8, 4><<<f.n_tiles, 256, 0, s>>>(f);
        close_of<T, 128, 64>(g.ak)<<<f.n_tiles, 256, 0, s>>>(f, la, g.len, g.alpha);
    }
    return cudaGetLastError();
}
template cudaError_t gen_finish_launch<double>(const GenLaunch &, const ListArgs &, const GenFinish &, bool, cudaStream_t);
template cudaError_t gen_finish_launch<float>(const GenLaunch &, const ListArgs &, const GenFinish &, bool, cudaStream_t);

}  // namespace dev
}  // namespace ssu
