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
void (*close_of(int ak))(const CloseArgs, const ListArgs) {
    switch (ak) {
    case 1: return close_strips_kernel<T, OpCloseGen<1>, BM, BN>;
    case 2: return close_strips_kernel<T, OpCloseGen<2>, BM, BN>;
    case 3: return close_strips_kernel<T, OpCloseGen<3>, BM, BN>;
    default: return close_strips_kernel<T, OpCloseGen<0>, BM, BN>;
    }
}

template <typename T, int BM, int BN>
cudaError_t close_launch(const GenLaunch &g, const ListArgs &la, const CloseArgs &c, cudaStream_t s) {
    const uint32_t strips = c.n_tiles * close_strips<BM, BN>(), most = 2 * static_cast<uint32_t>(g.n_sms);
    close_of<T, BM, BN>(g.ak)<<<strips < most ? strips : most, CTHREADS, close_smem(c.n_words), s>>>(c, la);
    return cudaGetLastError();
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
    for (int ak = 0; ak < 4; ak++)
        for (auto kernel : {close_of<double, 128, 64>(ak), close_of<double, 64, 64>(ak), close_of<float, 128, 64>(ak),
                            close_of<float, 64, 64>(ak)}) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       static_cast<int>(walk::kSharedMost));
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
    CloseArgs c{};
    c.tiles = f.tiles;
    c.n_tiles = f.n_tiles;
    c.tables = f.tables;
    c.tile_flags = f.tile_flags;
    c.close = f.close;
    c.len = g.len;
    c.n_words = g.n_words;
    c.alpha = g.alpha;
    c.out = f.out;
    if (small) {
        gen_finalize_kernel<T, 64, 64, 4, 4><<<f.n_tiles, 256, 0, s>>>(f);
        return close_launch<T, 64, 64>(g, la, c, s);
    }
    gen_finalize_kernel<T, 128, 64, 8, 4><<<f.n_tiles, 256, 0, s>>>(f);
    return close_launch<T, 128, 64>(g, la, c, s);
}
template cudaError_t gen_finish_launch<double>(const GenLaunch &, const ListArgs &, const GenFinish &, bool, cudaStream_t);
template cudaError_t gen_finish_launch<float>(const GenLaunch &, const ListArgs &, const GenFinish &, bool, cudaStream_t);

}  // namespace dev
}  // namespace ssu
