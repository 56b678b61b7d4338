// Instantiations and launches of the block-per-quartet kernel, one per ket
// class up to (ff).
#include "kernels.hpp"

#include <algorithm>

#include "device_common.cuh"
#include "eri_rows.cuh"
#include "engine.hpp"

namespace tlno_gpu {

#define TLNO_ROWS_KETS(X) \
    X(0, 0) X(1, 0) X(1, 1) X(2, 0) X(2, 1) X(2, 2) X(3, 0) X(3, 1) X(3, 2) X(3, 3)

void rows_upload(const dev::DevTables& t, const dev::CartTable& c, const dev::C2STable& s) {
    dev::upload_constant_tables(t, c, s);
#define TLNO_ROWS_ATTR(lc, ld)                                                                                  \
    TLNO_CUDA(cudaFuncSetAttribute(dev::eri_rows_jk_kernel<double, lc, ld>,                                     \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem));                \
    TLNO_CUDA(cudaFuncSetAttribute(dev::eri_rows_jk_kernel<float, lc, ld>,                                      \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBlockSmem));
    TLNO_ROWS_KETS(TLNO_ROWS_ATTR)
#undef TLNO_ROWS_ATTR
}

namespace {

// Test hook of reciprocals: out[2 i] = 1/x, out[2 i + 1] = 1/sqrt(x).
template <typename R>
__global__ void reciprocals_test_kernel(const double* x, int n, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    R inv, rs;
    dev::reciprocals(R(x[i]), inv, rs);
    out[2 * i] = double(inv);
    out[2 * i + 1] = double(rs);
}

template <typename R, int LC, int LD>
void launch(const dev::PlanView& pv, const dev::ClassLaunch& cl, int sms, cudaStream_t s) {
    // item slots per batch: 32 (64 take the shared memory of resident blocks),
    // halved while the block needs more than 100 KB
    dev::RowsLayout lay;
    int nb_items = 32;
    for (;;) {
        lay.init(cl.la, cl.lb, LC, LD, nb_items);
        if (lay.words * 8 <= 100 * 1024 || nb_items <= 16) break;
        nb_items /= 2;
    }
    const int bytes = lay.words * 8;
    int per_sm = 0;
    TLNO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dev::eri_rows_jk_kernel<R, LC, LD>, lay.threads,
                                                            bytes));
    const long long ntiles = cl.tile_end - cl.tile_begin;
    const int wave = sms * std::max(per_sm, 1);
    const int part = block_tile_part(ntiles, cl.bk, wave);
    const int grid = static_cast<int>(std::max(1LL, std::min<long long>(ntiles * ((cl.bk + part - 1) / part), wave)));
    dev::eri_rows_jk_kernel<R, LC, LD><<<grid, lay.threads, bytes, s>>>(pv, cl, nb_items, part);
    TLNO_CUDA(cudaGetLastError());
}

}  // namespace

void launch_reciprocals_test(const double* x, int n, bool fp32, double* out, cudaStream_t s) {
    if (fp32) reciprocals_test_kernel<float><<<(n + 127) / 128, 128, 0, s>>>(x, n, out);
    else reciprocals_test_kernel<double><<<(n + 127) / 128, 128, 0, s>>>(x, n, out);
    TLNO_CUDA(cudaGetLastError());
}

bool launch_eri_jk_rows(const dev::PlanView& pv, const dev::ClassLaunch& cl, bool fp32, int sms, cudaStream_t s) {
    if (cl.la > 3 || cl.la + cl.lb < 2) return false;
#define TLNO_ROWS_CASE(a, b)                             \
    if (cl.lc == a && cl.ld == b) {                      \
        if (fp32) launch<float, a, b>(pv, cl, sms, s);   \
        else launch<double, a, b>(pv, cl, sms, s);       \
        return true;                                     \
    }
    TLNO_ROWS_KETS(TLNO_ROWS_CASE)
#undef TLNO_ROWS_CASE
    return false;
}

}  // namespace tlno_gpu
