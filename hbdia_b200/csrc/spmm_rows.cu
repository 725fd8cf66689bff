// Launcher of the row-major SpMM (spmm_rows.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "args.cuh"
#include "hbdia_internal.hpp"
#include "spmm_rows.cuh"

namespace hbdia {
namespace {

template <typename VT, typename XT, int V, int G, int S>
void launch(const DevicePlan &P, const XT *X, int64_t ldx, XT *Y, int64_t ldy, int32_t k, cudaStream_t s) {
    auto kernel = dev::spmm_rows<VT, XT, V, G, S>;
    constexpr int threads = dev::kRowsWarps * 32;
    int sms = 0, perSm = 0;
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, P.device), "cudaDeviceGetAttribute");
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, threads, 0),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    const int64_t slabs = static_cast<int64_t>(P.numTiles) * (32 / (32 / G * S));
    const int64_t need = (slabs + dev::kRowsWarps - 1) / dev::kRowsWarps;
    const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(need, int64_t(sms) * std::max(1, perSm))));
    const int32_t vec = (reinterpret_cast<uintptr_t>(P.vals) & 15) == 0;
    kernel<<<grid, threads, 0, s>>>(make_args<VT, XT>(P), X, ldx, Y, ldy, k, vec);
}

}  // namespace

template <typename VT, typename XT>
void launch_spmm_rows(const DevicePlan &P, const XT *X, int64_t ldx, XT *Y, int64_t ldy, int32_t k, int32_t width,
                      void *stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    constexpr int VW = 16 / static_cast<int>(sizeof(XT));  // elements of a 16-byte access
    const bool wide = k % VW == 0 && ldx % VW == 0 && ldy % VW == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
    const int32_t w = std::min(width, k);
    if (wide) {
        if constexpr (VW == 2) {
            if (w <= 2) return launch<VT, XT, 2, 1, 1>(P, X, ldx, Y, ldy, k, s);
            if (w <= 4) return launch<VT, XT, 2, 2, 2>(P, X, ldx, Y, ldy, k, s);
            if (w <= 8) return launch<VT, XT, 2, 4, 4>(P, X, ldx, Y, ldy, k, s);
            if (w <= 16) return launch<VT, XT, 2, 8, 8>(P, X, ldx, Y, ldy, k, s);
            return launch<VT, XT, 2, 16, 8>(P, X, ldx, Y, ldy, k, s);
        } else {
            if (w <= 4) return launch<VT, XT, 4, 1, 1>(P, X, ldx, Y, ldy, k, s);
            if (w <= 8) return launch<VT, XT, 4, 2, 2>(P, X, ldx, Y, ldy, k, s);
            if (w <= 16) return launch<VT, XT, 4, 4, 4>(P, X, ldx, Y, ldy, k, s);
            return launch<VT, XT, 4, 8, 8>(P, X, ldx, Y, ldy, k, s);
        }
    }
    if (w <= 2) return launch<VT, XT, 1, 2, 2>(P, X, ldx, Y, ldy, k, s);
    if (w <= 4) return launch<VT, XT, 1, 4, 4>(P, X, ldx, Y, ldy, k, s);
    if (w <= 8) return launch<VT, XT, 1, 8, 8>(P, X, ldx, Y, ldy, k, s);
    if (w <= 16) return launch<VT, XT, 1, 16, 8>(P, X, ldx, Y, ldy, k, s);
    return launch<VT, XT, 1, 32, 8>(P, X, ldx, Y, ldy, k, s);
}

template void launch_spmm_rows<double, double>(const DevicePlan &, const double *, int64_t, double *, int64_t, int32_t, int32_t, void *);
template void launch_spmm_rows<float, double>(const DevicePlan &, const double *, int64_t, double *, int64_t, int32_t, int32_t, void *);
template void launch_spmm_rows<__nv_bfloat16, double>(const DevicePlan &, const double *, int64_t, double *, int64_t, int32_t, int32_t, void *);
template void launch_spmm_rows<float, float>(const DevicePlan &, const float *, int64_t, float *, int64_t, int32_t, int32_t, void *);

}  // namespace hbdia
