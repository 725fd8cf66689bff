// Launcher of the row-major SpMM (spmm_rows.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "args.cuh"
#include "hbdia_internal.hpp"
#include "spmm_rows.cuh"

namespace hbdia {

// 16-byte accesses: every row segment of X and Y begins and ends on a 16-byte boundary.
bool spmm_rows_wide(const void *X, int64_t ldx, const void *Y, int64_t ldy, int32_t k, int elem) {
    const int VW = 16 / elem;
    return k % VW == 0 && ldx % VW == 0 && ldy % VW == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
}

// Whether lanes sharing rows of X beat the kernels with one lane per row
// (spmm_kernels.cuh), which read whole 16-byte groups of a row where k is 2, 4 or
// 8 and keep more warps on an SM.  Those win where a row of X is a few bytes,
// where few loads are left to share (short lists), and on small matrices.
// B200, us, one lane per row -> shared rows, blockWidth 32 unless given:
//  * 8-byte x: k = 1 7-point 32^3 5.1 -> 6.1, 48^3 10.3 -> 8.2; k = 2 7-point
//    64^3 12.3 -> 14.4, 96^3 51.2 -> 35.4, 9 offsets 300 K rows 12.3 -> 15.3, 1 M
//    59.5 -> 41.6, 27-point 64^3 28.7 -> 23.5, FP32 storage 18.5 -> 22.6, 96^3
//    63.6 -> 59.1; k = 3 22.0 -> 20.5 at 27-point 48^3 and better elsewhere; k = 4
//    7-point 64^3 14.3 -> 16.4, 27-point 96^3 93.2 -> 100.7; k = 8 off a 16-byte
//    boundary 27-point 48^3 24.6 -> 27.8, 64^3 68.0 -> 49.6;
//  * 4-byte x: k = 1 27-point 64^3 16.4 -> 24.4, 96^3 69.9 -> 62.2, 7-point 96^3
//    30.8 -> 37.3; k = 2 always slower (27-point 96^3 40.1 -> 62.2); k = 3
//    27-point 64^3 25.7 -> 35.2, 96^3 110.7 -> 94.1; k = 4 7-point 64^3 10.3 ->
//    14.1, 27-point 64^3 22.6 -> 21.5; off a 16-byte boundary 64^3 16.4 -> 35.1;
//    k = 5 to 7 7-point 64^3 14.6 -> 20.3, 96^3 69.1 -> 53.2; with ldx = 8, whose
//    one-lane rows lie 32 bytes apart, k = 7 22.6 -> 21.5; k = 8 off a boundary
//    27-point 96^3 89.4 -> 117; k = 9 7-point 64^3 26.7 -> 31.0, 112^3 166 ->
//    154; k = 17 80^3 92.9 -> 115, 48^3 24.6 -> 26.6, 32^3 14.7 -> 12.3;
//  * wide blocks (one thread per row): up to 40^3 equal or better; FP64 k = 1
//    7-point 72^3 10.3 -> 18.5, k = 2 27-point 56^3 17.4 -> 18.4, 72^3 38.9 ->
//    28.8, k = 3 35.4 -> 45.0, k = 4 7-point 56^3 11.1 -> 12.4, 72^3 20.5 ->
//    18.4, k = 5 25.6 -> 28.2, k = 6 27-point 48^3 19.4 -> 24.6, 56^3 40.3 -> 36.3,
//    100^3 144 -> 156, k = 9 80^3 137 -> 154, k = 11 160 -> 155; float k = 4 7-point
//    72^3 13.8 -> 16.4, 27-point 35.8 -> 26.1, k = 6 39 -> 49, off a boundary 27-point
//    80^3 k = 9 90 -> 122, k = 13 120 -> 127, k = 15 142 -> 128, k = 17 187 -> 230, k =
//    23 281 -> 233.
// The rest is better with shared rows: 27-point 96^3 k = 16 0.31 of the time in
// FP64, 0.15 in float.
bool spmm_rows_pay(const DevicePlan &P, int32_t k, bool wide, int64_t ldx) {
    const int64_t n = P.n, tiles = P.numTiles;
    const int64_t work = P.totalOffsets * (P.bw / 32);  // offsets of 32-row tiles
    const bool isLong = work >= 16 * tiles, f32 = P.dtype == HBDIA_F32;
    if (P.bw != 32) {
        if (n <= (1 << 16)) return true;
        if (f32) return wide ? k >= 8 || (k == 4 && isLong) : k > 20 || (k > 13 && k < 17);
        if (k == 2) return wide && work >= 300000;
        if (k == 4) return wide && work >= 70000;
        if (k == 6) return wide && work >= 100000 && n <= 500000;
        return k >= 10 || (k == 8 && (wide || work >= 100000));
    }
    if (f32) {
        if (k == 1) return n >= 800000 && work >= 9 * tiles;
        if (k == 2) return false;
        if (k == 3) return n >= 800000;
        if (k == 4) return wide && isLong;
        if (k < 8) return work >= 190000 || ldx % 8 == 0;
        if (k == 8) return wide;
        const bool few = !wide && work < 12 * tiles;
        if (few && k <= 11) return n < 200000 || n > 700000;
        if (few && k >= 17 && k <= 19) return n < 100000;
        return true;
    }
    if (k == 1) return n >= (1 << 16);
    if (k == 2) return work >= (P.storage == HBDIA_STORE_NATIVE ? 150000 : 700000);
    if (k == 4) return false;
    return k != 8 || wide || n >= 200000;
}

namespace {

template <typename VT, typename XT, int V, int G, int S>
void launch(const DevicePlan &P, const XT *X, int64_t ldx, XT *Y, int64_t ldy, int32_t k, cudaStream_t s) {
    auto kernel = dev::spmm_rows<VT, XT, V, G, S>;
    const int64_t slabs = static_cast<int64_t>(P.numTiles) * (32 / (32 / G * S));
    int sms = 0;
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, P.device), "cudaDeviceGetAttribute");
    // 4 warps a CTA where a warp has few slabs: they reach every SM (27-point 32^3
    // FP64 k = 8 16.4 -> 12.5 us); 16 where there are many, whose neighbouring
    // slabs share lines in L1 (7-point 96^3 k = 12 112 -> 107)
    const bool small = !dev::rows_fixed_cta<XT, V, S>() && slabs <= 2 * int64_t(sms) * dev::kRowsWarps;
    const int threads = 32 * (small ? 4 : dev::kRowsWarps);
    // CTAs an SM holds: the kernel's own figure, the same on every B200, asked for once
    static std::atomic<int> held[2];
    int perSm = held[small].load(std::memory_order_relaxed);
    if (perSm == 0) {
        check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, threads, 0),
                   "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        perSm = std::max(1, perSm);
        held[small].store(perSm, std::memory_order_relaxed);
    }
    const int64_t need = (slabs + threads / 32 - 1) / (threads / 32);
    const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(need, int64_t(sms) * perSm)));
    const int32_t vec = (reinterpret_cast<uintptr_t>(P.vals) & 15) == 0;
    kernel<<<grid, threads, 0, s>>>(make_args<VT, XT>(P), X, ldx, Y, ldy, k, vec);
}

}  // namespace

template <typename VT, typename XT>
void launch_spmm_rows(const DevicePlan &P, const XT *X, int64_t ldx, XT *Y, int64_t ldy, int32_t k, int32_t width,
                      void *stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    constexpr int VW = 16 / static_cast<int>(sizeof(XT));  // elements of a 16-byte access
    const bool wide = spmm_rows_wide(X, ldx, Y, ldy, k, static_cast<int>(sizeof(XT)));
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
