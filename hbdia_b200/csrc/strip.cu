// The strip SpMV (spmv_strip.cuh): its descriptors, when it runs, its launch.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "args.cuh"
#include "hbdia_internal.hpp"
#include "spmv_strip.cuh"

namespace hbdia {
namespace {

constexpr int kStripWarps = 16;  // 128 registers a thread: 512 threads fill an SM's register file
constexpr int kStripGroup = 4;   // offsets per stage

// Stages per warp: 2 for 8-byte values (27-point 256^3 662 us, 3 stages 670),
// 3 for narrower ones, whose stages are smaller (4 stages: 2 % slower).
template <typename VT>
constexpr int strip_ring() {
    return sizeof(VT) == 8 ? 2 : 3;
}

// f(kernel, dynamic shared memory) of the instance for one layout: blockWidth 32, with its
// quad-interleaved forms, or a larger multiple of 32.
template <typename VT, typename XT, typename F>
void with_strip_kernel(const DevicePlan &P, F f) {
    constexpr int U = kStripGroup, D = strip_ring<VT>(), NW = kStripWarps;
    constexpr size_t smem = NW * dev::strip_warp_smem<VT, XT, U, D>();
    static_assert(smem <= 232448, "strip stages too large for one CTA");
    if constexpr (sizeof(VT) >= 4) {
        if (P.bw != 32) return f(dev::spmv_strip<VT, XT, U, D, NW, false, false>, smem);
    }
    if constexpr (sizeof(VT) < 8 && sizeof(XT) == 8) {
        if (P.quadLayout) return f(dev::spmv_strip<VT, XT, U, D, NW, true, true>, smem);
    }
    f(dev::spmv_strip<VT, XT, U, D, NW, false, true>, smem);
}

template <typename VT, typename XT>
void configure(const DevicePlan &P) {
    with_strip_kernel<VT, XT>(P, [](auto kernel, size_t smem) {
        check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                   "cudaFuncSetAttribute(strip SpMV)");
    });
}

// Whether a layout has enough work for the strip kernel to be the faster one.
// A warp's first strip waits for a chain of loads that the other kernels spread
// over four times as many warps (148 x 16 here).  B200, us, other kernel ->
// strip kernel:
//  * native values of blockWidth 32, from 4 strips a warp: 27-point FP64 80^3
//    (1.7) 24.8 -> 27.9, 96^3 (2.9) 38.4 -> 38.9, 112^3 (4.6) 61.7 -> 60.0; 9
//    offsets 950 K rows (3.1) 20.9 -> 21.6, 1.5 M (4.9) 31.6 -> 26.7, float
//    16.5 -> 17.3, 24.4 -> 20.5.  From 2 where the pipelined kernel's groups of
//    9 are mostly tails: 7-point 64^3 (0.9) 8.7 -> 10.3, 90^3 (2.4) 22.6 ->
//    17.8, 100^3 (3.3) 28.7 -> 20.6, float 22.9 -> 16.9;
//  * FP32 storage, from half a strip a warp and 32 K strip-offsets: 27-point
//    40^3 (13 K) 12.4 -> 14.4, 56^3 (37 K) 17.9 -> 14.4; 9 offsets 280 K rows
//    (20 K) 8.4 -> 9.5, 600 K (42 K) 13.3 -> 13.7, 1 M 19.9 -> 18.5; 7-point
//    70^3 (19 K) 11.0 -> 12.3, 80^3 (28 K) 16.0 -> 12.4;
//  * BF16 storage, from 1.5 and 48 K: 27-point 64^3 (0.9) 17.1 -> 18.5, 80^3
//    (1.7, 108 K) 26.6 -> 25.0; 9 offsets 500 K rows (35 K) 12.3 -> 14.3, 800 K
//    (56 K) 16.2 -> 16.5, 1.5 M 26.6 -> 22.9; 7-point 80^3 (28 K) 12.8 -> 14.4,
//    96^3 (48 K) 17.3 -> 16.5;
//  * wide blocks, from half a strip a warp: 27-point blockWidth 64 32^3 (0.1)
//    12.4 -> 14.4, 45^3 (0.3) equal, 64^3 (0.9) 22.6 -> 20.7.
// 16-byte copies need a 16-byte aligned value array (a caller's may not be), and
// the kernel ascending lists: a flag in it that turns the unchecked path off
// instead cost 1.6 % of BF16 131x127x125 (59.9 -> 60.8 us).
bool enough_strips(const DevicePlan &P, int sms) {
    const int64_t strips = (static_cast<int64_t>(P.numTiles) + 3) / 4, warps = int64_t(sms) * kStripWarps;
    const bool native = P.storage == HBDIA_STORE_NATIVE, bf16 = P.storage == HBDIA_STORE_BF16_SCALED;
    if (P.bw % 32 != 0 || P.n > (1 << 30) || (bf16 && P.bw != 32)) return false;
    if ((reinterpret_cast<uintptr_t>(P.vals) & 15) != 0 || !P.ascending) return false;
    if (native) return strips >= (P.bw != 32 ? warps / 2 : P.tailHeavy ? 2 * warps : 4 * warps);
    const int64_t stripOffsets = P.totalOffsets * (P.bw / 32) / 4;
    return bf16 ? strips >= warps * 3 / 2 && stripOffsets >= 48 * 1024 : strips >= warps / 2 && stripOffsets >= 32 * 1024;
}

// The least share of strips with one list: 27-point 300x4x1000 (75 %) 45.6 ->
// 53.7 us, 20x20x2000 (99 %) 36.0 -> 34.1.
constexpr double kUniformShare = 0.85;

}  // namespace

size_t strip_bytes(int32_t numTiles) { return (static_cast<size_t>(numTiles) + 3) / 4 * sizeof(int4) + 16; }

void make_strips(DevicePlan &P, void *where) {
    P.strips = nullptr;
    P.stripGrid = 0;
    int device = 0, sms = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    if (!enough_strips(P, sms)) return;
    const int32_t strips = (P.numTiles + 3) / 4;
    int4 *desc = static_cast<int4 *>(where);
    int32_t *counts = reinterpret_cast<int32_t *>(desc + strips), found[2] = {0, 0};
    check_cuda(cudaMemset(counts, 0, sizeof(found)), "cudaMemset(strips)");
    dev::strip_desc_kernel<<<static_cast<unsigned>((strips + 7) / 8), 256>>>(
        P.blkOff, P.offs, P.cooTile, P.scale, P.numBlocks, P.numTiles, P.bw / 32, P.nCoo > 0, desc, counts);
    check_cuda(cudaGetLastError(), "strip descriptors");
    check_cuda(cudaMemcpy(found, counts, sizeof(found), cudaMemcpyDeviceToHost), "cudaMemcpy(strips)");
    if (found[0] < kUniformShare * strips || found[1] != 0) return;
    P.strips = desc;
    P.stripGrid = static_cast<int32_t>(std::min<int64_t>((strips + kStripWarps - 1) / kStripWarps, sms));
    // here and not at the launch, which may be captured into a graph
    if (P.dtype == HBDIA_F32) configure<float, float>(P);
    else if (P.storage == HBDIA_STORE_F32) configure<float, double>(P);
    else if (P.storage == HBDIA_STORE_BF16_SCALED) configure<__nv_bfloat16, double>(P);
    else configure<double, double>(P);
}

template <typename VT, typename XT>
void launch_strip(const DevicePlan &P, const XT *x, XT *y, void *stream) {
    with_strip_kernel<VT, XT>(P, [&](auto kernel, size_t smem) {
        kernel<<<P.stripGrid, kStripWarps * 32, smem, static_cast<cudaStream_t>(stream)>>>(
            make_args<VT, XT>(P), static_cast<const int4 *>(P.strips), x, y);
    });
}

template void launch_strip<double, double>(const DevicePlan &, const double *, double *, void *);
template void launch_strip<float, double>(const DevicePlan &, const double *, double *, void *);
template void launch_strip<__nv_bfloat16, double>(const DevicePlan &, const double *, double *, void *);
template void launch_strip<float, float>(const DevicePlan &, const float *, float *, void *);

}  // namespace hbdia
