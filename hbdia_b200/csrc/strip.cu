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

// When the strip kernel is the faster one.  Two things decide it (strips a warp
// = strips / (SMs x 16); B200, 148 SMs, us, other kernel -> strip kernel):
//
// Enough strips.  A warp's first strip waits for a chain of loads that the other
// kernels spread over four times as many warps; long lists make up for it sooner
// than short ones (fewer than 16 offsets a block on average).
//
// Even shares.  Warp w takes strips w, w + W, ..., and a strip whose tiles differ
// costs about twice as much.  Where such strips recur with a period that divides
// W they all fall to the same warps: 27-point 64x64x400, 6 % of the strips, FP64
// 67.5 -> 96.3, float 44.0 -> 72.6.  `most` is the share that one warp in 256
// may exceed (a matrix's ends, chance extras), over the mean one; a last round
// that is nearly empty counts in it too.
//  * native values, 4 strips and 1.33: 27-point FP64 96^3 (2.9 strips) 37.0 ->
//    38.3, 108^3 (4.2; 1.50) 51.5 -> 60.8, 112^3 (4.6; 1.20) 57.4 -> 57.0, 20x20x4000
//    (1.14) 66.0 -> 63.3, 116^3 (1.28) 63.8 -> 65.3 and 124^3 (1.26) 78.5 -> 79.5,
//    the ones inside that lose (float 41.1 -> 40.7, 48.0 -> 47.2), 300x12x560 (1.37) 82.6 -> 83.5, 144^3 (1.02) 122 -> 113; float 108^3
//    34.2 -> 41.3, 112^3 and up 0.79-0.99 of it; 9 offsets 1.5 M rows (4.9;
//    1.01) FP64 28.9 -> 25.0, float 24.3 -> 20.3;
//  * native values where the pipelined kernel's groups of 9 are mostly tails, 2
//    and 1.75: 7-point FP64 86^3 (2.1; 1.88) 20.5 -> 21.1, 90^3 (2.4; 1.64) 22.6
//    -> 17.5, 100^3 28.7 -> 20.5, 64x64x400 (2.07) 44.4 -> 47.3, 128^3 56.0 ->
//    26.7; float 86^3 13.7 -> 16.5, 90^3 15.8 -> 13.4;
//  * FP32 storage, long lists 0.55 strips and 32 K strip-offsets, 2.25: 27-point
//    52^3 (0.46) 12.3 -> 14.4, 56^3 (0.58) 12.4-15.7 -> 14.4, 60^3 (0.71) 15.3 -> 14.4,
//    64x64x400 (1.87) 99.0 -> 79.2; short ones 2 strips and 2: 9 offsets 560 K
//    rows (1.85) 11.4 -> 12.3, 650 K (2.1) 14.9 -> 14.5, 7-point 85^3 (2.0) 15.9 ->
//    14.4;
//  * quad-interleaved FP32, which CG iterates on, half a strip and 32 K
//    strip-offsets whatever the shares: between a CG's vector kernels the strip
//    kernel is the faster one from there (solves of 27-point 56^3 6.5 -> 5.8 ms,
//    64^3 6.9 -> 6.1, 70^3 9.0 -> 7.8, 72^3 and up equal or better), though lone
//    products back to back are not before a strip a warp (56^3 12.3 -> 14.4 us,
//    64^3 13.3 -> 14.4, 72^3 24.4 -> 20.7; 9 offsets 600 K rows 11.2 -> 12.3, 800 K
//    15.2 -> 15.0);
//  * BF16 storage, 2.75 and 1.6: 27-point 88^3 (2.2) 29.3 -> 30.8,
//    96^3 (2.9; 1.22) 32.7 -> 30.8, 104^3 (1.55) 48.4 -> 46.9, 300x10x650 (1.38)
//    79.6 -> 82.6, 300x9x700 (1.46) 74.5 -> 66.8, 64x64x400 (1.87) 87.6 -> 96.6;
//    short lists 4 and 1.5: 9 offsets 1 M rows (3.3) 18.4 -> 19.8, 1.5 M (4.9)
//    23.1 -> 22.6, 7-point 104^3 (3.7; 1.59) 22.6 -> 24.6, 112^3 (4.6) 22.6 -> 22.4;
//  * quad-interleaved BF16, 2.75 and 1.35: 27-point 88^3 32.5 -> 32.7, 96^3 33.0 ->
//    32.6, 104^3 47.8 -> 49.2, 112^3 (1.20) 52.5 -> 45.3, 300x10x650 85.2 -> 88.6;
//    short lists 4.5 and 1.5: 9 offsets 1.25 M rows (4.1) 22.6 -> 23.5, 1.5 M 24.0
//    -> 23.4, 7-point 112^3 (4.6) 24.1 -> 23.4;
//  * wide blocks (against one row per thread), half a strip (4-byte x 3/4) and 2.25:
//    27-point blockWidth 64 FP64 45^3 (0.3) 14.4 -> 15.9, 54^3 (0.5) 18.9 -> 16.0,
//    float 54^3 11.9 -> 12.3, 64^3 (0.9) 14.2 -> 12.5; short lists 1.5 and 1.65:
//    7-point 64^3 (0.9) 8.2 -> 12.3, 80^3 (1.69) 14.4 -> 16.4,
//    96^3 (2.9; 1.33) 22.6 -> 20.9, 9 offsets 300 K rows (1.0) 10.3 -> 10.3, 500 K
//    (1.7; 1.21) 18.5 -> 15.0.
// BF16 values in wide blocks have no instance of the kernel.
struct StripRule {
    double strips, most;  // strips a warp at least, the share over the mean at most
};
StripRule strip_rule(const DevicePlan &P) {
    const bool isLong = P.totalOffsets >= 16 * static_cast<int64_t>(P.numBlocks);
    if (P.bw != 32) return isLong ? StripRule{P.dtype == HBDIA_F32 ? 0.75 : 0.5, 2.25} : StripRule{1.5, 1.65};
    if (P.storage == HBDIA_STORE_NATIVE) return P.tailHeavy ? StripRule{2.0, 1.75} : StripRule{4.0, 1.33};
    if (P.storage == HBDIA_STORE_BF16_SCALED) {
        if (P.quadLayout) return isLong ? StripRule{2.75, 1.35} : StripRule{4.5, 1.5};
        return isLong ? StripRule{2.75, 1.6} : StripRule{4.0, 1.5};
    }
    if (P.quadLayout) return StripRule{0.5, 1e9};
    return isLong ? StripRule{0.55, 2.25} : StripRule{2.0, 2.0};
}

// 16-byte copies need a 16-byte aligned value array (a caller's may not be), and
// the kernel ascending lists: a flag in it that turns the unchecked path off
// instead cost 1.6 % of BF16 131x127x125 (59.9 -> 60.8 us).
bool strips_possible(const DevicePlan &P) {
    if (P.bw % 32 != 0 || P.n <= 0 || P.n > (1 << 30) || (P.storage == HBDIA_STORE_BF16_SCALED && P.bw != 32)) return false;
    return (reinterpret_cast<uintptr_t>(P.vals) & 15) == 0 && P.ascending;
}
bool enough_strips(const DevicePlan &P, int sms) {
    const int64_t strips = (static_cast<int64_t>(P.numTiles) + 3) / 4, warps = int64_t(sms) * kStripWarps;
    if (P.storage == HBDIA_STORE_F32 && P.totalOffsets * (P.bw / 32) / 4 < 32 * 1024) return false;
    return strips >= strip_rule(P).strips * warps;
}

// The least share of strips with one list: 27-point 300x4x1000 (75 %) 45.6 ->
// 53.7 us, 300x9x700 (88 %) FP32 storage 77.1 -> 59.5.
constexpr double kUniformShare = 0.85;

}  // namespace

size_t strip_bytes(int32_t numTiles) { return (static_cast<size_t>(numTiles) + 3) / 4 * sizeof(int4) + 16; }

void make_strips(DevicePlan &P, void *where) {
    P.stripMem = where;
    P.strips = nullptr;
    P.stripGrid = 0;
    P.stripPays = false;
    int device = 0, sms = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    const bool enough = enough_strips(P, sms);
    if (!strips_possible(P) || !(enough || P.kernel == HBDIA_KERNEL_STRIP)) return;
    const int32_t strips = (P.numTiles + 3) / 4;
    int4 *desc = static_cast<int4 *>(where);
    int32_t *counts = reinterpret_cast<int32_t *>(desc + strips), found[3] = {0, 0, 0};
    check_cuda(cudaMemset(counts, 0, sizeof(found)), "cudaMemset(strips)");
    dev::strip_desc_kernel<<<static_cast<unsigned>((strips + 7) / 8), 256>>>(
        P.blkOff, P.offs, P.cooTile, P.scale, P.numBlocks, P.numTiles, P.bw / 32, P.nCoo > 0, desc, counts);
    check_cuda(cudaGetLastError(), "strip descriptors");
    const int32_t grid = static_cast<int32_t>(std::min<int64_t>((strips + kStripWarps - 1) / kStripWarps, sms)), W = grid * kStripWarps;
    const double mean = static_cast<double>(P.totalOffsets) * (P.bw / 32) / W;
    const int32_t limit = static_cast<int32_t>(std::min(strip_rule(P).most * mean, 2147483647.0));
    dev::strip_share_kernel<<<static_cast<unsigned>((W + 255) / 256), 256>>>(desc, P.blkOff, P.numBlocks, P.numTiles, P.bw / 32, W,
                                                                             limit, counts + 2);
    check_cuda(cudaGetLastError(), "strip shares");
    check_cuda(cudaMemcpy(found, counts, sizeof(found), cudaMemcpyDeviceToHost), "cudaMemcpy(strips)");
    if (found[1] != 0) return;
    P.stripPays = enough && found[0] >= kUniformShare * strips && found[2] <= W / 256;
    if (!P.stripPays && P.kernel != HBDIA_KERNEL_STRIP) return;
    P.strips = desc;
    P.stripGrid = grid;
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
