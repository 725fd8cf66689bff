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

// Whether the strip kernel is the faster one for a layout (B200, us):
//  * it needs enough strips for the SMs' 2368 warps, since a warp's first strip
//    waits for a chain of loads that the other kernels spread over four times
//    as many warps.  Native values of blockWidth 32 against the pipelined
//    kernel: 27-point FP64 80^3 (1.7 strips per warp) 27.9 against 24.8, 96^3
//    (2.9) 38.9 against 38.4, 112^3 (4.6) 60.0 against 61.7; float 80^3 20.6
//    against 18.6.  FP32 storage against the quad kernel: 40^3 (0.2) 14.4
//    against 12.4, 56^3 (0.6) 14.4 against 17.9; BF16 storage 64^3 (0.9) 18.5
//    against 17.1, 80^3 25.0 against 26.6.  Wide blocks against the
//    row-per-thread kernel: 32^3 (0.1) 14.4 against 12.4, 64^3 (0.9) 20.7
//    against 22.6;
//  * most strips must share one list: 27-point 300x4x1000 (75 % do) 53.7
//    against 45.6, 20x20x2000 (99 %) 34.1 against 36.0, 40^3 (88 %);
//  * 16-byte copies need a 16-byte aligned value array (a caller's may not be).
bool strip_pays(const DevicePlan &P, int sms) {
    const int64_t strips = (static_cast<int64_t>(P.numTiles) + 3) / 4, warps = int64_t(sms) * kStripWarps;
    const bool native = P.storage == HBDIA_STORE_NATIVE, bf16 = P.storage == HBDIA_STORE_BF16_SCALED;
    if (P.bw % 32 != 0 || P.n > (1 << 30) || (bf16 && P.bw != 32)) return false;
    if ((reinterpret_cast<uintptr_t>(P.vals) & 15) != 0) return false;
    const int64_t least = native && P.bw == 32 ? 3 * warps : bf16 ? warps * 3 / 2 : warps / 2;
    return strips >= least && P.uniformStrips >= 0.85 * static_cast<double>(strips);
}

}  // namespace

size_t strip_bytes(int32_t numTiles) { return (static_cast<size_t>(numTiles) + 3) / 4 * sizeof(int4) + 16; }

void make_strips(DevicePlan &P, void *where) {
    P.strips = nullptr;
    P.stripGrid = 0;
    P.uniformStrips = 0;
    if (P.bw % 32 != 0 || P.numTiles <= 0) return;
    const int32_t strips = (P.numTiles + 3) / 4;
    int4 *desc = static_cast<int4 *>(where);
    int32_t *uniform = reinterpret_cast<int32_t *>(desc + strips);
    check_cuda(cudaMemset(uniform, 0, sizeof(int32_t)), "cudaMemset(strips)");
    dev::strip_desc_kernel<<<static_cast<unsigned>((strips + 7) / 8), 256>>>(
        P.blkOff, P.offs, P.cooTile, P.numBlocks, P.numTiles, P.bw / 32, P.nCoo > 0, desc, uniform);
    check_cuda(cudaGetLastError(), "strip descriptors");
    check_cuda(cudaMemcpy(&P.uniformStrips, uniform, sizeof(int32_t), cudaMemcpyDeviceToHost), "cudaMemcpy(strips)");
    int device = 0, sms = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    if (!strip_pays(P, sms)) return;
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
