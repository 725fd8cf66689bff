// Strip SpMV: four 32-row tiles per warp, values streamed through shared
// memory (sm_100a).
//
// What bounds the product: HBM for 8-byte values; for narrower ones the
// instructions and latencies of a warp's products (about 14 instructions per
// stored offset of a 32-row tile).  The kernels that load values into registers
// (spmv_kernels.cuh, spmv_quad.cuh) keep a warp's loads of one group in flight
// and then none while its products are formed.  Here a warp owns a strip of 128
// rows (lane l: rows l, l + 32, l + 64, l + 96), one offset and one x address
// serve its four tiles, and the values arrive in a ring of D shared-memory
// stages of U offsets (cp.async, evict-first in L2), D - 1 stages ahead of the
// products and across strip ends, so copies are always in flight and hold no
// registers.  x comes through L1: the 16 warps of a CTA own 2048 consecutive
// rows, so neighbouring strips share its lines; one CTA per SM.
//
// Strips whose four tiles share one list of at most 32 offsets (nearly all of a
// stencil's or a banded matrix's) are marked in a descriptor made once per
// layout (strip_desc_kernel), which also holds their COO range: a warp reads 16
// bytes per strip instead of comparing four lists.  Other strips go tile by
// tile through the same ring, a stage holding up to 4 U offsets of one tile.
//
// The first 64 COO entries of a strip are loaded two strips ahead, their x one
// strip ahead, and their products wait in shared memory.
//
// B200, three matrices in turn, against the kernel used before (pipelined
// for native values, quad for narrow ones, row-per-thread for wide blocks):
//   FP64 27-point 256^3 735-746 -> 653-662 us (93 % of the measured copy
//   bandwidth), 128^3 88.0 -> 82.1, 7-point 128^3 55.4 -> 28.8;
//   float 27-point 129x121x133 61.2 -> 51.8; FP32 storage 27-point 128^3 69.7
//   -> 54.2, 200^3 246 -> 201, banded 8M rows 113.3 -> 94.6; BF16 storage
//   131x127x125 68.1 -> 60.3; 7-point 160^3 with blockWidth 64 98.3 -> 53.3,
//   27-point 128^3 with blockWidth 128 145 -> 83.0.
// Measured and left out: x windows of the CTA staged in shared memory by bulk
// copies (FP32 128^3 69 against 56 us: the windows take the ring's space),
// bulk L2 prefetch of the next strip's values (66 against 58), deeper rings
// (6 stages 60 against 56: less L1 for x), 24 warps with 80 registers (spills).
//
// Offsets ascend in every block: a list's ends bound the others.
//
// Arithmetic is the reference's, in the reference's order: per row, offsets
// ascending, stored zeros and columns outside [0, xn) skipped, fma; COO
// products summed from zero in list order with separately rounded multiply
// and add; y = dia + coo when the matrix has a remainder (+0 is added at rows
// without entries, which turns a sum of -0 into +0), else y = dia
// (src/Operations/HBDIASpMV.cu:42-88, src/Operations/HBDIASpMV.cpp:76-92).
#pragma once

#include <type_traits>

#include "spmv_kernels.cuh"

namespace hbdia {
namespace dev {

__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint64_t pol) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(pol) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// N list entries, four at a time; the list is 16-byte aligned there.
template <int N>
__device__ __forceinline__ void load_list(const int32_t *p, int32_t (&o)[N]) {
#pragma unroll
    for (int u = 0; u < N; u += 4) {
        const int4 t = *reinterpret_cast<const int4 *>(p + u);
        o[u] = t.x;
        o[u + 1] = t.y;
        o[u + 2] = t.z;
        o[u + 3] = t.w;
    }
}

// One strip (4 consecutive 32-row tiles), made once per layout: x = first
// offset index of the first tile's block; y = number of offsets when the four
// tiles share one list of at most 32 offsets, else -1; z, w = the strip's COO
// entries [z, w).  counts[0]: strips of one list; counts[1]: not zero when a
// block's scale is 0, infinite or NaN (add_product tells zeros by the stored
// value, which then is not what the widened one says).
inline __global__ void __launch_bounds__(256)
strip_desc_kernel(const int32_t *__restrict__ blkOff, const int32_t *__restrict__ offs,
                  const int32_t *__restrict__ cooTile, const float *__restrict__ scale, int32_t numBlocks, int32_t numTiles,
                  int32_t tilesPerBlock, int32_t hasCoo, int4 *__restrict__ desc, int32_t *__restrict__ counts) {
    const int lane = threadIdx.x & 31;
    const int32_t s = static_cast<int32_t>((static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) >> 5);
    const int32_t numStrips = (numTiles + 3) / 4;
    if (s >= numStrips) return;  // warp-uniform
    int32_t k0[4], K[4];
    for (int i = 0; i < 4; ++i) {
        const int32_t b = (s * 4 + i) / tilesPerBlock;
        k0[i] = b < numBlocks ? blkOff[b] : 0;
        K[i] = b < numBlocks && s * 4 + i < numTiles ? blkOff[b + 1] - k0[i] : 0;
    }
    bool uni = K[0] <= 32 && K[1] == K[0] && K[2] == K[0] && K[3] == K[0];
    int diff = 0;
    if (uni && lane < K[0])
        for (int i = 1; i < 4; ++i) diff |= offs[k0[i] + lane] != offs[k0[0] + lane];
    uni = uni && !__any_sync(kFull, diff);
    if (lane == 0) {
        int4 d;
        d.x = k0[0];
        d.y = uni ? K[0] : -1;
        d.z = hasCoo ? cooTile[min(s * 4, numTiles)] : 0;
        d.w = hasCoo ? cooTile[min(s * 4 + 4, numTiles)] : 0;
        desc[s] = d;
        if (uni) atomicAdd(counts, 1);
        if (scale)
            for (int i = 0; i < 4; ++i) {
                const int32_t b = (s * 4 + i) / tilesPerBlock;
                if (b >= numBlocks) break;
                const float sc = fabsf(scale[b]);
                if (!(sc > 0.0f && sc < __int_as_float(0x7f800000))) atomicOr(counts + 1, 1);
            }
    }
}

// *over += the warps of W whose share exceeds limit, in stored offsets of 32-row
// tiles, a strip of differing tiles counted twice (its tiles go one by one).
inline __global__ void __launch_bounds__(256)
strip_share_kernel(const int4 *__restrict__ desc, const int32_t *__restrict__ blkOff, int32_t numBlocks, int32_t numTiles,
                   int32_t tilesPerBlock, int32_t W, int32_t limit, int32_t *__restrict__ over) {
    const int32_t w = static_cast<int32_t>(blockIdx.x) * 256 + threadIdx.x;
    if (w >= W) return;
    int32_t sum = 0;
    for (int32_t s = w; s < (numTiles + 3) / 4; s += W) {
        const int32_t K = desc[s].y;
        if (K >= 0) {
            sum += 4 * K;
            continue;
        }
        for (int32_t t = s * 4; t < min(s * 4 + 4, numTiles); ++t) {
            const int32_t b = t / tilesPerBlock;
            if (b < numBlocks) sum += 2 * (blkOff[b + 1] - blkOff[b]);
        }
    }
    if (sum > limit) atomicAdd(over, 1);
}

// sum += v * x unless the stored value is zero, as one predicated FMA.
// For 8-byte values the product of a zero is made -0 instead, which leaves
// every sum as it is: x keeps its low word and takes the zero's negative for
// its high word, so the product is (+-0) * (-+tiny) = -0 whatever x holds, an
// infinity or NaN included.
__device__ __forceinline__ void add_product(double &sum, double v, float, double x) {
    const int hi = v != 0.0 ? __double2hiint(x) : __double2hiint(v) ^ 0x80000000;
    sum = fma_rn(v, __hiloint2double(hi, __double2loint(x)), sum);
}
__device__ __forceinline__ void add_product(double &sum, float v, float, double x) {
    asm("{\n\t.reg .pred p;\n\tsetp.neu.f32 p, %1, 0f00000000;\n\t@p fma.rn.f64 %0, %2, %3, %0;\n\t}"
        : "+d"(sum) : "f"(v), "d"(static_cast<double>(v)), "d"(x));
}
// (for a scale that is neither 0 nor infinite nor NaN: v * s is zero when v is)
__device__ __forceinline__ void add_product(double &sum, __nv_bfloat16 v, float s, double x) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p fma.rn.f64 %0, %2, %3, %0;\n\t}"
        : "+d"(sum) : "r"(__bfloat16_as_ushort(v) & 0x7fffu), "d"(widen<double>(v, s)), "d"(x));
}
__device__ __forceinline__ void add_product(float &sum, float v, float, float x) {
    asm("{\n\t.reg .pred p;\n\tsetp.neu.f32 p, %1, 0f00000000;\n\t@p fma.rn.f32 %0, %1, %2, %0;\n\t}"
        : "+f"(sum) : "f"(v), "f"(x));
}

template <typename VT, typename XT, int U, int D>
constexpr size_t strip_warp_smem() {
    return static_cast<size_t>(D) * U * 128 * sizeof(VT) + 192 * sizeof(XT) + 384;
}

template <typename VT, typename XT, int U, int D, int NW, bool QL, bool B32>
__global__ void __launch_bounds__(NW * 32, 1)
spmv_strip(const SpmvArgs<VT, XT> a, const int4 *__restrict__ desc, const XT *__restrict__ x, XT *__restrict__ y) {
    constexpr int RB = 32 * static_cast<int>(sizeof(VT));  // bytes of one offset of one tile
    constexpr int GB = U * 4 * RB;                         // bytes of one stage
    constexpr int PB = QL ? 512 : 128;                     // contiguous bytes per tile and copy instruction
    constexpr int NI = (GB + 511) / 512;
    constexpr int WU = 4 * U;  // offsets of one tile per stage when the tiles differ
    static_assert(U == 4, "the list is read four offsets at a time");
    static_assert(B32 || PB <= RB, "a copy instruction stays within one row");
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    unsigned char *ring = smem + w * (D * GB);
    XT *db = reinterpret_cast<XT *>(smem + NW * D * GB) + w * 192;  // row sums; COO products from 128 on
    int32_t *so = reinterpret_cast<int32_t *>(smem + NW * (D * GB + 192 * sizeof(XT))) + w * 96;  // offsets
    int32_t *sr = so + 32;                                                                        // COO rows
    XT *sv = db + 128;
    const uint32_t ringS = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
    const int32_t W = static_cast<int32_t>(gridDim.x) * NW;
    const int32_t numStrips = (a.numTiles + 3) >> 2;
    const uint32_t xn = static_cast<uint32_t>(a.xn);
    const int32_t m = B32 ? 1 : a.bw >> 5;                                       // tiles per block
    const int64_t rs = B32 ? RB : static_cast<int64_t>(a.bw) * sizeof(VT);       // bytes between a tile's offsets
    int32_t s = static_cast<int32_t>(blockIdx.x) * NW + w;
    if (s >= numStrips) return;  // warp-uniform
    const uint64_t pol = policy_evict_first();
    const int4 kNone = make_int4(0, 0, 0, 0);

    // block pointers of a strip's tiles, for strips whose tiles differ: lane
    // i < 4 the first offset index of tile i, lane 4 + i the end
    auto tileRange = [&](int32_t q) {
        int32_t kb = 0;
        const int32_t t = q * 4 + (lane & 3);
        const int32_t b = B32 ? t : t / m;
        if (lane < 8 && b < a.numBlocks && t < a.numTiles) kb = __ldg(a.blkOff + b + (lane >> 2));
        return kb;
    };
    struct Coo {
        int32_t r[2], c[2];
        XT v[2];
    };
    auto loadCoo = [&](int32_t q, int32_t c0, int32_t c1, Coo &f) {
        if (c1 <= c0) return;  // warp-uniform
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int32_t e = c0 + 32 * i + lane;
            if (i > 0 && c1 - c0 <= 32) return;  // warp-uniform
            if (e < c1) {
                f.r[i] = __ldg(a.cooRow + e) - q * 128;
                f.c[i] = __ldg(a.cooCol + e);
                f.v[i] = __ldg(a.cooVal + e);
            }
        }
    };

    // ---- copies: D - 1 groups ahead of the products, across strips
    const unsigned char *isrc = nullptr;
    int32_t is = s, irem = 0;  // the iterator's strip, and its offsets (wide: its tile's) left to copy
    int4 idesc = __ldg(desc + s);
    int32_t ikb = 0;
    int iTile = -1;            // -1: the four tiles together; else tile by tile
    uint32_t cst = 0, pst = (D - 1) * GB;  // stages of the next products and of the last, byte offsets
    const int blk = lane >> 3;
    const uint32_t ldst = ringS + (QL ? lane * 16u : static_cast<uint32_t>(blk * (U * RB) + (lane & 7) * 16));
    const int32_t lsub = QL ? lane * 16 : (lane & 7) * 16;
    // the iterator's strip begins (its descriptor in idesc)
    auto beginStrip = [&]() {
        if (idesc.y >= 0) {
            iTile = -1;
            irem = idesc.y;
            int64_t e;
            if (QL) e = static_cast<int64_t>(idesc.x) * 32;
            else if (B32) e = (static_cast<int64_t>(idesc.x) + blk * idesc.y) * 32;
            else {
                const int32_t t0 = is * 4, b0 = t0 / m, b = (t0 + blk) / m;
                e = (static_cast<int64_t>(idesc.x) + static_cast<int64_t>(b - b0) * idesc.y) * a.bw + (t0 + blk - b * m) * 32;
            }
            isrc = reinterpret_cast<const unsigned char *>(a.vals) + e * static_cast<int64_t>(sizeof(VT)) + lsub;
        } else {
            ikb = tileRange(is);
            iTile = 0;
            irem = 0;
        }
    };
    // wide: from iTile on, the next tile that has offsets; false at the strip's end
    auto wideTile = [&]() {
        for (; iTile < 4; ++iTile) {
            const int32_t k0 = __shfl_sync(kFull, ikb, iTile);
            irem = __shfl_sync(kFull, ikb, 4 + iTile) - k0;
            if (irem > 0) {
                int64_t e = static_cast<int64_t>(k0) * a.bw;
                if (!B32) e += static_cast<int64_t>((is * 4 + iTile) % m) * 32;
                isrc = reinterpret_cast<const unsigned char *>(a.vals) + e * static_cast<int64_t>(sizeof(VT)) +
                       (B32 ? lane * 16 : (lane * 16 / RB) * rs + (lane * 16) % RB);
                return true;
            }
        }
        irem = 0;
        return false;
    };
    int4 inext = is + W < numStrips ? __ldg(desc + is + W) : kNone;
    beginStrip();
    // one group's copies (none at the end of the work); always one commit
    auto issue = [&](uint32_t fill) {
        if (irem > U && iTile < 0) {  // a full group, and not the strip's last
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int64_t o = B32 ? static_cast<int64_t>(i) * PB : (i * PB / RB) * rs + (i * PB) % RB;
                cp_async16(ldst + fill + i * PB, isrc + o, pol);
            }
            cp_async_commit();
            isrc += QL ? U * 4 * RB : U * rs;
            irem -= U;
            return;
        }
        while (irem == 0 && is < numStrips) {
            if (iTile >= 0 && iTile < 4 && wideTile()) break;
            is += W;
            if (is >= numStrips) break;
            idesc = inext;
            inext = is + W < numStrips ? __ldg(desc + is + W) : kNone;
            beginStrip();
        }
        if (irem > 0) {
            if (iTile < 0) {
                const int32_t lim = (QL ? 4 : 1) * irem * RB - lsub;  // this lane's bytes left
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    const int64_t o = B32 ? static_cast<int64_t>(i) * PB : (i * PB / RB) * rs + (i * PB) % RB;
                    if (i * PB < lim) cp_async16(ldst + fill + i * PB, isrc + o, pol);
                }
                isrc += QL ? U * 4 * RB : U * rs;
                irem = max(irem - U, 0);
            } else {
                const int32_t lim = min(WU, irem) * RB - lane * 16;
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    const int64_t o = B32 ? static_cast<int64_t>(i) * 512 : (i * 512 / RB) * rs;
                    if (i * 512 < lim) cp_async16(ringS + fill + lane * 16 + i * 512, isrc + o, pol);
                }
                isrc += WU * rs;
                irem -= min(WU, irem);
                if (irem == 0) ++iTile;
            }
        }
        cp_async_commit();
    };
    // the next group's values have arrived and its stage may be read; the
    // stage read before it may be overwritten
    auto nextStage = [&]() {
        cp_async_wait<D - 2>();
        __syncwarp();
        const unsigned char *st = ring + cst;
        issue(pst);
        pst = cst;
        cst = cst == (D - 1) * GB ? 0 : cst + GB;
        return st;
    };

    int4 d0 = idesc;
    int4 d1 = s + W < numStrips ? __ldg(desc + s + W) : kNone;
    int4 d2 = s + 2 * W < numStrips ? __ldg(desc + s + 2 * W) : kNone;
    // products of a strip's first COO entries, kept in shared memory until its turn
    auto gatherCoo = [&](int32_t c0, int32_t c1, const Coo &f, XT (&cx)[2]) {
        if (c1 <= c0) return;  // warp-uniform
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (c0 + 32 * i + lane < c1) cx[i] = __ldg(x + f.c[i]);
    };
    auto storeCoo = [&](int32_t c0, int32_t c1, const Coo &f, const XT (&cx)[2]) {
        if (c1 <= c0) return;  // warp-uniform
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (c0 + 32 * i + lane < c1) {
                sr[32 * i + lane] = f.r[i];
                sv[32 * i + lane] = mul_rn(f.v[i], cx[i]);
            }
    };
    Coo co;
    loadCoo(s, d0.z, d0.w, co);
    {
        XT cx[2];
        gatherCoo(d0.z, d0.w, co, cx);
        storeCoo(d0.z, d0.w, co, cx);
    }
    loadCoo(s + W, d1.z, d1.w, co);
    so[lane] = lane < d0.y ? __ldg(a.offs + d0.x + lane) : 0;
#pragma unroll 1
    for (int i = 0; i < D - 1; ++i) issue(i * GB);
    __syncwarp();

    for (; s < numStrips; s += W) {
        const int32_t row0 = s * 128;
        const int32_t row = row0 + lane;
        const int32_t K = d0.y, c0 = d0.z, c1 = d0.w;
        // the next strip's COO products begin (columns loaded one strip ago)
        XT cx[2];
        gatherCoo(d1.z, d1.w, co, cx);
        const int4 d3 = s + 3 * W < numStrips ? __ldg(desc + s + 3 * W) : kNone;
        const int32_t on = lane < d1.y ? __ldg(a.offs + d1.x + lane) : 0;
        Coo cn;
        loadCoo(s + 2 * W, d2.z, d2.w, cn);
        float sc[4] = {1.0f, 1.0f, 1.0f, 1.0f};
        if constexpr (sizeof(VT) == 2) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (s * 4 + q < a.numBlocks) sc[q] = __ldg(a.scale + s * 4 + q);
        }
        XT sum[4] = {XT(0), XT(0), XT(0), XT(0)};
        const XT *xr = x + row;
        // narrow values: ask L2 for the x of this warp's next strip (at the middle
        // offset; the strips of a round together cover every row).  Banded 8M
        // rows 98.4 -> 94.6 us; nothing to gain, and 0.4 % to lose, where the
        // values are 8 bytes
        if constexpr (sizeof(VT) < 8) {
            constexpr int EPS = 32 / static_cast<int>(sizeof(XT));  // x elements of one sector
            if (lane < 128 / EPS) {
                const int64_t c = static_cast<int64_t>(row0) + static_cast<int64_t>(W) * 128 + lane * EPS + (K > 0 ? so[K >> 1] : 0);
                if (c >= 0 && c < a.xn) asm volatile("prefetch.global.L2 [%0];" ::"l"(x + c));
            }
        }
        if (K > 0) {
            const bool interior = int64_t(row0) + so[0] >= 0 && int64_t(row0) + 127 + so[K - 1] < int64_t(a.xn);
            // C offsets from g on: their x first, then their values
            auto step = [&](auto CNT, auto CHECK, int32_t g) {
                constexpr int C = decltype(CNT)::value;
                constexpr bool CK = decltype(CHECK)::value;
                XT xv[C][4];
                unsigned ok = 0;
                int32_t of[(C + 3) / 4 * 4];
                load_list(so + g, of);
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    const XT *xp = xr + of[u];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (CK) {
                            const bool in = static_cast<uint32_t>(row + of[u] + 32 * q) < xn;
                            xv[u][q] = XT(0);
                            if (in) xv[u][q] = __ldg(xp + 32 * q);
                            ok |= in ? 1u << (u * 4 + q) : 0u;
                        } else {
                            xv[u][q] = __ldg(xp + 32 * q);
                        }
                    }
                }
                const unsigned char *st = nextStage();
#pragma unroll
                for (int u = 0; u < C; ++u) {
                    VT v[4];
                    if constexpr (QL && sizeof(VT) == 4) {
                        const float4 f = reinterpret_cast<const float4 *>(st)[u * 32 + lane];
                        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
                    } else if constexpr (QL) {
                        const uint2 r = reinterpret_cast<const uint2 *>(st)[u * 32 + lane];
                        v[0] = __ushort_as_bfloat16(static_cast<unsigned short>(r.x & 0xffffu));
                        v[1] = __ushort_as_bfloat16(static_cast<unsigned short>(r.x >> 16));
                        v[2] = __ushort_as_bfloat16(static_cast<unsigned short>(r.y & 0xffffu));
                        v[3] = __ushort_as_bfloat16(static_cast<unsigned short>(r.y >> 16));
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = reinterpret_cast<const VT *>(st + (q * U + u) * RB)[lane];
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (!CK || (ok >> (u * 4 + q) & 1u)) add_product(sum[q], v[q], sc[q], xv[u][q]);
                }
            };
            auto all = [&](auto CHECK) {
                int32_t g = 0;
#pragma unroll 1
                for (; g + U <= K; g += U) step(std::integral_constant<int, U>(), CHECK, g);
                const int32_t rest = K - g;
                if (rest == 3) step(std::integral_constant<int, 3>(), CHECK, g);
                if (rest == 2) step(std::integral_constant<int, 2>(), CHECK, g);
                if (rest == 1) step(std::integral_constant<int, 1>(), CHECK, g);
            };
            if (interior) all(std::false_type());
            else all(std::true_type());
        } else if (K < 0) {
            // tiles that differ: one by one, up to WU offsets at a time
            const int32_t kb = tileRange(s);
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
                const int32_t k0 = __shfl_sync(kFull, kb, q), Kq = __shfl_sync(kFull, kb, 4 + q) - k0;
                const int32_t rq = row + 32 * q;
                const float sq = q == 0 ? sc[0] : q == 1 ? sc[1] : q == 2 ? sc[2] : sc[3];
                XT acc = XT(0);
#pragma unroll 1
                for (int32_t g = 0; g < Kq; g += WU) {
                    const int32_t cnt = min(WU, Kq - g);
                    const int32_t o = lane < cnt ? __ldg(a.offs + k0 + g + lane) : 0;
                    XT xv[WU];
                    unsigned ok = 0;
#pragma unroll
                    for (int u = 0; u < WU; ++u) {
                        const int32_t col = rq + __shfl_sync(kFull, o, u);
                        const bool in = u < cnt && static_cast<uint32_t>(col) < xn;
                        ok |= in ? 1u << u : 0u;
                        xv[u] = in ? __ldg(x + col) : XT(0);
                    }
                    const VT *st = reinterpret_cast<const VT *>(nextStage());
#pragma unroll
                    for (int u = 0; u < WU; ++u) {
                        const VT v = st[u * 32 + lane];
                        if (ok >> u & 1u) add_product(acc, v, sq, xv[u]);
                    }
                }
                if (q == 0) sum[0] = acc;
                else if (q == 1) sum[1] = acc;
                else if (q == 2) sum[2] = acc;
                else sum[3] = acc;
            }
        }

        // COO remainder: every row's sum starts from +0 (a row's own sum is never
        // -0, so adding the +0 first leaves rows with entries as they are);
        // the heads of row segments add their sums into db
        if (a.hasCoo) {
#pragma unroll
            for (int q = 0; q < 4; ++q) sum[q] = add_rn(sum[q], XT(0));
        }
        if (c1 > c0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) db[lane + 32 * q] = sum[q];
            __syncwarp();
            XT carry = XT(0);
            int32_t carryRow = -1;
#pragma unroll 1
            for (int32_t base = c0; base < c1; base += 32) {
                int32_t cr = 0x7fffffff;
                XT p = XT(0);
                const bool valid = base + lane < c1;
                if (valid) {
                    if (base <= c0 + 32) {
                        cr = sr[base - c0 + lane];
                        p = sv[base - c0 + lane];
                    } else {  // rare: more than 64 entries in the strip
                        cr = __ldg(a.cooRow + base + lane) - row0;
                        p = mul_rn(__ldg(a.cooVal + base + lane), __ldg(x + __ldg(a.cooCol + base + lane)));
                    }
                }
                const int32_t prevR = __shfl_up_sync(kFull, cr, 1);
                const bool cont = lane == 0 && cr == carryRow;  // continues the carried segment
                const bool head = valid && (lane == 0 || cr != prevR);
                if (lane == 0 && carryRow >= 0 && cr != carryRow) db[carryRow] = add_rn(db[carryRow], carry);
                XT c = head ? add_rn(cont ? carry : XT(0), p) : XT(0);
                const unsigned heads = __ballot_sync(kFull, head), some = __ballot_sync(kFull, valid);
                if (heads != some) {  // rows with several entries here: each head adds its followers in order
                    bool ext = head;
                    for (int t = 1; __any_sync(kFull, ext); ++t) {
                        const int32_t rt = __shfl_down_sync(kFull, cr, t & 31);
                        const XT pt = __shfl_down_sync(kFull, p, t & 31);
                        ext = ext && lane + t < 32 && rt == cr;
                        if (ext) c = add_rn(c, pt);
                    }
                }
                const bool last = base + 32 >= c1;
                const int lastHead = 31 - __clz(heads);
                if (!last) {  // the chunk's last segment may continue in the next chunk
                    carry = __shfl_sync(kFull, c, lastHead);
                    carryRow = __shfl_sync(kFull, cr, lastHead);
                }
                if (head && (last || lane != lastHead)) db[cr] = add_rn(db[cr], c);
                __syncwarp();
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) sum[q] = db[lane + 32 * q];
        }
        if (row0 + 128 <= a.n) {
#pragma unroll
            for (int q = 0; q < 4; ++q) __stcs(y + row + 32 * q, sum[q]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (row + 32 * q < a.n) __stcs(y + row + 32 * q, sum[q]);
        }
        __syncwarp();  // this strip's offsets and COO products have been read
        so[lane] = on;
        storeCoo(d1.z, d1.w, co, cx);
        d0 = d1;
        d1 = d2;
        d2 = d3;
        co = cn;
        __syncwarp();
    }
    cp_async_wait<0>();
}

}  // namespace dev
}  // namespace hbdia
