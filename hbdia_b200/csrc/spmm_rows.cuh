// Row-major multi-RHS product Y = A X (element (i, j) at X[i * ldx + j]) for
// block widths that are multiples of 32 (sm_100a).
//
// What bounds it: L1 wavefronts and the latency of the X rows.  One lane per
// row reads X at a stride of ldx, so every 16-byte request of a warp touches 32
// lines (the kernel used before: 94 % of the L1 wavefront rate, 12 % of HBM).
// Here G lanes share a row of X and a lane keeps S neighbouring rows by V
// columns: a request reads whole row segments, a lane's S values of one offset
// are one or a few wide loads, and three neighbouring offsets (a stencil's -1,
// 0, 1) read S + 2 rows of X instead of 3 S.  Other offsets' loads go out
// together too, 128 bytes of X a lane, the last ones of a list as groups of 4
// and 1-3: one at a time each of them is a round trip (7-point 96^3 k = 2 67.9
// -> 35.4 us, 27-point 96^3 k = 9 422 -> 252).  Up to 32 columns a pass, so that
// the values are read once.
//
// B200, before -> after: 7-point 128^3 FP64 k = 16 603 -> 221 us, k = 32 1200 ->
// 422, k = 5 341 -> 197; 27-point 128^3 k = 8 570 -> 338, k = 3 495 -> 253; 96^3
// k = 2 84.9 -> 78.0; float 27-point 96^3 k = 16 747 -> 115; FP32 storage 97^3 k
// = 16 882 -> 235.  Now bound by instructions and load latency with 16 warps of
// 128 registers an SM (27-point k = 8: 36 % issue active, 56 % of the L1
// wavefront rate).  Measured and left out: X and values by bulk copies through
// shared memory (k = 16 197-207, k = 32 375, but float k = 16 149 against 115),
// 4 rows a lane for 9 to 16 columns (258).
//
// Offsets ascend in every block (interior tiles are told by a list's ends).
// Column j is computed with exactly the SpMV's arithmetic (spmv_kernels.cuh).
#pragma once

#include <type_traits>

#include "spmv_kernels.cuh"

namespace hbdia {
namespace dev {

constexpr int kRowsWarps = 16;  // warps per CTA at most (128 registers a thread)

// N stored values from p on, p a multiple of their bytes up to 16 (vec) or of one value.
template <typename VT, int N>
__device__ __forceinline__ void ld_values(const VT *p, bool vec, VT (&v)[N]) {
    constexpr int B = N * static_cast<int>(sizeof(VT));
    if (vec) {
        if constexpr (B >= 16) {
#pragma unroll
            for (int i = 0; i < B / 16; ++i)
                reinterpret_cast<int4 *>(v)[i] = __ldcs(reinterpret_cast<const int4 *>(p) + i);
        } else if constexpr (B == 8) {
            *reinterpret_cast<int2 *>(v) = __ldcs(reinterpret_cast<const int2 *>(p));
        } else if constexpr (B == 4) {
            *reinterpret_cast<int *>(v) = __ldcs(reinterpret_cast<const int *>(p));
        } else {
            v[0] = ld_stream(p);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = ld_stream(p + i);
    }
}

__device__ __forceinline__ bool is_zero(double v) { return v == 0.0; }
__device__ __forceinline__ bool is_zero(float v) { return v == 0.0f; }
__device__ __forceinline__ bool is_zero(__nv_bfloat16 v) { return (__bfloat16_as_ushort(v) & 0x7fffu) == 0; }

// V neighbouring elements of X.
template <int V>
__device__ __forceinline__ void ld_x(const double *p, double (&x)[V]) {
    if constexpr (V == 2) {
        const double2 t = __ldg(reinterpret_cast<const double2 *>(p));
        x[0] = t.x;
        x[1] = t.y;
    } else {
        x[0] = __ldg(p);
    }
}
template <int V>
__device__ __forceinline__ void ld_x(const float *p, float (&x)[V]) {
    if constexpr (V == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
        x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
    } else {
        x[0] = __ldg(p);
    }
}

// The COO entries [c0, c1) of a tile for one slab (first row row0).  Each of
// the 32 rows has a mask of its entries among the 32 at hand; 32 / G entries'
// products are formed per request and kept in shared memory, and every lane
// adds those of its rows in list order; each row's sum is added to its
// accumulators once.  er, ec, ev: this lane's of the first 32 entries (row
// within the slab, column, value).
template <typename XT, int V>
struct RowsCoo {
    XT p[32 * V];      // 32 / G entries x G V columns
    uint32_t mask[32];
};
template <typename VT, typename XT, int V, int G, int S>
__device__ __forceinline__ void rows_coo(const SpmvArgs<VT, XT> &a, const XT *__restrict__ X, int64_t ldx, int32_t c0,
                                         int32_t c1, int32_t row0, int32_t er, int32_t ec, XT ev, int lane,
                                         RowsCoo<XT, V> &sm, XT (&acc)[S][V]) {
    constexpr int RPR = 32 / G, RS = RPR * S;
    const int grp = lane / G;
    XT sum[S][V];
#pragma unroll
    for (int t = 0; t < S; ++t)
#pragma unroll
        for (int v = 0; v < V; ++v) sum[t][v] = XT(0);
#pragma unroll 1
    for (int32_t base = c0; base < c1; base += 32) {
        const int cnt = min(32, c1 - base);
        if (base != c0 && lane < cnt) {
            er = __ldg(a.cooRow + base + lane) - row0;
            ec = __ldg(a.cooCol + base + lane);
            ev = __ldg(a.cooVal + base + lane);
        }
        sm.mask[lane] = 0;
        __syncwarp();
        if (lane < cnt && er >= 0 && er < RS) atomicOr(&sm.mask[er], 1u << lane);
        __syncwarp();
        uint32_t mk[S], any = 0;
#pragma unroll
        for (int t = 0; t < S; ++t) {
            mk[t] = sm.mask[grp * S + t];
            any |= mk[t];
        }
        any = __reduce_or_sync(kFull, any);  // the slab's entries
#pragma unroll 1
        for (int i0 = 0; i0 < cnt; i0 += RPR) {
            const uint32_t part = (RPR == 32 ? ~0u : ((1u << RPR) - 1u)) << i0;
            if (!(any & part)) continue;  // warp-uniform
            const int mine = i0 + grp;    // the entry whose x this lane's group reads
            const int32_t col = __shfl_sync(kFull, ec, mine & 31);
            const XT val = __shfl_sync(kFull, ev, mine & 31);
            if (any >> (mine & 31) & 1u) {
                XT p[V];
                ld_x<V>(X + static_cast<int64_t>(col) * ldx, p);
#pragma unroll
                for (int v = 0; v < V; ++v) sm.p[lane * V + v] = mul_rn(val, p[v]);
            }
            __syncwarp();
#pragma unroll
            for (int t = 0; t < S; ++t)
                for (uint32_t m = mk[t] & part; m; m &= m - 1) {
                    const XT *q = sm.p + ((__ffs(m) - 1 - i0) * G + lane % G) * V;
#pragma unroll
                    for (int v = 0; v < V; ++v) sum[t][v] = add_rn(sum[t][v], q[v]);
                }
            __syncwarp();
        }
    }
#pragma unroll
    for (int t = 0; t < S; ++t)
#pragma unroll
        for (int v = 0; v < V; ++v) acc[t][v] = add_rn(acc[t][v], sum[t][v]);
}

template <typename XT, int V>
__device__ __forceinline__ void st_y(XT *p, const XT (&v)[V]) {
    if constexpr (V == 4) __stcs(reinterpret_cast<float4 *>(p), make_float4(v[0], v[1], v[2], v[3]));
    else if constexpr (V == 2) __stcs(reinterpret_cast<double2 *>(p), make_double2(v[0], v[1]));
    else __stcs(p, v[0]);
}

// The DIA part of one slab with X and the values loaded into registers.
// first: this lane's of the block's first 32 offsets; xb: X at the lane's
// first row and column; vp: the lane's first value of the block's first offset.
template <typename VT, typename XT, int V, int G, int S>
__device__ __forceinline__ void rows_dia(const SpmvArgs<VT, XT> &a, const XT *__restrict__ xb, int64_t ldx, const TileMeta &mt,
                                         int32_t first, const VT *__restrict__ vp, float sc, int32_t row0, int32_t row,
                                         int lane, bool vec, XT (&acc)[S][V]) {
    constexpr int RS = 32 / G * S;
    for (int32_t kb = mt.k0; kb < mt.k1; kb += 32) {
        const int cnt = min(32, mt.k1 - kb);
        const int32_t myoff = kb == mt.k0 ? first : (lane < cnt ? __ldg(a.offs + kb + lane) : 0);
        // bit j: offsets j, j + 1, j + 2 are neighbours
        const int32_t o1 = __shfl_down_sync(kFull, myoff, 1), o2 = __shfl_down_sync(kFull, myoff, 2);
        const unsigned runs = __ballot_sync(kFull, lane + 2 < cnt && o1 == myoff + 1 && o2 == myoff + 2);
        const int32_t oF = __shfl_sync(kFull, myoff, 0), oL = __shfl_sync(kFull, myoff, cnt - 1);
        const bool interior = int64_t(row0) + oF >= 0 && int64_t(row0) + RS - 1 + oL < int64_t(a.xn);
        // L neighbouring offsets from j on (RUN: one after the other, so
        // that they share rows of X; else any)
        auto step = [&](auto LEN, auto RUNT, auto CHECK, int j) {
            constexpr int L = decltype(LEN)::value;
            constexpr bool RUN = decltype(RUNT)::value, CK = decltype(CHECK)::value;
            constexpr int N = RUN ? S + L - 1 : S * L;  // rows of X the lane reads
            XT xv[N][V];
            bool ok[N];
            int32_t off[L];
#pragma unroll
            for (int l = 0; l < L; ++l) off[l] = __shfl_sync(kFull, myoff, (j + l) & 31);
#pragma unroll
            for (int t = 0; t < N; ++t) {
                const int32_t o = RUN ? off[0] + t : off[t / S] + t % S;
                ok[t] = !CK || static_cast<uint32_t>(row + o) < static_cast<uint32_t>(a.xn);
                const XT *xp = xb + (RUN ? off[0] : off[t / S]) * ldx + (RUN ? t : t % S) * ldx;
                if (CK) {
#pragma unroll
                    for (int v = 0; v < V; ++v) xv[t][v] = XT(0);
                }
                if (ok[t]) ld_x<V>(xp, xv[t]);
            }
            // Up to 12 values at once: products without a zero test when the
            // warp holds no stored zero among them.  With 8 rows a lane
            // the vote, which waits for all of them, costs more than the
            // tests (7-point 128^3 k = 16: 221 against 200 us).
            constexpr int GL = S * L <= 16 ? L : 1;
            constexpr bool VOTE = !CK && S <= 4;
#pragma unroll
            for (int l0 = 0; l0 < L; l0 += GL) {
                VT vs[GL][S];
#pragma unroll
                for (int l = 0; l < GL; ++l)
                    ld_values<VT, S>(vp + static_cast<int64_t>(kb - mt.k0 + j + l0 + l) * a.bw, vec, vs[l]);
                bool nz = VOTE && (sizeof(VT) != 2 || sc != 0.0f);  // (scale 0: every widened value is zero)
                if constexpr (VOTE) {
#pragma unroll
                    for (int l = 0; l < GL; ++l)
#pragma unroll
                        for (int t = 0; t < S; ++t) nz = nz && !is_zero(vs[l][t]);
                }
                if (VOTE && __all_sync(kFull, nz)) {
#pragma unroll
                    for (int l = 0; l < GL; ++l)
#pragma unroll
                        for (int t = 0; t < S; ++t) {
                            const XT vv = widen<XT>(vs[l][t], sc);
#pragma unroll
                            for (int v = 0; v < V; ++v)
                                acc[t][v] = fma_rn(vv, xv[RUN ? t + l0 + l : (l0 + l) * S + t][v], acc[t][v]);
                        }
                } else {
#pragma unroll
                    for (int l = 0; l < GL; ++l)
#pragma unroll
                        for (int t = 0; t < S; ++t) {
                            const int i = RUN ? t + l0 + l : (l0 + l) * S + t;
                            const XT vv = widen<XT>(vs[l][t], sc);
                            if (ok[i] && vv != XT(0)) {
#pragma unroll
                                for (int v = 0; v < V; ++v) acc[t][v] = fma_rn(vv, xv[i][v], acc[t][v]);
                            }
                        }
                }
            }
        };
        auto all = [&](auto CHECK) {
            // any offsets at once: 128 bytes of X a lane
            constexpr int U = 128 / (S * V * static_cast<int>(sizeof(XT))) >= 8 ? 8 : 128 / (S * V * static_cast<int>(sizeof(XT)));
            constexpr bool RUNS = S >= 4;
            if constexpr (U == 1) {
#pragma unroll 1
                for (int j = 0; j < cnt;) {
                    if (runs >> j & 1u) {
                        step(std::integral_constant<int, 3>(), std::true_type(), CHECK, j);
                        j += 3;
                    } else {
                        step(std::integral_constant<int, 1>(), std::false_type(), CHECK, j);
                        ++j;
                    }
                }
                return;
            }
#pragma unroll 1
            for (int j = 0; j < cnt;) {
                const unsigned next = RUNS ? runs >> j : 0u;
                if (next & 1u) {
                    step(std::integral_constant<int, 3>(), std::true_type(), CHECK, j);
                    j += 3;
                    continue;
                }
                // offsets before the next run: a group of U, else of 4, else the rest
                const int left = next ? __ffs(next) - 1 : cnt - j;
                if (left >= U) {
                    step(std::integral_constant<int, U>(), std::false_type(), CHECK, j);
                    j += U;
                } else if (U > 4 && left >= 4) {
                    step(std::integral_constant<int, U < 4 ? 1 : 4>(), std::false_type(), CHECK, j);
                    j += 4;
                } else {
                    if (U > 3 && left == 3) step(std::integral_constant<int, U < 3 ? 1 : 3>(), std::false_type(), CHECK, j);
                    if (U > 2 && left == 2) step(std::integral_constant<int, U < 2 ? 1 : 2>(), std::false_type(), CHECK, j);
                    if (U > 1 && left == 1) step(std::integral_constant<int, 1>(), std::false_type(), CHECK, j);
                    j += left;
                }
            }
        };
        if (interior) all(std::false_type());
        else all(std::true_type());
    }
}

// Instances whose CTAs always have kRowsWarps warps.
template <typename XT, int V, int S>
__host__ __device__ constexpr bool rows_fixed_cta() {
    return S == 8 && V * sizeof(XT) == 16;
}

// One warp per slab of RS = (32 / G) S rows of a 32-row tile and C = G V
// columns: lane l holds rows (l / G) S .. + S - 1 of the slab and columns
// (l % G) V .. + V - 1, so one request of a warp reads 32 / G whole row
// segments of X, and a lane's S values of one offset are neighbours.
template <typename VT, typename XT, int V, int G, int S>
__global__ void __launch_bounds__(kRowsWarps * 32, 1)
spmm_rows(const SpmvArgs<VT, XT> a, const XT *__restrict__ X, int64_t ldx, XT *__restrict__ Y, int64_t ldy, int32_t k,
          int32_t vec) {
    __shared__ RowsCoo<XT, V> coo[kRowsWarps];
    constexpr int RPR = 32 / G;        // row segments per request
    constexpr int RS = RPR * S;        // rows of a slab
    constexpr int HALVES = 32 / RS;    // slabs per tile
    constexpr int C = G * V;
    const int lane = threadIdx.x & 31;
    const int grp = lane / G;
    const int c = (lane % G) * V;
    // (a constant where registers are scarce: 8 rows of 16 bytes a lane spill 44
    // bytes instead of 20 otherwise, 27-point 96^3 k = 16 258 -> 282 us)
    const int32_t warps = rows_fixed_cta<XT, V, S>() ? kRowsWarps : static_cast<int32_t>(blockDim.x >> 5);
    const int32_t W = static_cast<int32_t>(gridDim.x) * warps;
    const int32_t numSlabs = a.numTiles * HALVES;
    const int32_t m = a.bw >> 5;
    int32_t s = static_cast<int32_t>(blockIdx.x) * warps + (threadIdx.x >> 5);
    if (s >= numSlabs) return;  // warp-uniform

    auto loadMeta = [&](int32_t q) {
        TileMeta t{0, 0, 0, 0};
        if (q >= numSlabs) return t;
        const int32_t tile = q / HALVES, b = tile / m;
        if (b < a.numBlocks) {
            t.k0 = __ldg(a.blkOff + b);
            t.k1 = __ldg(a.blkOff + b + 1);
        }
        if (a.hasCoo) {
            t.c0 = __ldg(a.cooTile + tile);
            t.c1 = __ldg(a.cooTile + tile + 1);
        }
        return t;
    };
    TileMeta mt = loadMeta(s);
    int32_t offNext = lane < mt.k1 - mt.k0 ? __ldg(a.offs + mt.k0 + lane) : 0;
    for (; s < numSlabs; s += W) {
        const TileMeta mn = loadMeta(s + W);
        const int32_t tile = s / HALVES;
        const int32_t row0 = tile * 32 + (s % HALVES) * RS;  // the slab's first row
        const int32_t row = row0 + grp * S;                  // the lane's first row
        // first COO entries of the tile
        int32_t cr = 0x7fffffff, cc = 0;
        XT cv = XT(0);
        if (mt.c0 + lane < mt.c1) {
            cr = __ldg(a.cooRow + mt.c0 + lane) - row0;
            cc = __ldg(a.cooCol + mt.c0 + lane);
            cv = __ldg(a.cooVal + mt.c0 + lane);
        }
        const float sc = a.scale && tile / m < a.numBlocks ? __ldg(a.scale + tile / m) : 1.0f;
        // the lane's values of offset k of the block: vp + k * bw
        const VT *vp = a.vals + static_cast<int64_t>(mt.k0) * a.bw + (tile % m) * 32 + (row - tile * 32);
        const int32_t first = offNext;
        offNext = lane < mn.k1 - mn.k0 ? __ldg(a.offs + mn.k0 + lane) : 0;
        for (int32_t c0 = 0; c0 < k; c0 += C) {
            const bool on = c0 + c < k;
            const int32_t cx = on ? c : 0;  // lanes without a column read the first one's X
            const XT *xb = X + static_cast<int64_t>(row) * ldx + c0 + cx;
            XT acc[S][V];
#pragma unroll
            for (int t = 0; t < S; ++t)
#pragma unroll
                for (int v = 0; v < V; ++v) acc[t][v] = XT(0);
            rows_dia<VT, XT, V, G, S>(a, xb, ldx, mt, first, vp, sc, row0, row, lane, vec, acc);
            if (mt.c1 > mt.c0) {
                rows_coo<VT, XT, V, G, S>(a, X + c0 + cx, ldx, mt.c0, mt.c1, row0, cr, cc, cv, lane, coo[threadIdx.x >> 5], acc);
            } else if (a.hasCoo) {  // rows without entries add an empty sum: -0 becomes +0
#pragma unroll
                for (int t = 0; t < S; ++t)
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[t][v] = add_rn(acc[t][v], XT(0));
            }
            if (on) {
#pragma unroll
                for (int t = 0; t < S; ++t)
                    if (row + t < a.n) {
                        st_y<XT, V>(Y + static_cast<int64_t>(row + t) * ldy + c0 + c, acc[t]);
                    }
            }
        }
        mt = mn;
    }
}

}  // namespace dev
}  // namespace hbdia
