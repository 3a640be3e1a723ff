// kcna_pairs.cuh - canonical FP32 distances of the pairs of a small set of
// rows by one warp (the FP32 local join and the FP32 P2K join).
//
// A node of either join brings 20 to 60 rows and some hundred pairs.  A block
// per node with a 32 x 64 (or 128 x 64) tile computed every slot of the tile
// (four to eight times the pairs) and met several block barriers per node;
// measured on 150,001 x 128 rows it ran at 15 % of the FP32 rate.  Here a warp
// takes a node by itself: its rows in shared memory, 64 dimensions at a time,
// and the pairs as 4 x 4 micro-tiles dealt out to the lanes, so that only the
// edges of the micro-tiles are wasted and nothing but the warp waits.
//
// The four rows of a micro-tile's side are `step` apart, not adjacent: the
// lanes of one load then read neighbouring rows, which the row pitch (68
// floats) puts in distinct banks.  Rows past the end of a side read whatever
// lies there (inside the warp's region: three spare rows) and their results
// are not used.
#pragma once
#include "kcna_common.cuh"

namespace {

constexpr int PT_KC = 64;         // dimensions staged at a time
constexpr int PT_P = PT_KC + 4;   // row pitch in floats
constexpr int PT_SPARE = 3;       // rows a micro-tile may read past the set
constexpr int PT_MAXR = 4;        // micro-tiles per lane at most
constexpr int PT_MAXT = 32 * PT_MAXR;

// One micro-tile: rows a0 + x * as against rows b0 + y * bs, x, y in 0..3.
struct PairTile {
    int a0, as, b0, bs;
};

// Rows s_id[0, n) of dimensions [k0, k0 + kc) into s_x; the caller syncs.
__device__ __forceinline__ void pairs_stage(const RowsF32 &rows, const uint32_t *s_id, int n, int k0, int kc,
                                            float *s_x) {
    const int sh = kc <= 32 ? 3 : 4, lane = kcna_lane(); // 8 or 16 float4 per row
    const int c = 4 * (lane & ((1 << sh) - 1));
    if (c < kc)
        for (int r = lane >> sh; r < n; r += 32 >> sh) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_x + r * PT_P + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                         "l"(rows.p + (uint64_t)s_id[r] * rows.ld + k0 + c)
                         : "memory");
        }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void pairs_stage(const RowsB16 &rows, const uint32_t *s_id, int n, int k0, int kc,
                                            float *s_x) {
    const int sh = kc <= 32 ? 3 : 4, lane = kcna_lane();
    const int c = 4 * (lane & ((1 << sh) - 1));
    if (c < kc)
        for (int r = lane >> sh; r < n; r += 32 >> sh)
            *reinterpret_cast<float4 *>(s_x + r * PT_P + c) = rows.ld4(s_id[r], (k0 + c) >> 2);
}

// acc[r][4 x + y] = canonical distance of the lane's micro-tile r (on[r]).
template <int R, class RowsT>
__device__ __forceinline__ void pairs_distances(const RowsT &rows, const uint32_t *s_id, int n, float *s_x,
                                                const PairTile (&t)[R], const bool (&on)[R], float (&acc)[R][16]) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[r][i] = 0.f;
    for (int k0 = 0; k0 < rows.ld; k0 += PT_KC) {
        const int kc = min(PT_KC, rows.ld - k0);
        __syncwarp(); // the previous chunk is read
        pairs_stage(rows, s_id, n, k0, kc, s_x);
        __syncwarp();
        for (int k = 0; k < kc; k += 4) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (!on[r]) continue;
                float4 xa[4], xb[4];
                const float *pa = s_x + t[r].a0 * PT_P + k, *pb = s_x + t[r].b0 * PT_P + k;
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    xa[x] = *reinterpret_cast<const float4 *>(pa + x * t[r].as * PT_P);
                    xb[x] = *reinterpret_cast<const float4 *>(pb + x * t[r].bs * PT_P);
                }
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) acc[r][4 * x + y] = kcna_acc4(acc[r][4 * x + y], xa[x], xb[y]);
            }
        }
    }
    __syncwarp(); // the rows' region is free
}

} // namespace
