// kcna_pairs.cuh - canonical FP32 distances of the pairs of a small set of
// rows by one warp or one small block (the FP32 local join and the FP32 P2K
// join).
//
// A node of either join brings 20 to 60 rows and some hundred pairs.  A block
// of 256 threads per node with a 32 x 64 (or 128 x 64) tile computed every slot
// of the tile (four to eight times the pairs) and met a dozen block barriers
// per node; measured on 150,001 x 128 rows it ran at 15 % of the FP32 rate.
// Here the pairs are 4 x 4 micro-tiles dealt out to the lanes, so that only
// the edges of the micro-tiles are wasted, and a node of up to 64 rows is one
// warp's, so that nothing else waits for its loads.  The rows come 16
// dimensions at a time into two buffers (cp.async), the next chunk in flight
// while this one is used: with 32 at a time eleven warps instead of sixteen
// share an SM, and the joins took 3 to 25 % longer.
//
// The four rows of a micro-tile's side are `step` apart, not adjacent: the
// lanes of one load then read neighbouring rows, which the row pitch (20
// floats) puts in distinct banks.  Rows past the end of a side read whatever
// lies there (inside the group's region: three spare rows) and their results
// are not used.
#pragma once
#include "kcna_common.cuh"

namespace {

constexpr int PT_KC = 16;         // dimensions staged at a time
constexpr int PT_P = PT_KC + 4;   // row pitch in floats
constexpr int PT_SPARE = 3;       // rows a micro-tile may read past the set
constexpr int PT_MAXR = 3;        // micro-tiles per lane at most
__host__ __device__ constexpr int pairs_region(int rows) { return 2 * (rows + PT_SPARE) * PT_P; } // floats

// One micro-tile: rows a0 + x * as against rows b0 + y * bs, x, y in 0..3.
struct PairTile {
    int a0, as, b0, bs;
};

// NT threads (a warp, or a whole block) work on one set.
template <int NT> __device__ __forceinline__ int pairs_lane() { return NT == 32 ? kcna_lane() : (int)threadIdx.x; }
template <int NT> __device__ __forceinline__ void pairs_sync() {
    if (NT == 32)
        __syncwarp();
    else
        __syncthreads();
}

// Rows s_id[0, n), dimensions [k0, k0 + PT_KC) below ld, into s_x: 4 threads a row.
template <int NT>
__device__ __forceinline__ void pairs_stage(const RowsF32 &rows, const uint32_t *s_id, int n, int k0, float *s_x) {
    const int lane = pairs_lane<NT>(), c = 4 * (lane & 3);
    if (k0 + c < rows.ld) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_x + c);
        const float *src = rows.p + k0 + c;
        for (int r = lane >> 2; r < n; r += NT / 4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + r * (PT_P * 4)),
                         "l"(src + (uint64_t)s_id[r] * rows.ld)
                         : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int NT>
__device__ __forceinline__ void pairs_stage(const RowsB16 &rows, const uint32_t *s_id, int n, int k0, float *s_x) {
    const int lane = pairs_lane<NT>(), c = 4 * (lane & 3);
    if (k0 + c < rows.ld)
        for (int r = lane >> 2; r < n; r += NT / 4)
            *reinterpret_cast<float4 *>(s_x + r * PT_P + c) = rows.ld4(s_id[r], (k0 + c) >> 2);
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// acc[r][4 x + y] = canonical distance of the thread's micro-tile r (on[r]).
// s_x: pairs_region(rows >= n) floats, free again on return.  Every cp.async
// group this thread committed before the call has landed on return.
template <int NT, int R, class RowsT>
__device__ __forceinline__ void pairs_distances(const RowsT &rows, const uint32_t *s_id, int n, float *s_x,
                                                const PairTile (&t)[R], const bool (&on)[R], float (&acc)[R][16]) {
    const int half = (n + PT_SPARE) * PT_P; // one buffer
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[r][i] = 0.f;
    pairs_stage<NT>(rows, s_id, n, 0, s_x);
    int b = 0;
    for (int k0 = 0; k0 < rows.ld; k0 += PT_KC, b ^= 1) {
        if (k0 + PT_KC < rows.ld) {
            pairs_stage<NT>(rows, s_id, n, k0 + PT_KC, s_x + (b ^ 1) * half);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        pairs_sync<NT>(); // this chunk is there for every thread
        const float *x = s_x + b * half;
        const int kc = min(PT_KC, rows.ld - k0);
        for (int k = 0; k < kc; k += 4) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (!on[r]) continue;
                float4 xa[4], xb[4];
                const float *pa = x + t[r].a0 * PT_P + k, *pb = x + t[r].b0 * PT_P + k;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    xa[u] = *reinterpret_cast<const float4 *>(pa + u * t[r].as * PT_P);
                    xb[u] = *reinterpret_cast<const float4 *>(pb + u * t[r].bs * PT_P);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) acc[r][4 * u + v] = kcna_acc4(acc[r][4 * u + v], xa[u], xb[v]);
            }
        }
        pairs_sync<NT>(); // this chunk is read: its buffer takes the chunk after the next
    }
}

} // namespace
