// kcna_knn_tc.cu - the filter of the exact k-NN (kcna_knn.cu) on tcgen05 Gram
// tiles, d <= 128.
//
// For every query a bound T on the k-th smallest distance is known.  The
// canonical FP32 chain of every (query, row) pair takes 6.4 ms for 1,000
// queries against 1,000,000 x 128 rows at the FP32 rate (10.2 measured); but
// only the few thousand rows within T matter.  So the pairs are screened with
// the rows rounded to BF16 and FP32 accumulation, and a row's id is handed on
// unless its distance is certainly above T; the distances of those handed on
// are then computed canonically (knn_final_kernel).  What is certain: with
// q~, x~ the rounded rows, e their rounding errors' norms, G = <q~, x~> as
// computed and c (|q~|^2 + |x~|^2) a bound on its error and the norms',
//   d <= T  implies  |q~|^2 + |x~|^2 - 2 G <= (sqrt(T (1 + g)) + e_q + e_x)^2 + c (|q~|^2 + |x~|^2)
// (the triangle inequality; g: the chain's own rounding).  c = 2^-15 + d 2^-22
// allows sixteen-term sums that lose a bit each and FP32 sums of the squares.
// The test is written so that a NaN hands the row on.
//
// Persistent, one block of 16 warps per SM: a base tile of 256 rows is read
// from memory once, in FP32, rounded into the 128-byte swizzled K-major layout
// (its successor's rows wait in registers meanwhile) and meets all the query
// tiles of 128 (BF16, four buffers, from L2); the tensor cores fill one of two
// TMEM accumulators while the warps test the other: warp w reads the lanes
// (queries) of quarter w % 4 and the 64 columns (rows) of group w / 4.  The
// size above takes 1.07 ms, where every pair in FP32 took 10.2.  Nothing in it is
// busy (400,000 rows: issue 0.37 a cycle, tensor pipe 9 %, L2 6 %); the warps
// wait: for the place that the atomicAdd of a row handed on returns and for TMEM
// (long scoreboard, 3.6 cycles of an issue's 10), and at the barrier (1.8).
#include <algorithm>

#include "kcna_internal.h"
#include "kcna_tc.cuh"

using namespace kcna_tc;

namespace {

constexpr int FQ = 128, FB = 256;          // queries and base rows per tile (MMA M, N)
constexpr int FT = 512;                    // threads
constexpr int FQBUF = 4;                   // query tile buffers
constexpr uint32_t KBB = 128;              // bytes of a row inside one 64-element K block
constexpr uint32_t TILE_Q = FQ * KBB * 2, TILE_B = FB * KBB * 2;

struct FilterShared {
    alignas(16) float2 col[FB]; // of a base row: |x~|^2 (1 - c), e_x; read two rows at a time
    uint64_t full[2];           // accumulator written
    uint32_t tmem;
};

struct FilterArgs {
    const float *X;
    uint32_t n, ld;
    const uint16_t *Qh;   // rounded queries, 128 elements apart, rows up to a multiple of 128
    const float2 *qmeta;  // of a query: |q~|^2 (1 - c), sqrt(T (1 + g)) + e_q
    uint32_t m;
    float one_c;
    uint32_t *cand, *cnt; // ids handed on, `cap` per query
    uint32_t cap;
    int *err;
};

// norms of one row held by a warp, four elements per lane: rounded row to dst
// (8 bytes per lane), its squared norm and a bound on |x - x~|
__device__ __forceinline__ uint2 round4(float4 x, float &nn, float &ee) {
    const float v[4] = {x.x, x.y, x.z, x.w};
    uint32_t h[4];
    nn = ee = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat16 b = __float2bfloat16_rn(v[i]);
        h[i] = *reinterpret_cast<const uint16_t *>(&b);
        const float f = __uint_as_float(h[i] << 16), df = v[i] - f;
        nn = fmaf(f, f, nn);
        ee = fmaf(df, df, ee);
    }
    return make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
}
__device__ __forceinline__ float error_bound(float nn, float ee) {
    return sqrtf(ee) * (1.f + 1.f / 1024.f) + sqrtf(nn) * (1.f / 4194304.f) + 1e-18f;
}

// Queries: rounded rows (zero past ld and m) and their terms; warp per row.
__global__ void filter_queries_kernel(const float *__restrict__ Q, uint32_t m, uint32_t ld, uint32_t rows,
                                      const uint32_t *__restrict__ thresh, float one_g, float one_c,
                                      uint16_t *__restrict__ Qh, float2 *__restrict__ qmeta) {
    const uint32_t r = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= rows) return;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < m && 4u * lane < ld) x = reinterpret_cast<const float4 *>(Q + (uint64_t)r * ld)[lane];
    float nn, ee;
    reinterpret_cast<uint2 *>(Qh + (uint64_t)r * 128)[lane] = round4(x, nn, ee);
    nn = kcna_warp_sum(nn);
    ee = kcna_warp_sum(ee);
    if (lane == 0) {
        const float T = r < m ? __uint_as_float(thresh[r]) : 0.f;
        qmeta[r] = make_float2(nn * one_c, sqrtf(fmaf(T, one_g, 1e-36f)) * 1.00001f + error_bound(nn, ee));
    }
}

__global__ void __launch_bounds__(FT, 1) knn_filter_kernel(FilterArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t sB = (smem_u32(smem_raw) + 1023u) & ~1023u; // swizzled tiles need 1024-byte alignment
    unsigned char *tB = smem_raw + (sB - smem_u32(smem_raw));
    const uint32_t sQ = sB + TILE_B;
    FilterShared &S = *reinterpret_cast<FilterShared *>(tB + TILE_B + FQBUF * TILE_Q);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nkb = ((int)a.ld + 63) >> 6;
    const uint32_t nq = (a.m + FQ - 1) / FQ, ntiles = (a.n + FB - 1) / FB;
    if (warp == 0) tmem_alloc(&S.tmem, 2 * FB);
    if (tid == 0) {
        mbar_init(&S.full[0], 1);
        mbar_init(&S.full[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = S.tmem, idesc = idesc_bf16(FQ, FB);
    const int quarter = warp & 3, h = warp >> 2; // TMEM lane quarter, group of 64 columns

    constexpr int RW = FB / (FT / 32); // base rows per warp
    float4 nxt[RW];
    auto fetch = [&](uint32_t tile) { // this warp's rows of a base tile
#pragma unroll
        for (int i = 0; i < RW; ++i) {
            const uint64_t b = (uint64_t)tile * FB + warp * RW + i;
            nxt[i] = tile < ntiles && b < a.n && 4u * lane < a.ld
                         ? __ldg(reinterpret_cast<const float4 *>(a.X + b * a.ld) + lane)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto load_queries = [&](uint32_t qt) { // tile qt into its buffer, one cp.async group
        if (qt < nq) {
            const uint32_t dst = sQ + (qt % FQBUF) * TILE_Q;
#pragma unroll
            for (int i = 0; i < FQ * 16 / FT; ++i) {
                const uint32_t e = tid + FT * i, r = e >> 4, s = e & 15; // row, 16-byte segment
                if ((int)(s >> 3) < nkb)
                    cp_async16(dst + (s >> 3) * FQ * KBB + sw128_off(r, s & 7),
                               a.Qh + ((uint64_t)qt * FQ + r) * 128 + s * 8);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    bool ok = true;
    uint32_t used = 0; // products issued so far: accumulator used & 1
    fetch(blockIdx.x);
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        // every product of the previous tile is complete (its last epilogue waited for it)
#pragma unroll
        for (int i = 0; i < RW; ++i) {
            const uint32_t r = warp * RW + i;
            float nn, ee;
            const uint2 v = round4(nxt[i], nn, ee);
            const uint32_t seg = lane >> 1; // 16-byte segment of the row
            if ((int)(seg >> 3) < nkb)
                *reinterpret_cast<uint2 *>(tB + (seg >> 3) * FB * KBB + sw128_off(r, seg & 7) + (lane & 1) * 8) = v;
            nn = kcna_warp_sum(nn);
            ee = kcna_warp_sum(ee);
            if (lane == 0) S.col[r] = make_float2(nn * a.one_c, error_bound(nn, ee));
        }
        load_queries(0);
        load_queries(1);
        fetch(tile + gridDim.x);
        const uint32_t valid = min((uint32_t)FB, a.n - tile * FB);
        auto epilogue = [&](uint32_t qt, uint32_t u) { // test of product u, query tile qt
            const uint32_t q = qt * FQ + 32 * quarter + lane;
            const float2 qm = q < a.m ? a.qmeta[q] : make_float2(0.f, 0.f);
            ok = __all_sync(KCNA_FULL, mbar_wait(&S.full[u & 1], (u >> 1) & 1)) && ok;
            fence_after();
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int c0 = 64 * h + 16 * g;
                uint32_t raw[16];
                tmem_ld16_async(tmem + ((uint32_t)(32 * quarter) << 16) + (u & 1) * FB + c0, raw);
                tmem_wait_ld16(raw);
                uint32_t mask = 0;
#pragma unroll
                for (int x = 0; x < 16; x += 2) {
                    const float4 cm = *reinterpret_cast<const float4 *>(&S.col[c0 + x]);
                    const float r0 = qm.y + cm.y, r1 = qm.y + cm.w;
                    const float l0 = fmaf(-2.f, __uint_as_float(raw[x]), cm.x) + qm.x;
                    const float l1 = fmaf(-2.f, __uint_as_float(raw[x + 1]), cm.z) + qm.x;
                    mask |= (!(l0 > r0 * r0) ? 1u : 0u) << x;
                    mask |= (!(l1 > r1 * r1) ? 2u : 0u) << x;
                }
                if (q >= a.m) mask = 0;
                while (mask) {
                    const uint32_t x = __ffs(mask) - 1;
                    mask &= mask - 1;
                    if (c0 + x >= valid) break;
                    const uint32_t p = atomicAdd(a.cnt + q, 1u);
                    if (p < a.cap) a.cand[(uint64_t)q * a.cap + p] = tile * FB + c0 + x;
                }
            }
            fence_before();
        };
        for (uint32_t qt = 0; qt < nq; ++qt) {
            asm volatile("cp.async.wait_group 1;" ::: "memory"); // tile qt has landed
            fence_proxy_async();
            fence_before();
            if (__syncthreads_or(!ok)) { // also: the accumulator of product used - 2 is read
                ok = false;
                break;
            }
            if (tid == 0) {
                fence_after();
                const uint32_t q0 = sQ + (qt % FQBUF) * TILE_Q, d = tmem + (used & 1) * FB;
                for (int kb = 0; kb < nkb; ++kb)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        mma_bf16(d, desc_sw128(q0 + kb * FQ * KBB + kk * 32), desc_sw128(sB + kb * FB * KBB + kk * 32),
                                 idesc, (kb | kk) ? 1u : 0u);
                mma_commit(&S.full[used & 1]);
            }
            __syncwarp();
            load_queries(qt + 2); // its buffer was product used - 2's
            ++used;
            if (qt > 0) epilogue(qt - 1, used - 2);
        }
        if (ok) epilogue(nq - 1, used - 1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (__syncthreads_or(!ok)) { // the base tile may be overwritten
            ok = false;
            break;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 2 * FB);
    if (!ok) kcna_set_err(a.err, KCNA_DERR_SPIN);
}

} // namespace

// Hands on, for each of m queries, the ids of the rows that may lie within its
// bound thresh[q] (FP32 bits): cand (cap per query), cnt (zero at entry).
kcna_status kcna_knn_filter(kcna_ctx *c, const float *dQ, uint32_t m, const uint32_t *thresh, uint32_t *cand,
                            uint32_t *cnt, uint32_t cap) {
    if (c->ld > 128 || m == 0) return kcna_fail(c, KCNA_E_STATE, "k-NN filter: d <= 128");
    const uint32_t rows = (m + FQ - 1) / FQ * FQ;
    uint16_t *Qh = nullptr;
    float2 *qmeta = nullptr;
    const float cc = (float)(1.0 / 32768.0 + (double)c->ld / 4194304.0);
    const float g = (float)((c->ld + 2) * (2.0 / 16777216.0));
    kcna_status s = kcna_alloc(c, &Qh, (size_t)rows * 128, "rounded queries");
    if (s == KCNA_OK) s = kcna_alloc(c, &qmeta, rows, "query terms");
    if (s == KCNA_OK) {
        filter_queries_kernel<<<kcna_div_up((uint64_t)rows * 32, 256), 256, 0, c->stream>>>(
            dQ, m, c->ld, rows, thresh, 1.f + g, 1.f - cc, Qh, qmeta);
        KCNA_LAUNCHED(c);
        FilterArgs a{c->X, c->n, c->ld, Qh, qmeta, m, 1.f - cc, cand, cnt, cap, c->d_err};
        const size_t sm = 1024 + TILE_B + FQBUF * TILE_Q + sizeof(FilterShared);
        s = kcna_cuda_check(c, cudaFuncSetAttribute(knn_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)sm),
                            "knn filter smem attr");
        if (s == KCNA_OK) {
            const uint32_t grid = std::min((c->n + FB - 1) / FB, (uint32_t)std::max(c->num_sms, 1));
            knn_filter_kernel<<<grid, FT, sm, c->stream>>>(a);
            KCNA_LAUNCHED(c);
            s = kcna_cuda_check(c, cudaGetLastError(), "knn_filter_kernel");
        }
    }
    kcna_release(c, Qh); // later users run behind these kernels on the context's stream
    kcna_release(c, qmeta);
    return s;
}
