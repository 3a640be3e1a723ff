// kcna_knn.cu - exact k-NN (brute force) on the GPU.
//
// Replaces LinearSearch (src/kgraph.cpp:309-330, used by GenerateControl
// :363-387) and SearchOracle::search (:332-361): for each query, the k rows
// with the smallest squared L2 distance, ties broken by the lower id (the
// reference scans ids in order and inserts equal distances after existing
// ones, src/kgraph.cpp:227-260).
//
// Few rows or few queries (knn_bound_pays): two kernels,
//   1. a tiled distance kernel (32 queries x 128 rows per block, 4x4 register
//      micro-tiles, dimensions staged through shared memory in chunks of 32)
//      computing the canonical FMA-chain distance of every pair;
//   2. an exact selection kernel per query: three radix-histogram passes over
//      the distance bits find the k-th smallest distance T, then every row with
//      distance < T plus the lowest ids among rows with distance == T are kept
//      and sorted by (distance, id).
// Else: writing every distance and reading it four times costs more
// than computing it (7.3 of 17.7 ms for 1,000 queries against 1,000,000 x 128
// rows), and the computation itself can be spared for all but a few thousand
// rows per query:
//   1. distances to s rows, one drawn from every n / s consecutive ones (not
//      every (n / s)-th: in rows stored with a period, those can all belong to
//      a few clusters, and the lists of the other clusters' queries overflow);
//      the max(k, 32)-th smallest of them is a bound T on the k-th smallest of all;
//   2. the rows that may lie within T: screened on tensor cores where the work
//      is large and d <= 128 (kcna_knn_tc.cu), else by the tiled kernel, which
//      then keeps a pair only if its distance is at most T;
//   3. per query, canonical distances of the rows handed on (where 2 screened)
//      and the selection among them.
// s is chosen so that about 4,096 rows remain; the queries whose lists of 8,192
// overflow, or come up short (NaN), are gathered and done again together the
// first way.
// The size above: 2.05 ms a call (0.26 sample, 0.08 bounds, 1.07 screen, 0.58
// selection).
#include <algorithm>

#include "kcna_internal.h"
#include "kcna_sort.cuh"

namespace {

constexpr int TQ = 32, TB = 128, KC = 32, KCP = KC + 4;

// DT_ALL: every distance is written.  DT_FILTER: instead, (distance, id) is
// appended to the query's list when the distance is at most thresh[q].
// DT_SAMPLE: as DT_ALL, base row b being row sample_row(b, stride) of X.
enum { DT_ALL, DT_FILTER, DT_SAMPLE };
__device__ __forceinline__ uint64_t sample_row(uint64_t b, uint32_t stride) { // one of the rows [b, b + 1) * stride
    uint32_t h = (uint32_t)b * 0x9E3779B1u;
    h = (h ^ (h >> 15)) * 0x85EBCA77u;
    return b * stride + __umulhi(h ^ (h >> 13), stride);
}
struct DistOut {
    float *D;
    uint64_t ldD;
    const uint32_t *thresh;
    uint64_t *cand;
    uint32_t *cnt, cap;
};
template <int MODE>
__global__ void __launch_bounds__(256) dist_tile_kernel(const float *__restrict__ Q, uint32_t m,
                                                        const float *__restrict__ X, uint32_t n, uint32_t stride,
                                                        int ld, const uint32_t *__restrict__ q_self, DistOut o) {
    __shared__ __align__(16) float Qs[TQ][KCP];
    __shared__ __align__(16) float Xs[TB][KCP];
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const uint32_t q0 = blockIdx.y * TQ;
    const uint64_t b0 = (uint64_t)blockIdx.x * TB;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    auto row_of = [&](uint64_t b) { return MODE == DT_SAMPLE ? sample_row(b, stride) : b * stride; };

    for (int k0 = 0; k0 < ld; k0 += KC) {
        {   // Q chunk: 32 rows x 32 floats, one float4 per thread
            int r = tid >> 3, c = (tid & 7) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q0 + r < m && k0 + c < ld) v = *reinterpret_cast<const float4 *>(Q + (uint64_t)(q0 + r) * ld + k0 + c);
            *reinterpret_cast<float4 *>(&Qs[r][c]) = v;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) { // X chunk: 128 rows x 32 floats
            int idx = tid + s * 256;
            int r = idx >> 3, c = (idx & 7) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (b0 + r < n && k0 + c < ld) v = __ldg(reinterpret_cast<const float4 *>(X + row_of(b0 + r) * ld + k0 + c));
            *reinterpret_cast<float4 *>(&Xs[r][c]) = v;
        }
        __syncthreads();
        const int kend = min(KC, ld - k0);
        for (int k = 0; k < kend; k += 4) {
            float4 qa[4], xb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) qa[i] = *reinterpret_cast<const float4 *>(&Qs[ty + 8 * i][k]);
#pragma unroll
            for (int j = 0; j < 4; ++j) xb[j] = *reinterpret_cast<const float4 *>(&Xs[tx + 32 * j][k]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = kcna_acc4(acc[i][j], qa[i], xb[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t q = q0 + ty + 8 * i;
        if (q >= m) continue;
        uint32_t self = q_self ? q_self[q] : KCNA_NONE;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint64_t b = b0 + tx + 32 * j;
            if (b >= n) continue;
            const uint64_t row = row_of(b);
            const bool own = row == self;
            if (MODE != DT_FILTER) {
                o.D[(uint64_t)q * o.ldD + b] = own ? __uint_as_float(0x7F800000u) : acc[i][j];
            } else if (!own && __float_as_uint(acc[i][j]) <= o.thresh[q]) {
                const uint32_t p = atomicAdd(o.cnt + q, 1u);
                if (p < o.cap) o.cand[(uint64_t)q * o.cap + p] = ((uint64_t)__float_as_uint(acc[i][j]) << 32) | row;
            }
        }
    }
}

constexpr int SEL_T = 512;
constexpr int SEL_BINS = 4096;
constexpr int SEL_MAXK = 1024;
constexpr int SEL_TIES = 1024;
constexpr int SEL_QUICK = 256;

constexpr uint32_t KNN_CAP = 8192;       // rows handed on per query at most
constexpr uint32_t SEL_CACHE = 40960;    // a sample up to this length is read once, into shared memory

struct SelectShared {
    uint32_t hist[SEL_BINS];
    uint32_t scan[SEL_T / 32];
    int bin;
    uint32_t before, nout, ntie;
};

// Finds the bin holding the want-th (0-based) element, S.bin, and the number
// of elements in lower bins, S.before; nb bins (a multiple of SEL_T).
__device__ void find_bin(SelectShared &S, int nb, uint32_t want) {
    const int per = nb / SEL_T, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t local = 0;
    for (int i = 0; i < per; ++i) local += S.hist[threadIdx.x * per + i];
    uint32_t incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(KCNA_FULL, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) S.scan[warp] = incl;
    __syncthreads();
    for (int w = 0; w < warp; ++w) incl += S.scan[w];
    const uint32_t excl = incl - local;
    if (want >= excl && want < incl) {
        uint32_t run = excl;
        for (int i = 0; i < per; ++i) {
            const uint32_t h = S.hist[threadIdx.x * per + i];
            if (want < run + h) {
                S.bin = threadIdx.x * per + i;
                S.before = run;
                break;
            }
            run += h;
        }
    }
    __syncthreads();
}

// The want-th (0-based) smallest of the n words at(j), by the whole block:
// bits 31..20, 19..8, 7..0.
template <class At>
__device__ uint32_t kth_word(SelectShared &S, uint32_t n, uint32_t want, At at) {
    uint32_t prefix = 0;
    const int shifts[3] = {20, 8, 0};
    const int widths[3] = {12, 12, 8};
    for (int pass = 0; pass < 3; ++pass) {
        const int sh = shifts[pass], nb = 1 << widths[pass];
        for (int i = threadIdx.x; i < max(nb, SEL_T); i += SEL_T) S.hist[i] = 0;
        __syncthreads();
        const int hsh = sh + widths[pass];
        for (uint32_t j = threadIdx.x; j < n; j += SEL_T) {
            const uint32_t v = at(j);
            if (pass == 0 || (v >> hsh) == prefix) atomicAdd(&S.hist[(v >> sh) & (nb - 1)], 1u);
        }
        __syncthreads();
        find_bin(S, max(nb, SEL_T), want);
        prefix = (prefix << widths[pass]) | (uint32_t)S.bin;
        want -= S.before;
        __syncthreads();
    }
    return prefix;
}

// The k smallest (distance, id) of n entries, dist(j) and id(j), sorted, to
// out; by the whole block.
// Up to k = SEL_QUICK the k-th smallest of the threads' own minima bounds the
// k-th distance: k entries lie within it, and seldom more than a few over (the
// expected number at k = SEL_QUICK is 355).  Those alone are collected and
// sorted, with two reads of each entry and no histogram, whose atomics meet in
// a few bins as distances share their leading bits: one query, k = 10 of 20,000
// x 32 rows takes 57 us as a call, 68 with the histograms.  Larger k, or more than
// SEL_MAXK entries within the bound, take the histogram passes.
template <class Dist, class Id>
__device__ void select_k(SelectShared &S, uint64_t *s_out, uint64_t *s_tie, uint32_t n, uint32_t k, Dist dist, Id id,
                         uint32_t *out_ids, float *out_d, int *err) {
    if (k <= SEL_QUICK) {
        constexpr int U = 8; // loads in flight
        uint32_t lo = 0xFFFFFFFFu;
        for (uint32_t j0 = threadIdx.x; j0 < n; j0 += U * SEL_T) {
            uint32_t v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = j0 + u * SEL_T < n ? dist(j0 + u * SEL_T) : 0xFFFFFFFFu;
#pragma unroll
            for (int u = 0; u < U; ++u) lo = min(lo, v[u]);
        }
        s_tie[threadIdx.x] = lo;
        if (threadIdx.x == 0) S.nout = 0;
        kcna_cta_bitonic(s_tie, SEL_T); // syncs before and after
        const uint32_t bound = (uint32_t)s_tie[k - 1];
        for (uint32_t j0 = threadIdx.x; j0 < n; j0 += U * SEL_T) {
            uint32_t v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = j0 + u * SEL_T < n ? dist(j0 + u * SEL_T) : 0xFFFFFFFFu;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j0 + u * SEL_T < n && v[u] <= bound) {
                    const uint32_t p = atomicAdd(&S.nout, 1u);
                    if (p < SEL_MAXK) s_out[p] = ((uint64_t)v[u] << 32) | id(j0 + u * SEL_T);
                }
        }
        __syncthreads();
        const uint32_t got = S.nout;
        if (got <= SEL_MAXK) {
            const int gp = kcna_pow2_ceil_d((int)got);
            for (int i = got + threadIdx.x; i < gp; i += SEL_T) s_out[i] = KCNA_EMPTY_KEY;
            kcna_cta_bitonic(s_out, gp);
            for (uint32_t i = threadIdx.x; i < k; i += SEL_T) {
                out_ids[i] = (uint32_t)s_out[i];
                out_d[i] = __uint_as_float((uint32_t)(s_out[i] >> 32));
            }
            return;
        }
        __syncthreads(); // S.nout is written again below
    }
    const uint32_t T = kth_word(S, n, k - 1, dist); // k-th smallest distance bits
    if (threadIdx.x == 0) {
        S.nout = 0;
        S.ntie = 0;
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < n; j += SEL_T) {
        const uint32_t v = dist(j);
        if (v < T) {
            uint32_t p = atomicAdd(&S.nout, 1u);
            if (p < SEL_MAXK) s_out[p] = ((uint64_t)v << 32) | id(j);
        } else if (v == T) {
            uint32_t p = atomicAdd(&S.ntie, 1u);
            if (p < SEL_TIES) s_tie[p] = ((uint64_t)v << 32) | id(j);
        }
    }
    __syncthreads();
    uint32_t nless = S.nout, ntie = S.ntie;
    if (ntie > SEL_TIES) kcna_set_err(err, KCNA_DERR_TIES);
    if (nless >= k) kcna_set_err(err, KCNA_DERR_BOUNDS);
    ntie = min(ntie, (uint32_t)SEL_TIES);
    nless = min(nless, k);
    int tp = kcna_pow2_ceil_d((int)ntie);
    for (int i = ntie + threadIdx.x; i < tp; i += SEL_T) s_tie[i] = KCNA_EMPTY_KEY;
    kcna_cta_bitonic(s_tie, tp);
    uint32_t need = k - nless;
    for (uint32_t i = threadIdx.x; i < need; i += SEL_T) s_out[nless + i] = i < ntie ? s_tie[i] : KCNA_EMPTY_KEY;
    int kp = kcna_pow2_ceil_d((int)k);
    for (int i = k + threadIdx.x; i < kp; i += SEL_T) s_out[i] = KCNA_EMPTY_KEY;
    kcna_cta_bitonic(s_out, kp);
    for (uint32_t i = threadIdx.x; i < k; i += SEL_T) {
        uint64_t key = s_out[i];
        out_ids[i] = (uint32_t)key;
        out_d[i] = __uint_as_float((uint32_t)(key >> 32));
    }
}

__global__ void __launch_bounds__(SEL_T) select_kernel(const float *__restrict__ D, uint64_t ldD, uint32_t n,
                                                       uint32_t k, uint32_t q_base, uint32_t *__restrict__ out_ids,
                                                       float *__restrict__ out_d, int *err) {
    __shared__ SelectShared S;
    __shared__ uint64_t s_out[SEL_MAXK], s_tie[SEL_TIES];
    const uint32_t *row = reinterpret_cast<const uint32_t *>(D + (uint64_t)blockIdx.x * ldD);
    const uint64_t ob = (uint64_t)(q_base + blockIdx.x) * k;
    select_k(S, s_out, s_tie, n, k, [&](uint32_t j) { return row[j]; }, [](uint32_t j) { return j; }, out_ids + ob,
             out_d + ob, err);
}

// Bound of each query: the rank-th smallest of its s sampled distances; also
// clears the query's count.
template <bool CACHED>
__global__ void __launch_bounds__(SEL_T) knn_bound_kernel(const float *__restrict__ D, uint32_t s, uint32_t rank,
                                                          uint32_t *__restrict__ thresh, uint32_t *__restrict__ cnt) {
    extern __shared__ __align__(16) uint32_t s_row[];
    __shared__ SelectShared S;
    const uint32_t *row = reinterpret_cast<const uint32_t *>(D + (uint64_t)blockIdx.x * s);
    if (CACHED) {
#pragma unroll 8
        for (uint32_t j = threadIdx.x; j < s; j += SEL_T) s_row[j] = row[j];
        row = s_row;
        __syncthreads();
    }
    const uint32_t T = kth_word(S, s, rank - 1, [&](uint32_t j) { return row[j]; });
    if (threadIdx.x == 0) {
        thresh[blockIdx.x] = T;
        cnt[blockIdx.x] = 0;
    }
}

// Selection among the rows handed on; SCREENED: they are ids only, and their
// canonical distances are computed here, a row per thread, sixteen loads in
// flight.  A query with too many or too few goes to redo[1 ..], counted in redo[0].
template <bool SCREENED>
__global__ void __launch_bounds__(SEL_T) knn_final_kernel(const float *__restrict__ Q, const float *__restrict__ X,
                                                          int ld, const uint32_t *__restrict__ q_self,
                                                          const uint64_t *__restrict__ cand,
                                                          const uint32_t *__restrict__ cand_ids,
                                                          const uint32_t *__restrict__ cnt, uint32_t k, uint32_t q_base,
                                                          uint32_t *__restrict__ out_ids, float *__restrict__ out_d,
                                                          uint32_t *redo, int *err) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *s_key = reinterpret_cast<uint64_t *>(smem); // KNN_CAP (distance, id)
    float4 *s_q = reinterpret_cast<float4 *>(s_key + KNN_CAP); // SCREENED: the query
    __shared__ SelectShared S;
    __shared__ uint64_t s_out[SEL_MAXK], s_tie[SEL_TIES];
    const uint32_t q = blockIdx.x, n = cnt[q];
    const uint32_t self = q_self ? q_self[q] : KCNA_NONE;
    if (n > KNN_CAP || n < k) {
        if (threadIdx.x == 0) redo[1 + atomicAdd(redo, 1u)] = q;
        return;
    }
    if (SCREENED) {
        const int nv = ld >> 2;
        for (int i = threadIdx.x; i < nv; i += SEL_T) s_q[i] = reinterpret_cast<const float4 *>(Q + (uint64_t)q * ld)[i];
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < n; j += SEL_T) {
            const uint32_t id = cand_ids[(uint64_t)q * KNN_CAP + j];
            const float4 *x = reinterpret_cast<const float4 *>(X + (uint64_t)id * ld);
            float acc = 0.f;
            for (int k0 = 0; k0 < nv; k0 += 16) {
                float4 v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = __ldg(x + min(k0 + u, nv - 1));
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    if (k0 + u < nv) acc = kcna_acc4(acc, s_q[k0 + u], v[u]);
            }
            s_key[j] = ((uint64_t)(id == self ? 0x7F800000u : __float_as_uint(acc)) << 32) | id;
        }
    } else {
        for (uint32_t j = threadIdx.x; j < n; j += SEL_T) s_key[j] = cand[(uint64_t)q * KNN_CAP + j];
    }
    __syncthreads();
    const uint64_t ob = (uint64_t)(q_base + q) * k;
    select_k(S, s_out, s_tie, n, k, [&](uint32_t j) { return (uint32_t)(s_key[j] >> 32); },
             [&](uint32_t j) { return (uint32_t)s_key[j]; }, out_ids + ob, out_d + ob, err);
}

__global__ void gather_rows_kernel(const float *__restrict__ X, int ld, const uint32_t *__restrict__ ids, uint32_t m,
                                   uint32_t n, float *__restrict__ dst, int *err) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t total = (uint64_t)m * (ld / 4);
    if (t >= total) return;
    uint32_t r = (uint32_t)(t / (ld / 4)), c = (uint32_t)(t % (ld / 4));
    uint32_t id = ids[r];
    if (id >= n) {
        kcna_set_err(err, KCNA_DERR_BOUNDS);
        return;
    }
    reinterpret_cast<float4 *>(dst)[t] = reinterpret_cast<const float4 *>(X + (uint64_t)id * ld)[c];
}

// Entry i of the queries done again: the query to exclude for it, or its k results to their place.
__global__ void redo_self_kernel(const uint32_t *__restrict__ list, uint32_t m, const uint32_t *__restrict__ q_self,
                                 uint32_t *__restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) out[i] = q_self[list[i]];
}
__global__ void redo_place_kernel(const uint32_t *__restrict__ list, uint64_t entries, uint32_t k,
                                  const uint32_t *__restrict__ ids, const float *__restrict__ d,
                                  uint32_t *__restrict__ out_ids, float *__restrict__ out_d) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= entries) return;
    const uint64_t to = (uint64_t)list[t / k] * k + t % k;
    out_ids[to] = ids[t];
    out_d[to] = d[t];
}

} // namespace

kcna_status kcna_gather_rows(kcna_ctx *c, const uint32_t *d_ids, uint32_t m, float *dst) {
    uint64_t total = (uint64_t)m * (c->ld / 4);
    if (!total) return KCNA_OK;
    gather_rows_kernel<<<kcna_div_up(total, 256), 256, 0, c->stream>>>(c->X, c->ld, d_ids, m, c->n, dst, c->d_err);
    KCNA_LAUNCHED(c);
    return kcna_cuda_check(c, cudaGetLastError(), "gather_rows");
}

// Every distance written, then selected from.
static kcna_status knn_all(kcna_ctx *c, const float *dQ, uint32_t m, const uint32_t *q_self, uint32_t k,
                           uint32_t *d_out_ids, float *d_out_d) {
    // distance rows for a batch of queries; batch bounded to ~1 GiB of scratch
    uint64_t row_bytes = (uint64_t)c->n * sizeof(float);
    uint32_t batch = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(m, (1ull << 30) / row_bytes));
    batch = std::max<uint32_t>(batch - batch % TQ, std::min<uint32_t>(batch, TQ));
    batch = std::min<uint32_t>(batch, 65535u * TQ); // grid.y limit of the distance tiles
    void *buf = nullptr;
    KCNA_TRY(kcna_scratch(c, (uint64_t)batch * row_bytes, &buf));
    float *D = (float *)buf;
    for (uint32_t q0 = 0; q0 < m; q0 += batch) {
        uint32_t mb = std::min(batch, m - q0);
        dim3 grid(kcna_div_up(c->n, TB), kcna_div_up(mb, TQ));
        dist_tile_kernel<DT_ALL><<<grid, 256, 0, c->stream>>>(dQ + (uint64_t)q0 * c->ld, mb, c->X, c->n, 1, (int)c->ld,
                                                             q_self ? q_self + q0 : nullptr,
                                                             DistOut{D, c->n, nullptr, nullptr, nullptr, 0});
        KCNA_LAUNCHED(c);
        select_kernel<<<mb, SEL_T, 0, c->stream>>>(D, c->n, c->n, k, q0, d_out_ids, d_out_d, c->d_err);
        KCNA_LAUNCHED(c);
        KCNA_TRY(kcna_cuda_check(c, cudaGetLastError(), "knn kernels"));
    }
    return KCNA_OK;
}

// The m queries of `list` (of n_q) done again the first way, together: one by
// one, each was a pass over the base with 31 of a tile's 32 query places empty
// (60 of 1,000 queries, 200,000 x 64 rows: 5.6 ms a call against 2.2 for doing
// all 1,000 again, 0.94 so).
static kcna_status knn_redo(kcna_ctx *c, const float *dQ, uint32_t n_q, const uint32_t *q_self, uint32_t k,
                            const uint32_t *list, uint32_t m, uint32_t *d_out_ids, float *d_out_d) {
    if (m == n_q) return knn_all(c, dQ, n_q, q_self, k, d_out_ids, d_out_d);
    float *q = nullptr, *od = nullptr;
    uint32_t *self = nullptr, *oi = nullptr;
    kcna_status st = kcna_alloc(c, &q, (size_t)m * c->ld, "queries done again");
    if (st == KCNA_OK && q_self) st = kcna_alloc(c, &self, m, "queries done again");
    if (st == KCNA_OK) st = kcna_alloc(c, &oi, (size_t)m * k, "queries done again");
    if (st == KCNA_OK) st = kcna_alloc(c, &od, (size_t)m * k, "queries done again");
    if (st == KCNA_OK) {
        gather_rows_kernel<<<kcna_div_up((uint64_t)m * (c->ld / 4), 256), 256, 0, c->stream>>>(dQ, (int)c->ld, list, m, n_q,
                                                                                              q, c->d_err);
        KCNA_LAUNCHED(c);
        if (self) {
            redo_self_kernel<<<kcna_div_up(m, 256), 256, 0, c->stream>>>(list, m, q_self, self);
            KCNA_LAUNCHED(c);
        }
        st = knn_all(c, q, m, self, k, oi, od);
    }
    if (st == KCNA_OK) {
        redo_place_kernel<<<kcna_div_up((uint64_t)m * k, 256), 256, 0, c->stream>>>(list, (uint64_t)m * k, k, oi, od,
                                                                                    d_out_ids, d_out_d);
        KCNA_LAUNCHED(c);
        st = kcna_cuda_check(c, cudaGetLastError(), "redo_place_kernel");
    }
    kcna_release(c, q); // later users run behind these kernels on the context's stream
    kcna_release(c, self);
    kcna_release(c, oi);
    kcna_release(c, od);
    return st;
}

// Whether the rows within a bound are found on tensor cores: from about 0.1 ms of FP32 work on.
static bool knn_screened(const kcna_ctx *c, uint32_t m) {
    return c->ld <= 128 && (uint64_t)m * c->n * c->ld >= (1ull << 30);
}

// A bound per query from a sample, the rows that may lie within it, selection among those.
static kcna_status knn_bounded(kcna_ctx *c, const float *dQ, uint32_t m, const uint32_t *q_self, uint32_t k, uint32_t s,
                               uint32_t *d_out_ids, float *d_out_d) {
    // queries at a time: their sampled distances within 1 GiB, as the distances of knn_all are
    const uint32_t batch = std::min<uint32_t>(m, std::min<uint32_t>(2048, (uint32_t)((1ull << 30) / (s * 4ull)) & ~31u));
    const uint32_t rank = std::max<uint32_t>(k, 32), stride = c->n / s;
    const bool screened = knn_screened(c, m);
    uint64_t *cand = nullptr;
    uint32_t *words = nullptr; // bounds, counts, and the queries to do again behind their number
    kcna_status st = kcna_alloc(c, &cand, ((uint64_t)batch * KNN_CAP + (screened ? 1 : 0)) / (screened ? 2 : 1), "k-NN lists");
    if (st == KCNA_OK) st = kcna_alloc(c, &words, 3 * (size_t)batch + 1, "k-NN bounds");
    const bool cached = s <= SEL_CACHE;
    const size_t fsm = KNN_CAP * 8 + (screened ? (size_t)c->ld * 4 : 0);
    if (st == KCNA_OK && cached) st = kcna_allow_smem(c, knn_bound_kernel<true>, (size_t)s * 4, "knn smem attr");
    if (st == KCNA_OK)
        st = screened ? kcna_allow_smem(c, knn_final_kernel<true>, fsm, "knn smem attr")
                      : kcna_allow_smem(c, knn_final_kernel<false>, fsm, "knn smem attr");
    uint32_t q0 = 0;
    for (; q0 < m && st == KCNA_OK; q0 += batch) {
        const uint32_t mb = std::min(batch, m - q0);
        void *buf = nullptr; // asked for each time: knn_all below may move the scratch
        if ((st = kcna_scratch(c, (uint64_t)batch * s * 4, &buf)) != KCNA_OK) break;
        float *D = (float *)buf;
        const float *Q = dQ + (uint64_t)q0 * c->ld;
        const uint32_t *self = q_self ? q_self + q0 : nullptr;
        uint32_t *thresh = words, *cnt = words + batch, *redo = words + 2 * (size_t)batch;
        cudaMemsetAsync(redo, 0, 4, c->stream);
        dist_tile_kernel<DT_SAMPLE><<<dim3(kcna_div_up(s, TB), kcna_div_up(mb, TQ)), 256, 0, c->stream>>>(
            Q, mb, c->X, s, stride, (int)c->ld, self, DistOut{D, s, nullptr, nullptr, nullptr, 0});
        if (cached)
            knn_bound_kernel<true><<<mb, SEL_T, (size_t)s * 4, c->stream>>>(D, s, rank, thresh, cnt);
        else
            knn_bound_kernel<false><<<mb, SEL_T, 0, c->stream>>>(D, s, rank, thresh, cnt);
        c->launches += 2;
        if (screened) {
            if ((st = kcna_knn_filter(c, Q, mb, thresh, reinterpret_cast<uint32_t *>(cand), cnt, KNN_CAP)) != KCNA_OK) break;
            knn_final_kernel<true><<<mb, SEL_T, fsm, c->stream>>>(Q, c->X, (int)c->ld, self, nullptr,
                                                                  reinterpret_cast<uint32_t *>(cand), cnt, k, q0,
                                                                  d_out_ids, d_out_d, redo, c->d_err);
        } else {
            dist_tile_kernel<DT_FILTER><<<dim3(kcna_div_up(c->n, TB), kcna_div_up(mb, TQ)), 256, 0, c->stream>>>(
                Q, mb, c->X, c->n, 1, (int)c->ld, self, DistOut{nullptr, 0, thresh, cand, cnt, KNN_CAP});
            knn_final_kernel<false><<<mb, SEL_T, fsm, c->stream>>>(Q, c->X, (int)c->ld, self, cand, nullptr, cnt, k, q0,
                                                                   d_out_ids, d_out_d, redo, c->d_err);
            c->launches += 1;
        }
        c->launches += 1;
        uint32_t again = 0;
        st = kcna_cuda_check(c, cudaGetLastError(), "knn kernels");
        if (st == KCNA_OK) st = kcna_cuda_check(c, cudaMemcpyAsync(&again, redo, 4, cudaMemcpyDeviceToHost, c->stream), "d2h");
        if (st == KCNA_OK) st = kcna_cuda_check(c, cudaStreamSynchronize(c->stream), "knn sync");
        if (st == KCNA_OK && again)
            st = knn_redo(c, Q, mb, self, k, redo + 1, again, d_out_ids + (uint64_t)q0 * k, d_out_d + (uint64_t)q0 * k);
        if (st != KCNA_OK) break;
    }
    kcna_release(c, cand);
    kcna_release(c, words);
    if (st == KCNA_E_OOM) { // a nearly full device: the rest the first way
        c->err.clear();
        return knn_all(c, dQ + (uint64_t)q0 * c->ld, m - q0, q_self ? q_self + q0 : nullptr, k,
                       d_out_ids + (uint64_t)q0 * k, d_out_d + (uint64_t)q0 * k);
    }
    return st;
}

// Whether the bound pays, by the time of either way; 3,360 calls were timed
// both ways (8 to 960 dimensions, 16,384 to 2,000,000 rows, 1 to 4,000 queries, k =
// 10 to 1,000).  This takes the slower way by 0.3 % on average, 29 % at worst; a
// bound from 40,960 rows on took it by 29 %, at worst at nearly nine times the time
// (25,000 x 8 rows, 4,000 queries, k = 300: 4.7 ms against 0.54).
static bool knn_bound_pays(const kcna_ctx *c, uint32_t m, uint32_t k, uint64_t sample) {
    const double n = c->n, ld = c->ld, q = m, s = (double)sample;
    const bool passes = k > SEL_QUICK; // selection by histogram passes
    if (!knn_screened(c, m)) {
        // Every distance is computed either way; what is saved is writing and
        // selecting from them, against launches, the sample and the lists' atomics,
        // which short rows do not hide.  One query, k = 10, both ways: 41,000 x 960
        // rows 210 us (first way) and 306, 240,000 x 32 115 and 108, 700,000 x 128 415
        // and 319; 1,000 queries, 130,000 x 8: 430 and 1,147.
        const double from = passes ? (m <= 4 ? 65536 : 180000) : 262144;
        return n >= (ld <= 64 && m > (passes ? 16u : 4u) ? 2 * from : from);
    }
    // Microseconds, fitted; mean error 8 %.  First way: launches and waits, one
    // block's selection, and per pair the write, the selection and the FP32 chain.
    // Bound: the rows once, a pass over them per 128 queries, the sample, and a list
    // of about `len` rows a query, appended and rescored.
    const double len = std::max<uint32_t>(k, 32) * n / s;
    const double first = 57 + n * ((passes ? 7.4e-4 : 1.6e-4) + 1.3e-6 * ld + q * ((passes ? 4.9e-6 : 2e-6) + 7.2e-8 * ld));
    const double bound = 150 + n * (2.4e-6 * ld + 6.7e-5 * (m / 128 + 1)) + 2.9e-4 * s +
                         q * (0.08 + s * (5.6e-6 + 3.4e-8 * ld) + len * (8.7e-5 + 8.1e-7 * ld));
    return bound < first;
}

kcna_status kcna_knn_device(kcna_ctx *c, const float *dQ, uint32_t m, const uint32_t *q_self, uint32_t k,
                            uint32_t *d_out_ids, float *d_out_d) {
    if (k == 0 || k > SEL_MAXK || k > c->n) return kcna_fail(c, KCNA_E_ARG, "knn: k must be in [1, min(1024, n)]");
    if (q_self && k >= c->n) return kcna_fail(c, KCNA_E_ARG, "knn: k must be < n when self is excluded");
    // rows sampled for the bound: about 4,096 of n then lie within it
    const uint64_t s = std::max<uint64_t>(std::max<uint64_t>(2048, 2 * (uint64_t)k),
                                          (std::max<uint64_t>(k, 32) * c->n + 4095) / 4096);
    const bool bounded = 2 * s <= c->n && s <= (1u << 18) && knn_bound_pays(c, m, k, s);
    if (bounded) return knn_bounded(c, dQ, m, q_self, k, (uint32_t)s, d_out_ids, d_out_d);
    return knn_all(c, dQ, m, q_self, k, d_out_ids, d_out_d);
}
