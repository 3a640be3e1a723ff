// kcna_cagra.cu - CAGRA-style rank prune of the candidate pools into the graph.
//
// The reference's BuildCagra (src/kgraph.cpp:2818-2829; no build function
// calls it there) turns each node's K nearest pool entries into a graph of
// about K / 2 edges by counting detours instead of comparing distances:
//   route   (CagraComputeRoute, :2665-2757) route[j] = number of pairs (k, l)
//           with pool_i[k]'s own entry l equal to pool_i[j] and k, l < j;
//   keep    the prune_K = K / 2 entries with the fewest detours, equal counts
//           in rank order (sort_indexes, :62-76);
//   reverse (CagraReverse, :2759-2788) every kept edge i -> w gives w the entry
//           (i, rank of w in i's kept list), taken by increasing rank; equal
//           ranks by increasing source id (the reference sorts by rank alone,
//           leaving that order unspecified);
//   merge   (CagraMerge, :2790-2816) kept and reverse entries alternate until
//           prune_K are placed, one more when the last step places both;
//           a reverse entry carries d(i, source).
// With Ki = min(K, pool count), entries past a pool's count are absent.
//
// GPU form, four steps on the context's stream:
//   cagra_route_kernel  warp per node up to K = 64 (cagra_route_warps), else
//                       block per node: the node's first Ki pool ids in a
//                       shared-memory hash table (id -> rank), the K x K
//                       two-hop entries looked up in it (warp per one-hop
//                       node, lanes over its pool: coalesced 8-byte keys),
//                       detours counted with shared atomics, (route, rank)
//                       keys sorted, the kept ranks written and each kept
//                       target's in-degree counted;
//   exclusive scan of the in-degrees (kcna_graph.cu);
//   cagra_rev_fill_kernel  thread per kept edge: (rank << 32 | source) into
//                       the target's segment;
//   cagra_merge_warp_kernel / cagra_merge_kernel  warp per node with up to 256
//                       reverse entries, else (and for every node below
//                       CG_MERGE_WARPS of them) block per node: the smallest
//                       reverse keys (the segment sorted in shared memory, or
//                       streamed through a 1024-key best set for hubs), then
//                       the interleaved row with every slot's position computed
//                       in closed form.
// The routes are bound by issue (100,000 rows, K = 64: 0.76 a cycle, integer pipe
// 51 %).  A node's work is small (K = 64: 4,096 look-ups, some 32 reverse keys), so a
// block of 256 threads per node spent its time at barriers: 2.8 and 2.1 ms for
// 150,007 nodes at K = 64, 1.6 and 0.3 with a warp per node.
#include <algorithm>

#include "kcna_internal.h"
#include "kcna_sort.cuh"

namespace {

constexpr int CG_THREADS = 256;
constexpr uint32_t CG_EMPTY = 0xFFFFFFFFu;
constexpr int CG_BEST = 1024; // merge: best-set size when a segment is streamed

__device__ __forceinline__ uint32_t cg_hash(uint32_t id) { return (id * 0x9E3779B1u) >> 7; }

// Kept ranks of node i (fwd[i * PK + r] = pool index) and the kept targets'
// in-degrees; NT threads per node.  Shared, per node: sort keys[P2], ids[K],
// route[K], table keys[HS], table ranks[HS] (P2 = K rounded up to a power of
// two).  The K x K look-ups are what it does, most of them misses, and a warp
// takes as many steps as its unluckiest lane: HS = 8 P2 slots, an eighth full
// (2 P2: 3.5 ms for 150,007 nodes at K = 64 against 1.6; 28 against 19 ms a
// call at K = 200, 212 against 121 for 40,000 nodes at K = 1,000).
// Warp or block per node: whole calls for 150,007 nodes, warp / block, K = 64
// 2.26 / 2.82 ms, K = 100 8.3 / 6.0, for 11,132 nodes 0.30 / 0.32 and 0.81 /
// 0.55: from P2 = 128 on the tables of eight warps leave 24 warps an SM.  Few
// nodes leave SMs idle with a warp each: 600 nodes, K = 64 0.133 / 0.098 ms, 4,500
// 0.180 / 0.167, 9,000 0.231 / 0.240; K = 33, 2,000 0.121 / 0.114, 4,500 0.128 / 0.138;
// K = 16, 1,000 equal, 3,000 0.096 / 0.106.
constexpr uint32_t CG_WARP_K = 64;
constexpr bool cagra_route_warps(uint32_t N, uint32_t K) { return K <= CG_WARP_K && N >= 96 * K; }
// Merge: one launch with a block for every node below this many nodes, a warp a
// node and a second launch for the hubs from there on (600 nodes 0.092 / 0.098 ms a
// call, 1,000 equal, 2,000 0.139 / 0.129).
constexpr uint32_t CG_MERGE_WARPS = 1024;
constexpr uint32_t cagra_slots(uint32_t P2) { return 8 * P2; }
__host__ __device__ constexpr size_t cagra_route_bytes(uint32_t K, uint32_t P2, uint32_t HS) {
    return (size_t)P2 * 8 + (((size_t)K * 8 + 15) & ~(size_t)15) + (size_t)HS * 6;
}

template <int NT>
__global__ void __launch_bounds__(CG_THREADS) cagra_route_kernel(const uint64_t *__restrict__ pool,
                                                                 const uint32_t *__restrict__ pool_cnt, uint32_t cap,
                                                                 uint32_t N, uint32_t K, uint32_t PK, uint32_t P2,
                                                                 uint32_t HS, uint16_t *__restrict__ fwd,
                                                                 uint32_t *__restrict__ indeg,
                                                                 int *err) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NODES = CG_THREADS / NT, NW = NT / 32; // per block; warps per node
    const int tid = threadIdx.x % NT, warp = tid >> 5, lane = tid & 31;
    unsigned char *base = smem + (threadIdx.x / NT) * cagra_route_bytes(K, P2, HS);
    uint64_t *skey = reinterpret_cast<uint64_t *>(base);        // P2
    uint32_t *ids = reinterpret_cast<uint32_t *>(skey + P2);    // K
    uint32_t *route = ids + K;                                  // K
    uint32_t *hkey = reinterpret_cast<uint32_t *>(base + cagra_route_bytes(K, P2, HS) - (size_t)HS * 6); // HS
    uint16_t *hval = reinterpret_cast<uint16_t *>(hkey + HS);   // HS
    auto sync = [] {
        if (NT == 32)
            __syncwarp();
        else
            __syncthreads();
    };
    for (uint32_t i = blockIdx.x * NODES + threadIdx.x / NT; i < N; i += gridDim.x * NODES) {
        const uint32_t Ki = min(K, pool_cnt[i]);
        for (uint32_t h = tid; h < HS; h += NT) hkey[h] = CG_EMPTY;
        sync();
        for (uint32_t j = tid; j < Ki; j += NT) {
            const uint32_t id = kcna_key_id(pool[(uint64_t)i * cap + j]);
            ids[j] = id;
            route[j] = 0;
            uint32_t h = cg_hash(id) & (HS - 1);
            for (uint32_t probe = 0; probe < HS; ++probe, h = (h + 1) & (HS - 1))
                if (atomicCAS(&hkey[h], CG_EMPTY, id) == CG_EMPTY) {
                    hval[h] = (uint16_t)j;
                    break;
                }
        }
        sync();
        // two-hop entries: pool_i[k]'s entry l, looked up among pool_i's ranks
        // four one-hop nodes at a time: their counts and entries are in flight together
        for (uint32_t k0 = warp; k0 < Ki; k0 += 4 * NW) {
            uint32_t Kl[4], most = 0;
            const uint64_t *p1[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t k = k0 + u * NW, one = k < Ki ? ids[k] : 0u;
                if (one >= N) kcna_set_err(err, KCNA_DERR_BOUNDS);
                Kl[u] = k < Ki && one < N ? min(K, __ldg(pool_cnt + one)) : 0u;
                p1[u] = pool + (uint64_t)(one < N ? one : 0u) * cap;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) most = max(most, Kl[u]);
            for (uint32_t l = lane; l < most; l += 32) {
                uint64_t e[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) e[u] = l < Kl[u] ? __ldg(p1[u] + l) : 0u;
                uint32_t two[4], h[4], key[4]; // the first probes side by side
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    two[u] = l < Kl[u] ? kcna_key_id(e[u]) : CG_EMPTY;
                    h[u] = cg_hash(two[u]) & (HS - 1);
                    key[u] = hkey[h[u]];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    for (uint32_t probe = 0; probe < HS && key[u] != CG_EMPTY && key[u] != two[u]; ++probe) {
                        h[u] = (h[u] + 1) & (HS - 1);
                        key[u] = hkey[h[u]];
                    }
                    if (key[u] == CG_EMPTY || key[u] != two[u]) continue;
                    const uint32_t j = hval[h[u]];
                    if (j > max(k0 + u * NW, l)) atomicAdd(&route[j], 1u);
                }
            }
        }
        sync();
        for (uint32_t j = tid; j < P2; j += NT) skey[j] = j < Ki ? ((uint64_t)route[j] << 32) | j : ~0ull;
        if (NT == 32)
            kcna_warp_bitonic(skey, (int)P2);
        else
            kcna_cta_bitonic(skey, (int)P2);
        sync();
        const uint32_t nk = min(PK, Ki);
        for (uint32_t r = tid; r < nk; r += NT) {
            const uint32_t j = (uint32_t)(skey[r] & 0xFFFFFFFFull);
            fwd[(uint64_t)i * PK + r] = (uint16_t)j;
            const uint32_t w = ids[j];
            if (w < N)
                atomicAdd(indeg + w, 1u);
            else
                kcna_set_err(err, KCNA_DERR_BOUNDS);
        }
        sync(); // the next node reuses the arrays
    }
}

// Reverse entries: thread per kept edge (i, r) -> target's segment.
__global__ void cagra_rev_fill_kernel(const uint64_t *__restrict__ pool, const uint32_t *__restrict__ pool_cnt,
                                      uint32_t cap, uint32_t N, uint32_t K, uint32_t PK,
                                      const uint16_t *__restrict__ fwd, const uint64_t *__restrict__ off,
                                      uint32_t *__restrict__ cursor, uint64_t *__restrict__ rev) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (uint64_t)N * PK) return;
    const uint32_t i = (uint32_t)(t / PK), r = (uint32_t)(t % PK);
    if (r >= min(PK, min(K, pool_cnt[i]))) return;
    const uint32_t w = kcna_key_id(pool[(uint64_t)i * cap + fwd[t]]);
    if (w >= N) return; // counted as an error by the route kernel
    const uint64_t pos = off[w] + atomicAdd(cursor + w, 1u);
    rev[pos] = ((uint64_t)r << 32) | i;
}

// Row of node i: kept entry t at t + min(t, m), reverse entry t at
// min(t + 1, nk) + t; a step t runs while the row holds fewer than PK
// entries, size_before(t) = min(t, nk) + min(t, m).  s: the node's smallest
// reverse keys (rank, source) in order; NT threads.
template <class R>
struct CagraRow {
    R rows;
    const uint64_t *pool;
    const uint32_t *pool_cnt;
    uint32_t cap, N, K, PK;
    const uint16_t *fwd;
    const uint64_t *off, *rev;
    uint32_t *g_ids;
    float *g_dist;
    uint32_t *g_deg;
    uint32_t W;
    int *err;
};
template <int NT, class R>
__device__ __forceinline__ void cagra_row(const CagraRow<R> &a, uint32_t i, uint32_t nk, uint32_t m, uint32_t T,
                                          const uint64_t *s) {
    const uint32_t tid = threadIdx.x % NT, need = min(T, m), deg = min(T, nk) + need;
    if (deg > a.W) {
        if (tid == 0) kcna_set_err(a.err, KCNA_DERR_DEGREE);
        return;
    }
    uint32_t *gi = a.g_ids + (uint64_t)i * a.W;
    float *gd = a.g_dist + (uint64_t)i * a.W;
    for (uint32_t t = tid; t < min(T, nk); t += NT) {
        const uint64_t key = a.pool[(uint64_t)i * a.cap + a.fwd[(uint64_t)i * a.PK + t]];
        const uint32_t pos = t + min(t, m);
        gi[pos] = kcna_key_id(key);
        gd[pos] = kcna_key_dist(key);
    }
    for (uint32_t t = tid; t < need; t += NT) {
        const uint32_t src = (uint32_t)(s[t] & 0xFFFFFFFFull);
        const uint32_t pos = min(t + 1, nk) + t;
        gi[pos] = src;
        gd[pos] = rows_l2(a.rows, i, src);
    }
    for (uint32_t p = deg + tid; p < a.W; p += NT) gi[p] = 0xFFFFFFFFu;
    if (tid == 0) a.g_deg[i] = deg;
}
// steps of node i: they run while fewer than PK entries are placed
__device__ __forceinline__ uint32_t cagra_steps(uint32_t nk, uint32_t m, uint32_t PK) {
    uint32_t T = 0;
    while ((T < nk || T < m) && min(T, nk) + min(T, m) < PK) ++T;
    return T;
}

constexpr int CG_MW = 4;             // warps per block
constexpr uint32_t CG_WARP_REV = 256; // reverse entries a warp sorts

template <class R>
__global__ void __launch_bounds__(CG_MW * 32) cagra_merge_warp_kernel(CagraRow<R> a, uint32_t *list,
                                                                      uint32_t *list_cnt) {
    __shared__ uint64_t s_all[CG_MW][CG_WARP_REV];
    uint64_t *s = s_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    for (uint32_t i = blockIdx.x * CG_MW + (threadIdx.x >> 5); i < a.N; i += gridDim.x * CG_MW) {
        const uint32_t nk = min(a.PK, min(a.K, a.pool_cnt[i]));
        const uint64_t b = a.off[i];
        const uint32_t m = (uint32_t)(a.off[i + 1] - b);
        if (m > CG_WARP_REV) {
            if (lane == 0) list[atomicAdd(list_cnt, 1u)] = i;
            continue;
        }
        if (m <= 32) { // in registers
            const uint64_t k = kcna_warp_sort32((uint32_t)lane < m ? a.rev[b + lane] : ~0ull);
            if ((uint32_t)lane < m) s[lane] = k;
            __syncwarp();
        } else {
            for (uint32_t j = lane; j < m; j += 32) s[j] = a.rev[b + j];
            __syncwarp();
            kcna_warp_sort_n(s, (int)m);
        }
        cagra_row<32>(a, i, nk, m, cagra_steps(nk, m, a.PK), s);
        __syncwarp(); // the next node reuses the keys
    }
}

// the nodes of `list`, or all (null)
template <class R>
__global__ void __launch_bounds__(CG_THREADS) cagra_merge_kernel(CagraRow<R> a, const uint32_t *__restrict__ list,
                                                                 const uint32_t *__restrict__ list_cnt) {
    __shared__ uint64_t s[2 * CG_BEST];
    const int tid = threadIdx.x;
    const uint32_t n_list = list ? *list_cnt : a.N;
    for (uint32_t li = blockIdx.x; li < n_list; li += gridDim.x) {
        const uint32_t i = list ? list[li] : li;
        const uint32_t nk = min(a.PK, min(a.K, a.pool_cnt[i]));
        const uint64_t b = a.off[i];
        const uint32_t m = (uint32_t)(a.off[i + 1] - b);
        __syncthreads(); // the previous node's keys are read
        // the smallest (rank, source) keys in s[0 ..)
        if (m <= 2 * CG_BEST) {
            uint32_t p2 = 1;
            while (p2 < m) p2 <<= 1;
            for (uint32_t j = tid; j < p2; j += CG_THREADS) s[j] = j < m ? a.rev[b + j] : ~0ull;
            kcna_cta_bitonic(s, (int)p2);
        } else {
            for (uint32_t j = tid; j < CG_BEST; j += CG_THREADS) s[j] = ~0ull;
            for (uint32_t c0 = 0; c0 < m; c0 += CG_BEST) {
                __syncthreads();
                for (uint32_t j = tid; j < CG_BEST; j += CG_THREADS)
                    s[CG_BEST + j] = c0 + j < m ? a.rev[b + c0 + j] : ~0ull;
                kcna_cta_bitonic(s, 2 * CG_BEST);
            }
        }
        cagra_row<CG_THREADS>(a, i, nk, m, cagra_steps(nk, m, a.PK), s);
    }
}

} // namespace

kcna_status kcna_cagra_prune(kcna_ctx *c, const kcna_params *p) {
    if (!c->has_pools) return kcna_fail(c, KCNA_E_STATE, "prune: no pools (run NN-descent or set pools first)");
    const uint32_t K = p->K, PK = K / 2, N = c->n;
    if (K < 2 || K > c->cap || K > 1024)
        return kcna_fail(c, KCNA_E_ARG, "CAGRA prune: K must be in [2, min(pool capacity, 1024)]");
    KCNA_TRY(kcna_graph_alloc(c, std::max<uint32_t>(c->W, PK + 1)));
    uint32_t P2 = 1;
    while (P2 < K) P2 <<= 1;
    uint16_t *fwd = nullptr;
    uint32_t *indeg = nullptr, *cursor = nullptr;
    uint64_t *off = nullptr, *rev = nullptr;
    kcna_status s = KCNA_OK;
    auto cleanup = [&]() {
        kcna_release(c, fwd);
        kcna_release(c, indeg);
        kcna_release(c, cursor);
        kcna_release(c, off);
        kcna_release(c, rev);
    };
    if ((s = kcna_alloc(c, &fwd, (uint64_t)N * PK, "CAGRA kept ranks")) != KCNA_OK) return cleanup(), s;
    if ((s = kcna_alloc(c, &indeg, N, "CAGRA in-degrees")) != KCNA_OK) return cleanup(), s;
    if ((s = kcna_alloc(c, &cursor, N, "CAGRA cursors")) != KCNA_OK) return cleanup(), s;
    if ((s = kcna_alloc(c, &off, (uint64_t)N + 1, "CAGRA offsets")) != KCNA_OK) return cleanup(), s;
    if ((s = kcna_phase_begin(c)) != KCNA_OK) return cleanup(), s;
    cudaMemsetAsync(indeg, 0, (size_t)N * 4, c->stream);
    cudaMemsetAsync(cursor, 0, (size_t)N * 4, c->stream);
    const uint32_t sms = (uint32_t)std::max(c->num_sms, 1);
    auto route = [&](auto kern, uint32_t nodes) -> kcna_status { // nodes per block
        const uint32_t HS = cagra_slots(P2);
        const size_t sm = cagra_route_bytes(K, P2, HS) * nodes;
        int per_sm = 0;
        KCNA_TRY(kcna_allow_smem(c, kern, sm, "cagra smem attr"));
        KCNA_TRY(kcna_cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, CG_THREADS, sm),
                                 "cagra occupancy"));
        const uint32_t grid = std::min(kcna_div_up(N, nodes), sms * (uint32_t)std::max(per_sm, 1));
        kern<<<grid, CG_THREADS, sm, c->stream>>>(c->pool, c->pool_cnt, c->cap, N, K, PK, P2, HS, fwd, indeg, c->d_err);
        KCNA_LAUNCHED(c);
        return kcna_cuda_check(c, cudaGetLastError(), "cagra_route_kernel");
    };
    s = cagra_route_warps(N, K) ? route(cagra_route_kernel<32>, CG_THREADS / 32) : route(cagra_route_kernel<CG_THREADS>, 1);
    if (s != KCNA_OK) return cleanup(), s;
    uint64_t E = 0;
    if ((s = kcna_exclusive_scan_u32(c, indeg, N, off, &E)) != KCNA_OK) return cleanup(), s;
    if ((s = kcna_alloc(c, &rev, std::max<uint64_t>(E, 1), "CAGRA reverse entries")) != KCNA_OK) return cleanup(), s;
    cagra_rev_fill_kernel<<<kcna_div_up((uint64_t)N * PK, 256), 256, 0, c->stream>>>(c->pool, c->pool_cnt, c->cap, N,
                                                                                      K, PK, fwd, off, cursor, rev);
    KCNA_LAUNCHED(c);
    // nodes with many reverse entries are queued in the spent in-degrees
    uint32_t *list_cnt = reinterpret_cast<uint32_t *>(c->counters + 20);
    cudaMemsetAsync(list_cnt, 0, 4, c->stream);
    auto merge = [&](auto rows) {
        const CagraRow<decltype(rows)> a{rows, c->pool, c->pool_cnt, c->cap,  N,        K,        PK,   fwd,
                                         off,  rev,     c->g_ids,    c->g_dist, c->g_deg, c->W, c->d_err};
        if (N < CG_MERGE_WARPS) {
            cagra_merge_kernel<<<N, CG_THREADS, 0, c->stream>>>(a, nullptr, nullptr);
            KCNA_LAUNCHED(c);
            return;
        }
        cagra_merge_warp_kernel<<<std::min(kcna_div_up(N, CG_MW), sms * 12), CG_MW * 32, 0, c->stream>>>(a, indeg,
                                                                                                         list_cnt);
        cagra_merge_kernel<<<std::min(N, sms * 4), CG_THREADS, 0, c->stream>>>(a, indeg, list_cnt);
        c->launches += 2;
    };
    if (c->bf16_exact)
        merge(RowsB16{c->Xh, (int)c->ld});
    else
        merge(RowsF32{c->X, (int)c->ld});
    s = kcna_cuda_check(c, cudaGetLastError(), "CAGRA kernels");
    if (s == KCNA_OK) s = kcna_phase_end(c, KCNA_PHASE_PRUNE);
    if (s == KCNA_OK) s = kcna_cuda_check(c, cudaStreamSynchronize(c->stream), "CAGRA sync");
    cleanup();
    if (s == KCNA_OK) c->has_graph = true;
    return s;
}
