// kcna_nnd.cu - NN-descent on device-resident pools.
//
// Replaces the KGraphConstructor constructor loop (src/kgraph.cpp:1281-1459):
// init (:1001-1044), join (:1097-1117 with Nhood::join :970-987 and
// parallel_try_insert :948-967), update (:1118-1202) and the per-iteration
// statistics / stop rule (:1365-1426).
//
// GPU form of one iteration:
//   join    one warp per node n (a block for a node of more than 64 rows):
//           gather the node's new list A and old list B, compute every pair
//           of A x A (i < j) and A x B with the canonical FMA-chain distance
//           in register tiles (rows staged through shared memory), and emit
//           each pair to both endpoints' candidate buffers when it is within
//           that endpoint's radius.  Candidates of one target from one node
//           are written as one contiguous run after a single atomicAdd.
//   merge   the candidates a node's pool lacks, each once, put in by rank, the
//           best `limit` kept; new entries carry flag=new (the reference's
//           InsertIntoPool :261-298 semantics applied to a batch).
//           merge_set_kernel: four warps per node, the distinct ones in a
//           hash table, ranks from counts, no sort; merge_kernel: a block for
//           a node of more than 892; merge_warp_kernel: the few of a
//           refinement round, sorted by a warp.
//   sample  the update step: M (prefix holding S new entries), radiusM, the
//           forward new/old lists and reverse lists (atomics, capped buffers,
//           random subset of R chosen in the join).
// The reference inserts into locked pools while joining, so its result depends
// on thread timing; this batched form inserts all of an iteration's
// candidates at its end.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <random>

#include "kcna_internal.h"
#include "kcna_join.cuh"
#include "kcna_pairs.cuh"
#include "kcna_sort.cuh"

namespace {

// ---------------------------------------------------------------------------
// init: S random pool entries + 2S random ids as the first new list.
// GenRandom (src/kgraph.cpp:82-110): size values < N-size, sorted, made
// strictly increasing, shifted by a random offset mod N.  Done per warp with a
// bitonic sort and a prefix maximum (a[i] = i + max_{j<=i}(a[j]-j)).
// ---------------------------------------------------------------------------
__device__ void warp_gen_random(uint64_t seed, uint64_t stream, uint32_t size, uint32_t N, uint32_t *s_out,
                                uint64_t *s_tmp) {
    const int lane = kcna_lane();
    if (N == size) {
        for (uint32_t i = lane; i < size; i += 32) s_out[i] = i;
        __syncwarp();
        return;
    }
    int p = kcna_pow2_ceil_d((int)size);
    for (int i = lane; i < p; i += 32)
        s_tmp[i] = i < (int)size ? (uint64_t)(kcna_rand32(seed, stream, i) % (N - size)) : KCNA_EMPTY_KEY;
    kcna_warp_bitonic(s_tmp, p);
    // prefix max of a[j]-j over j, chunk by chunk of 32
    int64_t carry = INT64_MIN;
    for (uint32_t base = 0; base < size; base += 32) {
        uint32_t i = base + lane;
        int64_t v = i < size ? (int64_t)s_tmp[i] - (int64_t)i : INT64_MIN;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int64_t u = __shfl_up_sync(KCNA_FULL, v, o);
            if (lane >= o && u > v) v = u;
        }
        if (carry > v) v = carry;
        carry = __shfl_sync(KCNA_FULL, v, 31);
        if (i < size) s_out[i] = (uint32_t)((int64_t)i + v);
    }
    __syncwarp();
    uint32_t off = kcna_rand32(seed, stream, 0xFFFFFFull) % N;
    for (uint32_t i = lane; i < size; i += 32) s_out[i] = (uint32_t)(((uint64_t)s_out[i] + off) % N);
    __syncwarp();
}

// keep: entries a pool starts with, min(S, L).
__global__ void __launch_bounds__(128) init_kernel(const float *__restrict__ X, int ld, uint32_t N, uint32_t S,
                                                   uint32_t keep, uint32_t cap, uint64_t seed,
                                                   uint64_t *__restrict__ pool,
                                                   uint32_t *__restrict__ pool_cnt,
                                                   uint32_t *__restrict__ fwd_new, uint32_t fwd_new_cap,
                                                   uint32_t *__restrict__ fwd_new_cnt) {
    __shared__ uint32_t s_ids[4][128];
    __shared__ uint64_t s_tmp[4][128];
    const int w = threadIdx.x >> 5, lane = kcna_lane();
    const uint32_t n = blockIdx.x * 4 + w;
    if (n >= N) return;
    // first new list: 2S random ids (may include n itself, as in the reference)
    warp_gen_random(seed, (uint64_t)n * 4 + 0, 2 * S, N, s_ids[w], s_tmp[w]);
    for (uint32_t i = lane; i < 2 * S; i += 32) fwd_new[(uint64_t)n * fwd_new_cap + i] = s_ids[w][i];
    if (lane == 0) fwd_new_cnt[n] = 2 * S;
    __syncwarp();
    // pool: S+1 random ids, n dropped, of the first S the nearest `keep`
    warp_gen_random(seed, (uint64_t)n * 4 + 1, S + 1, N, s_ids[w], s_tmp[w]);
    uint64_t key = KCNA_EMPTY_KEY;
    {
        uint32_t r = lane <= (int)S ? s_ids[w][lane] : n;
        bool other = lane <= (int)S && r != n;
        unsigned mk = __ballot_sync(KCNA_FULL, other);
        int pos = __popc(mk & kcna_lanemask_lt());
        if (other && pos < (int)S) {
            float dd = kcna_l2_ldg(X + (uint64_t)r * ld, X + (uint64_t)n * ld, ld);
            key = kcna_key(dd, r, (uint32_t)(KCNA_FLAG_NEW | KCNA_FLAG_ISNEW));
        }
    }
    key = kcna_warp_sort32(key);
    uint64_t *pr = pool + (uint64_t)n * cap;
    for (uint32_t i = lane; i < cap; i += 32) pr[i] = (i == (uint32_t)lane && i < keep) ? key : KCNA_EMPTY_KEY;
    if (lane == 0) pool_cnt[n] = keep;
}

// ---------------------------------------------------------------------------
// join
// ---------------------------------------------------------------------------
constexpr int JT = 256;      // threads per join block
constexpr int JCOLS = 64;    // columns per tile chunk
constexpr int JKC = 32;      // floats per k chunk
constexpr int JKP = JKC + 4; // padded row pitch in shared memory

template <int RI, class R> // rows per thread = RI, tile rows = 32 * RI
__device__ void join_tiles(const JoinArgs &a, const R &rows, uint32_t node, const uint32_t *s_A, int na, const uint32_t *s_B, int nb,
                           float *s_As, float *s_Bs, float *s_D, const float *s_radA, unsigned *s_emit) {
    constexpr int RA = 32 * RI;
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3; // 8 col groups x 32 row groups
    const int ncol = na + nb;
    const int ld = a.ld;
    for (int c0 = 0; c0 < ncol; c0 += JCOLS) {
        // rows that can pair with this chunk: i < min(na, c0+JCOLS) (i < j inside A)
        const int rows_needed = min(na, c0 + JCOLS);
        float acc[RI][8];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
        for (int k0 = 0; k0 < ld; k0 += JKC) {
            // stage A rows (RA x 32 floats) and chunk columns (64 x 32 floats)
            for (int idx = tid; idx < RA * (JKC / 4); idx += JT) {
                int r = idx >> 3, c = (idx & 7) * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < rows_needed && k0 + c < ld) v = rows.ld4(s_A[r], (k0 + c) >> 2);
                *reinterpret_cast<float4 *>(s_As + r * JKP + c) = v;
            }
            for (int idx = tid; idx < JCOLS * (JKC / 4); idx += JT) {
                int r = idx >> 3, c = (idx & 7) * 4;
                int col = c0 + r;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (col < ncol && k0 + c < ld) {
                    uint32_t id = col < na ? s_A[col] : s_B[col - na];
                    v = rows.ld4(id, (k0 + c) >> 2);
                }
                *reinterpret_cast<float4 *>(s_Bs + r * JKP + c) = v;
            }
            __syncthreads();
            const int kend = min(JKC, ld - k0);
            for (int k = 0; k < kend; k += 4) {
                float4 ra[RI], cb[8];
#pragma unroll
                for (int i = 0; i < RI; ++i) ra[i] = *reinterpret_cast<const float4 *>(s_As + (ty + 32 * i) * JKP + k);
#pragma unroll
                for (int j = 0; j < 8; ++j) cb[j] = *reinterpret_cast<const float4 *>(s_Bs + (tx + 8 * j) * JKP + k);
#pragma unroll
                for (int i = 0; i < RI; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = kcna_acc4(acc[i][j], ra[i], cb[j]);
            }
            __syncthreads();
        }
        // distances of the chunk to shared memory: s_D[row][col], pitch JCOLS+1
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) s_D[(ty + 32 * i) * (JCOLS + 1) + tx + 8 * j] = acc[i][j];
        __syncthreads();
        // emission: warp w handles row targets, then column targets
        const int warp = tid >> 5, lane = tid & 31, nwarp = JT / 32;
        const int cend = min(JCOLS, ncol - c0);
        // row targets: A[i] receives column ids
        for (int i = warp; i < rows_needed; i += nwarp) {
            uint32_t tgt = s_A[i];
            float rad = s_radA[i];
            int cnt = 0;
            uint64_t keys[2];
            bool ok[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                int cl = lane + 32 * h, col = c0 + cl;
                ok[h] = false;
                if (cl < cend && (col >= na || i < col)) {
                    uint32_t id = col < na ? s_A[col] : s_B[col - na];
                    float dd = s_D[i * (JCOLS + 1) + cl];
                    if (id != tgt && dd <= rad) {
                        ok[h] = true;
                        keys[h] = kcna_key(dd, id, (uint32_t)(KCNA_FLAG_NEW | KCNA_FLAG_ISNEW));
                    }
                }
            }
            unsigned m0 = __ballot_sync(KCNA_FULL, ok[0]), m1 = __ballot_sync(KCNA_FULL, ok[1]);
            cnt = __popc(m0) + __popc(m1);
            if (cnt == 0) continue;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.cand_cnt + tgt, (uint32_t)cnt);
            base = __shfl_sync(KCNA_FULL, base, 0);
            const uint64_t s0 = (uint64_t)tgt * a.CB;
            if (ok[0]) {
                uint32_t p = base + __popc(m0 & kcna_lanemask_lt());
                if (p < a.CB) kcna_cand_put(a.cand, s0 + p, keys[0], node);
            }
            if (ok[1]) {
                uint32_t p = base + __popc(m0) + __popc(m1 & kcna_lanemask_lt());
                if (p < a.CB) kcna_cand_put(a.cand, s0 + p, keys[1], node);
            }
            if (lane == 0) atomicAdd(s_emit, (unsigned)cnt);
        }
        // column targets: column id receives row ids
        for (int cl = warp; cl < cend; cl += nwarp) {
            int col = c0 + cl;
            uint32_t tgt = col < na ? s_A[col] : s_B[col - na];
            float rad = __ldg(a.radius + tgt);
            unsigned mk[RI];
            uint64_t keys[RI];
            int cnt = 0;
#pragma unroll
            for (int h = 0; h < RI; ++h) {
                int i = lane + 32 * h;
                bool ok = false;
                if (i < rows_needed && (col >= na || i < col)) {
                    uint32_t id = s_A[i];
                    float dd = s_D[i * (JCOLS + 1) + cl];
                    if (id != tgt && dd <= rad) {
                        ok = true;
                        keys[h] = kcna_key(dd, id, (uint32_t)(KCNA_FLAG_NEW | KCNA_FLAG_ISNEW));
                    }
                }
                mk[h] = __ballot_sync(KCNA_FULL, ok);
                cnt += __popc(mk[h]);
            }
            if (cnt == 0) continue;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.cand_cnt + tgt, (uint32_t)cnt);
            base = __shfl_sync(KCNA_FULL, base, 0);
            const uint64_t s0 = (uint64_t)tgt * a.CB;
            uint32_t run = base;
#pragma unroll
            for (int h = 0; h < RI; ++h) {
                if (mk[h] & (1u << lane)) {
                    uint32_t p = run + __popc(mk[h] & kcna_lanemask_lt());
                    if (p < a.CB) kcna_cand_put(a.cand, s0 + p, keys[h], node);
                }
                run += __popc(mk[h]);
            }
            if (lane == 0) atomicAdd(s_emit, (unsigned)cnt);
        }
        __syncthreads();
    }
}

// Join of the nodes with more rows than the regions of join_warp_kernel and
// join_mid_kernel hold: block per node, persistent over the queue (from the end
// of `list` down).
template <class R>
__global__ void __launch_bounds__(JT, 3) join_kernel(JoinArgs a, R rows, const uint32_t *__restrict__ list,
                                                     const uint32_t *__restrict__ cnt) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *s_As = reinterpret_cast<float *>(smem);                // 128 x JKP
    float *s_Bs = s_As + 128 * JKP;                               // JCOLS x JKP
    float *s_D = s_Bs + JCOLS * JKP;                              // 128 x (JCOLS+1)
    float *s_radA = s_D + 128 * (JCOLS + 1);                      // capA
    uint32_t *s_A = reinterpret_cast<uint32_t *>(s_radA + a.capA); // capA
    uint32_t *s_B = s_A + a.capA;                                 // capB
    __shared__ unsigned s_emit;
    const uint32_t n_big = cnt[1];
    for (uint32_t bi = blockIdx.x; bi < n_big; bi += gridDim.x) {
        const uint32_t node = list[a.N - 1 - bi];
        __syncthreads(); // the previous node's lists and tiles are read
        // new list: forward new then a random subset (<= R) of reverse new
        uint32_t fn = min(a.fwd_new_cnt[node], a.fwd_new_cap);
        for (uint32_t i = threadIdx.x; i < fn; i += blockDim.x) s_A[i] = a.fwd_new[(uint64_t)node * a.fwd_new_cap + i];
        uint32_t fo = min(a.fwd_old_cnt[node], a.fwd_old_cap);
        for (uint32_t i = threadIdx.x; i < fo; i += blockDim.x) s_B[i] = a.fwd_old[(uint64_t)node * a.fwd_old_cap + i];
        __syncthreads();
        uint32_t rn = 0, ro = 0;
        if (a.iter > 0) {
            rn = take_reverse(a.rnew + (uint64_t)node * a.RB, a.rnew_cnt[node], a.R, s_A + fn);
            ro = take_reverse(a.rold + (uint64_t)node * a.RB, a.rold_cnt[node], a.R, s_B + fo);
            __syncthreads();
        }
        // at most 128 rows per tile; the forward list alone is <= S + R < 128 in practice
        const int na = (int)min(fn + rn, 128u), nb = (int)(fo + ro);
        for (int i = threadIdx.x; i < na; i += blockDim.x) s_radA[i] = __ldg(a.radius + s_A[i]);
        if (threadIdx.x == 0) {
            atomicAdd(a.counters + 0, (unsigned long long)((uint64_t)na * (na - 1) / 2 + (uint64_t)na * nb));
            atomicAdd(a.counters + 5, (unsigned long long)(na + nb));
            s_emit = 0;
        }
        __syncthreads();
        if (na <= 32)
            join_tiles<1>(a, rows, node, s_A, na, s_B, nb, s_As, s_Bs, s_D, s_radA, &s_emit);
        else if (na <= 64)
            join_tiles<2>(a, rows, node, s_A, na, s_B, nb, s_As, s_Bs, s_D, s_radA, &s_emit);
        else
            join_tiles<4>(a, rows, node, s_A, na, s_B, nb, s_As, s_Bs, s_D, s_radA, &s_emit);
        if (threadIdx.x == 0 && s_emit) atomicAdd(a.counters + 6, (unsigned long long)s_emit);
    }
}

// The same join for nodes of at most ROWS rows: NT threads per node (a warp for
// up to 64 rows, a block of four warps for up to 160), persistent.  The pairs
// are the 4 x 4 micro-tiles (kcna_pairs.cuh) of the upper triangle of A x A and
// of A x B.  The distances go to a matrix over the rows' region (both triangles
// of A x A), and each warp then takes its targets (target % warps): a count
// pass (ballots over the target's partners, kept by lane i of the i-th target),
// one atomicAdd per target with all of them in flight together, a write pass.
// A node's list lengths come with those of 31 others, its ids while the node
// before it is computed, its radii while its rows are.
// First the warp version walks all nodes and queues larger ones in `list`:
// those for the block version from the front (cnt[0]), those for join_kernel
// from the end (cnt[1]).  150,001 x 128 rows (28 rows a node): 20 ms a
// build against 47 for a block of 256 threads per node.
// 11.5 KB a warp: sixteen warps an SM, as many as the registers allow.  Instruction
// issue bounds it (60,000 x 128: 0.66 a cycle, FMA pipe 40 %, 18 to 19 of 32 lanes).
template <int NT, int ROWS>
struct JoinSet {
    float x[pairs_region(ROWS)]; // rows, then the distance matrix: row i at i * (n | 1)
    uint32_t id[2][ROWS];        // this node's ids and the next one's
    float rad[ROWS];
};
constexpr int JW_ROWS = 64, JM_ROWS = 160, JM_NT = 128;
using JoinWarp = JoinSet<32, JW_ROWS>;
using JoinMid = JoinSet<JM_NT, JM_ROWS>;

// sizes of one node's lists
struct JoinLists {
    uint32_t fn, rn, fo, ro;
    __device__ int na() const { return (int)(fn + rn); }
    __device__ int n() const { return (int)(fn + rn + fo + ro); }
    __device__ int tiles() const {
        const int ga = (na() + 3) >> 2;
        return ga * (ga + 1) / 2 + ga * ((int)(fo + ro + 3) >> 2);
    }
    template <int NT, int ROWS> __device__ bool fits() const {
        return n() <= ROWS && tiles() <= NT * PT_MAXR && na() * (n() | 1) <= pairs_region(ROWS);
    }
};
__device__ __forceinline__ JoinLists join_lists(const JoinArgs &a, uint32_t node) {
    JoinLists l;
    l.fn = min(a.fwd_new_cnt[node], a.fwd_new_cap);
    l.fo = min(a.fwd_old_cnt[node], a.fwd_old_cap);
    l.rn = a.iter > 0 ? min(a.rnew_cnt[node], a.R) : 0u; // the random subsets select_reverse_kernel left first
    l.ro = a.iter > 0 ? min(a.rold_cnt[node], a.R) : 0u;
    return l;
}
// ids of the node's set (A then B) by cp.async, one group
template <int NT>
__device__ __forceinline__ void join_load_ids(const JoinArgs &a, uint32_t node, const JoinLists &l, uint32_t *s_id) {
    const uint32_t na = l.fn + l.rn, n = na + l.fo + l.ro;
    for (uint32_t u = pairs_lane<NT>(); u < n; u += NT) {
        const uint32_t v = u - na;
        const uint32_t *src = u < l.fn   ? a.fwd_new + (uint64_t)node * a.fwd_new_cap + u
                              : u < na   ? a.rnew + (uint64_t)node * a.RB + (u - l.fn)
                              : v < l.fo ? a.fwd_old + (uint64_t)node * a.fwd_old_cap + v
                                         : a.rold + (uint64_t)node * a.RB + (v - l.fo);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(s_id + u)),
                     "l"(src)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int NT, int R, class RowsT>
__device__ __forceinline__ void join_set_tiles(const RowsT &rows, const uint32_t *s_id, float *s_x, int na, int n,
                                               int T) {
    const int lane = pairs_lane<NT>(), nb = n - na, GA = (na + 3) >> 2, GB = (nb + 3) >> 2;
    const int TA = GA * (GA + 1) / 2;
    PairTile t[R];
    bool on[R];
    float acc[R][16];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int k = lane + NT * r;
        on[r] = k < T;
        t[r] = PairTile{0, 0, 0, 0};
        if (on[r]) {
            if (k < TA) {
                int g = 0;
                while (k >= GA - g) k -= GA - g++;
                t[r] = PairTile{g, GA, g + k, GA};
            } else {
                k -= TA;
                t[r] = PairTile{k / GB, GA, na + k % GB, GB};
            }
        }
    }
    pairs_distances<NT, R>(rows, s_id, n, s_x, t, on, acc);
    const int dp = n | 1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (!on[r]) continue;
        const bool inA = t[r].b0 < na;
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const int i = t[r].a0 + x * t[r].as, j = t[r].b0 + y * t[r].bs;
                if (i >= na || j >= (inA ? na : n)) continue;
                s_x[i * dp + j] = acc[r][4 * x + y];
                if (inA) s_x[j * dp + i] = acc[r][4 * x + y];
            }
    }
}

// One node: ids in S.id[b] (landed and visible); the next node's ids are on
// their way into S.id[b ^ 1].
template <int NT, int ROWS, class RowsT>
__device__ __forceinline__ void join_set(const JoinArgs &a, const RowsT &rows, JoinSet<NT, ROWS> &S, int b,
                                         uint32_t node, const JoinLists &l, unsigned long long &emitted) {
    constexpr int NW = NT / 32, PB = ROWS / 32; // warps; ballots per target
    const int lane = kcna_lane(), warp = NW == 1 ? 0 : (int)(threadIdx.x >> 5);
    const int na = l.na(), n = l.n(), T = l.tiles();
    const uint32_t *id = S.id[b];
    constexpr int RL = (ROWS + NT - 1) / NT;
    float rad[RL];
#pragma unroll
    for (int u = 0; u < RL; ++u) { // consumed after the distances
        const int i = pairs_lane<NT>() + NT * u;
        rad[u] = i < n ? __ldg(a.radius + id[i]) : 0.f;
    }
    if (T <= NT)
        join_set_tiles<NT, 1>(rows, id, S.x, na, n, T);
    else if (T <= 2 * NT)
        join_set_tiles<NT, 2>(rows, id, S.x, na, n, T);
    else
        join_set_tiles<NT, PT_MAXR>(rows, id, S.x, na, n, T);
#pragma unroll
    for (int u = 0; u < RL; ++u) {
        const int i = pairs_lane<NT>() + NT * u;
        if (i < n) S.rad[i] = rad[u];
    }
    pairs_sync<NT>(); // matrix and radii, for every thread
    const int dp = n | 1;
    // whether partner p (a row of the set) enters target t's buffer
    auto dist = [&](int t, int p) { return t < na ? S.x[t * dp + p] : S.x[p * dp + t]; };
    auto emits = [&](int t, int p) {
        if (t < na ? p >= n || p == t : p >= na) return false;
        return id[p] != id[t] && dist(t, p) <= S.rad[t];
    };
    const int nt = (n - warp + NW - 1) / NW; // this warp's targets: warp + NW * i
    for (int i0 = 0; i0 < nt; i0 += 32) {
        uint32_t m[PB], base = 0u, cnt = 0u; // of target i0 + lane
#pragma unroll
        for (int v = 0; v < PB; ++v) m[v] = 0u;
        for (int i = i0; i < min(nt, i0 + 32); ++i) {
            const int t = warp + NW * i;
#pragma unroll
            for (int v = 0; v < PB; ++v) {
                const uint32_t bal = 32 * v < n ? __ballot_sync(KCNA_FULL, emits(t, lane + 32 * v)) : 0u;
                if (lane == i - i0) m[v] = bal;
            }
        }
#pragma unroll
        for (int v = 0; v < PB; ++v) cnt += __popc(m[v]);
        if (cnt) base = atomicAdd(a.cand_cnt + id[warp + NW * (i0 + lane)], cnt);
        emitted += cnt;
        for (int i = i0; i < min(nt, i0 + 32); ++i) {
            const int t = warp + NW * i;
            uint32_t at = __shfl_sync(KCNA_FULL, base, i - i0);
            const uint64_t s0 = (uint64_t)id[t] * a.CB;
#pragma unroll
            for (int v = 0; v < PB; ++v) {
                const uint32_t bits = __shfl_sync(KCNA_FULL, m[v], i - i0);
                const int p = lane + 32 * v;
                const uint32_t pos = at + __popc(bits & kcna_lanemask_lt());
                if (((bits >> lane) & 1u) && pos < a.CB)
                    kcna_cand_put(a.cand, s0 + pos,
                                  kcna_key(dist(t, p), id[p], (uint32_t)(KCNA_FLAG_NEW | KCNA_FLAG_ISNEW)), node);
                at += __popc(bits);
            }
        }
    }
    pairs_sync<NT>(); // the next node reuses the region
}

constexpr int JW_WARPS = 16; // of the warp version, one block an SM: they share nothing, but a block costs 1 KB

template <class RowsT>
__global__ void __launch_bounds__(JW_WARPS * 32, 1) join_warp_kernel(JoinArgs a, RowsT rows,
                                                                     uint32_t *__restrict__ list,
                                                                     uint32_t *__restrict__ cnt) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = kcna_lane();
    JoinWarp &S = reinterpret_cast<JoinWarp *>(smem)[threadIdx.x >> 5];
    unsigned long long pairs = 0, nrows = 0, emitted = 0;
    const uint32_t gw = blockIdx.x * JW_WARPS + (threadIdx.x >> 5), G = gridDim.x * JW_WARPS;
    // list sizes of 32 of this warp's nodes, one node per lane; the walk to the next node this version takes
    JoinLists mine{0u, 0u, 0u, 0u};
    uint64_t at = gw; // the next node to look at
    int j = 0;        // its place among the 32
    auto next = [&](JoinLists &l) -> uint32_t {
        for (; at < a.N; at += G) {
            if (j == 0) {
                const uint64_t q = at + (uint64_t)lane * G;
                mine = q < a.N ? join_lists(a, (uint32_t)q) : JoinLists{0u, 0u, 0u, 0u};
            }
            l.fn = __shfl_sync(KCNA_FULL, mine.fn, j);
            l.rn = __shfl_sync(KCNA_FULL, mine.rn, j);
            l.fo = __shfl_sync(KCNA_FULL, mine.fo, j);
            l.ro = __shfl_sync(KCNA_FULL, mine.ro, j);
            j = (j + 1) & 31;
            if (l.na() == 0) continue;
            if (!l.fits<32, JW_ROWS>()) {
                if (lane == 0) {
                    if (l.fits<JM_NT, JM_ROWS>())
                        list[atomicAdd(cnt, 1u)] = (uint32_t)at;
                    else
                        list[a.N - 1 - atomicAdd(cnt + 1, 1u)] = (uint32_t)at;
                }
                continue;
            }
            const uint32_t node = (uint32_t)at;
            at += G;
            return node;
        }
        return KCNA_NONE;
    };
    JoinLists l, ln;
    uint32_t node = next(l);
    if (node != KCNA_NONE) join_load_ids<32>(a, node, l, S.id[0]);
    for (int b = 0; node != KCNA_NONE; b ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        const uint32_t nn = next(ln);
        if (nn != KCNA_NONE) join_load_ids<32>(a, nn, ln, S.id[b ^ 1]);
        join_set<32, JW_ROWS>(a, rows, S, b, node, l, emitted);
        pairs += (unsigned long long)l.na() * (l.na() - 1) / 2 + (unsigned long long)l.na() * (l.fo + l.ro);
        nrows += (unsigned long long)l.n();
        node = nn;
        l = ln;
    }
    emitted = kcna_warp_sum(emitted);
    if (lane == 0) {
        atomicAdd(a.counters + 0, pairs);
        atomicAdd(a.counters + 5, nrows);
        atomicAdd(a.counters + 6, emitted);
    }
}

template <class RowsT>
__global__ void __launch_bounds__(JM_NT, 4) join_mid_kernel(JoinArgs a, RowsT rows, const uint32_t *__restrict__ list,
                                                            const uint32_t *__restrict__ cnt) {
    extern __shared__ __align__(16) unsigned char smem[];
    JoinMid &S = *reinterpret_cast<JoinMid *>(smem);
    const uint32_t n_mid = cnt[0];
    unsigned long long pairs = 0, nrows = 0, emitted = 0;
    for (uint32_t i = blockIdx.x; i < n_mid; i += gridDim.x) {
        const uint32_t node = list[i];
        const JoinLists l = join_lists(a, node);
        join_load_ids<JM_NT>(a, node, l, S.id[0]);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        join_set<JM_NT, JM_ROWS>(a, rows, S, 0, node, l, emitted);
        pairs += (unsigned long long)l.na() * (l.na() - 1) / 2 + (unsigned long long)l.na() * (l.fo + l.ro);
        nrows += (unsigned long long)l.n();
    }
    emitted = kcna_warp_sum(emitted);
    if (kcna_lane() == 0 && emitted) atomicAdd(a.counters + 6, emitted);
    if (threadIdx.x == 0 && nrows) {
        atomicAdd(a.counters + 0, pairs);
        atomicAdd(a.counters + 5, nrows);
    }
}

// ---------------------------------------------------------------------------
// merge: candidates of one node into its pool (batched InsertIntoPool)
// ---------------------------------------------------------------------------
constexpr int MT = 256;

struct MergeArgs {
    uint64_t *pool;
    uint32_t *pool_cnt;
    uint32_t cap, limit, K;
    float *radius;
    uint64_t *cand; // key and joiner per slot (kcna_cand_put)
    uint32_t *cand_cnt;
    uint32_t CB;
    unsigned long long *counters; // [1] flagged in top-K, [2] overflow, [3] inserted
    // found credit (NN-descent merges): the joiner of every candidate, and the
    // flags the merge sets.  The reference's join marks a node found when one
    // of the pairs its join evaluated was inserted below K by its
    // parallel_try_insert (src/kgraph.cpp:1107-1116); a pair several joiners
    // evaluate is inserted by the first to reach the pool, and only that one
    // is credited.  Here each distinct new entry placed at rank < K credits the
    // lowest joiner that emitted it (in the reference's increasing-node
    // parallel loop, in practice the first to reach the pair).  Crediting every
    // emitter instead over-credits: NN-descent then converges measurably
    // faster than the reference's (200k C2 rows: recall 0.9968 after six
    // iterations against the reference's 0.9943).
    uint32_t credit; // credit joiners (NN-descent merges)
    uint8_t *found;
    uint32_t n_nodes;
};

// Merge of a refinement round (no credit, few survivors): warp per node,
// survivors first.  Every candidate is looked up in the node's sorted pool by
// binary search (shared memory): a candidate equal to a pool entry, or one that
// would land at rank >= limit, is dropped.  Only the few survivors are sorted,
// deduplicated and merged, and only the pool entries they displace are written.
// A node with more than MW_SURV survivors is queued for the block merge
// (merge_kernel).  Same result as merging all candidates.  Persistent: each
// warp takes nodes grid-stride, so a block meets its barrier once at the end
// instead of waiting for its slowest node.
constexpr int MW_WARPS = 8, MW_SURV = 128; // five blocks share an SM
__host__ __device__ constexpr size_t merge_warp_bytes(uint32_t cap) {
    return ((size_t)cap * 8 + (size_t)MW_SURV * 8 + 16 + 15) & ~(size_t)15;
}

__global__ void __launch_bounds__(MW_WARPS * 32) merge_warp_kernel(MergeArgs a, uint32_t N, uint32_t *big_list,
                                                                  uint32_t *big_cnt) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = kcna_lane();
    const size_t per_warp = merge_warp_bytes(a.cap);
    unsigned char *base = smem + w * per_warp;
    uint64_t *s_pool = reinterpret_cast<uint64_t *>(base);
    uint64_t *s_sv = s_pool + a.cap;         // survivors (keys without flags)
    uint64_t *s_last = s_sv + MW_SURV;       // key landing at rank limit-1
    __shared__ unsigned long long s_stat[4]; // flagged, inserted, candidates, entries
    if (threadIdx.x < 4) s_stat[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t node = blockIdx.x * MW_WARPS + w; node < N; node += gridDim.x * MW_WARPS) {
        const uint32_t raw = a.cand_cnt[node];
        // a refinement round leaves most pools without candidates: their pool,
        // count and radius stand
        if (raw == 0) continue;
        const uint32_t nc = min(raw, a.CB);
        const uint32_t np = min(a.pool_cnt[node], a.limit);
        uint64_t *gp = a.pool + (uint64_t)node * a.cap;
        const uint64_t *gc = a.cand + 2 * (uint64_t)node * a.CB; // keys at even words
#pragma unroll 4
        for (uint32_t i = lane; i < np; i += 32) s_pool[i] = gp[i];
        // candidates in groups of 128 (four per lane), the next group's loads in
        // flight while this group is searched
        constexpr int CG = 4;
        uint64_t nxt[CG];
#pragma unroll
        for (int u = 0; u < CG; ++u) {
            const uint32_t j = 32 * u + lane;
            nxt[u] = j < nc ? gc[2 * j] : KCNA_EMPTY_KEY;
        }
        __syncwarp();
        // survivors: not in the pool, landing below limit
        uint32_t ns = 0;
        for (uint32_t b0 = 0; b0 < nc; b0 += 32 * CG) {
            uint64_t cur[CG];
#pragma unroll
            for (int u = 0; u < CG; ++u) {
                cur[u] = nxt[u];
                const uint32_t j = b0 + 32 * CG + 32 * u + lane;
                nxt[u] = j < nc ? gc[2 * j] : KCNA_EMPTY_KEY;
            }
#pragma unroll
            for (int u = 0; u < CG; ++u) {
                const uint32_t j = b0 + 32 * u + lane;
                bool surv = false;
                const uint64_t k = kcna_key_noflags(cur[u]);
                if (j < nc && k != KCNA_EMPTY_KEY_NOFLAGS) {
                    const int b = kcna_lower_bound(s_pool, (int)np, k);
                    surv = (uint32_t)b < a.limit && !(b < (int)np && (s_pool[b] >> 2) == (k >> 2));
                }
                const unsigned m = __ballot_sync(KCNA_FULL, surv);
                const uint32_t pos = ns + __popc(m & kcna_lanemask_lt());
                if (surv && pos < (uint32_t)MW_SURV) s_sv[pos] = k;
                ns += __popc(m);
            }
        }
        if (ns > (uint32_t)MW_SURV) {
            if (lane == 0) big_list[atomicAdd(big_cnt, 1u)] = node;
        } else {
            uint32_t nu = 0; // distinct survivors
            if (ns > 0) {
                __syncwarp();
                kcna_warp_sort_n(s_sv, (int)ns);
                // drop repeats among survivors (same distance and id are adjacent);
                // compaction moves entries down, so the previous key comes from
                // registers, not from the array being rewritten
                uint64_t carry = KCNA_EMPTY_KEY;
                for (uint32_t b0 = 0; b0 < ns; b0 += 32) {
                    const uint32_t j = b0 + lane;
                    const uint64_t k = j < ns ? s_sv[j] : KCNA_EMPTY_KEY;
                    uint64_t prev = __shfl_up_sync(KCNA_FULL, k, 1);
                    if (lane == 0) prev = carry;
                    const bool keep = j < ns && (j == 0 || (prev >> 2) != (k >> 2));
                    const unsigned m = __ballot_sync(KCNA_FULL, keep);
                    carry = __shfl_sync(KCNA_FULL, k, 31);
                    __syncwarp();
                    if (keep) s_sv[nu + __popc(m & kcna_lanemask_lt())] = k;
                    nu += __popc(m);
                    __syncwarp();
                }
            }
            const uint32_t newcnt = min(a.limit, np + nu);
            unsigned long long flagged = 0;
            if (lane == 0) *s_last = KCNA_EMPTY_KEY;
            __syncwarp();
            // pool entries: shifted by the survivors below them
            for (uint32_t i = lane; i < np; i += 32) {
                const uint64_t k = s_pool[i];
                const uint32_t sh = nu ? (uint32_t)kcna_lower_bound(s_sv, (int)nu, kcna_key_noflags(k)) : 0u;
                const uint32_t r = i + sh;
                if (r < newcnt) {
                    if (sh) gp[r] = k;
                    if (r < a.K && (k & KCNA_FLAG_NEW)) ++flagged;
                    if (r + 1 == a.limit) *s_last = k;
                }
            }
            // survivors at their rank
            unsigned long long placed = 0;
            for (uint32_t j = lane; j < nu; j += 32) {
                const uint64_t k = s_sv[j];
                const uint32_t r = j + (uint32_t)kcna_lower_bound(s_pool, (int)np, k);
                if (r < newcnt) {
                    gp[r] = k | KCNA_FLAG_NEW | KCNA_FLAG_ISNEW;
                    ++placed;
                    if (r < a.K) ++flagged;
                    if (r + 1 == a.limit) *s_last = k;
                }
            }
            flagged = kcna_warp_sum(flagged);
            placed = kcna_warp_sum(placed);
            __syncwarp();
            if (lane == 0) {
                if (flagged) atomicAdd(&s_stat[0], flagged);
                if (placed) atomicAdd(&s_stat[1], placed);
                atomicAdd(&s_stat[2], (unsigned long long)nc);
                atomicAdd(&s_stat[3], (unsigned long long)newcnt);
                if (raw > a.CB) atomicAdd(a.counters + 2, (unsigned long long)(raw - a.CB));
                a.pool_cnt[node] = newcnt;
                a.cand_cnt[node] = 0;
                a.radius[node] = newcnt >= a.limit ? kcna_key_dist(*s_last) : __uint_as_float(0x7F800000u);
            }
        }
        __syncwarp(); // the next node reuses this warp's shared memory
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_stat[0]) atomicAdd(a.counters + 1, s_stat[0]);
        if (s_stat[1]) atomicAdd(a.counters + 3, s_stat[1]);
        if (s_stat[2]) atomicAdd(a.counters + 7, s_stat[2]);
        if (s_stat[3]) atomicAdd(a.counters + 9, s_stat[3]);
    }
}

// In-place exclusive scan of data[0..n) by the whole block; data[n] receives
// the total.  s_warp holds blockDim.x/32 words.
__device__ uint32_t block_exclusive_scan(uint32_t *data, int n, uint32_t *s_warp) {
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int b = threadIdx.x * per;
    uint32_t local = 0;
    for (int i = 0; i < per && b + i < n; ++i) local += data[b + i];
    uint32_t incl = local;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t u = __shfl_up_sync(KCNA_FULL, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
            uint32_t t = s_warp[i];
            s_warp[i] = run;
            run += t;
        }
    }
    __syncthreads();
    uint32_t run = s_warp[w] + incl - local;
    for (int i = 0; i < per && b + i < n; ++i) {
        uint32_t t = data[b + i];
        data[b + i] = run;
        run += t;
    }
    if (threadIdx.x == blockDim.x - 1) data[n] = run;
    __syncthreads();
    return data[n];
}

// NN-descent's merge: a block of four warps per node, survivors first.  As in
// merge_warp_kernel every candidate is looked up in the node's sorted pool; in
// a converging NN-descent most are repeats.  The survivors go into a small hash
// table (open addressing on the id; one id has one distance, so equal keys are
// the same candidate emitted by several joiners), so that only distinct ones
// are merged; beside each stands the lowest joiner that emitted it (the slot's
// second word, fetched with the key), which is credited when the survivor
// lands at rank < K.
// Where the survivors land needs no sort: the search says between which pool
// entries each falls (its bucket), so bucket counts and their prefix sums give
// every pool entry its shift and every survivor its rank but for the order
// inside a bucket, which is counted (one or two entries; some fifty while the
// pools hold a dozen).
// What bounds it is the latency of dependent shared-memory steps: a warp per
// node issued every tenth cycle with three warps a scheduler, and a node's
// arrays (22 KB) allow no more.  Four warps share them here, nine blocks an SM
// (their 54 registers a thread allow no more either).  The pool lies as two arrays: the search reads the 4-byte distances
// only, and equal distances are told apart by the id once at the end.
// 400,003 rows, the four merges of a learned build: 58 ms with a warp per node
// and a sort of all survivors with their repeats, 26 ms now (9 nodes of each
// SM in flight; the table alone, with a warp per node, gave 50).  Now issue (0.65 to
// 0.74 a cycle) and shared memory (66 to 79 % of its cycles) are what is left.
// MS_H: table slots (a prime, for the double hashing).  A node with more than
// MS_CAP distinct survivors is queued for the block merge; the count is read
// before each warp's batch of 32, and the four warps' batches fit beside it.
constexpr int MS_NT = 128, MS_H = 1021, MS_CAP = MS_H - MS_NT - 1;
__host__ __device__ constexpr size_t merge_set_bytes(uint32_t cap) {
    return (size_t)MS_H * 8 + (size_t)cap * 8 + (size_t)MS_H * 4 + (size_t)(cap + 2) * 4 + (size_t)MS_H * 4;
}

__global__ void __launch_bounds__(MS_NT, 9) merge_set_kernel(MergeArgs a, uint32_t N, uint32_t *big_list,
                                                            uint32_t *big_cnt) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *s_sv = reinterpret_cast<uint64_t *>(smem);       // the table of distinct survivors (keys without flags)
    uint32_t *s_pd = reinterpret_cast<uint32_t *>(s_sv + MS_H);   // the pool: distance bits
    uint32_t *s_pi = s_pd + a.cap;                             // and id with flags
    uint32_t *s_joiner = s_pi + a.cap;                         // lowest joiner of a table slot
    uint32_t *s_off = s_joiner + MS_H;                            // cap + 2: bucket counts, starts, ends
    uint16_t *s_slot = reinterpret_cast<uint16_t *>(s_off + a.cap + 2), *s_b = s_slot + MS_H; // slots in bucket order; bucket of a slot
    __shared__ uint32_t s_warp[MS_NT / 32], s_flagged, s_placed;
    __shared__ uint64_t s_last; // key landing at rank limit-1
    __shared__ volatile uint32_t s_nu;
    const int tid = threadIdx.x, lane = tid & 31;
    unsigned long long t_flagged = 0, t_placed = 0, t_cand = 0, t_entries = 0; // thread 0
    auto clear_table = [&]() {
        for (int i = tid; i < MS_H; i += MS_NT) {
            s_sv[i] = KCNA_EMPTY_KEY;
            s_joiner[i] = KCNA_NONE;
        }
        for (uint32_t i = tid; i < a.cap + 2; i += MS_NT) s_off[i] = 0;
    };
    clear_table();
    uint32_t raw_n = blockIdx.x < N ? a.cand_cnt[blockIdx.x] : 0u; // of the next node, loaded a node ahead
    uint32_t np_n = blockIdx.x < N ? a.pool_cnt[blockIdx.x] : 0u;
    for (uint32_t node = blockIdx.x; node < N; node += gridDim.x) {
        const uint32_t raw = raw_n, np = min(np_n, a.limit);
        if (node + gridDim.x < N) {
            raw_n = a.cand_cnt[node + gridDim.x];
            np_n = a.pool_cnt[node + gridDim.x];
        }
        const uint32_t nc = min(raw, a.CB);
        uint64_t *gp = a.pool + (uint64_t)node * a.cap;
        const ulonglong2 *gc = reinterpret_cast<const ulonglong2 *>(a.cand) + (uint64_t)node * a.CB; // key, joiner
        // candidates in groups of 256 (two per thread), the next group's loads in
        // flight while this group is searched, the two searches side by side
        constexpr int CG = 2;
        ulonglong2 nxt[CG];
        auto fetch = [&](int u, uint32_t j) { nxt[u] = j < nc ? gc[j] : make_ulonglong2(KCNA_EMPTY_KEY, KCNA_NONE); };
#pragma unroll
        for (int u = 0; u < CG; ++u) fetch(u, MS_NT * u + tid);
#pragma unroll 4
        for (uint32_t i = tid; i < np; i += MS_NT) {
            const uint64_t k = gp[i];
            s_pd[i] = (uint32_t)(k >> 32);
            s_pi[i] = (uint32_t)k;
        }
        if (tid == 0) {
            s_nu = 0;
            s_flagged = s_placed = 0;
            s_last = KCNA_EMPTY_KEY;
        }
        __syncthreads();
        const int top = np ? 1 << (31 - __clz(np)) : 0, last = max((int)np - 1, 0); // largest step of the search
        for (uint32_t b0 = 0; b0 < nc; b0 += MS_NT * CG) {
            uint32_t d[CG], id[CG], joiner[CG];
            int b[CG];
            bool surv[CG];
#pragma unroll
            for (int u = 0; u < CG; ++u) {
                d[u] = (uint32_t)(nxt[u].x >> 32);
                id[u] = kcna_key_id(nxt[u].x);
                joiner[u] = (uint32_t)nxt[u].y;
                // a candidate, not the padding or a dropped one
                surv[u] = kcna_key_noflags(nxt[u].x) != KCNA_EMPTY_KEY_NOFLAGS;
                b[u] = 0;
                fetch(u, b0 + MS_NT * CG + MS_NT * u + tid);
            }
            // entries nearer than each candidate
            for (int step = top; step; step >>= 1) {
#pragma unroll
                for (int u = 0; u < CG; ++u) {
                    const int t = b[u] + step - 1;
                    const uint32_t v = s_pd[min(t, last)];
                    b[u] += (t <= last) & (v < d[u]) ? step : 0;
                }
            }
            // survivors, and what their table slot holds so far
            uint32_t h[CG];
            uint64_t seen[CG];
#pragma unroll
            for (int u = 0; u < CG; ++u) {
                h[u] = __umulhi(id[u] * 0x9E3779B1u, (uint32_t)MS_H);
                seen[u] = s_sv[h[u]];
                // entries at the candidate's distance: by id; its own twin drops it.  Mostly
                // one or two; in a longer run (few-valued rows: a hundred and more) the
                // place is sought by growing steps, then by halving ones
                const int stop = min((int)np, b[u] + 3);
                while (b[u] < stop && s_pd[b[u]] == d[u]) {
                    const uint32_t e = s_pi[b[u]] >> 2;
                    if (e >= id[u]) {
                        if (e == id[u]) surv[u] = false;
                        break;
                    }
                    ++b[u];
                }
                if (b[u] == stop && stop < (int)np) {
                    auto below = [&](int t) { return t < (int)np && s_pd[t] == d[u] && (s_pi[t] >> 2) < id[u]; };
                    int step = 1;
                    for (; below(b[u] + step - 1); step <<= 1) b[u] += step;
                    while (step >>= 1)
                        if (below(b[u] + step - 1)) b[u] += step;
                    if (b[u] < (int)np && s_pd[b[u]] == d[u] && (s_pi[b[u]] >> 2) == id[u]) surv[u] = false;
                }
                if ((uint32_t)b[u] >= a.limit) surv[u] = false;
            }
#pragma unroll
            for (int u = 0; u < CG; ++u) {
                bool fresh = false;
                if (s_nu > (uint32_t)MS_CAP) surv[u] = false; // table full: the block merge takes the node
                if (surv[u]) {
                    // double hashing: in a table three quarters full, runs of taken slots
                    // would keep a warp's unluckiest lane probing for tens of steps
                    const uint64_t k = ((uint64_t)d[u] << 32) | ((uint64_t)id[u] << 2);
                    uint32_t x = h[u];
                    const uint32_t step = 1u + __umulhi(id[u] * 0x85EBCA6Bu, (uint32_t)(MS_H - 1));
                    for (int probe = 0; probe < MS_H && seen[u] != k; ++probe) { // a slot is free, or holds k
                        if (seen[u] == KCNA_EMPTY_KEY) {
                            seen[u] = atomicCAS(reinterpret_cast<unsigned long long *>(s_sv + x), KCNA_EMPTY_KEY, k);
                            fresh = seen[u] == KCNA_EMPTY_KEY;
                            if (fresh || seen[u] == k) break;
                        }
                        x += step;
                        x -= x >= (uint32_t)MS_H ? (uint32_t)MS_H : 0u;
                        seen[u] = s_sv[x];
                    }
                    if (joiner[u] < s_joiner[x]) atomicMin(s_joiner + x, joiner[u]);
                    if (fresh) {
                        s_b[x] = (uint16_t)b[u];
                        atomicAdd(s_off + b[u], 1u);
                    }
                }
                const unsigned m = __ballot_sync(KCNA_FULL, fresh);
                if (m && lane == 0) atomicAdd(const_cast<uint32_t *>(&s_nu), (uint32_t)__popc(m));
            }
        }
        __syncthreads();
        const uint32_t nu = s_nu;
        if (nu > (uint32_t)MS_CAP) {
            if (tid == 0) big_list[atomicAdd(big_cnt, 1u)] = node;
        } else {
            const uint32_t newcnt = min(a.limit, np + nu);
            uint32_t flagged = 0, placed = 0;
            if (nu > 0) { // survivors in bucket order; s_off[b] ends as the end of bucket b
                block_exclusive_scan(s_off, (int)np + 1, s_warp);
                for (int i = tid; i < MS_H; i += MS_NT)
                    if (s_sv[i] != KCNA_EMPTY_KEY) s_slot[atomicAdd(s_off + s_b[i], 1u)] = (uint16_t)i;
                __syncthreads();
            }
            // pool entries: shifted by the survivors below them
#pragma unroll 4
            for (uint32_t i = tid; i < np; i += MS_NT) {
                const uint64_t k = ((uint64_t)s_pd[i] << 32) | s_pi[i];
                const uint32_t sh = s_off[i], r = i + sh; // all zero without survivors
                if (r < newcnt) {
                    if (sh) gp[r] = k;
                    if (r < a.K && (k & KCNA_FLAG_NEW)) ++flagged;
                    if (r + 1 == a.limit) s_last = k;
                }
            }
            // survivors at their rank
            for (uint32_t j = tid; j < nu; j += MS_NT) {
                const uint32_t slot = s_slot[j], b = s_b[slot], lo = b ? s_off[b - 1] : 0u, hi = s_off[b];
                const uint64_t k = s_sv[slot];
                uint32_t r = b + lo;
                if (hi - lo > 1) {
#pragma unroll 4
                    for (uint32_t x = lo; x < hi; ++x) r += s_sv[s_slot[x]] < k ? 1u : 0u;
                }
                if (r >= newcnt) continue;
                gp[r] = k | KCNA_FLAG_NEW | KCNA_FLAG_ISNEW;
                ++placed;
                if (r < a.K) {
                    ++flagged;
                    const uint32_t best = s_joiner[slot];
                    if (best < a.n_nodes) a.found[best] = 1;
                }
                if (r + 1 == a.limit) s_last = k;
            }
            flagged = kcna_warp_sum(flagged);
            placed = kcna_warp_sum(placed);
            if (lane == 0) {
                if (flagged) atomicAdd(&s_flagged, flagged);
                if (placed) atomicAdd(&s_placed, placed);
            }
            __syncthreads();
            if (tid == 0) {
                t_flagged += s_flagged;
                t_placed += s_placed;
                t_cand += nc;
                t_entries += newcnt;
                if (raw > a.CB) atomicAdd(a.counters + 2, (unsigned long long)(raw - a.CB));
                a.pool_cnt[node] = newcnt;
                a.cand_cnt[node] = 0;
                a.radius[node] = newcnt >= a.limit ? kcna_key_dist(s_last) : __uint_as_float(0x7F800000u);
            }
        }
        __syncthreads(); // the next node reuses the arrays
        if (nu > 0) clear_table();
    }
    if (tid == 0) {
        if (t_flagged) atomicAdd(a.counters + 1, t_flagged);
        if (t_placed) atomicAdd(a.counters + 3, t_placed);
        if (t_cand) atomicAdd(a.counters + 7, t_cand);
        if (t_entries) atomicAdd(a.counters + 9, t_entries);
    }
}

// Block merge of nodes with many survivors (queued by the two kernels above).
// Each candidate is placed by binary search into the gap of the sorted pool
// it falls in (its bucket: the number of pool entries below it); candidates
// equal to a pool entry or with bucket >= limit are dropped.  A counting sort
// by bucket then an insertion sort inside each bucket (block bitonic for the
// rare bucket above 32 entries) leave all candidates sorted, since buckets
// are ordered; duplicates are then adjacent.  Final position of pool entry i
// = i + kept candidates in buckets 0..i; of a kept candidate in bucket b =
// b + kept candidates before it.  Work is O(c log L + L) instead of a full
// sort of the candidates.
__global__ void __launch_bounds__(MT) merge_kernel(MergeArgs a, const uint32_t *big_list, const uint32_t *big_cnt) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int cbp = kcna_pow2_ceil_d((int)a.CB);
    uint64_t *s_pool = reinterpret_cast<uint64_t *>(smem); // cap
    uint64_t *s_c = s_pool + a.cap;                        // cbp (candidate keys, then bitonic scratch)
    uint64_t *s_sorted = s_c + cbp;                        // cbp
    uint32_t *s_b = reinterpret_cast<uint32_t *>(s_sorted + cbp); // cbp  bucket per candidate, then scratch
    uint32_t *s_ss = s_b + cbp;                            // cbp  joiner of each sorted candidate (credit)
    uint32_t *s_hist = s_ss + cbp;                         // cap + 2
    uint32_t *s_off = s_hist + a.cap + 2;                  // cap + 2
    uint32_t *s_giant = s_off + a.cap + 2;                 // cap + 2
    uint32_t *s_kept = reinterpret_cast<uint32_t *>(s_c);  // cbp + 1, once s_c's sorting is done
    const bool credit = a.credit != 0;
    __shared__ uint32_t s_warp[MT / 32];
    __shared__ uint32_t s_ngiant;
    __shared__ unsigned long long s_flagged;
    for (uint32_t bi = blockIdx.x; bi < *big_cnt; bi += gridDim.x) {
        __syncthreads();
        const uint32_t node = big_list[bi];
        const uint32_t raw = a.cand_cnt[node];
        const uint32_t nc = min(raw, a.CB);
        const uint32_t np = min(a.pool_cnt[node], a.limit);
        uint64_t *gp = a.pool + (uint64_t)node * a.cap;
        const uint64_t *gc = a.cand + 2 * (uint64_t)node * a.CB; // keys at even words
        if (threadIdx.x == 0) {
            s_flagged = 0;
            s_ngiant = 0;
        }
        for (uint32_t i = threadIdx.x; i < np; i += MT) s_pool[i] = gp[i];
        for (uint32_t i = threadIdx.x; i <= np + 1; i += MT) s_hist[i] = 0;
        __syncthreads();
        // bucket of every candidate
        for (uint32_t j = threadIdx.x; j < nc; j += MT) {
            const uint64_t k = kcna_key_noflags(gc[2 * j]);
            s_c[j] = k;
            const int b = kcna_lower_bound(s_pool, (int)np, k);
            const bool dup = b < (int)np && (s_pool[b] >> 2) == (k >> 2);
            if (dup || b >= (int)a.limit || k == KCNA_EMPTY_KEY_NOFLAGS) {
                s_b[j] = KCNA_NONE;
            } else {
                s_b[j] = (uint32_t)b;
                atomicAdd(&s_hist[b], 1u);
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i <= np; i += MT) s_off[i] = s_hist[i];
        __syncthreads();
        const uint32_t total = block_exclusive_scan(s_off, (int)np + 1, s_warp); // s_off[np+1] = total
        if (total == 0) { // nothing new: the pool stays as it is in memory
            unsigned long long f = 0;
            for (uint32_t i = threadIdx.x; i < np && i < a.K; i += MT) f += (s_pool[i] & KCNA_FLAG_NEW) ? 1 : 0;
            f = kcna_warp_sum(f);
            if ((threadIdx.x & 31) == 0 && f) atomicAdd(&s_flagged, f);
            __syncthreads();
            if (threadIdx.x == 0) {
                atomicAdd(a.counters + 1, s_flagged);
                if (raw > a.CB) atomicAdd(a.counters + 2, (unsigned long long)(raw - a.CB));
                atomicAdd(a.counters + 7, (unsigned long long)nc);
                atomicAdd(a.counters + 9, (unsigned long long)np);
                a.pool_cnt[node] = np;
                a.cand_cnt[node] = 0;
                a.radius[node] = np >= a.limit ? kcna_key_dist(s_pool[a.limit - 1]) : __uint_as_float(0x7F800000u);
            }
            continue;
        }
        for (uint32_t i = threadIdx.x; i <= np; i += MT) s_hist[i] = 0;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < nc; j += MT) {
            const uint32_t b = s_b[j];
            if (b != KCNA_NONE) {
                const uint32_t q = s_off[b] + atomicAdd(&s_hist[b], 1u);
                s_sorted[q] = s_c[j];
                s_ss[q] = credit ? (uint32_t)gc[2 * j + 1] : 0u;
            }
        }
        __syncthreads();
        // sort inside buckets, by key then joiner
        for (uint32_t b = threadIdx.x; b <= np; b += MT) {
            const uint32_t lo = s_off[b], hi = s_off[b + 1];
            if (hi - lo > 32) {
                s_giant[atomicAdd(&s_ngiant, 1u)] = b;
            } else {
                for (uint32_t x = lo + 1; x < hi; ++x) {
                    const uint64_t v = s_sorted[x];
                    const uint32_t vs = s_ss[x];
                    uint32_t y = x;
                    while (y > lo && (s_sorted[y - 1] > v || (s_sorted[y - 1] == v && s_ss[y - 1] > vs))) {
                        s_sorted[y] = s_sorted[y - 1];
                        s_ss[y] = s_ss[y - 1];
                        --y;
                    }
                    s_sorted[y] = v;
                    s_ss[y] = vs;
                }
            }
        }
        __syncthreads();
        const uint32_t ng = s_ngiant;
        for (uint32_t g = 0; g < ng; ++g) {
            const uint32_t b = s_giant[g];
            const uint32_t lo = s_off[b], len = s_off[b + 1] - lo;
            const int p2 = kcna_pow2_ceil_d((int)len);
            for (int i = threadIdx.x; i < p2; i += MT) {
                s_c[i] = i < (int)len ? s_sorted[lo + i] : KCNA_EMPTY_KEY;
                s_b[i] = i < (int)len ? s_ss[lo + i] : KCNA_NONE; // s_b is free after the scatter
            }
            kcna_cta_bitonic_kv(s_c, s_b, p2);
            for (uint32_t i = threadIdx.x; i < len; i += MT) {
                s_sorted[lo + i] = s_c[i];
                s_ss[lo + i] = s_b[i];
            }
            __syncthreads();
        }
        // duplicates among candidates are now adjacent
        for (uint32_t j = threadIdx.x; j < total; j += MT)
            s_kept[j] = (j == 0 || (s_sorted[j - 1] >> 2) != (s_sorted[j] >> 2)) ? 1u : 0u;
        __syncthreads();
        const uint32_t kept = block_exclusive_scan(s_kept, (int)total, s_warp);
        const uint32_t newcnt = min(a.limit, np + kept);
        unsigned long long flagged = 0, placed = 0;
        for (uint32_t i = threadIdx.x; i < np; i += MT) {
            const uint64_t k = s_pool[i];
            const uint32_t r = i + s_kept[s_off[i + 1]];
            if (r < newcnt) {
                gp[r] = k;
                if (r < a.K && (k & KCNA_FLAG_NEW)) ++flagged;
            }
        }
        for (uint32_t j = threadIdx.x; j < total; j += MT) {
            if (s_kept[j + 1] == s_kept[j]) continue; // duplicate
            // bucket of sorted position j: last b with s_off[b] <= j
            int lo = 0, hi = (int)np + 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (s_off[mid] <= j)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const uint32_t r = (uint32_t)lo + s_kept[j];
            if (r < newcnt) {
                gp[r] = s_sorted[j] | KCNA_FLAG_NEW | KCNA_FLAG_ISNEW;
                ++placed;
                if (r < a.K) {
                    ++flagged;
                    if (credit && s_ss[j] < a.n_nodes) a.found[s_ss[j]] = 1; // lowest joiner of this key
                }
            }
        }
        flagged = kcna_warp_sum(flagged);
        placed = kcna_warp_sum(placed);
        if ((threadIdx.x & 31) == 0 && flagged) atomicAdd(&s_flagged, flagged);
        if ((threadIdx.x & 31) == 0 && placed) atomicAdd(a.counters + 3, placed);
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicAdd(a.counters + 1, s_flagged);
            if (raw > a.CB) atomicAdd(a.counters + 2, (unsigned long long)(raw - a.CB));
            atomicAdd(a.counters + 7, (unsigned long long)nc);
            atomicAdd(a.counters + 9, (unsigned long long)newcnt);
            a.pool_cnt[node] = newcnt;
            a.cand_cnt[node] = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            a.radius[node] = newcnt >= a.limit ? kcna_key_dist(gp[a.limit - 1]) : __uint_as_float(0x7F800000u);
    }
}

// ---------------------------------------------------------------------------
// sample (update, src/kgraph.cpp:1118-1202)
// ---------------------------------------------------------------------------
__global__ void sample_m_kernel(const uint64_t *__restrict__ pool, const uint32_t *__restrict__ pool_cnt, uint32_t cap,
                                uint32_t N, uint32_t S, const uint8_t *__restrict__ found, uint32_t *__restrict__ Mv,
                                float *__restrict__ radiusM) {
    const uint32_t n = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = kcna_lane();
    if (n >= N) return;
    const uint64_t *pr = pool + (uint64_t)n * cap;
    uint32_t L = pool_cnt[n];
    uint32_t M = Mv[n];
    if (found[n]) {
        uint32_t maxl = min(M + S, L);
        uint32_t c = 0, l = maxl; // l: smallest prefix holding S flagged entries, else maxl
        for (uint32_t b = 0; b < maxl; b += 32) {
            uint32_t i = b + lane;
            bool f = i < maxl && (pr[i] & KCNA_FLAG_NEW);
            unsigned mk = __ballot_sync(KCNA_FULL, f);
            uint32_t tot = __popc(mk);
            if (c + tot >= S) {
                // position of the S-th flagged entry in this chunk
                uint32_t needed = S - c;
                unsigned mm = mk;
                for (uint32_t t = 1; t < needed; ++t) mm &= mm - 1;
                l = b + __ffs(mm);
                break;
            }
            c += tot;
        }
        M = l;
    }
    if (M == 0) M = min(1u, L); // the reference aborts here (BOOST_VERIFY, :1148)
    if (lane == 0) {
        Mv[n] = M;
        radiusM[n] = M > 0 ? kcna_key_dist(pr[M - 1]) : 0.f;
    }
}

__global__ void sample_lists_kernel(uint64_t *__restrict__ pool, uint32_t cap, uint32_t N,
                                    const uint32_t *__restrict__ Mv, const float *__restrict__ radiusM,
                                    uint32_t *__restrict__ fwd_new, uint32_t fwd_new_cap,
                                    uint32_t *__restrict__ fwd_new_cnt, uint32_t *__restrict__ fwd_old,
                                    uint32_t fwd_old_cap, uint32_t *__restrict__ fwd_old_cnt,
                                    uint32_t *__restrict__ rnew, uint32_t *__restrict__ rnew_cnt,
                                    uint32_t *__restrict__ rold, uint32_t *__restrict__ rold_cnt, uint32_t RB,
                                    unsigned long long *counters) {
    const uint32_t n = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = kcna_lane();
    if (n >= N) return;
    uint64_t *pr = pool + (uint64_t)n * cap;
    const uint32_t M = Mv[n];
    uint32_t cn = 0, co = 0;
    for (uint32_t b = 0; b < M; b += 32) {
        uint32_t l = b + lane;
        uint64_t k = l < M ? pr[l] : 0;
        bool valid = l < M;
        bool isnew = valid && (k & KCNA_FLAG_NEW);
        bool isold = valid && !(k & KCNA_FLAG_NEW);
        uint32_t id = kcna_key_id(k);
        float dd = kcna_key_dist(k);
        unsigned mn = __ballot_sync(KCNA_FULL, isnew), mo = __ballot_sync(KCNA_FULL, isold);
        if (isnew) {
            uint32_t p = cn + __popc(mn & kcna_lanemask_lt());
            if (p < fwd_new_cap) {
                fwd_new[(uint64_t)n * fwd_new_cap + p] = id;
                pr[l] = k & ~KCNA_FLAG_NEW; // used in a join from now on
            }
        }
        if (isold) {
            uint32_t p = co + __popc(mo & kcna_lanemask_lt());
            if (p < fwd_old_cap) fwd_old[(uint64_t)n * fwd_old_cap + p] = id;
        }
        // reverse edge n -> id only when n lies outside id's own join prefix
        if (valid && id < N && dd > radiusM[id]) {
            if (isnew) {
                uint32_t p = atomicAdd(rnew_cnt + id, 1u);
                if (p < RB)
                    rnew[(uint64_t)id * RB + p] = n;
                else
                    atomicAdd(counters + 12, 1ull); // dropped: which ones depends on timing
            } else {
                uint32_t p = atomicAdd(rold_cnt + id, 1u);
                if (p < RB)
                    rold[(uint64_t)id * RB + p] = n;
                else
                    atomicAdd(counters + 12, 1ull);
            }
        }
        cn += __popc(mn);
        co += __popc(mo);
    }
    if (lane == 0) {
        if (cn > fwd_new_cap) atomicAdd(counters + 4, (unsigned long long)(cn - fwd_new_cap));
        fwd_new_cnt[n] = min(cn, fwd_new_cap);
        fwd_old_cnt[n] = min(co, fwd_old_cap);
    }
}

// Random subset of R reverse entries (the reference shuffles rnn_* and keeps
// R, src/kgraph.cpp:1183-1201): each entry gets the priority
// hash(seed, iteration, node, id) and the R smallest priorities stay, in
// priority order.  The subset depends only on the set of entries, not on the
// order in which sample_lists_kernel's atomics appended them, so a run is
// reproducible as long as no list overflows RB.  Warp per list; lists of at
// most R entries are left as they are.
constexpr int SEL_WARPS = 8;
__global__ void __launch_bounds__(SEL_WARPS * 32) select_reverse_kernel(uint32_t *__restrict__ rnew,
                                                                       uint32_t *__restrict__ rnew_cnt,
                                                                       uint32_t *__restrict__ rold,
                                                                       uint32_t *__restrict__ rold_cnt, uint32_t N,
                                                                       uint32_t RB, uint32_t R, uint64_t seed,
                                                                       uint32_t iter, int P) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t *s = reinterpret_cast<uint64_t *>(smem) + (size_t)w * P;
    const uint64_t item = (uint64_t)blockIdx.x * SEL_WARPS + w; // list index: node * 2 + old
    if (item >= 2ull * N) return;
    const uint32_t node = (uint32_t)(item >> 1), old = (uint32_t)(item & 1);
    uint32_t *list = (old ? rold : rnew) + (uint64_t)node * RB;
    uint32_t *cnt = (old ? rold_cnt : rnew_cnt) + node;
    const uint32_t m = min(*cnt, RB);
    if (m <= R) {
        if (lane == 0) *cnt = m; // never more than the stored entries
        return;
    }
    const uint64_t stream = join_reverse_stream(iter, node, old);
    for (int i = lane; i < P; i += 32) {
        if (i < (int)m) {
            const uint32_t id = list[i];
            s[i] = ((uint64_t)kcna_rand32(seed, stream, id) << 32) | id;
        } else {
            s[i] = KCNA_EMPTY_KEY;
        }
    }
    kcna_warp_bitonic(s, P);
    for (uint32_t i = lane; i < R; i += 32) list[i] = (uint32_t)(s[i] & 0xFFFFFFFFull);
    if (lane == 0) *cnt = R;
}

// BF16 screen mode: every candidate the screening join emitted is recomputed
// with the canonical FP32 chain from the FP32 rows, unless its id is already
// in the target's pool: such a repeat carries the pool entry's own distance
// (the chain is symmetric), so the merge would drop it as equal to that entry,
// and it becomes an empty key without a recompute.  A recomputed candidate
// beyond the target's radius becomes an empty key too (the merges skip those).
// Warp per target: the target's row in shared memory and its first np pool
// ids (np = min(count, limit), the entries the merge compares against) in an
// open-addressing table of ht slots.  ht = 0 skips the repeat test.
// The candidates left after that test are queued, and a lane takes one row of
// 32 queued ones, eight 16-byte loads (a line) in flight: with a lane per
// candidate as they come, repeats left most lanes idle, and a line was asked
// for 16 bytes at a time after the table's share of the cache had lost it.
// 150,007 x 96, pools of 260, 1.7e8 recomputed
// pairs in six iterations: 32.6 ms before, 16.6 now.  (Adding the candidate ids to the table as well, to skip
// repeats within the buffer, was measured slower: the larger table costs
// occupancy and the inserts cost atomics.)
__global__ void __launch_bounds__(256) rescore_kernel(const float *__restrict__ X, int ld, uint32_t N,
                                                      uint64_t *__restrict__ cand, const uint32_t *__restrict__ cand_cnt,
                                                      uint32_t CB, const float *__restrict__ radius,
                                                      const uint64_t *__restrict__ pool,
                                                      const uint32_t *__restrict__ pool_cnt, uint32_t cap,
                                                      uint32_t limit, uint32_t ht, unsigned long long *rescored,
                                                      unsigned long long *repeats) {
    extern __shared__ __align__(16) float s_rows[]; // 8 warps x ld, then 8 warps x ht table slots
    __shared__ uint32_t s_queue[8][64];             // candidate indices waiting for their distance
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t t = blockIdx.x * 8 + w;
    if (t >= N) return;
    float *xt = s_rows + (size_t)w * ld;
    uint32_t *tab = reinterpret_cast<uint32_t *>(s_rows + (size_t)8 * ld) + (size_t)w * ht;
    for (int k = lane; k < ld; k += 32) xt[k] = X[(uint64_t)t * ld + k];
    if (ht) {
        for (uint32_t h = lane; h < ht; h += 32) tab[h] = KCNA_NONE;
        __syncwarp();
        const uint32_t np = min(pool_cnt[t], min(limit, cap));
        for (uint32_t i = lane; i < np; i += 32) {
            const uint32_t id = kcna_key_id(pool[(uint64_t)t * cap + i]);
            uint32_t h = (id * 0x9E3779B1u) & (ht - 1);
            for (uint32_t probe = 0; probe < ht; ++probe, h = (h + 1) & (ht - 1)) {
                const uint32_t old = atomicCAS(&tab[h], KCNA_NONE, id);
                if (old == KCNA_NONE || old == id) break;
            }
        }
    }
    __syncwarp();
    const uint32_t nc = min(cand_cnt[t], CB);
    const float rad = radius[t];
    uint64_t *buf = cand + 2 * (uint64_t)t * CB; // keys at even words
    const float4 *x4 = reinterpret_cast<const float4 *>(xt);
    unsigned long long n = 0, rep = 0;
    uint32_t *queue = s_queue[w];
    const int nv = ld >> 2;
    uint32_t queued = 0; // at most 31 stay between rounds
    for (uint32_t j0 = 0; j0 < nc; j0 += 32) {
        const uint32_t j = j0 + lane;
        bool want = false;
        if (j < nc) {
            const uint64_t k = buf[2 * j];
            if (kcna_key_noflags(k) != KCNA_EMPTY_KEY_NOFLAGS) {
                const uint32_t id = kcna_key_id(k);
                want = true;
                if (ht) {
                    uint32_t h = (id * 0x9E3779B1u) & (ht - 1);
                    for (uint32_t probe = 0; probe < ht; ++probe, h = (h + 1) & (ht - 1)) {
                        const uint32_t e = tab[h];
                        if (e == id) want = false;
                        if (e == id || e == KCNA_NONE) break;
                    }
                }
                if (!want) {
                    buf[2 * j] = KCNA_EMPTY_KEY;
                    ++rep;
                }
            }
        }
        const unsigned wm = __ballot_sync(KCNA_FULL, want);
        if (want) queue[queued + __popc(wm & ((1u << lane) - 1u))] = j;
        queued += __popc(wm);
        __syncwarp();
        const bool last = j0 + 32 >= nc;
        while (queued >= 32 || (last && queued)) {
            const uint32_t take = min(queued, 32u);
            if ((uint32_t)lane < take) {
                const uint32_t jq = queue[queued - take + lane];
                const uint64_t k = buf[2 * jq];
                const uint32_t id = kcna_key_id(k);
                const float4 *xc = reinterpret_cast<const float4 *>(X + (uint64_t)id * ld);
                float d = 0.f;
                for (int q0 = 0; q0 < nv; q0 += 8) {
                    float4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = __ldg(xc + min(q0 + u, nv - 1));
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (q0 + u < nv) d = kcna_acc4(d, x4[q0 + u], v[u]);
                }
                buf[2 * jq] = d <= rad ? kcna_key(d, id, kcna_key_flags(k)) : KCNA_EMPTY_KEY;
                ++n;
            }
            queued -= take;
            __syncwarp();
        }
    }
    n = kcna_warp_sum(n);
    rep = kcna_warp_sum(rep);
    if (lane == 0 && n) atomicAdd(rescored, n);
    if (lane == 0 && rep) atomicAdd(repeats, rep);
}

// control recall: |pool[0..min(cnt,K)) ∩ exact[0..K)| per control
__global__ void control_recall_kernel(const uint64_t *__restrict__ pool, const uint32_t *__restrict__ pool_cnt,
                                      uint32_t cap, const uint32_t *__restrict__ controls,
                                      const uint32_t *__restrict__ knn, uint32_t knn_k, uint32_t K,
                                      unsigned long long *out) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *s = reinterpret_cast<uint64_t *>(smem);
    const uint32_t c = blockIdx.x, id = controls[c];
    const int p = kcna_pow2_ceil_d((int)K);
    for (int i = threadIdx.x; i < p; i += blockDim.x) s[i] = i < (int)K ? knn[(uint64_t)c * knn_k + i] : KCNA_EMPTY_KEY;
    kcna_cta_bitonic(s, p);
    uint32_t lim = min(pool_cnt[id], K);
    unsigned long long f = 0;
    for (uint32_t i = threadIdx.x; i < lim; i += blockDim.x) {
        uint64_t q = kcna_key_id(pool[(uint64_t)id * cap + i]);
        int lb = kcna_lower_bound(s, (int)K, q);
        if (lb < (int)K && s[lb] == q) ++f;
    }
    f = kcna_warp_sum(f);
    if ((threadIdx.x & 31) == 0 && f) atomicAdd(out, f);
}

__global__ void set_radius_kernel(const uint64_t *__restrict__ pool, const uint32_t *__restrict__ pool_cnt,
                                  uint32_t cap, uint32_t N, uint32_t limit, float *__restrict__ radius) {
    uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    radius[n] = pool_cnt[n] >= limit ? kcna_key_dist(pool[(uint64_t)n * cap + limit - 1]) : __uint_as_float(0x7F800000u);
}

size_t join_smem_bytes(uint32_t capA, uint32_t capB) {
    return (size_t)(128 * JKP + JCOLS * JKP + 128 * (JCOLS + 1)) * sizeof(float) + (size_t)capA * 4 * 2 +
           (size_t)capB * 4;
}
size_t merge_smem_bytes(uint32_t cap, uint32_t CB) {
    size_t cp = (size_t)kcna_pow2_ceil((int)CB);
    return cap * 8 + cp * 8 * 2 + cp * 4 * 2 + (size_t)(cap + 2) * 4 * 3;
}

} // namespace

kcna_status kcna_nnd_alloc(kcna_ctx *c, const kcna_params *p, uint32_t maxl) {
    const uint64_t N = c->n;
    c->cap = maxl;
    c->S = p->S;
    c->Rr = p->R;
    // reverse-list buffer: 2R entries (at most 4 per join thread, 1024)
    const char *rb = getenv("KCNA_REV_CAP");
    c->RB = std::min<uint32_t>(std::max<uint32_t>(rb ? (uint32_t)atoi(rb) : 2 * p->R, std::max<uint32_t>(p->R, 32)), 1024);
    c->RB = (c->RB + 3) & ~3u; // rows of 16-byte multiples (bulk copies in the Gram-tile join)
    const char *cb = getenv("KCNA_CAND_CAP");
    uint32_t CB = cb ? (uint32_t)atoi(cb) : 4 * std::max<uint32_t>(p->L, 64);
    CB = std::min<uint32_t>(std::max<uint32_t>(CB, 64), 8192);
    c->CB = (uint32_t)kcna_pow2_ceil((int)CB);
    c->fwd_new_cap = (std::max<uint32_t>(2 * p->S, 64) + 3) & ~3u;
    c->fwd_old_cap = (std::max<uint32_t>(p->L, 1) + 3) & ~3u;
    // two spare entries: the tile prunes copy pool prefixes from an even index
    // in 16-byte units, which can reach one entry past the last row
    KCNA_TRY(kcna_alloc(c, &c->pool, N * c->cap + 2, "pool"));
    KCNA_TRY(kcna_alloc(c, &c->pool_cnt, N, "pool_cnt"));
    KCNA_TRY(kcna_alloc(c, &c->radius, N, "radius"));
    KCNA_TRY(kcna_alloc(c, &c->M, N, "M"));
    KCNA_TRY(kcna_alloc(c, &c->radiusM, N, "radiusM"));
    KCNA_TRY(kcna_alloc(c, &c->found, N, "found"));
    KCNA_TRY(kcna_alloc(c, &c->fwd_new, N * c->fwd_new_cap, "fwd_new"));
    KCNA_TRY(kcna_alloc(c, &c->fwd_new_cnt, N, "fwd_new_cnt"));
    KCNA_TRY(kcna_alloc(c, &c->fwd_old, N * c->fwd_old_cap, "fwd_old"));
    KCNA_TRY(kcna_alloc(c, &c->fwd_old_cnt, N, "fwd_old_cnt"));
    KCNA_TRY(kcna_alloc(c, &c->rnew, N * c->RB, "rnew"));
    KCNA_TRY(kcna_alloc(c, &c->rnew_cnt, N, "rnew_cnt"));
    KCNA_TRY(kcna_alloc(c, &c->rold, N * c->RB, "rold"));
    KCNA_TRY(kcna_alloc(c, &c->rold_cnt, N, "rold_cnt"));
    KCNA_TRY(kcna_alloc(c, &c->cand, 2 * N * c->CB, "candidate buffers"));
    KCNA_TRY(kcna_alloc(c, &c->cand_cnt, N, "cand_cnt"));
    KCNA_TRY(kcna_alloc(c, &c->big_list, N, "merge queue"));
    KCNA_TRY(kcna_alloc(c, &c->big_cnt, 2, "merge queue count"));
    if (!c->counters) KCNA_TRY(kcna_alloc(c, &c->counters, 64, "counters"));
    cudaStream_t s = c->stream;
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->cand_cnt, 0, N * 4, s), "memset"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->rnew_cnt, 0, N * 4, s), "memset"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->rold_cnt, 0, N * 4, s), "memset"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->fwd_old_cnt, 0, N * 4, s), "memset"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->found, 0, N, s), "memset"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->counters, 0, 64 * 8, s), "memset"));
    return KCNA_OK;
}

kcna_status kcna_cand_alloc(kcna_ctx *c, const kcna_params *p) {
    if (c->cand && c->cand_cnt && c->big_list && c->big_cnt && c->counters) return KCNA_OK;
    const uint64_t N = c->n;
    const char *cb = getenv("KCNA_CAND_CAP");
    uint32_t CB = cb ? (uint32_t)atoi(cb) : 4 * std::max<uint32_t>(p->L, 64);
    CB = std::min<uint32_t>(std::max<uint32_t>(CB, 64), 8192);
    c->CB = (uint32_t)kcna_pow2_ceil((int)CB);
    KCNA_TRY(kcna_alloc(c, &c->cand, 2 * N * c->CB, "candidate buffers"));
    KCNA_TRY(kcna_alloc(c, &c->cand_cnt, N, "cand_cnt"));
    KCNA_TRY(kcna_alloc(c, &c->big_list, N, "merge queue"));
    KCNA_TRY(kcna_alloc(c, &c->big_cnt, 2, "merge queue count"));
    if (!c->counters) KCNA_TRY(kcna_alloc(c, &c->counters, 64, "counters"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->cand_cnt, 0, N * 4, c->stream), "memset"));
    return KCNA_OK;
}

kcna_status kcna_nnd_init(kcna_ctx *c, const kcna_params *p) {
    if (p->S == 0 || p->S > 31) return kcna_fail(c, KCNA_E_ARG, "S must be in [1, 31]");
    KCNA_TRY(kcna_phase_begin(c));
    // the pools hold L entries, and M (how many the next lists come from) stays within a pool's count
    const uint32_t keep = std::min(p->S, p->L);
    init_kernel<<<kcna_div_up(c->n, 4), 128, 0, c->stream>>>(c->X, (int)c->ld, c->n, p->S, keep, c->cap, p->seed,
                                                           c->pool, c->pool_cnt, c->fwd_new, c->fwd_new_cap,
                                                           c->fwd_new_cnt);
    KCNA_LAUNCHED(c);
    KCNA_TRY(kcna_cuda_check(c, cudaGetLastError(), "init_kernel"));
    KCNA_TRY(kcna_pools_set_radius(c, p->L));
    // M = S (src/kgraph.cpp:1030)
    std::vector<uint32_t> Ms(c->n, keep);
    KCNA_TRY(kcna_cuda_check(c, cudaMemcpyAsync(c->M, Ms.data(), (size_t)c->n * 4, cudaMemcpyHostToDevice, c->stream),
                             "M init"));
    KCNA_TRY(kcna_phase_end(c, KCNA_PHASE_INIT));
    c->has_pools = true;
    return KCNA_OK;
}

kcna_status kcna_nnd_join(kcna_ctx *c, const kcna_params *p, int iter, uint64_t *n_comps) {
    JoinArgs a;
    a.X = c->X;
    a.ld = (int)c->ld;
    a.N = c->n;
    a.iter = (uint32_t)iter;
    a.seed = p->seed;
    a.R = p->R;
    a.RB = c->RB;
    a.fwd_new = c->fwd_new;
    a.fwd_new_cnt = c->fwd_new_cnt;
    a.fwd_new_cap = c->fwd_new_cap;
    a.fwd_old = c->fwd_old;
    a.fwd_old_cnt = c->fwd_old_cnt;
    a.fwd_old_cap = c->fwd_old_cap;
    a.rnew = c->rnew;
    a.rnew_cnt = c->rnew_cnt;
    a.rold = c->rold;
    a.rold_cnt = c->rold_cnt;
    a.radius = c->radius;
    a.cand = c->cand;
    a.cand_cnt = c->cand_cnt;
    a.CB = c->CB;
    a.found = c->found;
    a.counters = c->counters;
    a.capA = c->fwd_new_cap + std::min(p->R, c->RB);
    a.capB = c->fwd_old_cap + std::min(p->R, c->RB);
    a.err = c->d_err;
    size_t sm = join_smem_bytes(a.capA, a.capB);
    KCNA_TRY(kcna_allow_smem(c, join_kernel<RowsF32>, sm, "join smem attr"));
    KCNA_TRY(kcna_allow_smem(c, join_kernel<RowsB16>, sm, "join smem attr"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->counters, 0, 8 * 8, c->stream), "memset"));
    // found (src/kgraph.cpp:1104,1116): cleared for every node, then set by the
    // merge for the joiners whose candidates it inserts below K
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->found, 0, c->n, c->stream), "memset"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->big_cnt, 0, 8, c->stream), "memset"));
    KCNA_TRY(kcna_phase_begin(c));
    if ((c->gram_exact || c->bf16_screen) && kcna_join_tc_fits(a)) {
        KCNA_TRY(kcna_join_tc_launch(c, a));
        if (c->bf16_screen) {
            const uint32_t limit = std::min(p->L, c->cap);
            uint32_t ht = 64; // the pool ids at half load at most
            while (ht < 2 * limit) ht <<= 1;
            size_t rs = (size_t)8 * c->ld * 4 + (size_t)8 * ht * 4;
            if (rs > 160 * 1024) { // very long pools: recompute every candidate
                ht = 0;
                rs = (size_t)8 * c->ld * 4;
            }
            KCNA_TRY(kcna_allow_smem(c, rescore_kernel, rs, "rescore smem attr"));
            rescore_kernel<<<kcna_div_up(c->n, 8), 256, rs, c->stream>>>(
                c->X, (int)c->ld, c->n, c->cand, c->cand_cnt, c->CB, c->radius, c->pool, c->pool_cnt, c->cap, limit,
                ht, c->counters + 13, c->counters + 14);
            KCNA_LAUNCHED(c);
            KCNA_TRY(kcna_cuda_check(c, cudaGetLastError(), "rescore_kernel"));
        }
    } else {
        // the warp version queues larger nodes (in the merge's queue, idle here) for the other two
        auto launch = [&](auto rows) -> kcna_status {
            const uint32_t sms = (uint32_t)std::max(c->num_sms, 1);
            auto grid = [&](auto kern, int threads, size_t smem, uint32_t *out) -> kcna_status {
                int per_sm = 0;
                KCNA_TRY(kcna_allow_smem(c, kern, smem, "join smem attr"));
                KCNA_TRY(kcna_cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem),
                                         "join occupancy"));
                *out = std::min(kcna_div_up(c->n, threads == JM_NT ? 1 : threads / 32), sms * (uint32_t)std::max(per_sm, 1));
                return KCNA_OK;
            };
            auto warp_kern = join_warp_kernel<decltype(rows)>;
            auto mid_kern = join_mid_kernel<decltype(rows)>;
            const size_t wsm = JW_WARPS * sizeof(JoinWarp), msm = sizeof(JoinMid);
            uint32_t wg = 0, mg = 0;
            KCNA_TRY(grid(warp_kern, JW_WARPS * 32, wsm, &wg));
            KCNA_TRY(grid(mid_kern, JM_NT, msm, &mg));
            warp_kern<<<wg, JW_WARPS * 32, wsm, c->stream>>>(a, rows, c->big_list, c->big_cnt);
            mid_kern<<<mg, JM_NT, msm, c->stream>>>(a, rows, c->big_list, c->big_cnt);
            join_kernel<<<std::min(c->n, sms * 3), JT, sm, c->stream>>>(a, rows, c->big_list, c->big_cnt);
            c->launches += 3;
            return kcna_cuda_check(c, cudaGetLastError(), "join_kernel");
        };
        if (c->bf16_exact)
            KCNA_TRY(launch(RowsB16{c->Xh, (int)c->ld}));
        else
            KCNA_TRY(launch(RowsF32{c->X, (int)c->ld}));
    }
    KCNA_TRY(kcna_phase_end(c, KCNA_PHASE_JOIN));
    unsigned long long h[8] = {};
    KCNA_TRY(kcna_cuda_check(c, cudaMemcpyAsync(h, c->counters, 8 * 8, cudaMemcpyDeviceToHost, c->stream), "d2h"));
    KCNA_TRY(kcna_cuda_check(c, cudaStreamSynchronize(c->stream), "join sync"));
    if (n_comps) *n_comps = h[0];
    c->join_rows += h[5];
    c->cand_emitted += h[6];
    return KCNA_OK;
}

kcna_status kcna_merge(kcna_ctx *c, uint32_t limit, uint32_t K, uint64_t *overflow, uint64_t *flagged_topk,
                       uint64_t *merged, uint64_t *inserted, bool credit_found) {
    MergeArgs a;
    a.pool = c->pool;
    a.pool_cnt = c->pool_cnt;
    a.cap = c->cap;
    a.limit = std::min(limit, c->cap);
    a.K = K;
    a.radius = c->radius;
    a.cand = c->cand;
    a.cand_cnt = c->cand_cnt;
    a.CB = c->CB;
    a.counters = c->counters;
    a.credit = credit_found ? 1u : 0u;
    a.found = c->found;
    a.n_nodes = c->n;
    size_t sm = merge_smem_bytes(c->cap, c->CB);
    KCNA_TRY(kcna_allow_smem(c, merge_kernel, sm, "merge smem attr"));
    auto launch = [&](auto kern, int threads, uint32_t per_block, size_t smem) -> kcna_status {
        KCNA_TRY(kcna_allow_smem(c, kern, smem, "merge smem attr"));
        int per_sm = 0;
        KCNA_TRY(kcna_cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem),
                                 "merge occupancy"));
        const uint32_t grid = std::min(kcna_div_up(c->n, per_block),
                                       (uint32_t)std::max(c->num_sms, 1) * (uint32_t)std::max(per_sm, 1));
        KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->counters, 0, 10 * 8, c->stream), "memset"));
        KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->big_cnt, 0, 4, c->stream), "memset"));
        KCNA_TRY(kcna_phase_begin(c));
        kern<<<grid, threads, smem, c->stream>>>(a, c->n, c->big_list, c->big_cnt);
        return KCNA_OK;
    };
    if (!credit_found)
        KCNA_TRY(launch(merge_warp_kernel, MW_WARPS * 32, MW_WARPS, merge_warp_bytes(c->cap) * MW_WARPS));
    else
        KCNA_TRY(launch(merge_set_kernel, MS_NT, 1, merge_set_bytes(c->cap)));
    merge_kernel<<<std::max(1, c->num_sms) * 4, MT, sm, c->stream>>>(a, c->big_list, c->big_cnt);
    c->launches += 2;
    KCNA_TRY(kcna_cuda_check(c, cudaGetLastError(), "merge_kernel"));
    KCNA_TRY(kcna_phase_end(c, KCNA_PHASE_MERGE));
    unsigned long long h[10] = {};
    KCNA_TRY(kcna_cuda_check(c, cudaMemcpyAsync(h, c->counters, 10 * 8, cudaMemcpyDeviceToHost, c->stream), "d2h"));
    KCNA_TRY(kcna_cuda_check(c, cudaStreamSynchronize(c->stream), "merge sync"));
    c->cand_merged += h[7];
    c->pool_entries_merged += h[9];
    if (merged) *merged = h[7];
    if (inserted) *inserted = h[3];
    if (overflow) *overflow = h[2];
    if (flagged_topk) *flagged_topk = h[1];
    return KCNA_OK;
}

kcna_status kcna_nnd_sample(kcna_ctx *c, const kcna_params *p, int iter) {
    cudaStream_t s = c->stream;
    KCNA_TRY(kcna_phase_begin(c));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->rnew_cnt, 0, (size_t)c->n * 4, s), "memset"));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->rold_cnt, 0, (size_t)c->n * 4, s), "memset"));
    sample_m_kernel<<<kcna_div_up(c->n, 8), 256, 0, s>>>(c->pool, c->pool_cnt, c->cap, c->n, p->S, c->found, c->M,
                                                          c->radiusM);
    KCNA_LAUNCHED(c);
    sample_lists_kernel<<<kcna_div_up(c->n, 8), 256, 0, s>>>(c->pool, c->cap, c->n, c->M, c->radiusM, c->fwd_new,
                                                              c->fwd_new_cap, c->fwd_new_cnt, c->fwd_old,
                                                              c->fwd_old_cap, c->fwd_old_cnt, c->rnew, c->rnew_cnt,
                                                              c->rold, c->rold_cnt, c->RB, c->counters);
    KCNA_LAUNCHED(c);
    const int P = kcna_pow2_ceil((int)c->RB);
    KCNA_TRY(kcna_allow_smem(c, select_reverse_kernel, (size_t)SEL_WARPS * P * 8, "select smem attr"));
    select_reverse_kernel<<<kcna_div_up(2ull * c->n, SEL_WARPS), SEL_WARPS * 32, (size_t)SEL_WARPS * P * 8, s>>>(
        c->rnew, c->rnew_cnt, c->rold, c->rold_cnt, c->n, c->RB, p->R, p->seed, (uint32_t)iter, P);
    KCNA_LAUNCHED(c);
    KCNA_TRY(kcna_cuda_check(c, cudaGetLastError(), "sample kernels"));
    return kcna_phase_end(c, KCNA_PHASE_SAMPLE);
}

kcna_status kcna_pools_set_radius(kcna_ctx *c, uint32_t limit) {
    set_radius_kernel<<<kcna_div_up(c->n, 256), 256, 0, c->stream>>>(c->pool, c->pool_cnt, c->cap, c->n,
                                                                      std::min(limit, c->cap), c->radius);
    KCNA_LAUNCHED(c);
    return kcna_cuda_check(c, cudaGetLastError(), "set_radius");
}

// Controls: C random nodes and their exact MAXL-NN (GenerateControl,
// src/kgraph.cpp:363-387).  The nodes are the reference's own: the first C of
// 0..n-1 after std::random_shuffle driven by the C library's rand() in its
// initial state (the reference never seeds it), i.e. for i = 1..n-1 swap
// index[i] with index[rand() % (i + 1)].  The same generator runs here on a
// private state (random_r seeded with 1, the state rand() starts from), so
// the caller's rand() sequence is left alone; the order is cached per (n, C).
kcna_status kcna_controls_setup(kcna_ctx *c, const kcna_params *p, uint32_t maxl) {
    uint32_t C = std::min<uint32_t>(p->controls, c->n - 1);
    c->control_ids.clear();
    if (C == 0) return KCNA_OK;
    if (c->control_cache_n != c->n || c->control_cache.size() != C) {
        std::vector<uint32_t> idx(c->n);
        for (uint32_t i = 0; i < c->n; ++i) idx[i] = i;
        struct random_data rd;
        char state[128];
        std::memset(&rd, 0, sizeof rd);
        std::memset(state, 0, sizeof state);
        if (initstate_r(1u, state, sizeof state, &rd) != 0) return kcna_fail(c, KCNA_E_CUDA, "initstate_r failed");
        for (uint32_t i = 1; i < c->n; ++i) {
            int32_t r = 0;
            random_r(&rd, &r);
            std::swap(idx[i], idx[(uint32_t)r % (i + 1)]);
        }
        c->control_cache.assign(idx.begin(), idx.begin() + C);
        c->control_cache_n = c->n;
    }
    c->control_ids = c->control_cache;
    c->control_k = maxl;
    KCNA_TRY(kcna_alloc(c, &c->d_controls, C, "controls"));
    KCNA_TRY(kcna_alloc(c, &c->d_control_knn, (size_t)C * maxl, "control knn"));
    float *dd = nullptr, *rows = nullptr;
    KCNA_TRY(kcna_alloc(c, &dd, (size_t)C * maxl, "control dists"));
    KCNA_TRY(kcna_alloc(c, &rows, (size_t)C * c->ld, "control rows"));
    kcna_status st = kcna_phase_begin(c);
    if (st == KCNA_OK)
        st = kcna_cuda_check(c, cudaMemcpyAsync(c->d_controls, c->control_ids.data(), C * 4, cudaMemcpyHostToDevice,
                                                c->stream), "h2d");
    if (st == KCNA_OK) st = kcna_gather_rows(c, c->d_controls, C, rows);
    if (st == KCNA_OK) st = kcna_knn_device(c, rows, C, c->d_controls, maxl, c->d_control_knn, dd);
    if (st == KCNA_OK) st = kcna_phase_end(c, KCNA_PHASE_CONTROLS);
    kcna_release(c, dd);
    kcna_release(c, rows);
    return st;
}

kcna_status kcna_control_recall(kcna_ctx *c, uint32_t K, float *recall) {
    uint32_t C = (uint32_t)c->control_ids.size();
    if (C == 0) {
        *recall = 0.f;
        return KCNA_OK;
    }
    K = std::min(K, c->control_k);
    KCNA_TRY(kcna_phase_begin(c));
    KCNA_TRY(kcna_cuda_check(c, cudaMemsetAsync(c->counters + 8, 0, 8, c->stream), "memset"));
    size_t sm = (size_t)kcna_pow2_ceil((int)K) * 8;
    KCNA_TRY(kcna_allow_smem(c, control_recall_kernel, sm, "control recall smem attr"));
    control_recall_kernel<<<C, 256, sm, c->stream>>>(c->pool, c->pool_cnt, c->cap, c->d_controls, c->d_control_knn,
                                                     c->control_k, K, c->counters + 8);
    KCNA_LAUNCHED(c);
    KCNA_TRY(kcna_cuda_check(c, cudaGetLastError(), "control_recall"));
    KCNA_TRY(kcna_phase_end(c, KCNA_PHASE_CONTROLS));
    unsigned long long h = 0;
    KCNA_TRY(kcna_cuda_check(c, cudaMemcpyAsync(&h, c->counters + 8, 8, cudaMemcpyDeviceToHost, c->stream), "d2h"));
    KCNA_TRY(kcna_cuda_check(c, cudaStreamSynchronize(c->stream), "recall sync"));
    *recall = (float)((double)h / ((double)C * K));
    return KCNA_OK;
}

// The constructor loop of src/kgraph.cpp:1281-1459 with its stop rule
// (delta <= params.delta, recall >= params.recall, or I iterations).
kcna_status kcna_nndescent_run(kcna_ctx *c, const kcna_params *pin, kcna_stats *st) {
    kcna_params P = *pin;
    const uint32_t N = c->n;
    if (N < 3) return kcna_fail(c, KCNA_E_ARG, "need at least 3 rows");
    // parameter clamping, src/kgraph.cpp:1289-1327
    if (N <= P.controls) P.controls = N - 1;
    if (N <= P.L) P.L = N - 1;
    if (N <= P.S) P.S = N - 1;
    if (N <= P.search_L) P.search_L = N - 1;
    if (N <= P.search_K) P.search_K = N - 1;
    if (N <= P.K) {
        P.K = N - 1;
        P.loop_i = 0;
        P.S = N - 1;
        P.iterations = 0;
    }
    const uint32_t maxl = std::max(std::max(P.L, P.K), std::max(P.search_L, P.search_K));
    if (maxl > 1024) return kcna_fail(c, KCNA_E_ARG, "max(L, K, search_L, search_K) must be <= 1024");
    if (P.L == 0) return kcna_fail(c, KCNA_E_ARG, "L must be at least 1");
    st->maxl = maxl;
    KCNA_TRY(kcna_nnd_alloc(c, &P, maxl));
    KCNA_TRY(kcna_controls_setup(c, &P, maxl));
    // join iterations count from 1 when the first lists come from an update step
    int iter_base = 0;
    if (P.learned_seed) {
        KCNA_TRY(kcna_seed_learned(c, &P, st));
        KCNA_TRY(kcna_seed_finish(c, &P));
        KCNA_TRY(kcna_control_recall(c, P.K, &st->seed_recall));
        kcna_log(c, &P, "learned seed: %.1f ms (training %.1f ms), loss %.3f -> %.3f, recall %.4f", st->seed_total_ms,
                 st->seed_train_ms, st->seed_loss_first, st->seed_loss_last, st->seed_recall);
        KCNA_TRY(kcna_nnd_sample(c, &P, 1));
        iter_base = 1;
    } else {
        KCNA_TRY(kcna_nnd_init(c, &P));
    }
    uint64_t comps_total = 0;
    st->stop_condition = 0;
    st->iterations = 0;
    for (uint32_t it = 0; it < P.iterations; ++it) {
        uint64_t comps = 0, overflow = 0, flagged = 0, merged = 0, inserted = 0;
        const double j0 = c->phase_ms[KCNA_PHASE_JOIN], m0 = c->phase_ms[KCNA_PHASE_MERGE];
        KCNA_TRY(kcna_nnd_join(c, &P, (int)it + iter_base, &comps));
        KCNA_TRY(kcna_merge(c, P.L, P.K, &overflow, &flagged, &merged, &inserted, true));
        if (it < KCNA_MAX_ITERS) {
            st->iter_join_ms[it] = c->phase_ms[KCNA_PHASE_JOIN] - j0;
            st->iter_merge_ms[it] = c->phase_ms[KCNA_PHASE_MERGE] - m0;
            st->iter_cand[it] = merged;
            st->iter_inserted[it] = inserted;
        }
        comps_total += comps;
        float delta = (float)((double)flagged / ((double)N * P.K));
        float recall = 0.f;
        KCNA_TRY(kcna_control_recall(c, P.K, &recall));
        if (it < KCNA_MAX_ITERS) {
            st->iter_recall[it] = recall;
            st->iter_delta[it] = delta;
            st->iter_time[it] = kcna_now() - c->t0;
            st->iter_cand_overflow[it] = overflow;
        }
        st->iterations = it + 1;
        kcna_log(c, &P, "iteration %u recall %.4f delta %.4f comps %llu overflow %llu t %.3f", it + 1, recall, delta,
                 (unsigned long long)comps, (unsigned long long)overflow, kcna_now() - c->t0);
        KCNA_TRY(kcna_check_device_err(c, "nndescent"));
        if (delta <= P.delta) {
            st->stop_condition = 1;
            break;
        }
        if (recall >= P.recall) {
            st->stop_condition = 2;
            break;
        }
        if (it + 1 >= P.iterations) break;
        KCNA_TRY(kcna_nnd_sample(c, &P, (int)it + 1 + iter_base));
    }
    st->n_comps = comps_total;
    // pairs screened on Gram tiles; in screen mode the candidates among them were recomputed in FP32
    st->screened_pairs = (c->gram_exact || c->bf16_screen) ? comps_total : 0;
    unsigned long long resc = 0;
    KCNA_TRY(kcna_cuda_check(c, cudaMemcpyAsync(&resc, c->counters + 13, 8, cudaMemcpyDeviceToHost, c->stream), "d2h"));
    st->rescored_pairs = resc;
    unsigned long long rev_drop = 0;
    KCNA_TRY(kcna_cuda_check(c, cudaMemcpyAsync(&rev_drop, c->counters + 12, 8, cudaMemcpyDeviceToHost, c->stream), "d2h"));
    KCNA_TRY(kcna_cuda_check(c, cudaStreamSynchronize(c->stream), "sync"));
    st->rev_overflow = (uint32_t)std::min<unsigned long long>(rev_drop, 0xFFFFFFFFull);
    return KCNA_OK;
}
