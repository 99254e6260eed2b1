// RES row-wise sparsity estimator (sm_103a, FP64).
//
// Replaces the estimator loop of DynamicOptimizer::rows_sparse_optimal_matrix_chain_order
// (efficient/resmcm.cpp:506-517), getSparsities (:442-452) and
// compute_sparsities (:468-485):
//   r_ii[u] = min(1, |M_i[u]| / dim(vts[i+1]))
//   r_ij[u] = 1 - prod_{v in M_i[u]} (1 - r_{i+1,j}[v])          (j > i)
//   c_ij    = sum_u r_ij[u] * dim(vts[j+1])
// for i = len-1 .. 0.  dim(vts[j+1]) is the column count of M_j.
//
// One launch per level i computes every j > i at once, so each M_i is read
// once: a level stores q = 1 - r (r rounded first, then 1 - r rounded, the
// value the reference's next level forms), the len - i values of a row one
// after another (its own, then targets i + 1 ..), so the next level multiplies
// the gathered q directly, a row's gathers for all j are one contiguous run of
// doubles, and no level's table is wider than its targets.
// Mapping: lane (row, g, jo) multiplies the factors of entries g, g + G, ...
// of its row for target i + 1 + jo, and the G partial products of a row are
// combined with shuffles in a fixed order.  Sums of c_ij are per-warp, then
// per-block (fixed warp order), then a pass over the block partials (fixed
// order): the estimate is bit-for-bit reproducible run to run.
// Every multiply and add is an explicit round-to-nearest intrinsic, so no
// fused multiply-add changes the rounding against the reference's
// `tmp_rho *= (1 - r)` and `nnz += s * dim`.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <mutex>
#include <vector>

#include "internal.h"

namespace rmcm {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kEstThreads = 256;
constexpr int kMaxLen = 16;

struct LevelArgs {
    int32_t len;            // chain length (matrices)
    int32_t i;              // level
    int32_t nj;             // number of j > i (len - 1 - i)
    int32_t jp;             // lanes per group (power of two >= nj, >= 1)
    int32_t tile;           // rows a warp takes per step (1 .. 32)
    double dim_leaf;        // dim(vts[i+1]) = cols of M_i
    double dims[kMaxLen];   // dims[j] = cols of M_j
};

// prod over entries k = k0, k0 + G, ... < k1 of q_next[col_k * stride] (= 1 - r)
// for the rows that several warps share: eight independent partial products
// per lane, the next entries' columns loaded while the factors arrive, so one
// gather's latency a step of eight; combined in a fixed order.
__device__ __forceinline__ double factor_product(const DevCsr &M, const double *q_next, int32_t stride, int64_t k0,
                                                 int64_t k1, int G) {
    constexpr int U = 8;
    double p[U];
    int32_t v[U];
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = k0 + u * (int64_t)G < k1 ? __ldg(M.col + k0 + u * (int64_t)G) : -1;
#pragma unroll
    for (int u = 0; u < U; u++) {
        p[u] = v[u] >= 0 ? __ldg(q_next + (int64_t)v[u] * stride) : 1.0;
        const int64_t kn = k0 + (U + u) * (int64_t)G;
        v[u] = kn < k1 ? __ldg(M.col + kn) : -1;
    }
    for (int64_t k = k0 + U * (int64_t)G; k < k1; k += U * (int64_t)G) {
        double q[U];
#pragma unroll
        for (int u = 0; u < U; u++) q[u] = v[u] >= 0 ? __ldg(q_next + (int64_t)v[u] * stride) : 1.0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t kn = k + (U + u) * (int64_t)G;
            v[u] = kn < k1 ? __ldg(M.col + kn) : -1;
        }
#pragma unroll
        for (int u = 0; u < U; u++) p[u] = __dmul_rn(p[u], q[u]);
    }
    return __dmul_rn(__dmul_rn(__dmul_rn(p[0], p[1]), __dmul_rn(p[2], p[3])),
                     __dmul_rn(__dmul_rn(p[4], p[5]), __dmul_rn(p[6], p[7])));
}

// Rows per warp and chunk: 32 when that leaves a quarter of a full grid's
// warps (blocks_cap CTAs) with a chunk, fewer for shorter matrices.
inline int32_t level_tile(int64_t rows, int64_t blocks_cap) {
    const int64_t warps = blocks_cap * (kEstThreads / 32) / 4;
    int32_t t = 32;
    while (t > 1 && rows < warps * t) t >>= 1;
    return t;
}

// One level of one chain, as CTA `bid` of `nblk` (the same work split and
// summation order whether the CTA belongs to a one-chain launch or to a
// launch over many chains).
//
// Bound by the FP64 pipe: a warp's multiply holds it for many cycles whatever
// its active lanes, so lanes are packed.  The warp's rows take 1, 2, 4 ..
// groups of jp lanes, enough for four entries a lane (32 / jp groups at most),
// and are laid out group after group, the largest first: every step multiplies
// 32 / jp groups' entries, three multiplies and one per halving of the largest
// row in it.  Against a row per warp step (one to three of 32 lanes busy on
// most rows of a Zipf leaf) and 4,096 entries as one warp's share: a six-matrix
// chain over the 1,000,000 x 300,000 leaf with 20M entries 1,626 -> 715 us in
// all.
//
// A chunk's rows lie nch apart, so that neighbours of like length (rows sorted
// by degree, hubs numbered together) come to different CTAs: with 32
// consecutive rows a warp, one CTA held most of the long ones (100,000 rows of
// 60,000 / (rank + 10) entries, six matrices: 3,468 us so, 287 now).
// Rows of more than kWideLane entries a lane hold up their warp.  The CTA's
// warps multiply a slice of each together where one warp has more than twice
// the average of them; that costs a slice's combining multiplies and two
// barriers a row, so evenly long rows stay with their warps (3,000 rows of 900,
// five matrices: 199 us shared, 139 not) unless a slice is long itself.
constexpr int kWideLane = 64;

__device__ __forceinline__ void res_level_body(const DevCsr &M, const double *q_next, double *q_cur,
                                               const LevelArgs &la, double *partial, bool skip_long, int64_t bid,
                                               int64_t nblk) {
    constexpr int NW = kEstThreads / 32;
    if (la.nj == 0) {
        // the chain's last matrix: its own densities only, a row per thread
        for (int64_t u = bid * kEstThreads + threadIdx.x; u < M.rows; u += nblk * kEstThreads) {
            const double r = __ddiv_rn((double)(M.rowptr[u + 1] - M.rowptr[u]), la.dim_leaf);
            q_cur[u] = __dsub_rn(1.0, r > 1.0 ? 1.0 : r);
        }
        return;
    }
    __shared__ double s_tp[NW][32 * kMaxLen];   // tile products: [t * jp + jo]
    __shared__ double s_wide[NW][kMaxLen];      // slices of a wide row
    __shared__ uint8_t s_ord[NW][32];           // the warp's rows, most groups first
    __shared__ uint2 s_mask[NW];                // each warp's wide rows, the huge ones, and the former's entries
    __shared__ int32_t s_load[NW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int T = la.tile;                      // rows per warp and chunk (1 .. 32)
    const int jp = la.jp, qs = la.nj + 1;       // values per row of q_cur
    const int ng = 32 / jp;                     // groups per step
    const int emax = 31 - __clz(ng);
    const int64_t wide_min = kWideLane * (int64_t)ng;
    const int64_t nch = (M.rows + NW * T - 1) / (NW * T);   // chunks
    const int jo = lane & (jp - 1);             // target i + 1 + jo
    const bool active_j = jo < la.nj;
    const double dimj = active_j ? la.dims[la.i + 1 + jo] : 0.0;
    double term_sum = 0.0;                      // this lane's rows of target jo
    double *tp = s_tp[warp];
    for (int64_t c = bid; c < nch; c += nblk) {
        auto row_at = [&](int p) { return p * nch + c; };   // row of place p of the chunk
        const int nrow = __popc(__ballot_sync(kFull, lane < T && row_at(warp * T + lane) < M.rows));
        // r_ii of the tile's rows, a lane each (one division for T rows)
        int64_t my_a0 = 0, my_len = 0;
        if (lane < nrow) {
            const int64_t ul = row_at(warp * T + lane);
            my_a0 = M.rowptr[ul];
            my_len = M.rowptr[ul + 1] - my_a0;
            double r = __ddiv_rn((double)my_len, la.dim_leaf);
            r = r > 1.0 ? 1.0 : r;
            q_cur[ul * qs] = __dsub_rn(1.0, r);
        }
        const bool is_long = skip_long && my_len > kEstLongRow;   // a cluster of k_res_long takes it
        const uint32_t skipped = __ballot_sync(kFull, is_long);
        // wide rows that the CTA's warps multiply together
        uint32_t wide = __ballot_sync(kFull, !is_long && my_len > wide_min);
        const bool any_wide = __syncthreads_or(wide != 0);
        bool uneven = false;
        if (any_wide) {
            const uint32_t huge = __ballot_sync(kFull, !is_long && my_len > 16 * wide_min);
            const int load = __reduce_add_sync(kFull, (wide >> lane) & 1u ? (int)min(my_len, (int64_t)(INT_MAX >> 9)) : 0);
            if (lane == 0) {
                s_mask[warp] = make_uint2(wide, huge);
                s_load[warp] = load;
            }
            __syncthreads();
            int64_t most = 0, all = 0;
            for (int w = 0; w < NW; w++) {
                most = s_load[w] > most ? s_load[w] : most;
                all += s_load[w];
            }
            uneven = most * NW > 2 * all;
            if (!uneven) wide = huge;
        }
        // the row's groups: 2^e of them, -1 for none (its product is 1, or
        // another part of the kernel's)
        int e = -1;
        if (lane < nrow && my_len > 0 && !(((skipped | wide) >> lane) & 1u)) {
            e = my_len <= 4 ? 0 : 32 - __clz((int)((my_len + 3) / 4 - 1));
            e = e < emax ? e : emax;
        }
        if (lane < nrow && my_len == 0)
            for (int x = 0; x < la.nj; x++) tp[lane * jp + x] = 1.0;
        // class x's rows take groups base[x] .. in order of rank, from place[x]
        int base[6], place[6], groups = 0, placed = 0;
#pragma unroll
        for (int x = 5; x >= 0; x--) {
            const unsigned of = __ballot_sync(kFull, e == x);
            base[x] = groups;
            place[x] = placed;
            if (e == x) s_ord[warp][placed + __popc(of & lt_mask)] = (uint8_t)lane;
            groups += __popc(of) << x;
            placed += __popc(of);
        }
        __syncwarp();
        for (int s0 = 0; s0 < groups; s0 += ng) {
            // this lane's group, and the class it lies in: the least with
            // base <= s (bases ascend as classes descend)
            const bool live = s0 + lane / jp < groups;
            const int s = live ? s0 + lane / jp : groups - 1;
            int x = 5, bx = base[5], px = place[5];
#pragma unroll
            for (int y = 4; y >= 0; y--) {
                if (s >= base[y]) {
                    x = y;
                    bx = base[y];
                    px = place[y];
                }
            }
            const int t = s_ord[warp][px + ((s - bx) >> x)];
            const int G = 1 << x, g = (s - bx) & (G - 1);
            const int64_t a0 = __shfl_sync(kFull, my_a0, t);
            const int64_t rl = __shfl_sync(kFull, my_len, t);
            int64_t k = a0 + g;
            const int64_t k1 = live && active_j ? a0 + rl : a0;
            double p[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                p[u] = k + u * G < k1 ? __ldg(q_next + (int64_t)__ldg(M.col + k + u * G) * la.nj + jo) : 1.0;
            for (k += 4 * G; k < k1; k += 4 * G) {
                double q[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    q[u] = k + u * G < k1 ? __ldg(q_next + (int64_t)__ldg(M.col + k + u * G) * la.nj + jo) : 1.0;
#pragma unroll
                for (int u = 0; u < 4; u++) p[u] = __dmul_rn(p[u], q[u]);
            }
            double prod = __dmul_rn(__dmul_rn(p[0], p[1]), __dmul_rn(p[2], p[3]));
            // a row's groups are consecutive and aligned to their number: combine
            // them pairwise (fixed order); rows of fewer groups keep theirs
            const int most = __reduce_max_sync(kFull, live ? x : 0);
            for (int d = 0; d < most; d++) {
                const double o = __shfl_xor_sync(kFull, prod, jp << d);
                if (d < x) prod = __dmul_rn(prod, o);
            }
            if (live && g == 0 && active_j) tp[t * jp + jo] = prod;
        }
        // their products, warp by warp: every warp a slice
        if (any_wide) {
            const int G = 32 / jp, wg = lane / jp;
            for (int w = 0; w < NW; w++) {
                for (uint32_t m = uneven ? s_mask[w].x : s_mask[w].y; m; m &= m - 1) {
                    const int t = __ffs(m) - 1;
                    const int64_t u = row_at(w * T + t);
                    const int64_t a0 = M.rowptr[u], len = M.rowptr[u + 1] - a0;
                    const int64_t k0 = a0 + len * warp / NW, k1 = a0 + len * (warp + 1) / NW;
                    double prod = 1.0;
                    if (active_j) prod = factor_product(M, q_next + jo, la.nj, k0 + wg, k1, G);
                    for (int d = jp; d < 32; d <<= 1) prod = __dmul_rn(prod, __shfl_xor_sync(kFull, prod, d));
                    if (wg == 0 && active_j) s_wide[warp][jo] = prod;
                    __syncthreads();
                    if ((int)threadIdx.x < la.nj) {
                        double p = 1.0;
                        for (int x = 0; x < NW; x++) p = __dmul_rn(p, s_wide[x][threadIdx.x]);
                        s_tp[w][t * jp + threadIdx.x] = p;
                    }
                    __syncthreads();
                }
            }
        }
        __syncwarp();
        // per (row, target): r = 1 - prod, its term r * dim_j, and q = 1 - r
        // for the next level; a lane takes every (32 / jp)-th row
        if (active_j) {
            for (int t = lane / jp; t < nrow; t += 32 / jp) {
                if ((skipped >> t) & 1u) continue;
                const double r = __dsub_rn(1.0, tp[t * jp + jo]);
                q_cur[row_at(warp * T + t) * qs + 1 + jo] = __dsub_rn(1.0, r);
                term_sum = __dadd_rn(term_sum, __dmul_rn(r, dimj));
            }
        }
        __syncwarp();
    }
    // this warp's sums per target, over its lanes in a fixed order
    for (int d = jp; d < 32; d <<= 1) term_sum = __dadd_rn(term_sum, __shfl_xor_sync(kFull, term_sum, d));
    // block partials: partial[block * kMaxLen + jo]
    __shared__ double s_part[NW][kMaxLen];
    if (lane < jp && active_j) s_part[warp][jo] = term_sum;
    __syncthreads();
    if (threadIdx.x < la.nj) {
        double acc = 0.0;
        for (int w = 0; w < NW; w++) acc = __dadd_rn(acc, s_part[w][threadIdx.x]);
        partial[bid * kMaxLen + threadIdx.x] = acc;
    }
}

__global__ void __launch_bounds__(kEstThreads, 5) k_res_level(DevCsr M, const double *q_next, double *q_cur,
                                                           LevelArgs la, double *partial, bool skip_long) {
    res_level_body(M, q_next, q_cur, la, partial, skip_long, blockIdx.x, gridDim.x);
}

// Long rows (listed ascending): a CTA each, its warps multiplying the factors
// of one of as many equal slices of the row, combined in warp order; rows of
// more than kEstSpreadRow entries a cluster of CTAs, whose products (read
// through distributed shared memory) are combined in rank order.  The row's
// terms s * dim_j go to the partial of its place in the list, after the
// partials of k_res_level, so the reduction still adds them in a fixed order.
constexpr int kEstLongThreads = 256;
constexpr int kEstLongCluster = 8;
constexpr int64_t kEstSpreadRow = 8192;

__device__ __forceinline__ void res_long_row(const DevCsr &M, const double *q_next, double *q_cur, const LevelArgs &la,
                                             int64_t u, double *partial, int rank, int ranks) {
    constexpr int NW = kEstLongThreads / 32;
    __shared__ double s_prod[NW][kMaxLen];
    __shared__ double s_cta[kMaxLen];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = 32 / la.jp;
    const int g = lane / la.jp;
    const int jo = lane % la.jp;
    const bool active_j = jo < la.nj;
    const int64_t a0 = M.rowptr[u], len = M.rowptr[u + 1] - a0;
    const int slice = rank * NW + warp, slices = ranks * NW;
    const int64_t k0 = a0 + len * slice / slices, k1 = a0 + len * (slice + 1) / slices;
    double prod = 1.0;
    if (active_j) prod = factor_product(M, q_next + jo, la.nj, k0 + g, k1, G);
    for (int d = la.jp; d < 32; d <<= 1) {
        const double o = __shfl_xor_sync(kFull, prod, d);
        prod = __dmul_rn(prod, o);
    }
    if (g == 0 && active_j) s_prod[warp][jo] = prod;
    __syncthreads();
    double p = 1.0;
    if ((int)threadIdx.x < la.nj) {
        for (int w = 0; w < NW; w++) p = __dmul_rn(p, s_prod[w][threadIdx.x]);
        s_cta[threadIdx.x] = p;
    }
    if (ranks > 1) {
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        cluster.sync();
        if (rank == 0 && (int)threadIdx.x < la.nj)
            for (int c = 1; c < ranks; c++) p = __dmul_rn(p, cluster.map_shared_rank(s_cta, c)[threadIdx.x]);
        cluster.sync();   // the products are read: the CTAs may go on
    }
    if (rank == 0 && (int)threadIdx.x < la.nj) {
        const double sv = __dsub_rn(1.0, p);
        q_cur[u * (la.nj + 1) + 1 + threadIdx.x] = __dsub_rn(1.0, sv);   // q = 1 - r for the next level
        partial[threadIdx.x] = __dmul_rn(sv, la.dims[la.i + 1 + threadIdx.x]);
    }
    __syncthreads();   // s_prod is free
}

// The rows of places p0 .. p1 - 1 by one cluster: those a CTA takes alone dealt
// to its CTAs, then those that the cluster takes together.  row(place, ranks,
// rank) works on one of them; length(place) is its entries.
template <typename Length, typename Row>
__device__ __forceinline__ void res_long_rows(int64_t p0, int64_t p1, Length length, Row row) {
    const int rank = (int)cooperative_groups::this_cluster().block_rank();
    for (int64_t p = p0 + rank; p < p1; p += kEstLongCluster)
        if (length(p) <= kEstSpreadRow) row(p, 0, 1);
    for (int64_t p = p0; p < p1; p++)
        if (length(p) > kEstSpreadRow) row(p, rank, kEstLongCluster);
}

// Places a cluster takes: one while the device has room for a cluster each.
inline int32_t long_places(int64_t nlong, int sm_count) { return nlong <= 2 * sm_count ? 1 : kEstLongCluster; }

__global__ void __cluster_dims__(kEstLongCluster, 1, 1) __launch_bounds__(kEstLongThreads)
    k_res_long(DevCsr M, const double *q_next, double *q_cur, LevelArgs la, const int32_t *long_rows, int32_t nlong,
               int32_t places, double *partial) {
    const int64_t p0 = (int64_t)(blockIdx.x / kEstLongCluster) * places;
    res_long_rows(
        p0, min(p0 + places, (int64_t)nlong),
        [&](int64_t p) { return M.rowptr[long_rows[p] + 1] - M.rowptr[long_rows[p]]; },
        [&](int64_t p, int rank, int ranks) {
            res_long_row(M, q_next, q_cur, la, long_rows[p], partial + p * kMaxLen, rank, ranks);
        });
}

// One block, target jo: c[i*len + j] = sum over blocks (fixed pairwise order).
__device__ __forceinline__ void res_reduce_body(const double *partial, int32_t nblocks, int32_t len, int32_t i, int jo,
                                                double *c) {
    __shared__ double s[256];
    double acc = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) acc = __dadd_rn(acc, partial[(int64_t)b * kMaxLen + jo]);
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] = __dadd_rn(s[threadIdx.x], s[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) c[i * len + i + 1 + jo] = s[0];
}

// A CTA per target of one level.
__global__ void __launch_bounds__(256) k_res_reduce(const double *partial, int32_t nblocks, LevelArgs la, double *c) {
    res_reduce_body(partial, nblocks, la.len, la.i, blockIdx.x, c);
}

// Every estimate of a chain in one launch: CTA (j, i) sums level i's partials
// of target j, or clears an entry on or below the diagonal.
struct ReduceArgs {
    int32_t len;
    int32_t nblocks[kMaxLen];       // partials of each level
    int32_t first[kMaxLen];         // its first one
};

__global__ void __launch_bounds__(256) k_res_reduce_all(const double *partial, ReduceArgs ra, double *c) {
    const int i = blockIdx.y, j = blockIdx.x;
    if (j > i) res_reduce_body(partial + (int64_t)ra.first[i] * kMaxLen, ra.nblocks[i], ra.len, i, j - i - 1, c);
    else if (threadIdx.x == 0) c[i * ra.len + j] = 0.0;
}

// Many chains at once: job j is one level of one chain, exactly the launch
// the one-chain estimator makes for it (its CTAs are blocks first .. first +
// blocks - 1 of this grid), so every chain's estimates are bit-identical to
// rmcm_estimate's.
struct LevelJob {
    DevCsr M;
    const double *q_next;
    double *q_cur;
    double *partial;
    double *c;                  // the chain's len x len estimates
    const int32_t *long_rows;   // rows that k_res_long takes (nlong of them)
    LevelArgs la;
    int64_t first, blocks;      // CTAs of the level launch
    int64_t lfirst;             // its places among the long rows of the launch: lfirst .. lfirst + nlong - 1
    int32_t nlong;
};

__device__ __forceinline__ int find_job(const LevelJob *jobs, int njobs, int64_t b, bool longs) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((longs ? jobs[mid].lfirst : jobs[mid].first) <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(kEstThreads, 5) k_res_level_multi(const LevelJob *jobs, int32_t njobs) {
    const LevelJob &jb = jobs[find_job(jobs, njobs, blockIdx.x, false)];
    res_level_body(jb.M, jb.q_next, jb.q_cur, jb.la, jb.partial, jb.nlong > 0, (int64_t)blockIdx.x - jb.first,
                   jb.blocks);
}

__global__ void __cluster_dims__(kEstLongCluster, 1, 1) __launch_bounds__(kEstLongThreads)
    k_res_long_multi(const LevelJob *jobs, int32_t njobs, int64_t nlong, int32_t places) {
    const int64_t p0 = (int64_t)(blockIdx.x / kEstLongCluster) * places;
    res_long_rows(
        p0, min(p0 + places, nlong),
        [&](int64_t p) {
            const LevelJob &jb = jobs[find_job(jobs, njobs, p, true)];
            const int64_t u = jb.long_rows[p - jb.lfirst];
            return jb.M.rowptr[u + 1] - jb.M.rowptr[u];
        },
        [&](int64_t p, int rank, int ranks) {
            const LevelJob &jb = jobs[find_job(jobs, njobs, p, true)];
            res_long_row(jb.M, jb.q_next, jb.q_cur, jb.la, jb.long_rows[p - jb.lfirst],
                         jb.partial + (jb.blocks + p - jb.lfirst) * kMaxLen, rank, ranks);
        });
}

__global__ void __launch_bounds__(256) k_res_reduce_multi(const LevelJob *jobs) {
    const LevelJob &jb = jobs[blockIdx.x];
    if ((int)blockIdx.y < jb.la.nj)
        res_reduce_body(jb.partial, (int32_t)(jb.blocks + jb.nlong), jb.la.len, jb.la.i, blockIdx.y, jb.c);
}

}  // namespace

int32_t estimate(rmcm_handle *h, rmcm_mat *const *chain, int32_t len, double *c_dev) {
    if (len < 1 || len > kMaxLen) return set_error(h, RMCM_EINVAL, "estimate: chain length must be 1..16");
    cudaStream_t s = h->stream;
    int64_t max_rows = 1;
    for (int i = 0; i < len; i++) {
        if (!chain[i]) return set_error(h, RMCM_EINVAL, "estimate: null matrix");
        if (i + 1 < len && chain[i]->d.cols != chain[i + 1]->d.rows)
            return set_error(h, RMCM_EINVAL, "estimate: consecutive matrices do not chain");
        max_rows = std::max(max_rows, chain[i]->d.rows);
    }
    // grid is fixed by the row count only, so the reduction order is stable
    const int64_t blocks_cap = (int64_t)h->sm_count * 8;
    auto al = [](int64_t x) { return (x + 255) & ~255LL; };
    const int64_t rbytes = al(8 * max_rows * len);
    // block partials of every level, one after another, summed by one launch
    ReduceArgs ra{};
    ra.len = len;
    int64_t nparts = 0;
    for (int i = len - 1; i >= 0; i--) {
        const int64_t rows = chain[i]->d.rows, tile = level_tile(rows, blocks_cap);
        const int64_t blocks = std::max<int64_t>(
            1, std::min((rows + tile * (kEstThreads / 32) - 1) / (tile * (kEstThreads / 32)), blocks_cap));
        const int32_t nlong = i < len - 1 && chain[i]->n_est_long > 0 ? chain[i]->n_est_long : 0;
        ra.first[i] = (int32_t)nparts;
        ra.nblocks[i] = (int32_t)(blocks + nlong);
        nparts += blocks + nlong;
    }
    const int64_t pbytes = al(8 * nparts * kMaxLen);
    double *r_a = nullptr, *r_b = nullptr, *part = nullptr;
    RMCM_TRY(dev_alloc(h, (void **)&r_a, 2 * rbytes + pbytes));
    r_b = (double *)((char *)r_a + rbytes);
    part = (double *)((char *)r_a + 2 * rbytes);
    cudaError_t e = cudaSuccess;
    double *r_cur = r_a, *r_next = r_b;
    for (int i = len - 1; i >= 0 && e == cudaSuccess; i--) {
        const DevCsr &M = chain[i]->d;
        LevelArgs la{};
        la.len = len;
        la.i = i;
        la.nj = len - 1 - i;
        int jp = 1;
        while (jp < la.nj) jp <<= 1;
        la.jp = jp;
        la.dim_leaf = (double)M.cols;
        for (int j = 0; j < len; j++) la.dims[j] = (double)chain[j]->d.cols;
        la.tile = level_tile(M.rows, blocks_cap);
        // rows of more than kEstLongRow entries (known for uploaded matrices)
        // get a cluster of CTAs each
        const int32_t nlong = la.nj > 0 && chain[i]->n_est_long > 0 ? chain[i]->n_est_long : 0;
        const int32_t blocks = ra.nblocks[i] - nlong;
        double *lp = part + (int64_t)ra.first[i] * kMaxLen;
        k_res_level<<<(unsigned)blocks, kEstThreads, 0, s>>>(M, r_next, r_cur, la, lp, nlong > 0);
        h->launches++;
        if (nlong > 0) {
            const int32_t places = long_places(nlong, h->sm_count);
            k_res_long<<<(unsigned)((nlong + places - 1) / places * kEstLongCluster), kEstLongThreads, 0, s>>>(
                M, r_next, r_cur, la, chain[i]->est_long, nlong, places, lp + (int64_t)blocks * kMaxLen);
            h->launches++;
        }
        e = cudaGetLastError();
        std::swap(r_cur, r_next);
    }
    if (e == cudaSuccess) {
        k_res_reduce_all<<<dim3((unsigned)len, (unsigned)len), 256, 0, s>>>(part, ra, c_dev);
        h->launches++;
        e = cudaGetLastError();
    }
    dev_free(h, r_a, 2 * rbytes + pbytes);
    if (e != cudaSuccess) return cuda_error(h, e, "estimator launch");
    return RMCM_OK;
}


// Estimates of many chains, a launch per level step over all of them: step s
// runs level len_c - 1 - s of every chain c longer than s.  Job tables go to
// the device through the arena (persistent pinned host memory and device
// memory, so that a stream capture records copies that stay valid).
int32_t estimate_multi(rmcm_handle *h, const EstChain *chains, int32_t n, TableArena &arena) {
    cudaStream_t s = h->stream;
    const int64_t blocks_cap = (int64_t)h->sm_count * 8;
    auto al = [](int64_t x) { return (x + 255) & ~255LL; };
    int32_t max_len = 0;
    std::vector<int64_t> off(n + 1, 0);
    for (int32_t c = 0; c < n; c++) {
        const int32_t len = chains[c].len;
        if (len < 1 || len > kMaxLen) return set_error(h, RMCM_EINVAL, "estimate: chain length must be 1..16");
        max_len = std::max(max_len, len);
        int64_t max_rows = 1, long_cap = 0;
        for (int i = 0; i < len; i++) {
            max_rows = std::max(max_rows, chains[c].mats[i]->d.rows);
            long_cap = std::max<int64_t>(long_cap, chains[c].mats[i]->n_est_long);
        }
        off[c + 1] = off[c] + 2 * al(8 * max_rows * len) + al(8 * (blocks_cap + long_cap) * kMaxLen);
    }
    char *buf = nullptr;
    RMCM_TRY(dev_alloc(h, (void **)&buf, std::max<int64_t>(off[n], 256)));
    cudaError_t e = cudaSuccess;
    for (int32_t c = 0; c < n && e == cudaSuccess; c++)
        e = cudaMemsetAsync(chains[c].c_dev, 0, sizeof(double) * chains[c].len * chains[c].len, s);
    std::vector<LevelJob> jobs;
    for (int32_t st = 0; st < max_len && e == cudaSuccess; st++) {
        jobs.clear();
        int64_t nb = 0, nl = 0;
        for (int32_t c = 0; c < n; c++) {
            const int32_t len = chains[c].len;
            if (st >= len) continue;
            const int i = len - 1 - st;
            int64_t max_rows = 1;
            for (int q = 0; q < len; q++) max_rows = std::max(max_rows, chains[c].mats[q]->d.rows);
            const int64_t rbytes = al(8 * max_rows * len);
            // the one-chain estimator swaps its two level buffers every level
            double *ra = (double *)(buf + off[c]), *rb = (double *)(buf + off[c] + rbytes);
            double *r_cur = (st % 2 == 0) ? ra : rb, *r_next = (st % 2 == 0) ? rb : ra;
            const rmcm_mat *Mi = chains[c].mats[i];
            LevelJob jb{};
            jb.M = Mi->d;
            jb.q_next = r_next;
            jb.q_cur = r_cur;
            jb.partial = (double *)(buf + off[c] + 2 * rbytes);
            jb.c = chains[c].c_dev;
            jb.la.len = len;
            jb.la.i = i;
            jb.la.nj = len - 1 - i;
            int jp = 1;
            while (jp < jb.la.nj) jp <<= 1;
            jb.la.jp = jp;
            jb.la.dim_leaf = (double)Mi->d.cols;
            for (int q = 0; q < len; q++) jb.la.dims[q] = (double)chains[c].mats[q]->d.cols;
            jb.la.tile = level_tile(Mi->d.rows, blocks_cap);
            int64_t blocks = (Mi->d.rows + (int64_t)jb.la.tile * (kEstThreads / 32) - 1) /
                             ((int64_t)jb.la.tile * (kEstThreads / 32));
            jb.blocks = std::max<int64_t>(1, std::min(blocks, blocks_cap));
            jb.nlong = jb.la.nj > 0 && Mi->n_est_long > 0 ? Mi->n_est_long : 0;
            jb.long_rows = Mi->est_long;
            jb.first = nb;
            jb.lfirst = nl;
            nb += jb.blocks;
            nl += jb.nlong;
            jobs.push_back(jb);
        }
        void *hp = nullptr, *dp = nullptr;
        const int64_t tbytes = (int64_t)sizeof(LevelJob) * (int64_t)jobs.size();
        if (!arena.push(tbytes, &hp, &dp)) {
            dev_free(h, buf, std::max<int64_t>(off[n], 256));
            return set_error(h, RMCM_EINTERNAL, "estimate: job table arena full");
        }
        memcpy(hp, jobs.data(), tbytes);
        e = cudaMemcpyAsync(dp, hp, tbytes, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) break;
        k_res_level_multi<<<(unsigned)nb, kEstThreads, 0, s>>>((const LevelJob *)dp, (int32_t)jobs.size());
        h->launches++;
        if (nl > 0) {
            const int32_t places = long_places(nl, h->sm_count);
            k_res_long_multi<<<(unsigned)((nl + places - 1) / places * kEstLongCluster), kEstLongThreads, 0, s>>>(
                (const LevelJob *)dp, (int32_t)jobs.size(), nl, places);
            h->launches++;
        }
        if (st > 0) {   // (the first step is every chain's last level: no targets)
            k_res_reduce_multi<<<dim3((unsigned)jobs.size(), (unsigned)st), 256, 0, s>>>((const LevelJob *)dp);
            h->launches++;
        }
        e = cudaGetLastError();
    }
    dev_free(h, buf, std::max<int64_t>(off[n], 256));
    if (e != cudaSuccess) return cuda_error(h, e, "multi-chain estimator launch");
    return RMCM_OK;
}

// ---------------------------------------------------------------------------
// RES estimator for callers that cannot allocate device memory
// ---------------------------------------------------------------------------
//
// Some callers of this library may not call cudaMalloc (or any allocating
// routine) at the point where they need an estimate: a host framework that
// owns every byte of device memory through its own pool and forbids plugins
// from allocating behind its back, or a latency-critical serving loop that
// allows no allocation after start-up (an allocation can synchronise the
// device or fail under memory pressure at the worst moment).
// rmcm_estimate_noalloc serves them.  The caller passes
// its chain as plain device CSR arrays it already owns and a host array for
// the estimates; every temporary the estimator needs (two levels of row
// sparsities, per-block partial sums and the estimate matrix) lives in the
// file-scope array below, a fixed 32 MiB that every GPU which loads this
// library holds until the process exits.  The array's address is looked up
// once per device, on the first call made with that device current.

namespace {

constexpr int64_t kNoAllocScratchBytes = 32LL << 20;
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

struct NoAllocDevice {
    bool ready = false;
    unsigned char *scratch = nullptr;   // device address of g_noalloc_scratch
    int sm_count = 0;
};
std::mutex g_noalloc_mu;
NoAllocDevice g_noalloc_dev[128];

}  // namespace
}  // namespace rmcm

extern "C" RMCM_API int32_t rmcm_estimate_noalloc(int32_t len, const int64_t *rows, const int64_t *cols,
                                                  const int64_t *const *rowptr, const int32_t *const *col,
                                                  double *c_out, void *stream) {
    using namespace rmcm;
    if (len < 1 || len > kMaxLen || !rows || !cols || !rowptr || !col || !c_out) return RMCM_EINVAL;
    int64_t max_rows = 1;
    for (int i = 0; i < len; i++) {
        if (rows[i] < 0 || cols[i] < 0 || cols[i] > INT32_MAX || (rows[i] > 0 && !rowptr[i])) return RMCM_EINVAL;
        // two FP64 levels of len values per row must fit the array: refuse
        // before any size product can wrap around
        if (rows[i] > kNoAllocScratchBytes / (16 * (int64_t)len)) return RMCM_EINVAL;
        if (i + 1 < len && cols[i] != rows[i + 1]) return RMCM_EINVAL;
        max_rows = std::max(max_rows, rows[i]);
    }
    // set-up, once per device, with that device current
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return RMCM_ECUDA;
    NoAllocDevice nd;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        NoAllocDevice &d = g_noalloc_dev[dev];
        if (!d.ready) {
            void *ptr = nullptr;
            if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) {
                cudaGetLastError();
                return RMCM_ECUDA;
            }
            int sm = 0;
            if (cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sm <= 0) {
                cudaGetLastError();
                return RMCM_ECUDA;
            }
            d.scratch = (unsigned char *)ptr;
            d.sm_count = sm;
            d.ready = true;
        }
        nd = d;
    }
    // scratch layout: estimates | level r | level r' | block partials
    const int64_t blocks_cap = (int64_t)nd.sm_count * 8;
    auto al = [](int64_t x) { return (x + 255) & ~255LL; };
    const int64_t cbytes = al(8 * kMaxLen * kMaxLen);
    const int64_t rbytes = al(8 * max_rows * len);
    const int64_t pbytes = al(8 * blocks_cap * kMaxLen);
    if (cbytes + 2 * rbytes + pbytes > kNoAllocScratchBytes) return RMCM_EINVAL;   // chain too large
    cudaStream_t s = (cudaStream_t)stream;
    double *c_dev = (double *)nd.scratch;
    double *r_cur = (double *)(nd.scratch + cbytes);
    double *r_next = (double *)(nd.scratch + cbytes + rbytes);
    double *part = (double *)(nd.scratch + cbytes + 2 * rbytes);
    cudaError_t e = cudaMemsetAsync(c_dev, 0, sizeof(double) * len * len, s);
    for (int i = len - 1; i >= 0 && e == cudaSuccess; i--) {
        DevCsr M;
        M.rows = rows[i];
        M.cols = cols[i];
        M.rowptr = const_cast<int64_t *>(rowptr[i]);
        M.col = const_cast<int32_t *>(col[i]);
        LevelArgs la{};
        la.len = len;
        la.i = i;
        la.nj = len - 1 - i;
        int jp = 1;
        while (jp < la.nj) jp <<= 1;
        la.jp = jp;
        la.dim_leaf = (double)M.cols;
        for (int j = 0; j < len; j++) la.dims[j] = (double)cols[j];
        la.tile = level_tile(M.rows, blocks_cap);
        int64_t blocks = (M.rows + (int64_t)la.tile * (kEstThreads / 32) - 1) / ((int64_t)la.tile * (kEstThreads / 32));
        blocks = std::max<int64_t>(1, std::min(blocks, blocks_cap));
        k_res_level<<<(unsigned)blocks, kEstThreads, 0, s>>>(M, r_next, r_cur, la, part, false);
        if (la.nj > 0) k_res_reduce<<<(unsigned)la.nj, 256, 0, s>>>(part, (int32_t)blocks, la, c_dev);
        e = cudaGetLastError();
        std::swap(r_cur, r_next);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(c_out, c_dev, sizeof(double) * len * len, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return RMCM_ECUDA;
    }
    return RMCM_OK;
}
