// Rank-bin rows (outputs wider than a dense window, many products) without a
// bitmap of the whole output: the row's products are partitioned by column
// range into buckets of about two hundred (up to 330 in the largest rows) in
// shared memory, and a warp sorts and merges each bucket in registers
// (sort_rows.cuh).  Included by spgemm.cu.
#pragma once

constexpr int kBucketBits = 9;        // products a bucket may hold: 512
constexpr int kBucketMean = 200;      // products a bucket is meant for: a sort of 256 with room for their spread

// A CTA of NT threads holds 22 NT products at a time (the SM then takes 1024
// threads with uint32 counts) and partitions a row into at most NT buckets.
template <int NT>
struct BucketCap {
    static constexpr int value = 22 * NT;
};

// The rows a launch of k_bucket takes: more than `over` products, at most
// `upto`, [1] for rows whose B rows average kWideBucket positions or more, [0]
// for the others.  Each fill of the buckets is another pass over the row's
// entries, and the count is one before them.
struct BucketRange {
    int64_t over[2], upto[2];
    int32_t least2;   // only rows whose B rows average least2 / 2 positions or more
};
constexpr int kWideBucket = 32;

// Fills a row may take in a CTA of 128 and of 512 threads, by launch (few:
// 512 threads only).  Rows beyond are k_rank's, whose cost grows with the
// output's width instead (its bitmap, one CTA an SM beyond some 500,000
// columns).  2,000 rows, us, uint32: 8,000 products through B rows of 5, 300,000
// columns: k_rank 541, one fill of 512 threads 519, three of 128 789; through 40,
// 200,000 columns: 429, 351, 412.  8,000 rows of 4,000 through 40: k_rank 765,
// one fill of 512 703, two of 128 592.  16,000 products, two fills of 512: through
// 5 1,141 (k_rank 959), through 40 641 (688).  uint64 (half the CTAs an SM), 6,000
// through 20, 300,000 columns: k_rank 344, 512 threads 415, 128 404; a million
// columns: 546, 422, 410.  Through B rows of one position the entries cost more than
// the products: 3,000 rows of 2,500 on 60,000 columns 641 against 556, uint64 811
// against 592 (and through two 508 against 467), on a million 652 against 975.
inline BucketRange bucket_range(int nt, bool u64, int64_t cols, bool few) {
    constexpr int64_t c128 = BucketCap<128>::value, c512 = BucketCap<512>::value;
    const bool wide_output = !u64 || cols > (1 << 19);
    BucketRange small{{0, 0}, {c128, c128}, cols > (1 << 19) ? 0 : u64 && cols <= (1 << 17) ? 6 : 3};
    if (wide_output) {
        small.upto[1] = 2 * c128;
        if (u64) small.upto[0] = 2 * c128;
    }
    if (nt == 128) return small;
    BucketRange r{{0, 0}, {0, 0}, small.least2};
    if (!few) {
        r.over[0] = small.upto[0];
        r.over[1] = small.upto[1];
    }
    if (wide_output || few) r.upto[0] = r.upto[1] = c512;
    if (wide_output) r.upto[1] = 3 * c512;
    return r;
}

template <typename V, int NT>
struct BucketShared {
    uint32_t key[BucketCap<NT>::value];  // column << kBucketBits | place in the bucket (columns: 20 bits)
    V val[BucketCap<NT>::value];
    int32_t start[NT + 1];               // products before each bucket (of the whole row)
    int32_t fill[NT];                    // placed so far; then the bucket's merged length
    int64_t bs[NT];                      // entries of A whose B rows are shared by lanes: mid ones from the
    V va[NT];                            // front, long ones from the back
    int32_t len[NT];
    int32_t nmid[2], nlong[2];
    int32_t wsum[NT / 32];
    int32_t next_bucket, row, big, pass_end;
};

// Visits every product of A entries [a0, a1): visit(column, A value, B value);
// without VALS neither value is read.  Ends with a barrier.
template <bool VALS, int NT, typename V, typename Visit>
__device__ __forceinline__ void bucket_stream(const DevCsr &A, const DevCsr &B, bool a_ones, bool b_ones, int64_t a0,
                                              int64_t a1, BucketShared<V, NT> &sh, int &cur, Visit visit) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    const V *Bval = (const V *)B.val;
    // positions p, p + step, .. (four) of the B row at q, those below L; the
    // loads in flight together
    auto four = [&](int64_t q, int32_t p, int step, int32_t L, V x) {
        int32_t c[4];
        V y[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            c[u] = p + u * step < L ? __ldg(B.col + q + p + u * step) : 0;
            y[u] = 1;
            if (VALS && !b_ones) y[u] = p + u * step < L ? __ldg(Bval + q + p + u * step) : (V)0;
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (p + u * step < L) visit(c[u], x, y[u]);
    };
    for (int64_t k0 = a0; k0 < a1; k0 += NT) {
        const int64_t k = k0 + tid;
        int64_t bs = 0;
        int32_t len = 0;
        V va = 0;
        if (k < a1) {
            const int32_t a = A.col[k];
            bs = B.rowptr[a];
            len = (int32_t)(B.rowptr[a + 1] - bs);
            if (VALS) va = a_ones ? (V)1 : ((const V *)A.val)[k];
        }
        const unsigned mid = __ballot_sync(kFull, len > 0 && len <= kMidLen);
        const unsigned lng = __ballot_sync(kFull, len > kMidLen);
        if (mid | lng) {
            int base = 0;
            if (lane == 0 && mid) base = atomicAdd(&sh.nmid[cur], __popc(mid));
            if (lane == 1 && lng) base = atomicAdd(&sh.nlong[cur], __popc(lng));
            const int mb = __shfl_sync(kFull, base, 0), lb = __shfl_sync(kFull, base, 1);
            if (len > 0) {
                const int i = len > kMidLen ? NT - 1 - (lb + __popc(lng & lt_mask)) : mb + __popc(mid & lt_mask);
                sh.bs[i] = bs;
                sh.len[i] = len;
                sh.va[i] = va;
            }
        }
        __syncthreads();
        if (tid == 0) {   // the other counters serve the next step
            sh.nmid[cur ^ 1] = 0;
            sh.nlong[cur ^ 1] = 0;
        }
        const int nm = sh.nmid[cur], nl = sh.nlong[cur];
        int turn = warp;   // pieces of 128 positions of the long entries, dealt round robin
        for (int i = NT - 1; i >= NT - nl; i--) {
            const int64_t q = sh.bs[i];
            const int32_t L = sh.len[i];
            const V x = sh.va[i];
            const int np = (L + 127) >> 7;
            for (; turn < np; turn += NW) four(q, 128 * turn + lane, 32, L, x);
            turn -= np;
        }
        // eight lanes an entry, 32 positions a step
        for (int i = tid >> 3; i < nm; i += NT / 8) {
            const int64_t q = sh.bs[i];
            const int32_t L = sh.len[i];
            const V x = sh.va[i];
            for (int32_t p = tid & 7; p < L; p += 32) four(q, p, 8, L, x);
        }
        cur ^= 1;
        __syncthreads();
    }
}

// Bound by the sort's instructions (about three a product and column) and the
// latency of the gathers, which a bitmap of a million columns (128 KB and its
// prefixes: one CTA an SM) left uncovered.  Per row: a histogram of the
// products over the buckets, then per pass as many whole buckets as the
// products held allow: products to their buckets, a warp per bucket sorts and
// merges, the merged buckets go out in order.  A row with a bucket of more
// than 512 products is left to k_rank (done[r] stays 0).
template <typename V, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_bucket(DevCsr A, DevCsr B, bool a_ones, bool b_ones, DevCsr C,
                                                           const int32_t *rows, int32_t nrows, const int64_t *flops,
                                                           BucketRange take, int64_t *cnt, int *st,
                                                           uint8_t *bin_of, int32_t *next_row) {
    constexpr int NW = NT / 32, CAP = BucketCap<NT>::value;
    extern __shared__ __align__(16) unsigned char smem[];
    BucketShared<V, NT> &sh = *(BucketShared<V, NT> *)smem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 2) {
        sh.nmid[tid] = 0;
        sh.nlong[tid] = 0;
    }
    bool ovf = false;
    int cur = 0;
    int32_t ri = blockIdx.x;
    while (ri < nrows) {
        const int32_t r = rows[ri];
        const int64_t f = flops[r];
        const uint8_t flags = bin_of[r];
        __syncthreads();   // the row before is done with the shared words
        if (tid == 0) sh.row = (int32_t)gridDim.x + atomicAdd(next_row, 1);
        const int64_t a0 = A.rowptr[r], a1 = A.rowptr[r + 1];
        const bool wide = f >= kWideBucket * (a1 - a0);
        if (f <= (wide ? take.over[1] : take.over[0]) || f > (wide ? take.upto[1] : take.upto[0]) ||
            2 * f < take.least2 * (a1 - a0)) {
            __syncthreads();
            ri = sh.row;
            continue;
        }
        // bucket of column c: c * nb / columns, in 32-bit fixed point
        const int nb = (int)min((int64_t)NT, (f + kBucketMean - 1) / kBucketMean);
        const uint64_t scale = ((uint64_t)nb << 32) / (uint64_t)B.cols;
        auto bucket_of = [&](int32_t c) { return (int)(((uint64_t)(uint32_t)c * scale) >> 32); };
        for (int b = tid; b < nb; b += NT) sh.fill[b] = 0;
        if (tid == 0) sh.big = 0;
        __syncthreads();
        bucket_stream<false, NT>(A, B, a_ones, b_ones, a0, a1, sh, cur,
                             [&](int32_t c, V, V) { atomicAdd(&sh.fill[bucket_of(c)], 1); });
        // starts (at most NT buckets: one per thread)
        {
            const int n = tid < nb ? sh.fill[tid] : 0;
            if (n > (1 << kBucketBits)) sh.big = 1;
            const int incl = warp_incl_scan(n);
            if (lane == 31) sh.wsum[warp] = incl;
            __syncthreads();
            int base = 0;
            for (int w = 0; w < warp; w++) base += sh.wsum[w];
            if (tid < nb) sh.start[tid] = base + incl - n;
            if (tid == nb - 1) sh.start[nb] = base + incl;
        }
        __syncthreads();
        if (sh.big) {
            ri = sh.row;
            continue;
        }
        const int64_t base = C.rowptr[r];
        const int64_t rlen = C.rowptr[r + 1] - base;
        const bool checked = (flags & kRiskyBit) != 0;
        int64_t out = 0;
        for (int b0 = 0; b0 < nb;) {
            // buckets b0 .. b1 - 1: as many as CAP products take (at least one)
            const int p0 = sh.start[b0];
            if (tid == 0) sh.pass_end = nb;
            __syncthreads();
            if (tid >= b0 && tid < nb && sh.start[tid + 1] - p0 > CAP && sh.start[tid] - p0 <= CAP)
                sh.pass_end = tid;
            for (int b = tid; b < nb; b += NT) sh.fill[b] = 0;
            if (tid == 0) sh.next_bucket = b0;
            __syncthreads();
            const int b1 = sh.pass_end;
            bucket_stream<true, NT>(A, B, a_ones, b_ones, a0, a1, sh, cur, [&](int32_t c, V x, V y) {
                const int b = bucket_of(c);
                if (b < b0 || b >= b1) return;
                const int i = atomicAdd(&sh.fill[b], 1);
                const int at = sh.start[b] - p0 + i;
                sh.key[at] = (uint32_t)c << kBucketBits | (uint32_t)i;
                sh.val[at] = checked ? mul_chk(x, y, ovf) : (V)(x * y);
            });
            // a warp per bucket
            while (true) {
                int b = 0;
                if (lane == 0) b = atomicAdd(&sh.next_bucket, 1);
                b = __shfl_sync(kFull, b, 0);
                if (b >= b1) break;
                const int n = sh.fill[b], at = sh.start[b] - p0;
                int m = 0;
                if (n > 256) m = sort_merge<16, kBucketBits>(sh.key + at, sh.val + at, n, lane, checked, ovf);
                else if (n > 128) m = sort_merge<8, kBucketBits>(sh.key + at, sh.val + at, n, lane, checked, ovf);
                else if (n > 64) m = sort_merge<4, kBucketBits>(sh.key + at, sh.val + at, n, lane, checked, ovf);
                else if (n > 0) m = sort_merge<2, kBucketBits>(sh.key + at, sh.val + at, n, lane, checked, ovf);
                if (lane == 0) sh.fill[b] = m;
            }
            __syncthreads();
            // the merged buckets in order: a bucket's place is the scan of the
            // lengths before it
            {
                const bool in = tid >= b0 && tid < b1;
                const int m = in ? sh.fill[tid] : 0;
                const int incl = warp_incl_scan(m);
                if (lane == 31) sh.wsum[warp] = incl;
                __syncthreads();
                int before = 0, total = 0;
                for (int w = 0; w < NW; w++) {
                    if (w < warp) before += sh.wsum[w];
                    total += sh.wsum[w];
                }
                __syncthreads();   // (fill becomes the scan: lengths are in registers)
                if (in) sh.fill[tid] = before + incl;
                if (tid == 0) sh.pass_end = total;
                __syncthreads();
            }
            const int total = sh.pass_end;
            for (int b = b0 + warp; b < b1; b += NW) {
                const int at = sh.start[b] - p0, o1 = sh.fill[b], o0 = b > b0 ? sh.fill[b - 1] : 0;
                for (int i = lane; i < o1 - o0; i += 32) {
                    const int64_t o = out + o0 + i;
                    if (o < rlen) {
                        C.col[base + o] = (int32_t)sh.key[at + i];
                        ((V *)C.val)[base + o] = sh.val[at + i];
                    }
                }
            }
            out += total;
            b0 = b1;
            __syncthreads();
        }
        if (tid == 0) {
            // single pass (cnt given): the row's slots bound its entries
            if (cnt) cnt[r] = out;
            if (cnt ? out > rlen : out != rlen) raise_status(st, kInvariant);
            bin_of[r] = (uint8_t)(flags | kDoneBit);
        }
        ri = sh.row;
    }
    if (__syncthreads_or(ovf) && tid == 0) raise_status(st, kOverflow);
}
