// Rows of few products and wide outputs: a warp per row, expand - sort - merge
// in registers.  Included by spgemm.cu.
#pragma once

// BITS number a row's products (at most 1 << BITS): 8 and 10.
constexpr int kSortWarps = 4;

template <typename V, int BITS>
struct SortStage {
    uint32_t key[1 << BITS];  // column << BITS | product number; then the output's columns
    V val[1 << BITS];         // the products; then the output's counts
    int64_t bs[32];           // a chunk of 32 entries of A: B row start, length, value, first product
    int32_t len[32], pre[32];
    V va[32];
};

// Ascending sort of 32 R keys, key i = lane R + r in k[r], by merges of runs
// of kk / 2: the first step of a merge compares mirror images (i with its
// complement in the run of kk), which leaves every later step ascending, so
// that a pair of registers costs a minimum and a maximum and no direction.
// Partners less than R apart are registers of one lane, the others lie
// distance / R lanes away.
template <int R>
__device__ __forceinline__ void merge_sort(uint32_t (&k)[R], int lane) {
#pragma unroll
    for (int kk = 2; kk <= 32 * R; kk <<= 1) {
        if (kk <= R) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int o = r ^ (kk - 1);
                if (r > o) continue;
                const uint32_t lo = min(k[r], k[o]), hi = max(k[r], k[o]);
                k[r] = lo;
                k[o] = hi;
            }
        } else {
            const bool low = (lane & (kk / (2 * R))) == 0;
            uint32_t o[R];
#pragma unroll
            for (int r = 0; r < R; r++) o[r] = __shfl_xor_sync(kFull, k[R - 1 - r], kk / R - 1);
#pragma unroll
            for (int r = 0; r < R; r++) k[r] = low ? min(k[r], o[r]) : max(k[r], o[r]);
        }
#pragma unroll
        for (int j = kk >> 2; j > 0; j >>= 1) {
            if (j >= R) {
                const bool low = (lane & (j / R)) == 0;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint32_t o = __shfl_xor_sync(kFull, k[r], j / R);
                    k[r] = low ? min(k[r], o) : max(k[r], o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (r & j) continue;
                    const uint32_t lo = min(k[r], k[r | j]), hi = max(k[r], k[r | j]);
                    k[r] = lo;
                    k[r | j] = hi;
                }
            }
        }
    }
}

// Sorts n <= 32 R products (key: column << BITS | place of its product in val)
// by column, adds equal columns and leaves the row in key / val; returns its
// length.  The first product of a column stores its place in the row, the
// others add to it: most columns of such a row have one product.
template <int R, int BITS, typename V>
__device__ __forceinline__ int sort_merge(uint32_t *key, V *val, int n, int lane, bool checked, bool &ovf) {
    uint32_t k[R];
#pragma unroll
    for (int r = 0; r < R; r++) k[r] = lane * R + r < n ? key[lane * R + r] : 0xffffffffu;
    merge_sort<R>(k, lane);
    V v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = lane * R + r < n ? val[k[r] & ((1u << BITS) - 1u)] : (V)0;
    // heads of runs of one column (the n products sort to the front)
    const uint32_t before = __shfl_up_sync(kFull, k[R - 1], 1);
    uint32_t heads = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t p = r ? k[r - 1] : before;
        const bool first = r == 0 && lane == 0;
        if (lane * R + r < n && (first || (p >> BITS) != (k[r] >> BITS))) heads |= 1u << r;
    }
    const int incl = warp_incl_scan(__popc(heads));
    const int last = incl - __popc(heads) - 1;   // place of the run that is open before this lane
    const int total = __shfl_sync(kFull, incl, 31);
    __syncwarp();   // keys and products are in registers: their memory takes the row
#pragma unroll
    for (int r = 0; r < R; r++) {
        if ((heads >> r) & 1u) {
            const int pos = last + __popc(heads & ((2u << r) - 1u));
            key[pos] = k[r] >> BITS;
            val[pos] = v[r];
        }
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (lane * R + r < n && !((heads >> r) & 1u)) {
            V *sum = val + last + __popc(heads & ((2u << r) - 1u));
            if (checked) add_shared_chk(sum, v[r], ovf);
            else add_shared(sum, v[r]);
        }
    }
    __syncwarp();
    return total;
}

// Bound by instruction issue: the sort's compare-exchanges.  A key holds the
// column and the product's number, so the sort moves one register per product
// whatever the value type; the products wait in shared memory and are added
// where their columns come out.  Against a CTA with a hash table, whose barriers and shared-memory
// sort these rows took before: 52,860 rows of 68 products on 131,071 columns
// 355 -> 71 us, 25,195 uint64 rows of 120 258 -> 57 us; up to 1,024 products
// 581 -> 330 us (a wave of 64 chains).
template <typename V, int BITS>
__device__ __forceinline__ void sort_rows(const DevCsr &A, const DevCsr &B, bool a_ones, bool b_ones, const DevCsr &C,
                                          const int32_t *rows, int32_t nrows, int64_t *cnt, int *st,
                                          const uint8_t *bin_of, int64_t first, int64_t nwarps) {
    constexpr int MAX = 1 << BITS;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SortStage<V, BITS> &sg = ((SortStage<V, BITS> *)smem)[warp];
    const V *Aval = (const V *)A.val;
    const V *Bval = (const V *)B.val;
    bool ovf = false;
    for (int64_t wi = first; wi < nrows; wi += nwarps) {
        const int32_t r = rows[wi];
        const int64_t a0 = A.rowptr[r], a1 = A.rowptr[r + 1];
        const bool checked = (bin_of[r] & kRiskyBit) != 0;
        int n = 0;
        for (int64_t k0 = a0; k0 < a1; k0 += 32) {
            const int64_t k = k0 + lane;
            int64_t bs = 0;
            int32_t len = 0;
            V va = 0;
            if (k < a1) {
                const int32_t a = A.col[k];
                bs = B.rowptr[a];
                len = (int32_t)(B.rowptr[a + 1] - bs);
                va = a_ones ? (V)1 : Aval[k];
            }
            const int32_t incl = warp_incl_scan(len);
            sg.bs[lane] = bs;
            sg.len[lane] = len;
            sg.pre[lane] = n + incl - len;
            sg.va[lane] = va;
            n += __shfl_sync(kFull, incl, 31);
            const int entries = a1 - k0 < 32 ? (int)(a1 - k0) : 32;
            __syncwarp();
            auto stage = [&](int i, int first, int step) {
                const int64_t q = sg.bs[i];
                const int32_t L = sg.len[i], p0 = sg.pre[i];
                const V x = sg.va[i];
                for (int32_t p = first; p < L; p += step) {
                    const int at = p0 + p;
                    const V y = b_ones ? (V)1 : __ldg(Bval + q + p);
                    const int32_t c = __ldg(B.col + q + p);
                    if (at < MAX) {   // (the bin holds no longer row)
                        sg.key[at] = (uint32_t)c << BITS | (uint32_t)at;
                        sg.val[at] = checked ? mul_chk(x, y, ovf) : (V)(x * y);
                    }
                }
            };
            // eight lanes a B row, all 32 for one of more than 64 positions
            for (int i = lane >> 3; i < entries; i += 4)
                if (sg.len[i] <= 64) stage(i, lane & 7, 8);
            __syncwarp();
            for (unsigned wide = __ballot_sync(kFull, len > 64); wide; wide &= wide - 1)
                stage(__ffs(wide) - 1, lane, 32);
            __syncwarp();
        }
        if (n > MAX) {
            if (lane == 0) raise_status(st, kInvariant);
            n = MAX;
        }
        const int total = n <= MAX / 2 ? sort_merge<MAX / 64, BITS>(sg.key, sg.val, n, lane, checked, ovf)
                                       : sort_merge<MAX / 32, BITS>(sg.key, sg.val, n, lane, checked, ovf);
        const int64_t base = C.rowptr[r];
        const int64_t rlen = C.rowptr[r + 1] - base;
        if (lane == 0) {
            // single pass (cnt given): the row's slots bound its entries
            if (cnt) cnt[r] = total;
            if (cnt ? (int64_t)total > rlen : rlen != total) raise_status(st, kInvariant);
        }
        const int lim = (int)((int64_t)total < rlen ? (int64_t)total : rlen);
        for (int i = lane; i < lim; i += 32) {
            C.col[base + i] = (int32_t)sg.key[i];
            ((V *)C.val)[base + i] = sg.val[i];
        }
        __syncwarp();
    }
    if (__any_sync(kFull, ovf) && lane == 0) raise_status(st, kOverflow);
}

template <typename V, int BITS>
__global__ void __launch_bounds__(kSortWarps * 32) k_sort(DevCsr A, DevCsr B, bool a_ones, bool b_ones, DevCsr C,
                                                          const int32_t *rows, int32_t nrows, int64_t *cnt, int *st,
                                                          const uint8_t *bin_of) {
    sort_rows<V, BITS>(A, B, a_ones, b_ones, C, rows, nrows, cnt, st, bin_of,
                       (int64_t)blockIdx.x * kSortWarps + (threadIdx.x >> 5), (int64_t)gridDim.x * kSortWarps);
}
