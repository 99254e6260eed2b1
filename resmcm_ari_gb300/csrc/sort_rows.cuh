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

// Ascending bitonic sort of 32 R keys, key i = lane R + r in k[r]: partners
// less than R apart are registers of one lane, the others R / distance lanes
// away.
template <int R>
__device__ __forceinline__ void bitonic_sort(uint32_t (&k)[R], int lane) {
#pragma unroll
    for (int kk = 2; kk <= 32 * R; kk <<= 1) {
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
            if (j >= R) {
                const int d = j / R;
                const bool up = kk >= 32 * R || (lane & (kk / R)) == 0;
                const bool keep_min = ((lane & d) == 0) == up;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint32_t o = __shfl_xor_sync(kFull, k[r], d);
                    k[r] = keep_min ? min(k[r], o) : max(k[r], o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (r & j) continue;
                    // (the run's direction: bit kk of lane R + r)
                    const bool up = kk >= 32 * R || (kk >= R ? (lane & (kk / R)) == 0 : (r & kk) == 0);
                    const uint32_t lo = min(k[r], k[r | j]), hi = max(k[r], k[r | j]);
                    k[r] = up ? lo : hi;
                    k[r | j] = up ? hi : lo;
                }
            }
        }
    }
}

// Sorts the staged products (n <= 32 R of them) by column, adds equal columns
// and leaves the row in sg.key / sg.val; returns its length.
template <int R, int BITS, typename V>
__device__ __forceinline__ int sort_merge(SortStage<V, BITS> &sg, int n, int lane, bool &ovf) {
    uint32_t k[R];
#pragma unroll
    for (int r = 0; r < R; r++) k[r] = lane * R + r < n ? sg.key[lane * R + r] : 0xffffffffu;
    bitonic_sort<R>(k, lane);
    V v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = lane * R + r < n ? sg.val[k[r] & ((1u << BITS) - 1u)] : (V)0;
    // heads of runs of one column; (n products sort to the front)
    const uint32_t before = __shfl_up_sync(kFull, k[R - 1], 1);
    uint32_t heads = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t p = r ? k[r - 1] : before;
        const bool first = r == 0 && lane == 0;
        if (lane * R + r < n && (first || (p >> BITS) != (k[r] >> BITS))) heads |= 1u << r;
    }
    int incl = __popc(heads);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += o;
    }
    const int pos0 = incl - __popc(heads);
    const int total = __shfl_sync(kFull, incl, 31);
    // the part of this lane before its first head belongs to a run of an
    // earlier lane: suffix sums over lanes, stopping at lanes with a head
    auto add = [&](V &s, V x) {
        s += x;
        ovf |= s < x;
    };
    V lead = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (!(heads & ((2u << r) - 1u))) add(lead, v[r]);
    }
    bool stop = heads != 0;
    V tail = lead;   // lead of this lane and of the lanes after it up to (including) the first with a head
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const V o = __shfl_down_sync(kFull, tail, d);
        const bool os = __shfl_down_sync(kFull, stop, d);
        if (lane + d < 32 && !stop) {
            add(tail, o);
            stop = os;
        }
    }
    V next = __shfl_down_sync(kFull, tail, 1);
    if (lane == 31) next = 0;
    __syncwarp();   // keys and products are in registers: the stage takes the row
    int pos = pos0 - 1;
    V sum = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if ((heads >> r) & 1u) {
            if (pos >= pos0) sg.val[pos] = sum;
            pos++;
            sg.key[pos] = k[r] >> BITS;
            sum = v[r];
        } else if (pos >= pos0) {
            add(sum, v[r]);
        }
    }
    if (pos >= pos0) {
        add(sum, next);
        sg.val[pos] = sum;
    }
    __syncwarp();
    return total;
}

// Bound by instruction issue: the sort's compare-exchanges.  A key holds the
// column and the product's number, so the sort moves one register per product
// whatever the value type; the products wait in shared memory and are added
// after it.  Against a CTA with a hash table, whose barriers and shared-memory
// sort these rows took before: 52,860 rows of 68 products on 131,071 columns
// 355 -> 71 us, 25,195 uint64 rows of 120 258 -> 57 us; up to 1,024 products
// 581 -> 440 us (a wave of 64 chains).
template <typename V, int BITS>
__global__ void __launch_bounds__(kSortWarps * 32) k_sort(DevCsr A, DevCsr B, bool a_ones, bool b_ones, DevCsr C,
                                                          const int32_t *rows, int32_t nrows, int64_t *cnt, int *st,
                                                          const uint8_t *bin_of) {
    constexpr int MAX = 1 << BITS;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SortStage<V, BITS> &sg = ((SortStage<V, BITS> *)smem)[warp];
    const V *Aval = (const V *)A.val;
    const V *Bval = (const V *)B.val;
    bool ovf = false;
    for (int64_t wi = (int64_t)blockIdx.x * kSortWarps + warp; wi < nrows; wi += (int64_t)gridDim.x * kSortWarps) {
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
        const int total = n <= MAX / 2 ? sort_merge<MAX / 64, BITS>(sg, n, lane, ovf)
                                       : sort_merge<MAX / 32, BITS>(sg, n, lane, ovf);
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
