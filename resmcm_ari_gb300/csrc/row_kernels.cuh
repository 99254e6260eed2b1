// Row kernels of the rows that need neither overflow checks nor presence
// bytes: every input value of the product is >= 1 and no count of the row can
// overflow, so a counter > 0 marks a column and every add is a plain one.
// The general kernels (k_warp, k_dense) keep the other rows.
//
//   k_row_warp    a warp per row, a window of its own (outputs <= 2048 wide)
//   k_row_window  a CTA of 128 .. 1024 threads per row (one window wide)
//
// A window of uint64 counters is two planes of 32-bit words, low halves
// first.  A row whose counts all fit 32 bits (kNarrowBit) adds to the low
// plane only, with adds that return nothing; the others add the low halves
// first and what carries to the high ones (add_shared's two steps).  Planes
// keep consecutive columns in consecutive banks, where 8-byte counters put
// two columns of 32 on one bank.
//
// Measured against the general kernels, which these rows took before (kernel
// time on one GB300): uint64 products of 50,000-vertex types onto 1,000
// columns 3.0 -> 0.55 ms (566M multiply-adds, two a chain) and 3.2 -> 0.97 ms
// (1000 x 1000 x 1000, full); 30,000 rows onto 30,000 columns through 50
// (146M) 1.73 -> 0.94 ms; the light rows beside the 20,000 x 1,000,000 x 2,000
// tensor-core product 5.8 -> 2.6 ms; one million rows of a user's items onto
// 2,000 columns 0.83 -> 0.36 ms.
//
// Included by spgemm.cu.
#pragma once

// How the products of one entry of A are spread, by the length of its B row:
// up to kOwnLen positions by the thread that read the entry, up to kMidLen by
// kGroup lanes, each with four positions in flight, longer ones by whole warps.  A
// lane reading a row of ten by itself touches a sector per position and
// array; the L1, not the instruction rate, bounds such rows.
constexpr int kOwnLen = 4;
constexpr int kMidLen = 64;
constexpr int kGroup = 4;

// Right operand of a row kernel: columns and values, or (PK) one 32-bit word
// per entry: column in the low cbits, value - addend above them (a matrix of
// ones is its column array with cbits 31 and addend 1).
template <typename V>
struct RowB {
    const int64_t *rowptr;
    const int32_t *col;
    const V *val;
    const uint32_t *words;
    int32_t cbits;
    uint32_t addend;
};

// An entry of B as loaded; taken apart only where it is used, so that loads
// stay in flight together.
template <typename V, bool PK>
struct Entry {
    int32_t c;
    V v;
    __device__ __forceinline__ void clear() { c = 0; v = 0; }
    __device__ __forceinline__ void load(const RowB<V> &B, int64_t q) {
        c = __ldg(B.col + q);
        v = __ldg(B.val + q);
    }
    __device__ __forceinline__ int32_t col(const RowB<V> &) const { return c; }
    __device__ __forceinline__ V value(const RowB<V> &) const { return v; }
};
template <typename V>
struct Entry<V, true> {
    uint32_t w;
    __device__ __forceinline__ void clear() { w = 0; }
    __device__ __forceinline__ void load(const RowB<V> &B, int64_t q) { w = __ldg(B.words + q); }
    __device__ __forceinline__ int32_t col(const RowB<V> &B) const { return (int32_t)(w & ((1u << B.cbits) - 1u)); }
    __device__ __forceinline__ V value(const RowB<V> &B) const { return (V)((w >> B.cbits) + B.addend); }
};

// Counters of W columns in shared memory.
template <typename V>
struct Window {
    uint32_t *lo, *hi;   // hi: uint64 only
    __device__ __forceinline__ Window(void *p, int32_t W) : lo((uint32_t *)p), hi((uint32_t *)p + W) {}
    template <bool NARROW>
    __device__ __forceinline__ void add(int32_t c, V v) const {
        if (NARROW || sizeof(V) == 4) {
            atomicAdd(lo + c, (uint32_t)v);
        } else {
            const uint32_t l = (uint32_t)v;
            const uint32_t old = atomicAdd(lo + c, l);
            const uint32_t h = (uint32_t)((uint64_t)v >> 32) + (old > 0xffffffffu - l ? 1u : 0u);
            if (h) atomicAdd(hi + c, h);
        }
    }
    __device__ __forceinline__ V get(int c) const {
        return sizeof(V) == 4 ? (V)lo[c] : (V)((uint64_t)hi[c] << 32 | lo[c]);
    }
    __device__ __forceinline__ void set(int c, V v) const {
        lo[c] = (uint32_t)v;
        if (sizeof(V) == 8) hi[c] = (uint32_t)((uint64_t)v >> 32);
    }
};

// A thread's E entries of A from k (stride `step`, below a1): B row starts and
// lengths and A values.  Loads past the end go to the row's first entry and
// count for nothing: a branch around the dependent loads would keep them from
// being in flight together.
template <int E, typename V>
__device__ __forceinline__ void load_entries(const DevCsr &A, const V *aval, const RowB<V> &B, int64_t a0, int64_t k,
                                             int step, int64_t a1, int64_t (&bs)[E], int32_t (&len)[E], V (&va)[E]) {
    int32_t a[E];
    int64_t be[E];
#pragma unroll
    for (int u = 0; u < E; u++) a[u] = __ldg(A.col + (k + u * step < a1 ? k + u * step : a0));
    if (aval) {
#pragma unroll
        for (int u = 0; u < E; u++) va[u] = __ldg(aval + (k + u * step < a1 ? k + u * step : a0));
    } else {
#pragma unroll
        for (int u = 0; u < E; u++) va[u] = 1;
    }
#pragma unroll
    for (int u = 0; u < E; u++) {
        bs[u] = __ldg(B.rowptr + a[u]);
        be[u] = __ldg(B.rowptr + a[u] + 1);
    }
#pragma unroll
    for (int u = 0; u < E; u++) len[u] = k + u * step < a1 ? (int32_t)(be[u] - bs[u]) : 0;
}

// The short ones (up to kOwnLen positions) among a thread's E entries, a
// position of each per step.
template <bool NARROW, bool PK, int E, typename V>
__device__ __forceinline__ void add_own(const RowB<V> &B, const int64_t (&bs)[E], const int32_t (&len)[E],
                                        const V (&va)[E], const Window<V> &win) {
#pragma unroll
    for (int i = 0; i < kOwnLen; i++) {
        Entry<V, PK> e[E];
        bool any = false;
#pragma unroll
        for (int u = 0; u < E; u++) {
            e[u].clear();
            const bool ok = i < len[u] && len[u] <= kOwnLen;
            any |= ok;
            if (ok) e[u].load(B, bs[u] + i);
        }
        if (!any) break;
#pragma unroll
        for (int u = 0; u < E; u++)
            if (i < len[u] && len[u] <= kOwnLen) win.template add<NARROW>(e[u].col(B), (V)(va[u] * e[u].value(B)));
    }
}

// Adds va * B[q0 .. q0 + n) from kGroup lanes (sub = 0 .. kGroup - 1), four
// positions a lane in flight.
template <bool NARROW, bool PK, typename V>
__device__ __forceinline__ void add_group(const RowB<V> &B, int64_t q0, int32_t n, V va, const Window<V> &win,
                                          int sub) {
    for (int32_t p = sub; p < n; p += 4 * kGroup) {
        Entry<V, PK> e[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            e[u].clear();
            if (p + u * kGroup < n) e[u].load(B, q0 + p + u * kGroup);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (p + u * kGroup < n) win.template add<NARROW>(e[u].col(B), (V)(va * e[u].value(B)));
    }
}

// Adds va * (up to 128 positions from q0), four per lane: whole blocks
// without predicates.
template <bool NARROW, bool PK, typename V>
__device__ __forceinline__ void add_block(const RowB<V> &B, int64_t q0, int32_t left, V va, const Window<V> &win,
                                          int lane) {
    Entry<V, PK> e[4];
    if (left >= 128) {
#pragma unroll
        for (int u = 0; u < 4; u++) e[u].load(B, q0 + 32 * u + lane);
#pragma unroll
        for (int u = 0; u < 4; u++) win.template add<NARROW>(e[u].col(B), (V)(va * e[u].value(B)));
    } else {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            e[u].clear();
            if (32 * u + lane < left) e[u].load(B, q0 + 32 * u + lane);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (32 * u + lane < left) win.template add<NARROW>(e[u].col(B), (V)(va * e[u].value(B)));
    }
}

// Writes the nonzero counters of columns [c0, c0 + 128) at pos.., columns
// ascending, and clears them; returns the entries written.
template <typename V>
__device__ __forceinline__ int emit_block(const Window<V> &win, int c0, int64_t pos, int64_t lim, int32_t *col,
                                          V *val, int lane, unsigned lt_mask) {
    V v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = win.get(c0 + 32 * u + lane);
    if (!__any_sync(kFull, (v[0] | v[1] | v[2] | v[3]) != 0)) return 0;
    int n = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const unsigned bits = __ballot_sync(kFull, v[u] != 0);
        if (v[u] != 0) {
            const int64_t o = pos + n + __popc(bits & lt_mask);
            if (o < lim) {
                col[o] = c0 + 32 * u + lane;
                val[o] = v[u];
            }
            win.set(c0 + 32 * u + lane, 0);
        }
        n += __popc(bits);
    }
    return n;
}

// ---- a warp per row ---------------------------------------------------------
//
// Bound by instruction issue and by the latency of the chain row -> A entry ->
// B row -> counter; no block barrier, so an SM carries as many rows as its
// windows allow, and the row's products need no search.
constexpr int kWarpEntries = 4;   // entries of A a lane holds at a time

template <typename V>
struct WarpList {
    int64_t bs[32 * kWarpEntries];
    V va[32 * kWarpEntries];
    int32_t len[32 * kWarpEntries];
};

template <bool NARROW, bool PK, typename V>
__device__ __forceinline__ void row_warp_products(const DevCsr &A, const V *aval, const RowB<V> &B, int64_t a0,
                                                  int64_t a1, const Window<V> &win, WarpList<V> &sl, int lane) {
    constexpr int E = kWarpEntries;
    const unsigned lt_mask = (1u << lane) - 1u;
    for (int64_t k0 = a0; k0 < a1; k0 += 32 * E) {
        int64_t bs[E];
        int32_t len[E];
        V va[E];
        load_entries<E>(A, aval, B, a0, k0 + lane, 32, a1, bs, len, va);
        // listed: mid entries from the front, long ones from the back
        int nm = 0, nl = 0;
#pragma unroll
        for (int u = 0; u < E; u++) {
            const unsigned mid = __ballot_sync(kFull, len[u] > kOwnLen && len[u] <= kMidLen);
            const unsigned lng = __ballot_sync(kFull, len[u] > kMidLen);
            if (len[u] > kOwnLen) {
                const int i = len[u] > kMidLen ? 32 * E - 1 - (nl + __popc(lng & lt_mask)) : nm + __popc(mid & lt_mask);
                sl.bs[i] = bs[u];
                sl.len[i] = len[u];
                sl.va[i] = va[u];
            }
            nm += __popc(mid);
            nl += __popc(lng);
        }
        add_own<NARROW, PK, E>(B, bs, len, va, win);
        __syncwarp();
        for (int i = lane / kGroup; i < nm; i += 32 / kGroup)
            add_group<NARROW, PK>(B, sl.bs[i], sl.len[i], sl.va[i], win, lane % kGroup);
        __syncwarp();
        for (int j = 0; j < nl; j++) {
            const int i = 32 * E - 1 - j;
            const int64_t q = sl.bs[i];
            const int32_t L = sl.len[i];
            const V av = sl.va[i];
            for (int32_t p = 0; p < L; p += 128) add_block<NARROW, PK>(B, q + p, L - p, av, win, lane);
        }
        __syncwarp();   // the list is free again
    }
}

template <typename V, bool PK>
__device__ __forceinline__ void warp_window_rows(const DevCsr &A, const V *aval, const RowB<V> &B, const DevCsr &C,
                                                 const int32_t *rows, int32_t nrows, int32_t W, int64_t *cnt,
                                                 const uint8_t *bin_of, int *st, int64_t first, int64_t nwarps) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    __shared__ WarpList<V> lists[kWarpWarps];
    const Window<V> win((V *)smem + (int64_t)warp * W, W);
    WarpList<V> &sl = lists[warp];
    for (int i = lane; i < W; i += 32) win.set(i, 0);
    __syncwarp();
    for (int64_t wi = first; wi < nrows; wi += nwarps) {
        const int32_t r = rows[wi];
        const int64_t a0 = A.rowptr[r], a1 = A.rowptr[r + 1];
        const uint8_t flags = bin_of[r];
        if (flags & kRiskyBit) continue;   // left to k_warp
        if (sizeof(V) == 4 || (flags & kNarrowBit)) row_warp_products<true, PK>(A, aval, B, a0, a1, win, sl, lane);
        else row_warp_products<false, PK>(A, aval, B, a0, a1, win, sl, lane);
        __syncwarp();   // every product has landed in the window
        const int64_t base = C.rowptr[r];
        const int64_t rlen = C.rowptr[r + 1] - base;
        int64_t pos = 0;
        for (int c0 = 0; c0 < W; c0 += 128)
            pos += emit_block(win, c0, pos, rlen, C.col + base, (V *)C.val + base, lane, lt_mask);
        if (lane == 0) {
            // single pass (cnt given): the row's slots bound its entries
            if (cnt) cnt[r] = pos;
            if (cnt ? pos > rlen : pos != rlen) raise_status(st, kInvariant);
        }
        __syncwarp();
    }
}

template <typename V, bool PK>
__global__ void __launch_bounds__(kWarpWarps * 32, 8) k_row_warp(DevCsr A, const V *aval, RowB<V> B, DevCsr C,
                                                                 const int32_t *rows, int32_t nrows, int32_t W,
                                                                 int64_t *cnt, const uint8_t *bin_of, int *st) {
    warp_window_rows<V, PK>(A, aval, B, C, rows, nrows, W, cnt, bin_of, st,
                            (int64_t)blockIdx.x * kWarpWarps + (threadIdx.x >> 5), (int64_t)gridDim.x * kWarpWarps);
}

// ---- a CTA per row ------------------------------------------------------------
//
// Row ri of the list goes to slot ri (its own number with by_row) of the
// row-padded temporary T (stride tstride), its length to cnt.  The CTA takes
// up to four entries of A per thread and step: entries with short B rows are
// added by their thread, the others listed in shared memory, mid entries
// (kGroup lanes each) from the front and long ones from the back.  With at
// least two long entries per warp, warps take them one at a time; with fewer,
// every entry is dealt to the warps in pieces of 128 positions, so a row of a
// few long B rows (a 30,000-vertex type joined through 50) keeps every warp
// busy.
// Rows are taken from a counter (next_row, zeroed by the caller), the next one
// while a row is worked on: rows of Zipf-distributed work dealt in a fixed
// order left 40% of the SM time idle (2-hop uint64 product of a 50,000-vertex
// type onto 1,000 columns).
// With S the row starts from its tensor-core part, and A holds the row's
// other entries only (lcnt of them).

// Entries of A per thread and step: as many as a list of 1024 holds.
template <int NT>
struct RowEntries {
    static constexpr int value = NT >= 1024 ? 1 : NT == 512 ? 2 : 4;
};

template <int NT, typename V>
struct RowLists {
    static constexpr int N = NT * RowEntries<NT>::value;
    int64_t bs[N];
    V va[N];
    int32_t len[N];
    int32_t nmid[2], nlong[2], ctr[2];
};

template <bool NARROW, bool PK, int NT, typename V>
__device__ __forceinline__ void row_window_products(const DevCsr &A, const V *aval, const RowB<V> &B, int64_t a0,
                                                    int64_t a1, const Window<V> &win, RowLists<NT, V> &sl, int &cur) {
    constexpr int NW = NT / 32, E = RowEntries<NT>::value, N = NT * E;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    for (int64_t k0 = a0; k0 < a1; k0 += N) {
        int64_t bs[E];
        int32_t len[E];
        V va[E];
        load_entries<E>(A, aval, B, a0, k0 + tid, NT, a1, bs, len, va);
#pragma unroll
        for (int u = 0; u < E; u++) {
            const unsigned mid = __ballot_sync(kFull, len[u] > kOwnLen && len[u] <= kMidLen);
            const unsigned lng = __ballot_sync(kFull, len[u] > kMidLen);
            if (mid | lng) {
                int base = 0;
                if (lane == 0 && mid) base = atomicAdd(&sl.nmid[cur], __popc(mid));
                if (lane == 1 && lng) base = atomicAdd(&sl.nlong[cur], __popc(lng));
                const int mb = __shfl_sync(kFull, base, 0), lb = __shfl_sync(kFull, base, 1);
                if (len[u] > kOwnLen) {
                    const int i = len[u] > kMidLen ? N - 1 - (lb + __popc(lng & lt_mask)) : mb + __popc(mid & lt_mask);
                    sl.bs[i] = bs[u];
                    sl.len[i] = len[u];
                    sl.va[i] = va[u];
                }
            }
        }
        add_own<NARROW, PK, E>(B, bs, len, va, win);
        __syncthreads();
        // the other counters serve the next step: clear them between the two
        // barriers, while nobody uses them
        if (tid == 0) {
            sl.nmid[cur ^ 1] = 0;
            sl.nlong[cur ^ 1] = 0;
            sl.ctr[cur ^ 1] = 0;
        }
        const int nm = sl.nmid[cur], nl = sl.nlong[cur];
        if (nl >= 2 * NW) {
            while (true) {
                int i = 0;
                if (lane == 0) i = atomicAdd(&sl.ctr[cur], 1);
                i = N - 1 - __shfl_sync(kFull, i, 0);
                if (i < N - nl) break;
                const int64_t q = sl.bs[i];
                const int32_t L = sl.len[i];
                const V av = sl.va[i];
                for (int32_t p = 0; p < L; p += 128) add_block<NARROW, PK>(B, q + p, L - p, av, win, lane);
            }
        } else {
            int turn = warp;   // pieces of all entries dealt round robin
            for (int i = N - 1; i >= N - nl; i--) {
                const int64_t q = sl.bs[i];
                const int32_t L = sl.len[i];
                const V av = sl.va[i];
                const int np = (L + 127) >> 7;
                for (; turn < np; turn += NW)
                    add_block<NARROW, PK>(B, q + 128 * (int64_t)turn, L - 128 * turn, av, win, lane);
                turn -= np;
            }
        }
        for (int i = tid / kGroup; i < nm; i += NT / kGroup)
            add_group<NARROW, PK>(B, sl.bs[i], sl.len[i], sl.va[i], win, tid % kGroup);
        cur ^= 1;
        __syncthreads();   // the list is free; after the last step, every product has landed
    }
}

// CTAs an SM should hold: warps cover the gathers' latency, so uint32 rows of a
// packed B run with 40 to 51 registers (40 to 48 warps; 1.4G multiply-adds
// through 500 B rows of 1,700 took 778 us at 64 registers and 32 warps, 520 in
// k_dense at 40).  The other forms would spill.
template <typename V, int NT, bool PK>
constexpr int row_window_ctas() {
    return sizeof(V) == 4 && PK ? (NT == 128 ? 10 : NT == 256 ? 6 : NT == 512 ? 3 : 1)
                                : (NT == 128 ? 8 : NT == 256 ? 4 : NT == 512 ? 2 : 1);
}

template <typename V, int NT, bool PK>
__global__ void __launch_bounds__(NT, row_window_ctas<V, NT, PK>())
    k_row_window(DevCsr A, const V *aval, RowB<V> B, DevCsr T, const int32_t *rows, int32_t nrows, int64_t tstride,
                 int32_t W, int32_t ncols, int64_t *cnt, const uint8_t *bin_of, const V *S, int64_t gld,
                 const int32_t *lcnt, int32_t *next_row, bool by_row) {
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    const Window<V> win(smem, W);
    __shared__ RowLists<NT, V> sl;
    __shared__ int32_t s_tot[NW];
    __shared__ int32_t s_row;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    for (int i = tid; i < W; i += NT) win.set(i, 0);
    if (tid < 2) {
        sl.nmid[tid] = 0;
        sl.nlong[tid] = 0;
        sl.ctr[tid] = 0;
    }
    // warps own contiguous ranges of 128-column blocks
    const int blocks = W >> 7, bper = (blocks + NW - 1) / NW;
    const int b0 = min(warp * bper, blocks), b1 = min(b0 + bper, blocks);
    int cur = 0;
    int32_t ri = blockIdx.x;
    while (ri < nrows) {
        const int32_t r = rows[ri];
        const int64_t a0 = A.rowptr[r], a1 = lcnt ? a0 + lcnt[r] : A.rowptr[r + 1];
        const uint8_t flags = bin_of[r];
        __syncthreads();   // the window is clear, every thread has its row
        if (tid == 0) s_row = (int32_t)gridDim.x + atomicAdd(next_row, 1);
        if (flags & kRiskyBit) {   // left to k_dense
            __syncthreads();
            ri = s_row;
            continue;
        }
        if (S) {
            const V *g = S + (int64_t)r * gld;
            for (int c = tid; c < ncols; c += NT) win.set(c, g[c]);
            __syncthreads();
        }
        if (sizeof(V) == 4 || (flags & kNarrowBit)) row_window_products<true, PK>(A, aval, B, a0, a1, win, sl, cur);
        else row_window_products<false, PK>(A, aval, B, a0, a1, win, sl, cur);
        int mine = 0;
        for (int b = b0; b < b1; b++) {
#pragma unroll
            for (int u = 0; u < 4; u++) mine += win.get(b * 128 + 32 * u + lane) != 0;
        }
        mine = __reduce_add_sync(kFull, mine);
        if (lane == 0) s_tot[warp] = mine;
        __syncthreads();
        int64_t pos = 0, total = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const int t = s_tot[w];
            if (w < warp) pos += t;
            total += t;
        }
        const int64_t slot = (int64_t)(by_row ? r : ri) * tstride;
        int32_t *oc = T.col + slot;
        V *ov = (V *)T.val + slot;
        for (int b = b0; b < b1; b++) pos += emit_block(win, b * 128, pos, tstride, oc, ov, lane, lt_mask);
        if (tid == 0) cnt[r] = total;
        ri = s_row;
    }
}
