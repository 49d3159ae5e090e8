// The reference's comparison sorts reproduced on the device: @order and
// @group keys of the types its radix and merge sorts do not take (bool, i8,
// i16, f32, f64, the date and time types) and lists of columns holding them.
//
//   lib_partition / lib_quicksort_other  src/horseir/v3/backend/h_libs.cc:409-442
//   lib_quicksort_char                   h_libs.cc:386-407
//   lib_order_by_sorted                  h_libs.cc:604-617
//   lib_quicksort_list                   h_libs.cc:637-697
//   lib_order_by_vector                  h_libs.cc:730-736
//
// The quicksort is unstable but deterministic, and the order it leaves equal
// keys in is the reference's result, so it is reproduced step for step.  One
// partition of a range [lo, hi) with the first element as pivot P computes:
//   * c = the number of elements of (lo, hi) comparing <= P; j = lo + c;
//   * the elements > P inside (lo, j] and the elements <= P inside (j, hi)
//     are equally many, and the k-th of the first (counted from the left)
//     trades places with the k-th of the second (counted from the right):
//     these are exactly the pairs the reference's two scans meet;
//   * then x[lo] and x[j] trade places, unless every element compares equal
//     to P (leftSame), in which case nothing moves and the range is done;
//   * the recursion continues on [lo, j) and [j+1, hi).
// Ranges are independent, so every range of one recursion depth is
// partitioned at once: a flag pair per element (<= P, < P), one scan over
// all ranges, the trade partners from the scan's ranks, and the next depth's
// ranges.  Depths repeat until no range of two or more elements is left.
//
// The same step runs at three scales: ranges above QS_BLOCK elements together
// in global memory (all depths in one launch of resident blocks while the
// elements fit them, else four launches a depth), ranges of up to QS_BLOCK in one
// CTA's shared memory and ranges of up to 32 in one warp's registers, both to
// their end without another launch.  (With every depth in global memory 114K
// random rows took 48 depths of five launches: what bounded the call was
// launch latency.)
// A NaN key makes the reference's comparator non-reflexive and its scans
// leave the range (undefined behaviour), so NaN keys return E_NOT_IMPL.
#include "dev_common.cuh"

namespace hg {

template <typename K>
I radix_sort(const K* keys, long long n, const K** kres, const unsigned** vres, const unsigned* init_vals);
I compact_rows(const uint8_t* mask, long long n, long long* out, long long* count);

constexpr unsigned QS_DONE = 0xffffffffu;
constexpr int QS_THREADS = 256, QS_ITEMS = 8, QS_TILE = QS_THREADS * QS_ITEMS;
constexpr int QS_WARP = 32;         // largest range one warp sorts
constexpr int QS_BLOCK = 4096;      // largest range one CTA sorts in shared memory
// CTAs of QB_ITEMS elements a thread: of 32 threads for ranges of up to 128
// elements, 128 for up to 512 and 1024 for up to QS_BLOCK
constexpr int QB_ITEMS = 4, QB_CLASSES = 3;
__host__ __device__ constexpr int qb_threads(int c) { return c == 0 ? 32 : c == 1 ? 128 : 1024; }
__host__ __device__ constexpr int qb_rows(int c) { return qb_threads(c) * QB_ITEMS; }
static_assert(qb_rows(QB_CLASSES - 1) == QS_BLOCK, "the largest CTA takes the largest listed range");
// A range handed to a CTA or a warp: positions [lo, hi), the recursion depth
// at which it was made, and which of the sort's two buffers holds its elements.
// Both buffers are free for them: a depth reads one and writes the other, and
// later depths touch neither at the positions of a listed range.
struct QsRange {
    unsigned lo, hi, depth, buf;
};
// ... as it is listed.  The depth fits: no more than the rows of a small sort,
// or 2^36 by the rows of a large one, either way below 2^19.
struct QsEntry {
    unsigned lo, rest;  // size - 1, buffer << 12, depth << 13
    __device__ __forceinline__ QsRange range() const {
        return QsRange{lo, lo + (rest & 4095u) + 1, rest >> 13, (rest >> 12) & 1u};
    }
};
static_assert(QS_BLOCK <= 4096, "packing of QsEntry::rest");
// counters of one sort, in device memory
struct QsCounters {
    unsigned nblock[QB_CLASSES], nwarp;  // ranges listed for CTAs of each size and for warps
    unsigned nbig;           // ranges the sort starts with that neither takes
    unsigned depth;          // recursion depth reached by the listed ranges
    unsigned nrev, nan;      // segments to reverse; a NaN key was seen
};
// Ranges for warps are listed from the front of `ends` and those for the
// smallest CTAs from its back: they hold at least 2 and 33 of the n rows each
// and share none, so n / 2 + 1 entries are enough for both.
struct QsLists {
    QsEntry *ends, *block[QB_CLASSES];  // block[0]: the last entry of `ends`
    QsCounters* cnt;
    __device__ __forceinline__ QsEntry& warp_entry(unsigned i) const { return ends[i]; }
    __device__ __forceinline__ QsEntry& block_entry(int c, unsigned i) const {
        return c == 0 ? *(block[0] - i) : c == 1 ? block[1][i] : block[2][i];
    }
};
__device__ __forceinline__ void qs_list(const QsLists& q, unsigned lo, unsigned hi, unsigned depth, unsigned buf) {
    const unsigned m = hi - lo;
    const QsEntry e{lo, (m - 1) | (buf << 12) | (depth << 13)};
    if (m > QS_WARP) {
        const int c = m <= qb_rows(0) ? 0 : m <= qb_rows(1) ? 1 : 2;
        q.block_entry(c, atomicAdd(&q.cnt->nblock[c], 1u)) = e;
    } else {
        q.warp_entry(atomicAdd(&q.cnt->nwarp, 1u)) = e;
    }
}
// A recursion deeper than max(8192, 2^36 / n) levels, rounded up to a multiple
// of 8 (first-element pivots on nearly ordered keys, where the reference's own
// sort is quadratic) is refused, which bounds a call to about 2^36 element
// visits.
static long long qs_max_levels(long long n) {
    const long long m = (1LL << 36) / (n > 0 ? n : 1);
    return ((m > 8192 ? m : 8192) + 7) / 8 * 8;
}
// Depths issued between two reads of the active count: a random range of n rows
// needs about 2 log2(n / QS_BLOCK) of them to come down to QS_BLOCK at its
// worst place, keys of few values a handful.  So the first round is short and
// the second holds the rest of that estimate; a depth after the last one
// (`prev` counts nothing left) writes nothing, and above QS_DIRECT tiles reads
// nothing either.  A wait costs some 25 us, a depth 30 us at 1M rows and 1.1 ms
// at 40M.  Keys of five values, with the whole estimate in one round and now:
// 2M rows 0.68 and 0.38 ms, 10M 3.5 and 2.0, 60M 26.8 and 8.4; random keys 0.81
// and 0.84 ms at 700K rows, even from 2M on.
constexpr int QS_ROUND1 = 8, QS_ROUND = 4, QS_MAX_ROUND = 64;
static int qs_second_round(long long n) {
    int d = 2;
    for (long long m = n; m > QS_BLOCK && d < QS_MAX_ROUND; m >>= 1) d += 2;
    return d - QS_ROUND1 > QS_ROUND ? d - QS_ROUND1 : QS_ROUND;
}
__device__ __forceinline__ bool qs_idle(const unsigned* prev) { return prev && *prev == 0; }

__device__ __forceinline__ long long qs_ival(const void* p, int typ, long long i) {
    switch (typ) {
    case H_B: return ((const uint8_t*)p)[i];
    case H_J: case H_C: return ((const int8_t*)p)[i];
    case H_H: return ((const int16_t*)p)[i];
    case H_I: case H_M: case H_D: case H_U: case H_W: case H_T: return ((const int32_t*)p)[i];
    default: return ((const long long*)p)[i];
    }
}

// An unsigned image of element i that orders as lib_quicksort_cmp_item
// (h_libs.cc:455-488) compares: integers (chars signed) by value, floats by
// value with -0.0 == +0.0.  Descending keys are complemented, so one
// ascending comparison of images serves both directions.
__device__ __forceinline__ unsigned long long qs_image(const void* p, int typ, long long i, unsigned* nanflag) {
    if (typ == H_F || typ == H_E) {
        double f = typ == H_F ? (double)((const float*)p)[i] : ((const double*)p)[i];
        if (f != f) { *nanflag = 1u; return 0; }
        if (f == 0.0) f = 0.0;
        const unsigned long long b = (unsigned long long)__double_as_longlong(f);
        return (b >> 63) ? ~b : (b | (1ull << 63));
    }
    return (unsigned long long)qs_ival(p, typ, i) ^ (1ull << 63);
}

__device__ __forceinline__ int qs_cmp(unsigned long long a, unsigned long long b) { return a < b ? -1 : (a > b ? 1 : 0); }

// img[p] = image of col[perm[p]] (perm null: row p)
__global__ void k_qs_image(const void* __restrict__ col, int typ, const unsigned* __restrict__ perm, long long n,
                           unsigned long long flip, unsigned long long* __restrict__ img, unsigned* nanflag,
                           uint8_t* __restrict__ up, uint8_t* __restrict__ down) {
    grid_entry();
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        img[p] = qs_image(col, typ, perm ? (long long)perm[p] : p, nanflag) ^ flip;
        if (up) up[p] = down[p] = 0;  // for k_qs_updown (a clear between kernels costs the chain 4 us)
    }
}

// rows in order; with `seg` also the one segment of a list's first column;
// the sort's counters cleared
__global__ void k_qs_iota(unsigned* __restrict__ v, long long n, unsigned* __restrict__ seg, long long* __restrict__ starts,
                          QsCounters* cnt) {
    grid_entry();
    const long long me = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long p = me; p < n; p += (long long)gridDim.x * blockDim.x) {
        v[p] = (unsigned)p;
        if (seg) seg[p] = 0;
    }
    if (me == 0) {
        *cnt = QsCounters{};
        if (seg) starts[0] = 0;
    }
}

// ---- one recursion depth over all ranges
// flag pair of position p: (x[p] <= P) + ((x[p] < P) << 32), 0 for the pivot
// itself and for finished positions.  Counts stay below 2^32, so the two
// halves of a packed prefix never carry into each other.
__device__ __forceinline__ unsigned long long qs_flag(const unsigned* __restrict__ lo, const unsigned long long* __restrict__ K,
                                                      long long p) {
    const unsigned l = lo[p];
    if (l == QS_DONE || (long long)l == p) return 0;
    const int c = qs_cmp(K[p], K[l]);
    return (unsigned long long)(c <= 0) | ((unsigned long long)(c < 0) << 32);
}

__global__ void __launch_bounds__(QS_THREADS) k_qs_count(const unsigned* __restrict__ lo, const unsigned long long* __restrict__ K,
                                                         long long n, unsigned long long* __restrict__ tile_sum,
                                                         const unsigned* __restrict__ prev) {
    grid_entry();
    if (qs_idle(prev)) return;
    __shared__ unsigned long long ws[QS_THREADS / 32];
    const long long base = (long long)blockIdx.x * QS_TILE + (long long)threadIdx.x * QS_ITEMS;
    unsigned long long s = 0;
#pragma unroll
    for (int k = 0; k < QS_ITEMS; k++)
        if (base + k < n) s += qs_flag(lo, K, base + k);
    s = warp_sum(s);
    if (lane_id() == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < QS_THREADS / 32; w++) t += ws[w];
        tile_sum[blockIdx.x] = t;
    }
}

// The tile sums before each tile: up to QS_DIRECT tiles every block of
// k_qs_prefix adds them up itself, beyond that they are scanned first, in place:
// that adding up grows with the square of the tiles.  Random f64 keys, ms, added
// up and scanned: 4M rows 3.45 and 3.52, 8M 7.19 and 7.24, 16M 16.37 and 16.27,
// 60M 71.5 and 66.9, 150M 201 and 166.
constexpr long long QS_DIRECT = 4096;
__global__ void __launch_bounds__(1024) k_qs_scan_sums(unsigned long long* __restrict__ ts, long long nt,
                                                       const unsigned* __restrict__ prev) {
    grid_entry();
    if (qs_idle(prev)) return;
    constexpr int PER = 4;
    __shared__ unsigned long long ws[32];
    const unsigned lane = lane_id(), w = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (long long b = 0; b < nt; b += 1024 * PER) {
        const long long at = b + (long long)threadIdx.x * PER;
        unsigned long long v[PER], sum = 0;
#pragma unroll
        for (int k = 0; k < PER; k++) v[k] = at + k < nt ? ts[at + k] : 0ull;
#pragma unroll
        for (int k = 0; k < PER; k++) sum += v[k];
        const unsigned long long incl = warp_incl_scan64(sum);
        if (lane == 31) ws[w] = incl;
        __syncthreads();
        const unsigned long long x = ws[lane], xi = warp_incl_scan64(x);  // every warp scans the warps' totals
        unsigned long long off = carry + __shfl_sync(0xffffffffu, xi - x, w) + incl - sum;
        carry += __shfl_sync(0xffffffffu, xi, 31);
#pragma unroll
        for (int k = 0; k < PER; k++) {
            if (at + k < nt) ts[at + k] = off;
            off += v[k];
        }
        __syncthreads();
    }
}

// S[p] = exclusive prefix of the flag pairs; S[n] = total
__global__ void __launch_bounds__(QS_THREADS) k_qs_prefix(const unsigned* __restrict__ lo, const unsigned long long* __restrict__ K,
                                                          long long n, const unsigned long long* __restrict__ tile_sum,
                                                          int scanned, unsigned long long* __restrict__ S,
                                                          const unsigned* __restrict__ prev) {
    grid_entry();
    const bool idle = qs_idle(prev);  // not looked at before the loads below are in flight
    __shared__ unsigned long long ws[QS_THREADS / 32], wb[QS_THREADS / 32];
    const long long base = (long long)blockIdx.x * QS_TILE + (long long)threadIdx.x * QS_ITEMS;
    unsigned long long v[QS_ITEMS], s = 0;
#pragma unroll
    for (int k = 0; k < QS_ITEMS; k++) {
        v[k] = base + k < n ? qs_flag(lo, K, base + k) : 0;
        s += v[k];
    }
    unsigned long long before = 0;
    if (scanned) before = threadIdx.x == 0 ? tile_sum[blockIdx.x] : 0ull;
    else
        for (long long t = threadIdx.x; t < blockIdx.x; t += QS_THREADS) before += tile_sum[t];
    before = warp_sum(before);
    const unsigned long long incl = warp_incl_scan64(s);
    if (lane_id() == 31) ws[threadIdx.x >> 5] = incl;
    if (lane_id() == 0) wb[threadIdx.x >> 5] = before;
    __syncthreads();
    unsigned long long off = incl - s;
#pragma unroll
    for (unsigned w = 0; w < QS_THREADS / 32; w++) off += wb[w] + (w < (threadIdx.x >> 5) ? ws[w] : 0ull);
    if (idle) return;
#pragma unroll
    for (int k = 0; k < QS_ITEMS; k++) {
        if (base + k < n) S[base + k] = off;
        off += v[k];
    }
    if (base < n && base + QS_ITEMS >= n) S[n] = off;  // the thread of the last element
}

__device__ __forceinline__ unsigned qs_le(unsigned long long s) { return (unsigned)s; }
__device__ __forceinline__ unsigned qs_lt(unsigned long long s) { return (unsigned)(s >> 32); }

// trade[lo + k] = the k-th element > P inside (lo, j] from the left;
// trade[hi - 1 - k] = the k-th element <= P inside (j, hi) from the right
// (They are equally many, at most half of (lo, hi), so neither side's slots
// reach the other's.  A slot outside [lo, hi) would mean inconsistent ranges and
// is recorded, not written.)
__global__ void k_qs_pos(const unsigned* __restrict__ lo, const unsigned* __restrict__ hi,
                         const unsigned long long* __restrict__ K, const unsigned long long* __restrict__ S, long long n,
                         unsigned* __restrict__ trade, const unsigned* __restrict__ prev, unsigned* derr) {
    grid_entry();
    if (qs_idle(prev)) return;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const unsigned l = lo[p];
        if (l == QS_DONE || (long long)l == p) continue;
        const unsigned h = hi[p];
        const unsigned le_lo = qs_le(S[l]), le_hi = qs_le(S[h]), le_p = qs_le(S[p]);
        const long long j = (long long)l + (le_hi - le_lo);
        const int c = qs_cmp(K[p], K[l]);
        long long slot;
        if (p <= j && c > 0) slot = (long long)l + (long long)(p - l - 1) - (long long)(le_p - le_lo);
        else if (p > j && c <= 0) slot = (long long)h - (long long)le_hi + (long long)le_p;
        else continue;
        if (slot >= (long long)l && slot < (long long)h) trade[slot] = (unsigned)p;
        else flag_error(derr, DERR_INDEX);
    }
}

// Moves every element of the partitioned ranges to its place, records the
// next depth's range of every element (or its final place; ranges of up to
// QS_BLOCK elements go to the lists) and counts the elements still in a larger
// range.  buf: which buffer K2 and P2 are.
__global__ void k_qs_move(unsigned* __restrict__ lo, unsigned* __restrict__ hi, const unsigned long long* __restrict__ K,
                          const unsigned* __restrict__ P, const unsigned long long* __restrict__ S, long long n,
                          const unsigned* __restrict__ trade, unsigned long long* __restrict__ K2,
                          unsigned* __restrict__ P2, unsigned* __restrict__ fin, const unsigned* prev, unsigned* active, unsigned depth, unsigned buf, QsLists lists,
                          unsigned* derr) {
    grid_entry();
    if (qs_idle(prev)) return;
    unsigned still = 0;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const unsigned l = lo[p];
        if (l == QS_DONE) continue;
        const unsigned h = hi[p];
        const unsigned long long sl = S[l], sh = S[h];
        const unsigned cle = qs_le(sh) - qs_le(sl);
        const long long j = (long long)l + cle;
        if (cle == h - l - 1 && qs_lt(sh) == qs_lt(sl)) {  // leftSame: every element equals the pivot
            fin[p] = P[p];
            lo[p] = QS_DONE;
            continue;
        }
        const unsigned long long kp = K[l];
        // the partner's slot of the k-th element > P in (l, j] counted from the
        // left, or of the k-th element <= P in (j, h) counted from the right
        auto left = [&](long long x) { return (long long)h - 1 - (x - l - 1) + (long long)(qs_le(S[x]) - qs_le(sl)); };
        auto right = [&](long long x) { return (long long)l + (long long)qs_le(sh) - (long long)qs_le(S[x]) - 1; };
        long long q = p, slot = -1;
        bool trades = false;
        if (p == (long long)l) {
            q = j;
            if (j > (long long)l && qs_cmp(K[j], kp) > 0) { slot = left(j); trades = true; }
        } else if (p == j) {
            q = l;
        } else {
            const int c = qs_cmp(K[p], kp);
            if (p < j && c > 0) { slot = left(p); trades = true; }
            else if (p > j && c <= 0) { slot = right(p); trades = true; }
        }
        if (trades) {
            if (slot >= (long long)l && slot < (long long)h) q = trade[slot];
            else { flag_error(derr, DERR_INDEX); q = p; }
        }
        if (q < (long long)l || q >= (long long)h) { flag_error(derr, DERR_INDEX); q = p; }
        long long nl, nh;
        if (p < j) { nl = l; nh = j; } else { nl = j + 1; nh = h; }
        if (p == j || nh - nl < 2) {
            fin[p] = P[q];
            lo[p] = QS_DONE;
        } else if (nh - nl <= QS_BLOCK) {
            P2[p] = P[q];
            K2[p] = K[q];
            lo[p] = QS_DONE;
            if (p == nl) qs_list(lists, (unsigned)nl, (unsigned)nh, depth + 1, buf);
        } else {
            P2[p] = P[q];
            K2[p] = K[q];
            lo[p] = (unsigned)nl;
            hi[p] = (unsigned)nh;
            still++;
        }
    }
    still = warp_sum(still);
    if (lane_id() == 0 && still) atomicAdd(active, still);
}

// ---- every depth of a sort whose elements the chip's threads hold: one launch
// Thread t of block b keeps E elements in registers, those of positions
// b * per + k * 1024 + t (per = 1024 E), and the blocks pass the same four
// steps as above, depth after depth, with a barrier over the grid where a step
// reads what other blocks wrote: after the block-relative prefixes, after the
// trade partners and after the moves.  What bounds a depth is latency, three
// barriers and half a dozen dependent loads: 8 us, against 13 to 15 for the
// four launches (114K random rows, 15 depths: 0.12 ms against 0.22, and no
// host waits between).  Loads of shared arrays bypass L1 (ld.cg).  A barrier
// that gives up ends the block with DERR_TIMEOUT; the others then give up too.
constexpr int QD_THREADS = 1024, QD_WARPS = QD_THREADS / 32, QD_ROUND = 256, QD_MAX_BLOCKS = 256;
struct QsDepths {
    unsigned *lo, *hi;
    unsigned long long* K[2];  // images and rows by position, of even and odd depths of this launch
    unsigned* P[2];
    unsigned long long *S, *ts;  // block-relative prefixes, the blocks' totals
    unsigned *trade, *fin;
    unsigned *act, *bar;  // elements left after each depth of this launch; the barrier's arrivals (all zero)
    unsigned* done;       // depths run, then elements left
    QsLists lists;
    unsigned* derr;
    unsigned n, level, maxd, buf;  // buf: which buffer K[0] and P[0] are
};
__device__ __forceinline__ bool qd_barrier(unsigned* bar, unsigned& target, unsigned* derr) {
    __shared__ bool ok;
    target += gridDim.x;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = true;
        atomicAdd(bar, 1u);
        long long spins = 0;
        unsigned v;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if (++spins > SPIN_LIMIT) { flag_error(derr, DERR_TIMEOUT); ok = false; break; }
        }
    }
    __syncthreads();
    return ok;
}
template <int E>
__global__ void __launch_bounds__(QD_THREADS, 1) k_qs_depths(const __grid_constant__ QsDepths a) {
    grid_entry();
    constexpr int SHIFT = E == 2 ? 11 : 12;
    static_assert(1 << SHIFT == QD_THREADS * E, "positions of a block");
    __shared__ unsigned long long wsum[E * QD_WARPS];    // per round and warp: the flag pairs before it in the block
    __shared__ unsigned long long pre[QD_MAX_BLOCKS + 1];  // the flag pairs before each block; [gridDim.x]: all
    const unsigned lane = lane_id(), w = threadIdx.x >> 5, C = gridDim.x, n = a.n;
    const unsigned base = (blockIdx.x << SHIFT) + threadIdx.x;
    unsigned lo[E], hi[E], row[E], target = 0;
    unsigned long long key[E];
#pragma unroll
    for (int k = 0; k < E; k++) {
        const unsigned p = base + k * QD_THREADS;
        lo[k] = QS_DONE;
        hi[k] = row[k] = 0;
        key[k] = 0;
        if (p < n) {
            lo[k] = a.lo[p];
            if (lo[k] != QS_DONE) {
                hi[k] = a.hi[p];
                key[k] = a.K[0][p];
                row[k] = a.P[0][p];
            }
        }
    }
    unsigned d = 0, left = 0;
    while (d < a.maxd) {
        const unsigned long long* K = a.K[d & 1];
        const unsigned* P = a.P[d & 1];
        unsigned long long rel[E], kp[E];
        int c[E];
#pragma unroll
        for (int k = 0; k < E; k++) kp[k] = lo[k] != QS_DONE ? __ldcg(K + lo[k]) : 0;
#pragma unroll
        for (int k = 0; k < E; k++) {
            const bool in = lo[k] != QS_DONE && lo[k] != base + k * QD_THREADS;
            c[k] = qs_cmp(key[k], kp[k]);
            const unsigned le = __ballot_sync(0xffffffffu, in && c[k] <= 0), lt = __ballot_sync(0xffffffffu, in && c[k] < 0);
            rel[k] = (unsigned long long)__popc(le & lanemask_lt()) | ((unsigned long long)__popc(lt & lanemask_lt()) << 32);
            if (lane == 0) wsum[k * QD_WARPS + w] = (unsigned long long)__popc(le) | ((unsigned long long)__popc(lt) << 32);
        }
        __syncthreads();
        if (w == 0) {
            unsigned long long v[E], sum = 0;
#pragma unroll
            for (int q = 0; q < E; q++) {
                v[q] = wsum[lane * E + q];
                sum += v[q];
            }
            unsigned long long off = warp_incl_scan64(sum);
            if (lane == 31) a.ts[blockIdx.x] = off;
            off -= sum;
#pragma unroll
            for (int q = 0; q < E; q++) {
                wsum[lane * E + q] = off;
                off += v[q];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < E; k++) {
            const unsigned p = base + k * QD_THREADS;
            rel[k] += wsum[k * QD_WARPS + w];
            if (p < n) a.S[p] = rel[k];  // of finished positions too: a range may end at one
        }
        if (!qd_barrier(a.bar, target, a.derr)) return;
        if (w == 0) {
            constexpr int PER = QD_MAX_BLOCKS / 32;
            unsigned long long v[PER], sum = 0;
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const unsigned b = lane * PER + q;
                v[q] = b < C ? __ldcg(a.ts + b) : 0;
            }
#pragma unroll
            for (int q = 0; q < PER; q++) sum += v[q];
            unsigned long long off = warp_incl_scan64(sum) - sum;
#pragma unroll
            for (int q = 0; q < PER; q++) {
                pre[lane * PER + q] = off;
                off += v[q];
            }
            if (lane == 31) pre[QD_MAX_BLOCKS] = off;
        }
        __syncthreads();
        auto prefix = [&](unsigned x) { return x >= n ? pre[C] : __ldcg(a.S + x) + pre[x >> SHIFT]; };
        unsigned long long sl[E], sh[E];
#pragma unroll
        for (int k = 0; k < E; k++) {
            const bool on = lo[k] != QS_DONE;
            rel[k] += pre[blockIdx.x];
            sl[k] = on ? prefix(lo[k]) : 0;
            sh[k] = on ? prefix(hi[k]) : 0;
        }
#pragma unroll
        for (int k = 0; k < E; k++) {
            const unsigned l = lo[k], p = base + k * QD_THREADS;
            if (l == QS_DONE || l == p) continue;
            const unsigned le_p = qs_le(rel[k]);
            const long long j = (long long)l + (qs_le(sh[k]) - qs_le(sl[k]));
            long long slot;
            if (p <= j && c[k] > 0) slot = (long long)l + (long long)(p - l - 1) - (long long)(le_p - qs_le(sl[k]));
            else if (p > j && c[k] <= 0) slot = (long long)hi[k] - (long long)qs_le(sh[k]) + (long long)le_p;
            else continue;
            if (slot >= (long long)l && slot < (long long)hi[k]) a.trade[slot] = p;
            else flag_error(a.derr, DERR_INDEX);
        }
        if (!qd_barrier(a.bar, target, a.derr)) return;
        unsigned still = 0;
#pragma unroll
        for (int k = 0; k < E; k++) {
            const unsigned l = lo[k], p = base + k * QD_THREADS, h = hi[k];
            if (l == QS_DONE) continue;
            const unsigned cle = qs_le(sh[k]) - qs_le(sl[k]);
            const long long j = (long long)l + cle;
            if (cle == h - l - 1 && qs_lt(sh[k]) == qs_lt(sl[k])) {  // leftSame: every element equals the pivot
                a.fin[p] = row[k];
                lo[k] = QS_DONE;
                continue;
            }
            auto left = [&](long long x, unsigned le_x) { return (long long)h - 1 - (x - l - 1) + (long long)(le_x - qs_le(sl[k])); };
            long long q = p, slot = -1;
            bool trades = false;
            if (p == l) {
                q = j;
                if (j > (long long)l && qs_cmp(__ldcg(K + j), kp[k]) > 0) {
                    slot = left(j, qs_le(prefix((unsigned)j)));
                    trades = true;
                }
            } else if (p == j) {
                q = l;
            } else if (p < j && c[k] > 0) {
                slot = left(p, qs_le(rel[k]));
                trades = true;
            } else if (p > j && c[k] <= 0) {
                slot = (long long)l + (long long)qs_le(sh[k]) - (long long)qs_le(rel[k]) - 1;
                trades = true;
            }
            if (trades) {
                if (slot >= (long long)l && slot < (long long)h) q = __ldcg(a.trade + slot);
                else { flag_error(a.derr, DERR_INDEX); q = p; }
            }
            if (q < (long long)l || q >= (long long)h) { flag_error(a.derr, DERR_INDEX); q = p; }
            if (q != (long long)p) {
                row[k] = __ldcg(P + q);
                key[k] = __ldcg(K + q);
            }
            unsigned nl = l, nh = (unsigned)j;
            if (p >= j) { nl = (unsigned)j + 1; nh = h; }
            if (p == j || nh - nl < 2) {
                a.fin[p] = row[k];
                lo[k] = QS_DONE;
            } else {
                a.P[(d & 1) ^ 1][p] = row[k];
                a.K[(d & 1) ^ 1][p] = key[k];
                if (nh - nl <= (unsigned)QS_BLOCK) {
                    lo[k] = QS_DONE;
                    if (p == nl) qs_list(a.lists, nl, nh, a.level + d + 1, a.buf ^ (d & 1) ^ 1);
                } else {
                    lo[k] = nl;
                    hi[k] = nh;
                    still++;
                }
            }
        }
        still = warp_sum(still);
        if (lane == 0 && still) atomicAdd(a.act + d, still);
        if (!qd_barrier(a.bar, target, a.derr)) return;
        left = __ldcg(a.act + d);
        d++;
        if (left == 0) break;
    }
    if (left)
#pragma unroll
        for (int k = 0; k < E; k++) {
            const unsigned p = base + k * QD_THREADS;
            if (p < n) {
                a.lo[p] = lo[k];
                a.hi[p] = hi[k];
            }
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.done[0] = d;
        a.done[1] = left;
    }
}

// ---- one warp's range: m <= 32 elements, element i in lane i (key k, row p).
// Partitions it to its end; p is then the row of position `lane`.  sl/sr: the
// warp's 32 slots for each side of the trades.  Returns the depths it took.
__device__ __forceinline__ unsigned qs_warp_range(unsigned long long k, unsigned& p, unsigned m, volatile uint8_t* sl,
                                                  volatile uint8_t* sr) {
    const unsigned lane = lane_id();
    unsigned lo = lane < m ? 0u : lane, hi = m, depths = 0;
    bool act = lane < m && m > 1;
    while (__any_sync(0xffffffffu, act)) {
        depths++;
        const unsigned long long kp = __shfl_sync(0xffffffffu, k, lo);
        const int c = act ? qs_cmp(k, kp) : 0;
        const unsigned le = __ballot_sync(0xffffffffu, act && lane != lo && c <= 0);
        const unsigned lt = __ballot_sync(0xffffffffu, act && lane != lo && c < 0);
        const unsigned seg = (hi >= 32 ? 0xffffffffu : (1u << hi) - 1u) & ~((1u << lo) - 1u);  // the range's lanes
        const unsigned cle = __popc(le & seg), j = act ? lo + cle : lane;
        const bool same = cle == hi - lo - 1 && !(lt & seg);
        auto below = [&](unsigned x) { return (unsigned)__popc(le & seg & ((1u << x) - 1u)); };  // le elements before x
        const bool up = act && !same && lane != lo && lane <= j && c > 0, down = act && !same && lane > j && c <= 0;
        if (up) sl[lo + (lane - lo - 1) - below(lane)] = (uint8_t)lane;
        if (down) sr[lo + cle - below(lane) - 1] = (uint8_t)lane;
        const unsigned long long kj = __shfl_sync(0xffffffffu, k, j);
        __syncwarp();
        unsigned q = lane;
        if (act && !same) {
            if (lane == lo) q = (j > lo && qs_cmp(kj, kp) > 0) ? sr[lo + (j - lo - 1) - below(j)] : j;
            else if (lane == j) q = lo;
            else if (up) q = sr[lo + (lane - lo - 1) - below(lane)];
            else if (down) q = sl[lo + cle - below(lane) - 1];
        }
        __syncwarp();
        k = __shfl_sync(0xffffffffu, k, q);
        p = __shfl_sync(0xffffffffu, p, q);
        if (act) {
            if (lane < j) hi = j;
            else if (lane > j) lo = j + 1;
            if (same || lane == j || hi - lo < 2) act = false;
        }
    }
    return depths;
}

// the listed ranges of 2 to 32 elements, one warp each
__global__ void __launch_bounds__(256) k_qs_warps(QsLists lists, const unsigned long long* __restrict__ K0,
                                                  const unsigned* __restrict__ P0,
                                                  const unsigned long long* __restrict__ K1,
                                                  const unsigned* __restrict__ P1, unsigned* __restrict__ fin) {
    grid_entry();
    __shared__ uint8_t slots[8][64];
    const unsigned lane = lane_id(), w = threadIdx.x >> 5, n = lists.cnt->nwarp;
    unsigned deep = 0;
    for (unsigned r = blockIdx.x * 8 + w; r < n; r += gridDim.x * 8) {
        const QsRange g = lists.warp_entry(r).range();
        const unsigned m = g.hi - g.lo;
        unsigned long long k = 0;
        unsigned p = 0;
        if (lane < m) {
            k = (g.buf ? K1 : K0)[g.lo + lane];
            p = (g.buf ? P1 : P0)[g.lo + lane];
        }
        const unsigned d = g.depth + qs_warp_range(k, p, m, slots[w], slots[w] + 32);
        deep = d > deep ? d : deep;
        if (lane < m) fin[g.lo + lane] = p;
    }
    if (lane == 0 && deep) atomicMax(&lists.cnt->depth, deep);
}

// The listed ranges of 33 to QS_BLOCK elements, one CTA each, in shared memory:
// position w * 128 + 32 k + lane of the range belongs to item k of the thread,
// so the prefixes are ballots.  Ranges that reach 32 elements wait in a list
// for the CTA's warps.  What bounds a depth is instruction issue, some 14K warp
// instructions for 4096 rows (ncu), and its five barriers: so the warps' totals
// are scanned with shuffles (one word a lane; each thread adding up all 32 of
// them was a fifth of the instructions), and a warp without a live element
// only passes the prefix on (ranges of a 114K-row sort: 0.108 -> 0.097 ms).
// Short ranges take small CTAs, many to an SM: with 1024 threads for every
// range a list order over 10M rows in segments of 40, 100 or 300 rows took 10.4,
// 9.7 and 6.2 ms, and takes 2.0, 2.0 and 2.2.
template <int C>
struct QsBlockSmem {
    static constexpr int ROWS = qb_rows(C), WARPS = qb_threads(C) / 32;
    unsigned long long K[ROWS];
    unsigned P[ROWS];
    unsigned S[ROWS + 1];             // exclusive prefix: (<= P) in the low half, (< P) in the high half
    unsigned short L[ROWS], R[ROWS];
    unsigned small[ROWS / 2];         // lo | (size - 1) << 12 | depth << 17
    unsigned wt[32];
    uint8_t slots[WARPS][64];
    unsigned nsmall, depth;
};
static_assert(QS_BLOCK <= 4096 && QS_WARP <= 32, "packing of QsBlockSmem::small");
template <int C>
__global__ void __launch_bounds__(qb_threads(C), C == 0 ? 24 : 1024 / qb_threads(C))
k_qs_blocks(const __grid_constant__ QsLists lists, const unsigned long long* __restrict__ K0,
            const unsigned* __restrict__ P0, const unsigned long long* __restrict__ K1, const unsigned* __restrict__ P1,
            unsigned* __restrict__ fin, int low, unsigned* derr) {
    grid_entry();
    extern __shared__ __align__(16) unsigned char qb_smem[];
    using Smem = QsBlockSmem<C>;
    Smem& sm = *reinterpret_cast<Smem*>(qb_smem);
    const unsigned lane = lane_id(), w = threadIdx.x >> 5, p0 = w * (32 * QB_ITEMS) + lane;
    auto le = [](unsigned s) { return s & 0xffffu; };
    auto lt = [](unsigned s) { return s >> 16; };
    unsigned cnt[C + 1], n = 0;
#pragma unroll
    for (int c = 0; c <= C; c++) {
        cnt[c] = lists.cnt->nblock[c];
        if (c >= low) n += cnt[c];
    }
    for (unsigned r = blockIdx.x; r < n; r += gridDim.x) {
        int c = C;  // the lists one after another, the longest ranges first
        unsigned at = r;
#pragma unroll
        for (int q = C; q > 0; q--)
            if (c == q && at >= cnt[q]) {
                at -= cnt[q];
                c = q - 1;
            }
        const QsRange g = lists.block_entry(c, at).range();
        const unsigned m = g.hi - g.lo;
        if (threadIdx.x == 0) sm.nsmall = sm.depth = 0;
        unsigned long long key[QB_ITEMS];
        unsigned row[QB_ITEMS], lo[QB_ITEMS], hi[QB_ITEMS], act = 0;
#pragma unroll
        for (int k = 0; k < QB_ITEMS; k++) {
            const unsigned p = p0 + 32 * k;
            key[k] = 0;
            row[k] = lo[k] = hi[k] = 0;
            if (p < m) {
                key[k] = (g.buf ? K1 : K0)[g.lo + p];
                row[k] = (g.buf ? P1 : P0)[g.lo + p];
                hi[k] = m;
                act |= 1u << k;
                sm.K[p] = key[k];
                sm.P[p] = row[k];
            }
        }
        __syncthreads();
        unsigned depths = 0;
        for (; __syncthreads_or((int)act); depths++) {
            unsigned pre[QB_ITEMS], run = 0;
            int c[QB_ITEMS];
            // a warp without a live element only passes the prefix on
            const bool live = __any_sync(0xffffffffu, act != 0);
#pragma unroll
            for (int k = 0; k < QB_ITEMS; k++) {
                pre[k] = 0;
                c[k] = 2;
            }
            if (live) {
#pragma unroll
                for (int k = 0; k < QB_ITEMS; k++) {
                    const unsigned p = p0 + 32 * k;
                    const bool a = (act >> k) & 1u;
                    c[k] = a && p != lo[k] ? qs_cmp(key[k], sm.K[lo[k]]) : 2;  // 2: the pivot, or finished
                    const unsigned ble = __ballot_sync(0xffffffffu, c[k] <= 0), blt = __ballot_sync(0xffffffffu, c[k] < 0);
                    pre[k] = run + ((unsigned)__popc(ble & lanemask_lt()) | ((unsigned)__popc(blt & lanemask_lt()) << 16));
                    run += (unsigned)__popc(ble) | ((unsigned)__popc(blt) << 16);
                }
            }
            if (lane == 0) sm.wt[w] = run;
            __syncthreads();
            // every warp scans the warps' totals for itself
            const unsigned wt = lane < Smem::WARPS ? sm.wt[lane] : 0u, wi = warp_incl_scan(wt);
            const unsigned base = __shfl_sync(0xffffffffu, wi - wt, w), all = __shfl_sync(0xffffffffu, wi, 31);
#pragma unroll
            for (int k = 0; k < QB_ITEMS; k++)
                if (p0 + 32 * k < m) sm.S[p0 + 32 * k] = base + pre[k];
            if (threadIdx.x == 0) sm.S[m] = all;
            __syncthreads();
            if (live)
#pragma unroll
            for (int k = 0; k < QB_ITEMS; k++) {
                if (!((act >> k) & 1u) || c[k] == 2) continue;
                const unsigned p = p0 + 32 * k, l = lo[k];
                const unsigned le_lo = le(sm.S[l]), le_hi = le(sm.S[hi[k]]), le_p = le(base + pre[k]);
                const unsigned j = l + (le_hi - le_lo);
                if (p <= j && c[k] > 0) sm.L[l + (p - l - 1) - (le_p - le_lo)] = (unsigned short)p;
                else if (p > j && c[k] <= 0) sm.R[l + (le_hi - le_p) - 1] = (unsigned short)p;
            }
            __syncthreads();
            unsigned long long nkey[QB_ITEMS];
            unsigned nrow[QB_ITEMS];
            if (live)
#pragma unroll
            for (int k = 0; k < QB_ITEMS; k++) {
                nkey[k] = key[k];
                nrow[k] = row[k];
                if (!((act >> k) & 1u)) continue;
                const unsigned p = p0 + 32 * k, l = lo[k], h = hi[k];
                const unsigned sl = sm.S[l], sh = sm.S[h], cle = le(sh) - le(sl), j = l + cle;
                if (cle == h - l - 1 && lt(sh) == lt(sl)) {  // leftSame: every element equals the pivot
                    lo[k] = hi[k] = 0;
                    continue;
                }
                unsigned q = p;
                if (p == l) {
                    q = j;
                    if (j > l && qs_cmp(sm.K[j], key[k]) > 0) q = sm.R[l + (j - l - 1) - (le(sm.S[j]) - le(sl))];
                } else if (p == j) {
                    q = l;
                } else if (p < j && c[k] > 0) {
                    q = sm.R[l + (p - l - 1) - (le(base + pre[k]) - le(sl))];
                } else if (p > j && c[k] <= 0) {
                    q = sm.L[l + (le(sh) - le(base + pre[k])) - 1];
                }
                if (q < l || q >= h) { flag_error(derr, DERR_INDEX); q = p; }
                nkey[k] = sm.K[q];
                nrow[k] = sm.P[q];
                if (p < j) hi[k] = j;
                else { lo[k] = p == j ? j : j + 1; if (p == j) hi[k] = j; }  // an empty range for the pivot's place
            }
            __syncthreads();
            if (live)
#pragma unroll
            for (int k = 0; k < QB_ITEMS; k++) {
                if (!((act >> k) & 1u)) continue;
                const unsigned p = p0 + 32 * k, sz = hi[k] - lo[k];
                key[k] = nkey[k];
                row[k] = nrow[k];
                sm.K[p] = key[k];
                sm.P[p] = row[k];
                if (sz > QS_WARP) continue;
                act &= ~(1u << k);
                if (sz < 2) fin[g.lo + p] = row[k];
                else if (p == lo[k]) sm.small[atomicAdd(&sm.nsmall, 1u)] = p | ((sz - 1) << 12) | ((depths + 1) << 17);
            }
        }
        // every range of 2 to 32 elements left in the CTA
        unsigned deep = depths;
        const unsigned ns = sm.nsmall;
        for (unsigned q = w; q < ns; q += Smem::WARPS) {
            const unsigned v = sm.small[q], a = v & 4095u, mm = ((v >> 12) & 31u) + 1;
            unsigned long long k = 0;
            unsigned p = 0;
            if (lane < mm) {
                k = sm.K[a + lane];
                p = sm.P[a + lane];
            }
            const unsigned d = (v >> 17) + qs_warp_range(k, p, mm, sm.slots[w], sm.slots[w] + 32);
            deep = d > deep ? d : deep;
            if (lane < mm) fin[g.lo + a + lane] = p;
        }
        if (lane == 0) atomicMax(&sm.depth, deep);
        __syncthreads();
        if (threadIdx.x == 0) atomicMax(&lists.cnt->depth, g.depth + sm.depth);
        __syncthreads();
    }
}

// ---- ranges (segments) of a list sort
// seg[p] = index of the segment holding position p (starts ascending)
__global__ void k_qs_segid(const long long* __restrict__ starts, long long ns, long long n, unsigned* __restrict__ seg,
                           QsCounters* cnt) {
    grid_entry();
    if (blockIdx.x == 0 && threadIdx.x == 0) *cnt = QsCounters{};  // the next column's
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        long long a = 0, b = ns - 1;  // last start <= p
        while (a < b) {
            const long long m = (a + b + 1) >> 1;
            if (starts[m] <= p) a = m; else b = m - 1;
        }
        seg[p] = (unsigned)a;
    }
}
// lib_order_by_sorted per segment: up[s] / down[s] = some neighbour pair rises / falls
__global__ void k_qs_updown(const unsigned long long* __restrict__ img, const unsigned* __restrict__ seg, long long n,
                            uint8_t* __restrict__ up, uint8_t* __restrict__ down) {
    grid_entry();
    for (long long p = 1 + blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const unsigned s = seg[p];
        if (s != seg[p - 1]) continue;
        const unsigned long long a = img[p - 1], b = img[p];
        if (a < b && !up[s]) up[s] = 1;
        if (a > b && !down[s]) down[s] = 1;
    }
}
enum : uint8_t { QS_SORT = 0, QS_KEEP = 1, QS_REVERSE = 2 };
// mode of each segment: an ascending-ordered segment (rises, never falls)
// is kept; for a descending key (images complemented) a segment whose values
// ascend (images fall, never rise) is reversed; every other one is sorted, and
// listed when it holds min_len or more elements (those above QS_BLOCK are only
// counted)
__global__ void k_qs_mode(const uint8_t* __restrict__ up, const uint8_t* __restrict__ down,
                          const long long* __restrict__ starts, long long ns, long long n, int desc, int min_len,
                          uint8_t* __restrict__ mode, QsLists lists) {
    grid_entry();
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < ns; s += (long long)gridDim.x * blockDim.x) {
        uint8_t m = QS_SORT;
        if (!desc && up[s] && !down[s]) m = QS_KEEP;
        if (desc && down[s] && !up[s]) { m = QS_REVERSE; atomicAdd(&lists.cnt->nrev, 1u); }
        mode[s] = m;
        const long long a = starts[s], b = s + 1 < ns ? starts[s + 1] : n;
        if (m == QS_SORT && b - a >= min_len) {
            if (b - a > QS_BLOCK) atomicAdd(&lists.cnt->nbig, 1u);
            else qs_list(lists, (unsigned)a, (unsigned)b, 0, 0);
        }
    }
}
// the only range of a vector sort (one thread)
__global__ void k_qs_whole(long long n, QsLists lists) {
    grid_entry();
    if (n > QS_BLOCK) lists.cnt->nbig = 1;
    else if (n >= 2) qs_list(lists, 0, (unsigned)n, 0, 0);
}
// the listed segments of 2 to 32 elements in stable order, one warp each: an
// element's place is the number of smaller images and of equal ones before it
__global__ void __launch_bounds__(256) k_qs_stable_small(QsLists lists, const unsigned long long* __restrict__ img,
                                                         unsigned* __restrict__ perm) {
    grid_entry();
    const unsigned lane = lane_id(), n = lists.cnt->nwarp;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += (gridDim.x * blockDim.x) >> 5) {
        const QsRange g = lists.warp_entry(r).range();
        const unsigned m = g.hi - g.lo;
        const unsigned long long k = lane < m ? img[g.lo + lane] : ~0ull;
        const unsigned row = lane < m ? perm[g.lo + lane] : 0u;
        unsigned at = 0;
        for (unsigned j = 0; j < m; j++) {
            const unsigned long long kj = __shfl_sync(0xffffffffu, k, j);
            at += kj < k || (kj == k && j < lane);
        }
        __syncwarp();
        if (lane < m) perm[g.lo + at] = row;
    }
}
__global__ void k_qs_reverse(const unsigned* __restrict__ perm, const unsigned* __restrict__ seg,
                             const long long* __restrict__ starts, long long ns, long long n, const uint8_t* __restrict__ mode,
                             unsigned* __restrict__ out) {
    grid_entry();
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const unsigned s = seg[p];
        long long q = p;
        if (mode[s] == QS_REVERSE) {
            const long long a = starts[s], b = s + 1 < ns ? starts[s + 1] : n;
            q = a + b - 1 - p;
        }
        out[p] = perm[q];
    }
}
// range of each position for the quicksort's depths in global memory (with
// `lo`): its segment when that is sorted and larger than QS_BLOCK.  Positions
// of segments that are not sorted keep their row.
__global__ void k_qs_ranges(const unsigned* __restrict__ seg, const long long* __restrict__ starts, long long ns, long long n,
                            const uint8_t* __restrict__ mode, const unsigned* __restrict__ perm,
                            unsigned* __restrict__ lo, unsigned* __restrict__ hi, unsigned* __restrict__ fin,
                            unsigned* __restrict__ act, int nact) {
    grid_entry();
    if (act && blockIdx.x == 0)
        for (int i = threadIdx.x; i < nact; i += blockDim.x) act[i] = 0;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const unsigned s = seg ? seg[p] : 0;
        const long long a = seg ? starts[s] : 0, b = seg ? (s + 1 < ns ? starts[s + 1] : n) : n;
        const bool sorted = !(mode && mode[s] != QS_SORT) && b - a >= 2;
        if (!sorted) fin[p] = perm[p];
        if (lo) {
            lo[p] = sorted && b - a > QS_BLOCK ? (unsigned)a : QS_DONE;
            hi[p] = (unsigned)b;
        }
    }
}
// stable sort of the segments in (segment, image) order: the key of a
// position that must not move (a kept, reversed or small char segment) is 0
__global__ void k_qs_skey(const unsigned long long* __restrict__ img, const unsigned* __restrict__ seg,
                          const long long* __restrict__ starts, long long ns, long long n, const uint8_t* __restrict__ mode,
                          int min_len, unsigned long long* __restrict__ key) {
    grid_entry();
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const unsigned s = seg[p];
        const long long a = starts[s], b = s + 1 < ns ? starts[s + 1] : n;
        key[p] = (mode[s] == QS_SORT && b - a >= min_len) ? img[p] : 0;
    }
}
__global__ void k_qs_gather_seg(const unsigned* __restrict__ seg, const unsigned* __restrict__ pos, long long n,
                                unsigned* __restrict__ out) {
    grid_entry();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = seg[pos[i]];
}
__global__ void k_qs_permute(const unsigned* __restrict__ perm, const unsigned* __restrict__ pos, long long n,
                             unsigned* __restrict__ out) {
    grid_entry();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = perm[pos[i]];
}
// lib_quicksort_char below ten elements (h_libs.cc:388-390): the all-pairs
// exchange on a[rtn[i]] > a[rtn[j]], one thread per sorted segment
__global__ void k_qs_char_small(const int8_t* __restrict__ a, const long long* __restrict__ starts, long long ns, long long n,
                                const uint8_t* __restrict__ mode, unsigned* __restrict__ perm) {
    grid_entry();
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < ns; s += (long long)gridDim.x * blockDim.x) {
        const long long lo = starts[s], hi = s + 1 < ns ? starts[s + 1] : n;
        if (mode[s] != QS_SORT || hi - lo >= 10 || hi - lo < 2) continue;
        unsigned r[10];
        const int m = (int)(hi - lo);
        for (int i = 0; i < m; i++) r[i] = perm[lo + i];
        for (int i = 0; i < m; i++)
            for (int j = 0; j < m; j++)
                if (a[r[i]] > a[r[j]]) { const unsigned t = r[i]; r[i] = r[j]; r[j] = t; }
        for (int i = 0; i < m; i++) perm[lo + i] = r[i];
    }
}
// run heads of the next column: a new segment or a new image value
__global__ void k_qs_heads(const unsigned long long* __restrict__ img, const unsigned* __restrict__ seg, long long n,
                           uint8_t* __restrict__ head) {
    grid_entry();
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
        head[p] = p == 0 || seg[p] != seg[p - 1] || img[p] != img[p - 1];
}

static unsigned qs_grid(long long n) {
    unsigned g = grid_for(n, 256);
    return g > (unsigned)g_sms * 16 ? (unsigned)g_sms * 16 : g;
}

static I qs_too_deep(long long levels) {
    return set_error(E_NOT_IMPL, "the reference's quicksort recursion is deeper than %lld levels here "
                     "(first-element pivots on nearly ordered keys)", levels);
}

static I qs_lists_alloc(long long n, QsLists* q) {
    bool ok = true;
    const size_t ends = (size_t)(n / 2 + 1);
    q->ends = (QsEntry*)salloc(ends * sizeof(QsEntry));
    ok = ok && q->ends;
    q->block[0] = q->ends + (ends - 1);
    for (int c = 1; c < QB_CLASSES; c++) {  // the class's shortest range: one more than the class below holds
        q->block[c] = (QsEntry*)salloc((size_t)(n / qb_rows(c - 1) + 1) * sizeof(QsEntry));
        ok = ok && q->block[c];
    }
    q->cnt = (QsCounters*)salloc(sizeof(QsCounters));
    return ok && q->cnt ? 0 : E_DEVICE_OOM;
}

// NaN keys, from counters already read back
static I qs_nan_check(const QsCounters& h) {
    if (h.nan) return set_error(E_NOT_IMPL, "NaN sort key: the reference's quicksort compares NaN as greater than "
                                "itself and scans outside the range");
    return 0;
}

// Launches k_qs_depths when n elements fit one block per SM of at most 4 per
// thread; *took = false when they do not, or the device does not take the blocks
// together.  @order of random f64 keys, us, with four launches a depth and
// with this: 6000 rows 182 and 162, 20K 225 and 191, 114K 351 and 287, 300K 407
// and 326, 600K 635 and 511; with 8 per thread (the registers spill) 600K 767,
// 1.2M 1064 against 1045.  (The CTA tier has since become 5 to 10 us faster on
// either side.)
static I qs_depths_launch(long long n, QsDepths& q, bool* took) {
    void* args[] = {&q};
    *took = false;
    const long long most = (long long)(g_sms < QD_MAX_BLOCKS ? g_sms : QD_MAX_BLOCKS) * QD_THREADS;
    const int e = n <= 2 * most ? 2 : 4;
    if (n > e * most) return 0;
    HG_CHECK(last_launch_error());  // of the launches before, while the error is theirs
    const void* kern = e == 2 ? (const void*)k_qs_depths<2> : (const void*)k_qs_depths<4>;
    LaunchScope ls("qs_depths");
    const cudaError_t rc = launch_cooperative_args(kern, grid_for(n, QD_THREADS * e), QD_THREADS, 0, args);
    *took = rc == cudaSuccess;
    if (*took) return 0;
    cudaGetLastError();  // the refused launch's own
    if (rc == cudaErrorCooperativeLaunchTooLarge || rc == cudaErrorNotSupported) return 0;
    HG_CU(rc);
    return 0;
}

// the ranges of classes low to C, in CTAs of class C
template <int C>
static I qs_blocks(const QsLists& lists, const QsCounters& h, int low, const unsigned long long* img, const unsigned* perm,
                   const unsigned long long* K2, const unsigned* P2, unsigned* fin) {
    unsigned n = 0;
    for (int c = low; c <= C; c++) n += h.nblock[c];
    if (!n) return 0;
    const int dsm = (int)sizeof(QsBlockSmem<C>);
    // the attribute belongs to the current device's context: set it on every call (a host-side write)
    HG_CU(cudaFuncSetAttribute(k_qs_blocks<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, dsm));
    const unsigned cap = (unsigned)g_sms * (2048 / qb_threads(C));
    HG_LAUNCH(C == 0 ? "qs_blocks_128" : C == 1 ? "qs_blocks_512" : "qs_blocks", n < cap ? n : cap, qb_threads(C), (size_t)dsm,
              k_qs_blocks<C>, lists, img, perm, K2, P2, fin, low, g_derr);
    return last_launch_error();
}
// Short ranges have launches of their own, in small CTAs, when a class has more
// than QB_OWN ranges a SM.  Fewer go with the class above: the launches follow
// one another, each as long as its deepest range, while large CTAs that would
// stand idle take them at once (100K random keys 0.27 ms, 0.33 with three
// launches; 114K rows in segments of 300, some 2.5 a SM: 0.226 and 0.192).
constexpr unsigned QB_OWN0 = 2, QB_OWN1 = 2;
static I qs_all_blocks(const QsLists& lists, const QsCounters& h, const unsigned long long* img, const unsigned* perm,
                       const unsigned long long* K2, const unsigned* P2, unsigned* fin) {
    const bool own0 = h.nblock[0] > QB_OWN0 * g_sms;
    const bool own1 = h.nblock[1] + (own0 ? 0 : h.nblock[0]) > QB_OWN1 * g_sms;
    HG_CHECK(qs_blocks<2>(lists, h, own1 ? 2 : own0 ? 1 : 0, img, perm, K2, P2, fin));
    if (own1) HG_CHECK(qs_blocks<1>(lists, h, own0 ? 1 : 0, img, perm, K2, P2, fin));
    if (own0) HG_CHECK(qs_blocks<0>(lists, h, 0, img, perm, K2, P2, fin));
    return 0;
}

// The quicksort of every sorted range at once.  perm/img: the elements in
// their current order (consumed); lists/h: the ranges listed so far and their
// counters as the host has read them; seg, starts, mode: the segments, for
// those too large to list (null: the whole).  On return fin holds every
// position's row.
static I qs_run(long long n, unsigned* perm, unsigned long long* img, const unsigned* seg, const long long* starts,
                long long ns, const uint8_t* mode, const QsLists& lists, QsCounters* h, unsigned* fin) {
    ScratchScope ss;  // the next column of a list takes the same memory
    const unsigned g = qs_grid(n);
    const long long max_levels = qs_max_levels(n);
    unsigned long long* K2 = nullptr;  // the second buffer (img and perm are the first)
    unsigned* P2 = nullptr;
    unsigned *lo = nullptr, *hi = nullptr;
    if (h->nbig) {
        lo = (unsigned*)salloc((size_t)n * 4);
        hi = (unsigned*)salloc((size_t)n * 4);
        if (!lo || !hi) return E_DEVICE_OOM;
    }
    unsigned* act = nullptr;  // counts of a round's depths, then k_qs_depths' barrier and result
    constexpr int nact = QD_ROUND + 3;
    if (h->nbig) {
        act = (unsigned*)salloc(nact * 4);
        if (!act) return E_DEVICE_OOM;
    }
    bool act_clear = true;  // k_qs_ranges has cleared them
    HG_LAUNCH("qs_ranges", g, 256, 0, k_qs_ranges, seg, starts, ns, n, mode, perm, lo, hi, fin, act, nact);
    if (h->nbig) {
        const long long nt = (n + QS_TILE - 1) / QS_TILE;
        const bool scan = nt > QS_DIRECT;
        P2 = (unsigned*)salloc((size_t)n * 4);
        K2 = (unsigned long long*)salloc((size_t)n * 8);
        unsigned long long* S = (unsigned long long*)salloc((size_t)(n + 1) * 8);
        unsigned long long* ts = (unsigned long long*)salloc((size_t)(nt > QD_MAX_BLOCKS ? nt : QD_MAX_BLOCKS) * 8);
        unsigned* trade = (unsigned*)salloc((size_t)n * 4);
        if (!P2 || !K2 || !S || !ts || !trade) return E_DEVICE_OOM;
        // the ranges listed at the start are read from perm/img, which the
        // depths below reuse only at the positions of larger ranges
        unsigned* Pc = perm;
        unsigned long long* Kc = img;
        int round = 0, rounds = 0;
        bool resident = true;  // k_qs_depths takes the depths, while the elements fit the chip's threads
        for (long long level = 0;; level += round) {
            if (level >= max_levels) return qs_too_deep(max_levels);
            if (resident) {
                round = (int)(max_levels - level < QD_ROUND ? max_levels - level : QD_ROUND);
                if (!act_clear) HG_CU(cudaMemsetAsync(act, 0, nact * 4, g_stream));
                act_clear = false;
                QsDepths q{lo, hi, {Kc, Kc == img ? K2 : img}, {Pc, Pc == perm ? P2 : perm}, S, ts, trade, fin,
                           act, act + QD_ROUND, act + QD_ROUND + 1, lists, g_derr, (unsigned)n, (unsigned)level,
                           (unsigned)round, Kc == img ? 0u : 1u};
                HG_CHECK(qs_depths_launch(n, q, &resident));
                if (resident) {
                    unsigned res[2];
                    HG_CHECK(rb_queue(res, q.done, 8));
                    HG_CHECK(rb_queue(h, lists.cnt, sizeof *h));
                    HG_CU(stream_sync());
                    if (res[0] == 0) {  // a barrier gave up
                        HG_CHECK(check_device_errors());
                        return set_error(E_DEVICE, "the quicksort's grid barrier did not complete");
                    }
                    if (res[1] == 0) break;
                    if (res[0] & 1) {
                        Kc = q.K[1];
                        Pc = q.P[1];
                    }
                    round = (int)res[0];
                    continue;
                }
            }
            round = rounds == 0 ? QS_ROUND1 : rounds == 1 ? qs_second_round(n) : QS_ROUND;
            rounds++;
            if (level + round > max_levels) round = (int)(max_levels - level);
            HG_CU(cudaMemsetAsync(act, 0, QS_MAX_ROUND * 4, g_stream));
            for (int d = 0; d < round; d++) {
                // (a round begins with elements left; where a depth takes microseconds
                // only the kernel that hides the look does it)
                const unsigned *left = d ? act + d - 1 : nullptr, *prev = scan ? left : nullptr;
                HG_LAUNCH("qs_count", (unsigned)nt, QS_THREADS, 0, k_qs_count, lo, Kc, n, ts, prev);
                if (scan) HG_LAUNCH("qs_scan_sums", 1, 1024, 0, k_qs_scan_sums, ts, nt, prev);
                HG_LAUNCH("qs_prefix", (unsigned)nt, QS_THREADS, 0, k_qs_prefix, lo, Kc, n, ts, scan ? 1 : 0, S, left);
                HG_LAUNCH("qs_pos", g, 256, 0, k_qs_pos, lo, hi, Kc, S, n, trade, prev, g_derr);
                unsigned* Pn = Pc == perm ? P2 : perm;
                unsigned long long* Kn = Kc == img ? K2 : img;
                HG_LAUNCH("qs_move", g, 256, 0, k_qs_move, lo, hi, Kc, Pc, S, n, trade, Kn, Pn, fin, prev, act + d,
                          (unsigned)(level + d), Kn == img ? 0u : 1u, lists, g_derr);
                Pc = Pn;
                Kc = Kn;
            }
            HG_CHECK(last_launch_error());
            unsigned left = 0;
            HG_CHECK(rb_queue(&left, act + round - 1, 4));
            HG_CHECK(rb_queue(h, lists.cnt, sizeof *h));
            HG_CU(stream_sync());
            if (left == 0) break;
        }
    }
    HG_CHECK(qs_all_blocks(lists, *h, img, perm, K2, P2, fin));
    if (h->nwarp) {
        const unsigned cap = 16u * (unsigned)g_sms, want = grid_for(h->nwarp, 8);
        HG_LAUNCH("qs_warps", want < cap ? want : cap, 256, 0, k_qs_warps, lists, img, perm, K2, P2, fin);
    }
    HG_CHECK(last_launch_error());
    // read again with the caller's next wait, for qs_depth_check
    return rb_queue(h, lists.cnt, sizeof *h);
}
// after the wait that follows a qs_run: the depths of the listed ranges count
static I qs_depth_check(long long n, const QsCounters& h) {
    return (long long)h.depth > qs_max_levels(n) ? qs_too_deep(qs_max_levels(n)) : 0;
}

static I qs_image_of(const void* col, I typ, const unsigned* perm, long long n, bool desc, unsigned long long* img,
                     unsigned* nanflag, uint8_t* up = nullptr, uint8_t* down = nullptr) {
    if (n > 0)
        HG_LAUNCH("qs_image", qs_grid(n), 256, 0, k_qs_image, col, (int)typ, perm, n, desc ? ~0ull : 0ull, img, nanflag, up,
                  down);
    return last_launch_error();
}

// lib_order_by_vector (h_libs.cc:730-736) on a key its quicksort sorts:
// rows 0..n-1 in order, then lib_quicksort_other over [0, n).
I qs_sort_vector(const void* col, I typ, long long n, bool asc, const unsigned** perm_out) {
    if (n >= (1LL << 31)) return set_error(E_NOT_IMPL, "quicksort order of 2^31 or more rows");
    unsigned* perm = (unsigned*)salloc((size_t)(n > 0 ? n : 1) * 4);
    unsigned* fin = (unsigned*)salloc((size_t)(n > 0 ? n : 1) * 4);
    unsigned long long* img = (unsigned long long*)salloc((size_t)(n > 0 ? n : 1) * 8);
    QsLists lists;
    if (!perm || !fin || !img) return E_DEVICE_OOM;
    HG_CHECK(qs_lists_alloc(n, &lists));
    *perm_out = fin;
    if (n == 0) return 0;
    HG_LAUNCH("qs_iota", qs_grid(n), 256, 0, k_qs_iota, perm, n, nullptr, nullptr, lists.cnt);
    HG_CHECK(qs_image_of(col, typ, nullptr, n, !asc, img, &lists.cnt->nan));
    HG_LAUNCH("qs_whole", 1, 1, 0, k_qs_whole, n, lists);
    QsCounters h;
    HG_CHECK(rb_queue(&h, lists.cnt, sizeof h));
    HG_CU(stream_sync());
    HG_CHECK(qs_nan_check(h));
    HG_CHECK(qs_run(n, perm, img, nullptr, nullptr, 0, nullptr, lists, &h, fin));
    HG_CHECK(check_device_errors());
    return qs_depth_check(n, h);
}

// lib_quicksort_list (h_libs.cc:637-697) over nc columns: for each column in
// turn, every run of rows equal on the columns before it is checked by
// lib_order_by_sorted (kept, or reversed for a descending column whose values
// ascend) and otherwise sorted -- i32/i64 columns by the stable merge sort,
// char columns by lib_quicksort_char, the rest by the quicksort -- and its
// runs of equal values form the next column's ranges.  *checked: the device
// error word has been read since the last pass that can set it.
I qs_sort_list(int nc, const void* const* cols, const I* typs, const B* asc, long long n, const unsigned** perm_out,
               bool* checked) {
    *checked = true;
    if (n >= (1LL << 31)) return set_error(E_NOT_IMPL, "quicksort order of 2^31 or more rows");
    const size_t nn = (size_t)(n > 0 ? n : 1);
    unsigned* perm = (unsigned*)salloc(nn * 4);
    unsigned* tmp = (unsigned*)salloc(nn * 4);
    unsigned* seg = (unsigned*)salloc(nn * 4);
    unsigned long long* img = (unsigned long long*)salloc(nn * 8);
    long long* starts = (long long*)salloc(nn * 8);
    uint8_t* flags = (uint8_t*)salloc(nn * 3);
    QsLists lists;
    if (!perm || !tmp || !seg || !img || !starts || !flags) return E_DEVICE_OOM;
    HG_CHECK(qs_lists_alloc(n, &lists));
    *perm_out = perm;
    if (n == 0) return 0;
    uint8_t* up = flags;
    uint8_t* down = flags + nn;
    uint8_t* mode = flags + 2 * nn;
    unsigned* nanflag = &lists.cnt->nan;
    const unsigned g = qs_grid(n);
    HG_LAUNCH("qs_iota", g, 256, 0, k_qs_iota, perm, n, seg, starts, lists.cnt);
    long long ns = 1;  // segments: runs of rows equal on the columns sorted so far
    for (int c = 0; c < nc; c++) {
        const I typ = typs[c];
        const bool desc = asc && !asc[c];
        if (typ == H_C && desc)
            return set_error(E_NOT_IMPL, "descending char column in a list order (the reference indexes past the range)");
        const bool stable = typ == H_I || typ == H_L || typ == H_C;
        bool ran = false;  // a quicksort whose counters the next wait reads into h
        HG_CHECK(qs_image_of(cols[c], typ, perm, n, desc, img, nanflag, up, down));
        // lib_order_by_sorted
        HG_LAUNCH("qs_updown", g, 256, 0, k_qs_updown, img, seg, n, up, down);
        HG_LAUNCH("qs_mode", qs_grid(ns), 256, 0, k_qs_mode, up, down, starts, ns, n, desc ? 1 : 0, typ == H_C ? 10 : 2,
                  mode, lists);
        QsCounters h;
        HG_CHECK(rb_queue(&h, lists.cnt, sizeof h));
        HG_CU(stream_sync());
        HG_CHECK(qs_nan_check(h));
        if (h.nrev) {
            HG_LAUNCH("qs_reverse", g, 256, 0, k_qs_reverse, perm, seg, starts, ns, n, mode, tmp);
            unsigned* t = perm; perm = tmp; tmp = t;
            HG_CHECK(qs_image_of(cols[c], typ, perm, n, desc, img, nanflag));
        }
        if (!h.nbig && !h.nblock[0] && !h.nblock[1] && !h.nblock[2] && (!h.nwarp || stable)) {
            // nothing is left to sort, or only short segments in stable order
            if (h.nwarp) {
                const unsigned cap = 16u * (unsigned)g_sms, want = grid_for(h.nwarp, 8);
                HG_LAUNCH("qs_stable_small", want < cap ? want : cap, 256, 0, k_qs_stable_small, lists, img, perm);
            }
            if (typ == H_C)
                HG_LAUNCH("qs_char_small", qs_grid(ns), 256, 0, k_qs_char_small, (const int8_t*)cols[c], starts, ns, n,
                          mode, perm);
        } else
        if (stable) {
            // stable by (segment, image): radix sort on the image, then on
            // the segment index; kept, reversed and small char segments have
            // key 0 and do not move
            unsigned long long* key = (unsigned long long*)salloc(nn * 8);
            unsigned* sk = (unsigned*)salloc(nn * 4);
            if (!key || !sk) return E_DEVICE_OOM;
            HG_LAUNCH("qs_skey", g, 256, 0, k_qs_skey, img, seg, starts, ns, n, mode, typ == H_C ? 10 : 2, key);
            const unsigned long long* k1;
            const unsigned* pos1;
            *checked = c + 1 < nc;  // the next column's waits read the error word
            HG_CHECK(radix_sort<unsigned long long>(key, n, &k1, &pos1, nullptr));
            HG_LAUNCH("qs_gather_seg", g, 256, 0, k_qs_gather_seg, seg, pos1, n, sk);
            const unsigned* k2;
            const unsigned* pos2;
            HG_CHECK(radix_sort<unsigned>(sk, n, &k2, &pos2, pos1));
            HG_LAUNCH("qs_permute", g, 256, 0, k_qs_permute, perm, pos2, n, tmp);
            unsigned* t = perm; perm = tmp; tmp = t;
            if (typ == H_C)
                HG_LAUNCH("qs_char_small", qs_grid(ns), 256, 0, k_qs_char_small, (const int8_t*)cols[c], starts, ns, n,
                          mode, perm);
        } else {
            HG_CHECK(qs_run(n, perm, img, seg, starts, ns, mode, lists, &h, tmp));
            ran = true;
            unsigned* t = perm; perm = tmp; tmp = t;
        }
        if (c + 1 < nc) {  // the runs of equal values become the next column's segments
            HG_CHECK(qs_image_of(cols[c], typ, perm, n, desc, img, nanflag));
            HG_LAUNCH("qs_heads", g, 256, 0, k_qs_heads, img, seg, n, up);
            HG_CHECK(compact_rows(up, n, starts, &ns));  // waits, and reads the device errors
            if (ran) HG_CHECK(qs_depth_check(n, h));
            HG_LAUNCH("qs_segid", g, 256, 0, k_qs_segid, starts, ns, n, seg, lists.cnt);
        } else if (ran) {
            HG_CHECK(check_device_errors());
            HG_CHECK(qs_depth_check(n, h));
        }
    }
    HG_CHECK(last_launch_error());
    *perm_out = perm;
    return 0;
}

}  // namespace hg
