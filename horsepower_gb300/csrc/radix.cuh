// The counted radix pass: one stable counting-sort pass over one digit.
//
// The rows are cut into chunks of consecutive tiles, one CTA each (as many
// chunks as CTAs fit on the chip).  A pass is three launches:
//   count    every chunk's digit counts, digit-major, and the digits' totals
//   scan     each (digit, chunk)'s first output position
//   scatter  each CTA walks its tiles in order: it ranks a tile's rows by
//            digit, puts the tile into digit order in shared memory and writes
//            each digit's run behind the one before it.
// No CTA waits for another, and only chunks x digits counts exist (0.6 MB),
// whereas a look-back or per-tile counts cost a status word per tile and
// digit.  A digit's output is written front to back by each CTA, so the
// sectors that a run leaves half written are completed from L2 by the same
// CTA's next tile.
//
// A row travels as one 64-bit record, its remaining key bits above its row id:
// the tile is staged and written with one 8-byte access per row, and a run of
// 16 rows is 128 bytes.  (60M rows, one pass: 0.36 ms with 32-bit keys and row
// ids in two arrays, 0.28 ms as records.)  When key and row id together exceed
// 64 bits by no more than the first digit, the first pass drops that digit
// from the records; wider keys take the two-array pass.  The key source is a
// template parameter, so the first pass reads the columns themselves (packed
// and range-compressed in registers) and no key array is made.
//
// What bounds a pass is the ranking: without it the same kernel moves 150M
// records in 0.40 ms, with it in 0.585 (8-bit digits) and 0.676 (9 bits); the
// ballots are half of its 70 instructions a row, and the warp's counter of a
// digit is read and written once a row, a chain through shared memory (ncu:
// short scoreboard 3.8 of 11.5 cycles an instruction, DRAM 51%).
// __match_any_sync, peers or counters by shared-memory atomics and other tiles
// were all slower or even.  A pass's count takes 0.20 ms.  150M rows: @order
// of (i64 key, i32 secondary) 11.2 -> 5.0 ms and @group of the i64 keys 6.0 ->
// 3.5 ms against look-back passes over separate keys and row ids.
#pragma once
#include "dev_common.cuh"

namespace hg {

// ---- key sources: key(i) of row i
template <typename K>
struct RxKeys {  // an array of keys
    using key_t = K;
    const K* p;
    __device__ __forceinline__ K operator()(long long i) const { return p[i]; }
};
struct RxLow32 {  // the low 32 bits of an i64 column
    using key_t = unsigned;
    const long long* p;
    __device__ __forceinline__ unsigned operator()(long long i) const { return (unsigned)(unsigned long long)p[i]; }
};
// Two i32/i64 columns, each range-compressed (v - lo, or hi - v when
// descending) and packed: the second in the low bits.
struct RxPair {
    using key_t = unsigned long long;
    const void* p0;
    const void* p1;
    long long o0, o1;  // lo, or hi when descending
    int w0, w1;        // the column is i64
    int d0, d1;        // descending
    int shift;         // of the first column
    __device__ __forceinline__ static unsigned long long part(const void* p, int w, int d, long long o, long long i) {
        const long long v = w ? ((const long long*)p)[i] : (long long)((const int*)p)[i];
        return d ? (unsigned long long)o - (unsigned long long)v : (unsigned long long)v - (unsigned long long)o;
    }
    __device__ __forceinline__ unsigned long long operator()(long long i) const {
        return (part(p0, w0, d0, o0, i) << shift) | part(p1, w1, d1, o1, i);
    }
};
struct RxRec {  // records written by an earlier pass
    using key_t = unsigned long long;
    const unsigned long long* p;
    __device__ __forceinline__ unsigned long long operator()(long long i) const { return p[i]; }
};

// chunk c of C covers tiles [rx_first_tile(c), rx_first_tile(c + 1)) of ntiles
__device__ __forceinline__ unsigned rx_first_tile(unsigned ntiles, unsigned c, unsigned C) {
    return (unsigned)(((unsigned long long)ntiles * c) / C);
}

// hides a value's origin from the optimiser, so that what was computed from it
// before is computed again instead of held in registers across a phase
__device__ __forceinline__ void rx_forget(unsigned long long& v) { asm volatile("" : "+l"(v)); }

// The lanes whose BITS-bit digit equals this lane's (every lane takes part).
// Each ballot comes from a predicate set straight from the bit, and the same
// predicate turns the ballot round for a lane whose bit is clear: 3.5
// instructions a bit.  These four instructions are those of CUB's MatchAny
// (util_ptx.cuh, BSD-3-Clause).  With an all-ones word per bit as the mask of
// both, as the compiler makes of the C++ form, a bit takes 5 (150M rows, 8-bit
// pass: 0.69 ms against 0.585).
template <int BITS>
__device__ __forceinline__ unsigned rx_match(unsigned d) {
    unsigned same[BITS], peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < BITS; b++)
        asm volatile(
            "{\n.reg .pred p;\n.reg .b32 t;\n"
            "and.b32 t, %1, %2;\nsetp.ne.u32 p, t, 0;\n"
            "vote.sync.ballot.b32 %0, p, 0xffffffff;\n"
            "@!p not.b32 %0, %0;\n}"
            : "=r"(same[b]) : "r"(d), "r"(1u << b));
#pragma unroll
    for (int b = 0; b < BITS; b++) peers &= same[b];
    return peers;
}

// Eight-bit digits: three CTAs per SM of 16 rows per thread; with four (64
// registers) the records spill and larger tiles make fewer warps.  Nine-bit
// digits: two of 24, so that a digit's run in a tile is 12 rows instead of 8
// and the bigger histogram's registers do not spill.  One pass over 150M
// records, ms, 8 and 9 bits:  3 x 16 0.585 and 0.84;  3 x 12 0.63, 1.01;
// 2 x 20 0.61, 0.71;  2 x 24 0.60, 0.676;  2 x 28 0.61, 0.71;  2 x 32 0.67,
// 0.75;  4 x 10 0.73, 1.2.
constexpr long long RX_MAX_ROWS = 0xffffffffll;  // counts, positions and row ids are 32 bits wide
constexpr int RX_THREADS = 256, RX_WARPS = RX_THREADS / 32, RX_MAX_PER_SM = 3, RX_MAX_DIGITS = 512;
template <int BITS>
struct RxShape {
    static constexpr int PER_SM = BITS > 8 ? 2 : RX_MAX_PER_SM, ITEMS = BITS > 8 ? 24 : 16;
    static constexpr int TILE = RX_THREADS * ITEMS;
};
constexpr int RX_KV_ITEMS = 12, RX_KV_TILE = RX_THREADS * RX_KV_ITEMS;

// counts[d * C + c] = rows of chunk c with digit d; tot[d] += them (tot zeroed before)
template <typename SRC, int BITS, int ITEMS>
__global__ void __launch_bounds__(RX_THREADS) k_rx_count(SRC src, unsigned n, unsigned ntiles, int shift, int bits,
                                                         unsigned* __restrict__ counts, unsigned* __restrict__ tot) {
    grid_entry();
    using K = typename SRC::key_t;
    constexpr int D = 1 << BITS, TILE = RX_THREADS * ITEMS;
    __shared__ unsigned wh[RX_WARPS][D];
    for (int i = threadIdx.x; i < RX_WARPS * D; i += RX_THREADS) (&wh[0][0])[i] = 0;
    __syncthreads();
    const unsigned dmask = (1u << bits) - 1, w = threadIdx.x >> 5;
    const unsigned t1 = rx_first_tile(ntiles, blockIdx.x + 1, gridDim.x);
    for (unsigned t = rx_first_tile(ntiles, blockIdx.x, gridDim.x); t < t1; t++) {
        const long long base = (long long)t * TILE + threadIdx.x;
        if ((long long)(t + 1) * TILE <= (long long)n) {
            K key[ITEMS];
#pragma unroll
            for (int k = 0; k < ITEMS; k++) key[k] = src(base + k * RX_THREADS);
#pragma unroll
            for (int k = 0; k < ITEMS; k++) atomicAdd(&wh[w][(unsigned)(key[k] >> shift) & dmask], 1u);
        } else {
            for (int k = 0; k < ITEMS; k++) {
                const long long i = base + k * RX_THREADS;
                if (i < (long long)n) atomicAdd(&wh[w][(unsigned)(src(i) >> shift) & dmask], 1u);
            }
        }
    }
    __syncthreads();
    for (unsigned d = threadIdx.x; d <= dmask; d += RX_THREADS) {
        unsigned c = 0;
#pragma unroll
        for (int q = 0; q < RX_WARPS; q++) c += wh[q][d];
        counts[d * gridDim.x + blockIdx.x] = c;
        if (c) atomicAdd(&tot[d], c);
    }
}

// one block per digit: counts[d * C ..] becomes its exclusive scan, from the
// rows of all lower digits (positions fit 32 bits: row ids do)
__global__ void __launch_bounds__(256) k_rx_scan(unsigned* __restrict__ counts, unsigned C,
                                                 const unsigned* __restrict__ tot) {
    grid_entry();
    __shared__ unsigned ws[8], wb[8];
    const unsigned lane = lane_id(), w = threadIdx.x >> 5, d = blockIdx.x;
    unsigned below = 0;
    for (unsigned q = threadIdx.x; q < d; q += 256) below += tot[q];
    below = warp_sum(below);
    if (lane == 0) wb[w] = below;
    __syncthreads();
    unsigned carry = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) carry += wb[q];
    for (unsigned c0 = 0; c0 < C; c0 += 256) {
        const unsigned c = c0 + threadIdx.x;
        const unsigned v = c < C ? counts[d * C + c] : 0u;
        const unsigned incl = warp_incl_scan(v);
        if (lane == 31) ws[w] = incl;
        __syncthreads();
        unsigned before = 0, all = 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            if (q < (int)w) before += ws[q];
            all += ws[q];
        }
        if (c < C) counts[d * C + c] = carry + before + incl - v;
        carry += all;
        __syncthreads();
    }
}

// The digit histogram of a ranked tile: wh[w][d] = rows of warp w with digit d
// becomes the first place in the tile of warp w's rows of digit d; gl[d] = the
// output position of a row of digit d less its place in the tile, from gofs[d],
// the digit's next output position, which moves on.
template <int D>
__device__ __forceinline__ void rx_tile_offsets(unsigned short (*wh)[D], unsigned* gofs, unsigned* gl, unsigned* ws) {
    constexpr int PER = D / RX_THREADS;  // adjacent digits per thread
    const unsigned lane = lane_id(), w = threadIdx.x >> 5;
    unsigned ct[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const unsigned d = threadIdx.x * PER + j;
        ct[j] = 0;
#pragma unroll
        for (int q = 0; q < RX_WARPS; q++) {
            const unsigned x = wh[q][d];
            wh[q][d] = (unsigned short)ct[j];
            ct[j] += x;
        }
        sum += ct[j];
    }
    const unsigned incl = warp_incl_scan(sum);
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    unsigned start = incl - sum;
#pragma unroll
    for (int q = 0; q < RX_WARPS; q++)
        if (q < (int)w) start += ws[q];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const unsigned d = threadIdx.x * PER + j;
#pragma unroll
        for (int q = 0; q < RX_WARPS; q++) wh[q][d] = (unsigned short)(wh[q][d] + start);
        const unsigned g = gofs[d];
        gl[d] = g - start;
        gofs[d] = g + ct[j];
        start += ct[j];
    }
}

// What a record pass reads and writes.
//   first (SRC not RxRec): record = ((key >> drop) & kmask) << rb | row id,
//     the row id being vin[i] or, without vin, i; digit = (key >> kshift) &
//     dmask.  `cut`: the digit is not in the record and is staged beside it.
//   later: digit = (record >> kshift) & dmask.
//   mode RX_REC: the records to out; RX_V64: the row ids to perm64 (at n - 1 -
//     pos when `reverse`); RX_KV64: these and the keys (record >> rb) to out as
//     KW-byte words; RX_KV: the keys and the u32 row ids (vout).
enum { RX_REC = 0, RX_V64 = 1, RX_KV64 = 2, RX_KV = 3 };
struct RxPass {
    const unsigned* vin;
    void* out;
    unsigned* vout;
    long long* perm64;
    unsigned long long kmask;
    unsigned n, ntiles;
    int kshift, bits, rb, drop, cut, mode, reverse, kw;
    const unsigned* offs;
    unsigned* derr;
};
template <typename SRC, int BITS>
__global__ void __launch_bounds__(RX_THREADS, RxShape<BITS>::PER_SM) k_rx_scatter(SRC src, RxPass a) {
    grid_entry();
    constexpr bool FIRST = !std::is_same<SRC, RxRec>::value;
    constexpr int D = 1 << BITS, RX_ITEMS = RxShape<BITS>::ITEMS, RX_TILE = RxShape<BITS>::TILE;
    extern __shared__ __align__(16) unsigned char rx_smem[];
    unsigned long long* stage = reinterpret_cast<unsigned long long*>(rx_smem);  // the tile in digit order
    unsigned short* sdig = reinterpret_cast<unsigned short*>(stage + RX_TILE);   // its digits, when dropped
    __shared__ __align__(16) unsigned short wh[RX_WARPS][D];
    __shared__ unsigned gofs[D], gl[D], ws[RX_WARPS];
    const unsigned lane = lane_id(), w = threadIdx.x >> 5, n = a.n;
    const unsigned dmask = (1u << a.bits) - 1;
    for (unsigned d = threadIdx.x; d < D; d += RX_THREADS) gofs[d] = d <= dmask ? a.offs[d * gridDim.x + blockIdx.x] : 0u;
    const unsigned t1 = rx_first_tile(a.ntiles, blockIdx.x + 1, gridDim.x);
    unsigned t = rx_first_tile(a.ntiles, blockIdx.x, gridDim.x);
    const bool dropped = FIRST && a.cut;
    unsigned long long rec[RX_ITEMS];  // FIRST: the key until it is staged
    // a lane's rows of tile tt: w * 32 * RX_ITEMS + k * 32 + lane.  Rows past
    // the end take the highest digit: they come last in the tile and are
    // never written.
    auto load = [&](unsigned tt) {
        const long long wb = (long long)tt * RX_TILE + w * (32 * RX_ITEMS) + lane;
        if ((long long)(tt + 1) * RX_TILE <= (long long)n) {
#pragma unroll
            for (int k = 0; k < RX_ITEMS; k++) rec[k] = (unsigned long long)src(wb + k * 32);
        } else {
            const int left = (int)((long long)n - wb);
#pragma unroll
            for (int k = 0; k < RX_ITEMS; k++) {
                rec[k] = ~0ull;
                if (k * 32 < left) rec[k] = (unsigned long long)src(wb + k * 32);
            }
        }
    };
    static_assert(sizeof(wh) % (16 * RX_THREADS) == 0, "the zeroing covers wh");
    if (t < t1) load(t);
    for (; t < t1; t++) {
#pragma unroll
        for (int q = 0; q < (int)(sizeof(wh) / 16 / RX_THREADS); q++)
            reinterpret_cast<uint4*>(&wh[0][0])[threadIdx.x + q * RX_THREADS] = make_uint4(0, 0, 0, 0);
        __syncthreads();  // also: the previous tile's writes have read gl and the staged rows
        unsigned rank[RX_ITEMS / 2];  // of rows 2j and 2j + 1 in the low and high halves
#pragma unroll
        for (int k = 0; k < RX_ITEMS; k++) {
            const unsigned d = (unsigned)(rec[k] >> a.kshift) & dmask;
            const unsigned peers = rx_match<BITS>(d);
            const unsigned before = __popc(peers & lanemask_lt());
            const unsigned pre = wh[w][d];
            __syncwarp();
            if (before == 0) wh[w][d] = (unsigned short)(pre + __popc(peers));
            __syncwarp();
            if (k & 1) rank[k / 2] |= (pre + before) << 16;
            else rank[k / 2] = pre + before;
        }
        __syncthreads();
        rx_tile_offsets<D>(wh, gofs, gl, ws);
        __syncthreads();
        const unsigned row0 = t * RX_TILE + w * (32 * RX_ITEMS) + lane;
#pragma unroll
        for (int k = 0; k < RX_ITEMS; k++) {
            rx_forget(rec[k]);
            const unsigned d = (unsigned)(rec[k] >> a.kshift) & dmask;
            const unsigned at = wh[w][d] + ((k & 1) ? rank[k / 2] >> 16 : rank[k / 2] & 0xffffu);
            if constexpr (FIRST) {
                unsigned row = row0 + k * 32;
                if (a.vin) row = row < n ? a.vin[row] : 0u;
                stage[at] = (((rec[k] >> a.drop) & a.kmask) << a.rb) | row;
                if (dropped) sdig[at] = (unsigned short)d;
            } else {
                stage[at] = rec[k];
            }
        }
        __syncthreads();
        const unsigned tn = n - t * RX_TILE < RX_TILE ? n - t * RX_TILE : (unsigned)RX_TILE;
        if (t + 1 < t1) load(t + 1);  // in flight while this tile is written
        // FIRST: the digit's place in a record is the key's, drop included
        const int rshift = FIRST ? a.rb + a.kshift - a.drop : a.kshift;
        const unsigned rowmask = a.rb >= 32 ? 0xffffffffu : (1u << a.rb) - 1;
#pragma unroll 4
        for (int k = 0; k < RX_ITEMS; k++) {
            const unsigned i = threadIdx.x + k * RX_THREADS;
            if (i < tn) {
                const unsigned long long r = stage[i];
                const unsigned d = dropped ? sdig[i] : (unsigned)(r >> rshift) & dmask;
                const unsigned pos = gl[d] + i;
                if (pos >= n) {  // inconsistent counts: an error, not a store
                    flag_error(a.derr, DERR_INDEX);
                    continue;
                }
                if (a.mode == RX_REC) {
                    ((unsigned long long*)a.out)[pos] = r;
                    continue;
                }
                const unsigned row = (unsigned)r & rowmask;
                if (a.mode != RX_V64) {
                    if (a.kw == 8) ((unsigned long long*)a.out)[pos] = r >> a.rb;
                    else ((unsigned*)a.out)[pos] = (unsigned)(r >> a.rb);
                }
                if (a.mode == RX_KV) a.vout[pos] = row;
                else a.perm64[a.reverse ? n - 1 - pos : pos] = (long long)row;
            }
        }
    }
}

// The same for 64-bit keys that leave no room for a row id: keys and row ids
// in two arrays.  mode: RX_KV, RX_KV64 or RX_V64.
__global__ void __launch_bounds__(RX_THREADS, RX_MAX_PER_SM)
k_rx_scatter_kv(const unsigned long long* __restrict__ kin, RxPass a) {
    grid_entry();
    constexpr int D = 256, ITEMS = RX_KV_ITEMS, TILE = RX_KV_TILE;
    extern __shared__ __align__(16) unsigned char rx_smem[];
    unsigned long long* skey = reinterpret_cast<unsigned long long*>(rx_smem);
    unsigned* sval = reinterpret_cast<unsigned*>(skey + TILE);
    __shared__ __align__(16) unsigned short wh[RX_WARPS][D];
    __shared__ unsigned gofs[D], gl[D], ws[RX_WARPS];
    const unsigned lane = lane_id(), w = threadIdx.x >> 5, n = a.n;
    const unsigned dmask = (1u << a.bits) - 1;
    gofs[threadIdx.x] = threadIdx.x <= dmask ? a.offs[threadIdx.x * gridDim.x + blockIdx.x] : 0u;
    const unsigned t1 = rx_first_tile(a.ntiles, blockIdx.x + 1, gridDim.x);
    for (unsigned t = rx_first_tile(a.ntiles, blockIdx.x, gridDim.x); t < t1; t++) {
        const long long wb = (long long)t * TILE + w * (32 * ITEMS) + lane;
        const int left = (int)((long long)n - wb < TILE ? (long long)n - wb : TILE);
        unsigned long long key[ITEMS];
        unsigned val[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            key[k] = ~0ull;
            val[k] = 0;
            if (k * 32 < left) {
                key[k] = kin[wb + k * 32];
                val[k] = a.vin ? a.vin[wb + k * 32] : (unsigned)(wb + k * 32);
            }
        }
        static_assert(sizeof(wh) == 16 * RX_THREADS, "one 16-byte store per thread clears wh");
        reinterpret_cast<uint4*>(&wh[0][0])[threadIdx.x] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        unsigned rank[ITEMS / 2];
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const unsigned d = (unsigned)(key[k] >> a.kshift) & dmask;
            const unsigned peers = rx_match<8>(d);
            const unsigned before = __popc(peers & lanemask_lt());
            const unsigned pre = wh[w][d];
            __syncwarp();
            if (before == 0) wh[w][d] = (unsigned short)(pre + __popc(peers));
            __syncwarp();
            if (k & 1) rank[k / 2] |= (pre + before) << 16;
            else rank[k / 2] = pre + before;
        }
        __syncthreads();
        rx_tile_offsets<D>(wh, gofs, gl, ws);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            rx_forget(key[k]);
            const unsigned d = (unsigned)(key[k] >> a.kshift) & dmask;
            const unsigned at = wh[w][d] + ((k & 1) ? rank[k / 2] >> 16 : rank[k / 2] & 0xffffu);
            skey[at] = key[k];
            sval[at] = val[k];
        }
        __syncthreads();
        const unsigned tn = n - t * TILE < TILE ? n - t * TILE : (unsigned)TILE;
#pragma unroll 4
        for (int k = 0; k < ITEMS; k++) {
            const unsigned i = threadIdx.x + k * RX_THREADS;
            if (i < tn) {
                const unsigned long long kk = skey[i];
                const unsigned pos = gl[(unsigned)(kk >> a.kshift) & dmask] + i;
                if (pos >= n) {
                    flag_error(a.derr, DERR_INDEX);
                    continue;
                }
                if (a.mode != RX_V64) ((unsigned long long*)a.out)[pos] = kk;
                if (a.mode == RX_KV) a.vout[pos] = sval[i];
                else a.perm64[a.reverse ? n - 1 - pos : pos] = (long long)sval[i];
            }
        }
    }
}

}  // namespace hg
