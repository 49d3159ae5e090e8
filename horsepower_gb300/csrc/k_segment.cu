// Segmented aggregation: the interpreter chain
//     raze(each(@sum|@avg|@min|@max|@len, each_right(@index, x, groups)))
// (h_primitive.cc:1818-1904 each/each_right, :935-955 raze, per-group
// pfnIndex :43-94 and pfnSum/pfnAvg/pfnReduce/pfnLen :656-847) and its fused
// form, the peephole functions of the pattern pass (optimizer/pattern.cc:
// 63-105 FP1/2/5/6/7, emitter :180-219), exported as hgpuGroupSum & co.
//
// Per-group semantics follow the interpreter (ints sum in i64, avg in f64,
// min/max keep the type, empty groups give the pfnReduce sentinels).  Every
// group is reduced with the fixed-order tile tree of dev_common.cuh, so the
// chain and the fused entry points are bit-identical to each other and to a
// plain @sum of the gathered vector.
//
// GB300 layout: the rows of all groups are one device array with group
// starts (the @group output), so a group is a contiguous segment.  Groups of
// up to 4096 rows are reduced by one warp each; longer groups are split into
// 4096-row chunks reduced by one CTA each, and their chunk partials are
// reduced again the same way.
#include <limits>
#include <vector>

#include "dev_common.cuh"

namespace hg {

I scan_exclusive(const unsigned* in, long long n, unsigned long long* out, unsigned long long* total_h);
I compact_rows(const uint8_t* mask, long long n, long long* out, long long* count);

enum { AG_SUM = 0, AG_AVG = 1, AG_MIN = 2, AG_MAX = 3, AG_LEN = 4 };
enum { OP_SUM = 0, OP_MIN = 1, OP_MAX = 2 };

template <typename A, int OP>
__device__ __forceinline__ A sop(A a, A b) {
    if constexpr (OP == OP_SUM) {
        if constexpr (std::is_same<A, double>::value) return __dadd_rn(a, b);
        else if constexpr (std::is_same<A, float>::value) return __fadd_rn(a, b);
        else return (A)((unsigned long long)a + (unsigned long long)b);
    } else if constexpr (OP == OP_MIN) return (a < b) ? a : b;
    else return (a > b) ? a : b;
}
// The values of a 256-lane tile's 8 warps at once, x[v] = this lane's value of
// warp v, folded as one xor butterfly (offsets 16, 8, 4, 2, 1) per warp and
// then ((w0, w1), (w2, w3)), ((w4, w5), (w6, w7)); the result is valid in lane
// 0.  A butterfly adds in all 32 lanes though half of them hold a copy after
// each step; here the first three steps give the freed half another warp's
// values instead (lane bit 16 picks warps 0-3 or 4-7, bit 8 then bit 4 halve
// again), so 8 warps cost 4 + 2 + 1 + 1 + 1 operations and 3 for the tile
// instead of 40 and 7.  GB300 issues an FP64 instruction every 19 cycles per
// SM, which is what bounds these folds.  Every operand pair, and its order in
// lane 0's tree, is that of the separate butterflies.
template <typename A, int OP>
__device__ __forceinline__ A sop_lane(A own, A other, bool upper) {
    if constexpr (OP == OP_SUM) return sop<A, OP>(own, other);  // commutes bit for bit
    else return upper ? sop<A, OP>(other, own) : sop<A, OP>(own, other);
}
template <typename A, int OP>
__device__ __forceinline__ A stile8(const A (&x)[8]) {
    const unsigned lane = lane_id();
    const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
    A a[4], b[2], c;
#pragma unroll
    for (int i = 0; i < 4; i++)
        a[i] = sop_lane<A, OP>(u16 ? x[i + 4] : x[i], __shfl_xor_sync(0xffffffffu, u16 ? x[i] : x[i + 4], 16), u16);
#pragma unroll
    for (int i = 0; i < 2; i++)
        b[i] = sop_lane<A, OP>(u8 ? a[i + 2] : a[i], __shfl_xor_sync(0xffffffffu, u8 ? a[i] : a[i + 2], 8), u8);
    c = sop_lane<A, OP>(u4 ? b[1] : b[0], __shfl_xor_sync(0xffffffffu, u4 ? b[0] : b[1], 4), u4);
    c = sop_lane<A, OP>(c, __shfl_xor_sync(0xffffffffu, c, 2), lane & 2);
    c = sop_lane<A, OP>(c, __shfl_xor_sync(0xffffffffu, c, 1), lane & 1);
    // lanes 4v .. 4v+3 hold warp v's value
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) c = sop<A, OP>(c, __shfl_down_sync(0xffffffffu, c, o));
    return c;
}
// ... when warps 4 to 7 hold nothing but the identity
template <typename A, int OP>
__device__ __forceinline__ A stile4(const A (&x)[8], A ident) {
    const unsigned lane = lane_id();
    const bool u16 = lane & 16, u8 = lane & 8;
    A a[2], b;
#pragma unroll
    for (int i = 0; i < 2; i++)
        a[i] = sop_lane<A, OP>(u16 ? x[i + 2] : x[i], __shfl_xor_sync(0xffffffffu, u16 ? x[i] : x[i + 2], 16), u16);
    b = sop_lane<A, OP>(u8 ? a[1] : a[0], __shfl_xor_sync(0xffffffffu, u8 ? a[0] : a[1], 8), u8);
    b = sop_lane<A, OP>(b, __shfl_xor_sync(0xffffffffu, b, 4), lane & 4);
    b = sop_lane<A, OP>(b, __shfl_xor_sync(0xffffffffu, b, 2), lane & 2);
    b = sop_lane<A, OP>(b, __shfl_xor_sync(0xffffffffu, b, 1), lane & 1);
    // lanes 8v .. 8v+7 hold warp v's value
    b = sop<A, OP>(b, __shfl_down_sync(0xffffffffu, b, 8));
    b = sop<A, OP>(b, __shfl_down_sync(0xffffffffu, b, 16));
    return sop<A, OP>(b, ident);
}
// the same for a block of 256 threads, thread t holding lane t & 31 of warp
// t >> 5: valid in thread 0 (sh is free again after the caller's next barrier)
template <typename A, int OP>
__device__ __forceinline__ A sblock8(A acc, A* sh) {
    sh[threadIdx.x] = acc;
    __syncthreads();
    A r = acc;
    if (threadIdx.x < 32) {
        A x[8];
#pragma unroll
        for (int v = 0; v < 8; v++) x[v] = sh[v * 32 + threadIdx.x];
        r = stile8<A, OP>(x);
    }
    return r;
}

// N elements of one lane, STRIDE apart: positions first + k * STRIDE, k = 0 ..
// N - 1, those below `end` loaded (row numbers first, then the values, so all N
// gathers are in flight together).
template <typename T, bool GATHER, int STRIDE, int N>
__device__ __forceinline__ void seg_load(const T* __restrict__ src, const long long* __restrict__ rows, long long nx,
                                         long long first, long long end, T (&v)[N], bool& bad) {
    if constexpr (GATHER) {
        long long r[N];
#pragma unroll
        for (int k = 0; k < N; k++) {
            const long long j = first + (long long)k * STRIDE;
            r[k] = j < end ? rows[j] : 0;
        }
#pragma unroll
        for (int k = 0; k < N; k++) {
            const bool in = first + (long long)k * STRIDE < end;
            const bool ok = r[k] >= 0 && r[k] < nx;
            bad |= in && !ok;
            v[k] = (in && ok) ? src[r[k]] : T(0);
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) {
            const long long j = first + (long long)k * STRIDE;
            v[k] = j < end ? src[j] : T(0);
        }
    }
}
// the 16 elements of one lane of a 256-lane tile
template <typename T, bool GATHER>
__device__ __forceinline__ void seg_load16(const T* __restrict__ src, const long long* __restrict__ rows, long long nx,
                                           long long first, long long end, T (&v)[16], bool& bad) {
    seg_load<T, GATHER, 256>(src, rows, nx, first, end, v, bad);
}

// The columns one launch reduces over the same segments: block row blockIdx.y
// takes column blockIdx.y.
// (a __grid_constant__ parameter where that saves the stack frame that an index
// into a copy takes; k_seg_mid, which has no register left, is faster without)
constexpr int SEG_MANY = 4;
template <typename T, typename A>
struct SegIO {
    const T* src[SEG_MANY];
    A* out[SEG_MANY];
};

// Segments by size class, so that each is reduced by the narrowest unit that
// reproduces the tile tree exactly: sizes 0-1, 2, 3-4, 5-8, 9-16, 17-32
// (classes 0-5), 33-4096 (6) and longer (7).
constexpr int SEG_CLASSES = 8;
static_assert(SEG_PLAN_HDR_BYTES == (SEG_CLASSES + 2) * 8, "plan header layout");
__device__ __forceinline__ int seg_class(long long m) {
    if (m <= 1) return 0;
    if (m > TILE_SUM) return 7;
    if (m > 32) return 6;
    return 32 - __clz((int)(m - 1));  // ceil(log2 m): 2 -> 1, 3-4 -> 2, ..., 17-32 -> 5
}
// pass 1: segments per class (cnt[c]) and the 4096-element chunks of the long
// ones, in all (*nch)
__global__ void k_seg_class_count(const long long* __restrict__ starts, long long ng, long long total,
                                  unsigned* __restrict__ cnt, unsigned long long* __restrict__ nch) {
    grid_entry();
    __shared__ unsigned sc[SEG_CLASSES];
    __shared__ unsigned long long snch;
    if (threadIdx.x < SEG_CLASSES) sc[threadIdx.x] = 0;
    if (threadIdx.x == 0) snch = 0;
    __syncthreads();
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g < ng) {
        const long long m = ((g + 1 < ng) ? starts[g + 1] : total) - starts[g];
        atomicAdd(&sc[seg_class(m)], 1u);
        if (m > TILE_SUM) atomicAdd(&snch, (unsigned long long)((m + TILE_SUM - 1) / TILE_SUM));
    }
    __syncthreads();
    if (threadIdx.x < SEG_CLASSES && sc[threadIdx.x]) atomicAdd(&cnt[threadIdx.x], sc[threadIdx.x]);
    if (threadIdx.x == 0 && snch) atomicAdd(nch, snch);
}
// pass 2: the segment ids of class c at ids[off_c ...] (off_c = segments of
// lower classes; order inside a class is immaterial); cur[c] counts the
// places taken
__global__ void k_seg_class_ids(const long long* __restrict__ starts, long long ng, long long total,
                                const unsigned* __restrict__ cnt, unsigned* __restrict__ cur,
                                unsigned* __restrict__ ids) {
    grid_entry();
    __shared__ unsigned sc[SEG_CLASSES], sbase[SEG_CLASSES];
    if (threadIdx.x < SEG_CLASSES) sc[threadIdx.x] = 0;
    __syncthreads();
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    int c = 0;
    unsigned local = 0;
    if (g < ng) {
        c = seg_class(((g + 1 < ng) ? starts[g + 1] : total) - starts[g]);
        local = atomicAdd(&sc[c], 1u);
    }
    __syncthreads();
    if (threadIdx.x < SEG_CLASSES) {
        unsigned off = 0;
        for (int k = 0; k < (int)threadIdx.x; k++) off += cnt[k];
        sbase[threadIdx.x] = sc[threadIdx.x] ? off + atomicAdd(&cur[threadIdx.x], sc[threadIdx.x]) : 0;
    }
    __syncthreads();
    if (g < ng) ids[sbase[c] + local] = (unsigned)g;
}

// Segments of classes 0-5 in one launch.  Class c (at most P = 2^c
// elements): the segment's elements sit in lanes 0..m-1 of warp 0 of the
// 256-lane tile and every other lane and warp holds the identity, so the
// tile tree reduces to the xor butterfly over the first P lanes.  Here a lane
// holds up to four of a segment's places, L = P / 4 apart (one lane a segment
// of up to 4, eight of up to 32): the butterfly's first two steps are its own
// and the rest go over L lanes.  What bounds the kernel is latency (segment
// id, start, row id and value are loads one behind the other) and the FP64
// unit, which takes a warp's instruction every 19 cycles however few lanes
// matter: four loads in flight per lane, and 1.5 additions a segment of 17 to
// 32 rows against 6 with one place per lane.  5.8M groups of 1 to 32 rows (18M
// rows) of a 150M-row Zipf grouping: 0.65-0.77 ms with one place per lane,
// 0.555-0.69 now, where the values' random sectors take 0.40 (the chip loads 41 to
// 45 G/s of them from columns of 1 GB and more, whatever is in flight; so
// four sets of segments at a time, or a pipeline over the four loads, gained
// nothing).
constexpr int SEG_LANE_ITEMS = 4;
__host__ __device__ constexpr int seg_lanes(int c) { return c <= 2 ? 1 : (1 << c) / SEG_LANE_ITEMS; }  // L of class c
template <typename T, typename A, int OP, bool GATHER>
__global__ void __launch_bounds__(256) k_seg_warps(const __grid_constant__ SegIO<T, A> io,
                                                   const long long* __restrict__ rows, long long nx, const long long* __restrict__ starts, long long ng,
                                                   long long total, const unsigned* __restrict__ ids,
                                                   const unsigned* __restrict__ cnt, A ident,
                                                   unsigned* derr) {
    grid_entry();
    const T* __restrict__ src = io.src[blockIdx.y];
    A* __restrict__ out = io.out[blockIdx.y];
    __shared__ long long wfirst[7];  // first warp of each class 0-5; wfirst[6] = warps in all
    __shared__ unsigned cfirst[6], ccnt[6];  // first id and number of ids of each class
    if (threadIdx.x == 0) {
        long long w = 0;
        unsigned o = 0;
        for (int c = 0; c < 6; c++) {
            wfirst[c] = w;
            cfirst[c] = o;
            ccnt[c] = cnt[c];
            const long long per = 32 / seg_lanes(c);  // segments per warp
            w += ((long long)cnt[c] + per - 1) / per;
            o += cnt[c];
        }
        wfirst[6] = w;
    }
    __syncthreads();
    const unsigned lane = lane_id();
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5), wend = wfirst[6];
    bool bad = false;
    for (long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < wend; w += warps) {
        int c = 0;
        while (c < 5 && w >= wfirst[c + 1]) c++;
        const int lb = c <= 2 ? 0 : c - 2;  // log2 of the lanes of a segment
        const unsigned l = lane & ((1u << lb) - 1);
        const long long k = (w - wfirst[c]) * (32 >> lb) + (lane >> lb);
        const bool have = k < (long long)ccnt[c];
        const unsigned g = ids[cfirst[c] + (have ? k : 0)];  // a class without segments has no warps
        const long long s = starts[g], e = ((long long)g + 1 < ng) ? starts[g + 1] : total;
        const long long m = have ? e - s : 0;
        bool in[SEG_LANE_ITEMS];
        long long at[SEG_LANE_ITEMS];
        T v[SEG_LANE_ITEMS];
#pragma unroll
        for (int q = 0; q < SEG_LANE_ITEMS; q++) {
            at[q] = l + ((unsigned)q << lb);
            in[q] = at[q] < m;
            at[q] += s;
        }
        if constexpr (GATHER) {
#pragma unroll
            for (int q = 0; q < SEG_LANE_ITEMS; q++) at[q] = in[q] ? rows[at[q]] : 0;
#pragma unroll
            for (int q = 0; q < SEG_LANE_ITEMS; q++) {
                const bool ok = at[q] >= 0 && at[q] < nx;
                bad |= in[q] && !ok;
                in[q] = in[q] && ok;
            }
        }
#pragma unroll
        for (int q = 0; q < SEG_LANE_ITEMS; q++) v[q] = in[q] ? src[at[q]] : T(0);
        A x[SEG_LANE_ITEMS];
#pragma unroll
        for (int q = 0; q < SEG_LANE_ITEMS; q++) {
            x[q] = ident;
            if (in[q]) x[q] = sop<A, OP>(ident, (A)v[q]);
        }
        A acc = x[0];
        if (c == 1) acc = sop<A, OP>(x[0], x[1]);
        else if (c >= 2) acc = sop<A, OP>(sop<A, OP>(x[0], x[2]), sop<A, OP>(x[1], x[3]));
        for (int o = (1 << lb) >> 1; o > 0; o >>= 1) acc = sop<A, OP>(acc, __shfl_xor_sync(0xffffffffu, acc, o));
        if (l == 0 && have) out[g] = acc;
    }
    if (bad) flag_error(derr, DERR_INDEX);
}

// Class 6 (33 to 4096 elements).  What bounds it is the latency of the row
// and value loads, so each lane has up to 16 of each in flight: a warp takes a
// segment of up to 512 elements (two per lane of the 256-lane tile) and loads
// all 8 virtual warps at once; the block's longer segments are taken one after
// another by all 8 warps, warp v as virtual warp v.  (One warp walking the 8
// virtual warps in turn, for every size: 0.98 ms against 0.61 ms for the
// 157K mid-size groups of a 150M-row Zipf grouping.)  WALK: rounds of eight such
// segments are k_seg_walk's (an instance of its own: looking for them costs
// groups of 50 rows 2%).
template <typename T, typename A, int OP, bool GATHER, bool WALK>
__global__ void __launch_bounds__(256, 4) k_seg_mid(SegIO<T, A> io, const long long* __restrict__ rows,
                                                 long long nx, const long long* __restrict__ starts, long long ng,
                                                 long long total, const unsigned* __restrict__ ids,
                                                 const unsigned* __restrict__ cnt, A ident,
                                                 unsigned* derr) {
    grid_entry();
    const T* __restrict__ src = io.src[blockIdx.y];
    A* __restrict__ out = io.out[blockIdx.y];
    __shared__ unsigned first;
    __shared__ long long sbig[8];  // per warp: its segment when that is longer than 512, else -1
    __shared__ A ws[256];
    if (threadIdx.x == 0) {
        unsigned o = 0;
        for (int c = 0; c < 6; c++) o += cnt[c];
        first = o;
    }
    __syncthreads();
    const long long n6 = cnt[6];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    bool bad = false;
    // neighbouring segments go to different blocks: a Zipf grouping's long
    // groups are neighbours, and a block takes its long segments in turn
    for (long long w0 = blockIdx.x; w0 < n6; w0 += (long long)gridDim.x * 8) {
        const long long w = w0 + (long long)gridDim.x * warp;
        long long g = -1, s = 0, e = 0;
        if (w < n6) {
            g = ids[first + w];
            s = starts[g];
            e = (g + 1 < ng) ? starts[g + 1] : total;
        }
        const long long m = e - s;
        if (lane == 0) sbig[warp] = m > 512 ? g : -1;
        if (g >= 0 && m <= 512) {
            T x[16];  // x[v + 8 k]: element k of lane `lane` of virtual warp v
            seg_load<T, GATHER, 32>(src, rows, nx, s + lane, e, x, bad);
            A acc[8], r;
#pragma unroll
            for (int v = 0; v < 8; v++) {
                acc[v] = ident;
                if (v * 32 >= m) continue;  // the whole warp: no FP64 issue for absent elements
                if (v * 32 + (int)lane < m) acc[v] = sop<A, OP>(acc[v], (A)x[v]);
            }
            if (m > 256) {
#pragma unroll
                for (int v = 0; v < 8; v++)
                    if (256 + v * 32 + (int)lane < m) acc[v] = sop<A, OP>(acc[v], (A)x[v + 8]);
            }
            if (m <= 128) r = stile4<A, OP>(acc, ident);
            else r = stile8<A, OP>(acc);
            if (lane == 0) out[g] = r;
        }
        __syncthreads();
        int nq = 8;
        if constexpr (WALK) {
            nq = 0;  // all eight are k_seg_walk's
            for (int q = 0; q < 8; q++)
                if (sbig[q] < 0) nq = 8;
        }
        for (int q = 0; q < nq; q++) {
            const long long gb = sbig[q];  // the same in every warp
            if (gb < 0) continue;
            const long long sb = starts[gb], eb = (gb + 1 < ng) ? starts[gb + 1] : total;
            T x[16];
            seg_load16<T, GATHER>(src, rows, nx, sb + threadIdx.x, eb, x, bad);
            A acc = ident;
#pragma unroll
            for (int k = 0; k < 16; k++)
                if (sb + (long long)k * 256 + threadIdx.x < eb) acc = sop<A, OP>(acc, (A)x[k]);
            acc = sblock8<A, OP>(acc, ws);
            if (threadIdx.x == 0) out[gb] = acc;
            __syncthreads();
        }
        __syncthreads();  // sbig is rewritten by the next round
    }
    if (bad) flag_error(derr, DERR_INDEX);
}

// The rounds of k_seg_mid whose eight segments are all longer than 512, when
// there are several rounds to a block and the class can average more than 512
// rows (seg_reduce): each warp walks a segment of its own, 256 elements (a lane's
// element of each of the 8 virtual warps) at a time.  A grouping's row lists
// are ascending, so the warps of the chip walk through the column side by side
// and meet in its sectors, where a segment read at once takes them from all of
// the column.  Groups of 1000 rows, f64 sums: 60M rows 1.25 ms by k_seg_mid
// alone and 1.15 so, 150M rows 3.25 and 3.03; of 3000, 150M rows 3.24 and 2.93.
// With one round to a block it is the other way round (20M rows in groups of
// 1000: 0.42 and 0.71 ms).  Five blocks an SM spill (3.25 ms at 150M rows).
template <typename T, typename A, int OP, bool GATHER>
__global__ void __launch_bounds__(256, 4) k_seg_walk(const __grid_constant__ SegIO<T, A> io,
                                                     const long long* __restrict__ rows, long long nx,
                                                     const long long* __restrict__ starts, long long ng,
                                                     long long total, const unsigned* __restrict__ ids,
                                                     const unsigned* __restrict__ cnt, A ident, unsigned* derr) {
    grid_entry();
    const T* __restrict__ src = io.src[blockIdx.y];
    A* __restrict__ out = io.out[blockIdx.y];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    unsigned first = 0;
    for (int c = 0; c < 6; c++) first += cnt[c];
    const long long n6 = cnt[6];
    bool bad = false;
    for (long long w0 = blockIdx.x; w0 < n6; w0 += (long long)gridDim.x * 8) {
        const long long w = w0 + (long long)gridDim.x * (lane & 7);  // lane q looks at warp q's segment
        long long g = 0, s = 0, e = 0;
        if (w < n6) {
            g = ids[first + w];
            s = starts[g];
            e = (g + 1 < ng) ? starts[g + 1] : total;
        }
        if (!__all_sync(0xffffffffu, e - s > 512)) continue;
        g = __shfl_sync(0xffffffffu, g, warp);
        s = __shfl_sync(0xffffffffu, s, warp);
        e = __shfl_sync(0xffffffffu, e, warp);
        A acc[8];
#pragma unroll
        for (int v = 0; v < 8; v++) acc[v] = ident;
#pragma unroll 1
        for (long long b = s; b < e; b += 256) {
            T x[8];
            seg_load<T, GATHER, 32>(src, rows, nx, b + lane, e, x, bad);
#pragma unroll
            for (int v = 0; v < 8; v++)
                if (b + v * 32 + (int)lane < e) acc[v] = sop<A, OP>(acc[v], (A)x[v]);
        }
        const A r = stile8<A, OP>(acc);
        if (lane == 0) out[g] = r;
    }
    if (bad) flag_error(derr, DERR_INDEX);
}

// The chunk partials of the long segments, one CTA per segment of at most
// 4096 partials (the caller checks): thread t holds partials t, t + 256, ...
// exactly as the tile tree places them (the order k_seg_mid's virtual warps
// follow, whatever size class would have scheduled the segment); the result
// goes straight to the segment's slot of out.
template <typename A, int OP>
__global__ void __launch_bounds__(256) k_seg_partials(const A* __restrict__ parts, const long long* __restrict__ pstarts,
                                                      const long long* __restrict__ big, long long nbig,
                                                      long long nchunks, A ident, const __grid_constant__ SegIO<A, A> io) {
    grid_entry();
    __shared__ A ws[256];
    const long long g = blockIdx.x;
    const A* __restrict__ part = parts + (size_t)blockIdx.y * (size_t)nchunks;
    A* __restrict__ out = io.out[blockIdx.y];
    const long long s = pstarts[g], e = (g + 1 < nbig) ? pstarts[g + 1] : nchunks;
    bool bad = false;
    A v[16];
    seg_load16<A, false>(part, nullptr, 0, s + threadIdx.x, e, v, bad);
    A acc = ident;
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (s + k * 256 + threadIdx.x < e) acc = sop<A, OP>(acc, v[k]);
    acc = sblock8<A, OP>(acc, ws);
    if (threadIdx.x == 0) out[big[g]] = acc;
}

// one CTA per 4096-element chunk of the long segments, each from its
// descriptor (one 16-byte load; finding the chunk by a binary search over the
// segments instead put seven dependent loads before its first row)
template <typename T, typename A, int OP, bool GATHER>
__global__ void __launch_bounds__(256, 4) k_seg_chunk(const __grid_constant__ SegIO<T, A> io,
                                                      const long long* __restrict__ rows, long long nx, const ChunkDesc* __restrict__ order, A ident,
                                                      A* __restrict__ part, unsigned* derr) {
    grid_entry();
    const T* __restrict__ src = io.src[blockIdx.y];
    part += (size_t)blockIdx.y * gridDim.x;
    __shared__ A ws[256];
    const ChunkDesc d = order[blockIdx.x];
    const long long base = d.first, e = d.first + d.len;
    bool bad = false;
    T v[16];
    seg_load16<T, GATHER>(src, rows, nx, base + threadIdx.x, e, v, bad);
    A acc = ident;
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (base + k * 256 + threadIdx.x < e) acc = sop<A, OP>(acc, (A)v[k]);
    acc = sblock8<A, OP>(acc, ws);
    if (threadIdx.x == 0) part[d.chunk] = acc;
    if (bad) flag_error(derr, DERR_INDEX);
}

// The long segments of a list from the ids of their class: big[k], the first
// chunk of each (c0, and as i64 in ps), in one block (a list of 2^31 rows has
// fewer than 2^19 of them).
__global__ void __launch_bounds__(1024) k_big_plan(const long long* __restrict__ starts, long long ng, long long total,
                                                   const unsigned* __restrict__ ids, long long nbig,
                                                   long long* __restrict__ big, unsigned long long* __restrict__ c0,
                                                   long long* __restrict__ ps) {
    grid_entry();
    __shared__ unsigned long long wsum[32];
    __shared__ unsigned long long carry;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (long long b = 0; b < nbig; b += 1024) {
        const long long k = b + threadIdx.x;
        long long g = 0;
        unsigned long long n = 0;
        if (k < nbig) {
            g = ids[k];
            const long long m = ((g + 1 < ng) ? starts[g + 1] : total) - starts[g];
            n = (unsigned long long)((m + TILE_SUM - 1) / TILE_SUM);
        }
        const unsigned long long incl = warp_incl_scan64(n);
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const unsigned long long x = wsum[lane];
            wsum[lane] = warp_incl_scan64(x) - x;
        }
        __syncthreads();
        const unsigned long long first = carry + wsum[warp] + incl - n;
        if (k < nbig) {
            big[k] = g;
            c0[k] = first;
            ps[k] = (long long)first;
        }
        __syncthreads();
        if (threadIdx.x == 1023) carry = first + n;
        __syncthreads();
    }
}
// The descriptors of a general list's chunks, one thread each, and for a
// gather the order in which they run: by the region of the source column that
// their middle row lies in (nx >> shift < CHUNK_BUCKETS regions), so that the
// CTAs resident together gather from one region in every segment and a sector
// fetched for one is still in L2 for the others.  A counting sort: the
// descriptors and the regions' counts, the regions' first places, the
// descriptors placed.  Only the schedule depends on the order, so chunks of
// one region may come in any order, and a row outside the column only puts
// its chunk into the first or last region.  (150M Zipf rows, 25K chunks of
// 1640 segments: ranking every chunk against every segment took 0.12 ms.)
// Without `region` the descriptors stay in segment order.
constexpr int CHUNK_BUCKETS = 4096;
__global__ void k_chunk_desc(const long long* __restrict__ rows, const long long* __restrict__ starts, long long ng,
                             long long total, const long long* __restrict__ big,
                             const unsigned long long* __restrict__ c0, long long nbig, long long nchunks, int shift,
                             ChunkDesc* __restrict__ desc, unsigned short* __restrict__ region,
                             unsigned* __restrict__ hist) {
    grid_entry();
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nchunks) return;
    long long lo = 0, hi = nbig - 1;  // the long segment owning chunk t
    while (lo < hi) {
        const long long mid = (lo + hi + 1) >> 1;
        if ((long long)c0[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const long long g = big[lo], s = starts[g], e = (g + 1 < ng) ? starts[g + 1] : total;
    const long long first = s + (t - (long long)c0[lo]) * TILE_SUM;
    const long long len = e - first < TILE_SUM ? e - first : TILE_SUM;
    desc[t] = ChunkDesc{first, (unsigned)len, (unsigned)t};
    if (region) {
        const long long r = rows[first + len / 2] >> shift;
        const unsigned b = r < 0 ? 0u : (r >= CHUNK_BUCKETS ? CHUNK_BUCKETS - 1u : (unsigned)r);
        region[t] = (unsigned short)b;
        atomicAdd(&hist[b], 1u);
    }
}
__global__ void __launch_bounds__(1024) k_chunk_regions(unsigned* __restrict__ hist) {
    grid_entry();
    __shared__ unsigned wsum[32];
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    uint4* h4 = reinterpret_cast<uint4*>(hist);  // CHUNK_BUCKETS = 4 per thread
    const uint4 v = h4[threadIdx.x];
    const unsigned n = v.x + v.y + v.z + v.w, incl = warp_incl_scan(n);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const unsigned x = wsum[lane];
        wsum[lane] = warp_incl_scan(x) - x;
    }
    __syncthreads();
    const unsigned o = wsum[warp] + incl - n;
    h4[threadIdx.x] = make_uint4(o, o + v.x, o + v.x + v.y, o + v.x + v.y + v.z);
}
__global__ void k_chunk_place(const ChunkDesc* __restrict__ desc, const unsigned short* __restrict__ region,
                              long long nchunks, unsigned* __restrict__ next, ChunkDesc* __restrict__ order) {
    grid_entry();
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t < nchunks) order[atomicAdd(&next[region[t]], 1u)] = desc[t];
}
template <typename A>
__global__ void k_scatter_big(const A* __restrict__ r, const long long* __restrict__ big, long long nbig, A* __restrict__ out) {
    grid_entry();
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nbig; k += (long long)gridDim.x * blockDim.x)
        out[big[k]] = r[k];
}
// The chunk order of a list that @group plans itself (at most
// CHUNK_ORDER_SMALL_SEGS long segments, all in shared memory): a segment's
// rows are spread over the whole source column, so running one segment's
// chunks after another's would sweep the column once per segment.  Instead
// chunk (k, c) of long segment k (n_k chunks) runs at the rank of its relative
// position (2c + 1) / (2 n_k), ties to the lower k.  Only the schedule
// changes; each chunk's partial lands at its own index as before.
constexpr long long CHUNK_ORDER_SMALL_SEGS = 64;
// below this many elements the values of a list fit in L2 whatever the
// order, and the general plan builds none (it costs three launches)
constexpr long long CHUNK_ORDER_MIN_TOTAL = 4ll << 20;
// order[rank of chunk t] = chunk t's descriptor, for chunk t of nchunks (c0:
// the long segments' first chunks; seg_first/seg_end(k): long segment k's
// element range)
template <typename SegRange>
__device__ __forceinline__ void chunk_rank(const unsigned long long* c0, long long nbig, unsigned long long nchunks,
                                           long long t, ChunkDesc* __restrict__ order, SegRange range) {
    long long lo = 0, hi = nbig - 1;  // the long segment owning chunk t
    while (lo < hi) {
        long long mid = (lo + hi + 1) >> 1;
        if ((long long)c0[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const long long k = lo, c = t - (long long)c0[k];
    const long long nk = (long long)((k + 1 < nbig ? c0[k + 1] : nchunks) - c0[k]);
    long long rank = c;
    for (long long k2 = 0; k2 < nbig; k2++) {
        if (k2 == k) continue;
        const long long n2 = (long long)((k2 + 1 < nbig ? c0[k2 + 1] : nchunks) - c0[k2]);
        // chunks c2 of segment k2 placed before (k, c): (2 c2 + 1) n_k < (2c + 1) n2, or equal and k2 < k
        const long long x = (2 * c + 1) * n2 + (k2 < k ? 1 : 0);
        const long long q = x <= 0xffffffffll ? (long long)((unsigned)(x - 1) / (unsigned)nk) : (x - 1) / nk;
        const long long cnt = (q + 1) / 2;
        rank += cnt < n2 ? cnt : n2;
    }
    long long sf, se;
    range(k, sf, se);
    const long long first = sf + c * TILE_SUM;
    const long long len = se - first < TILE_SUM ? se - first : TILE_SUM;
    order[rank] = ChunkDesc{first, (unsigned)len, (unsigned)t};
}
// The whole plan of a list of at most SEG_PLAN_SMALL segments in one CTA of
// 1024 threads (four consecutive segments each): the class counts and ids
// of seg_classes, then the long segments in ascending order with their
// first chunks (an exclusive scan over the threads) and the chunk order.
// hdr = {the 8 class counts, nbig, nchunks}.
__global__ void __launch_bounds__(1024) k_seg_plan_small(const long long* __restrict__ starts, long long ng,
                                                         long long total, unsigned* __restrict__ cc,
                                                         unsigned* __restrict__ ids, long long* __restrict__ big,
                                                         unsigned long long* __restrict__ c0, long long* __restrict__ ps,
                                                         ChunkDesc* __restrict__ order, unsigned long long* __restrict__ hdr) {
    grid_entry();
    __shared__ unsigned sc[SEG_CLASSES], soff[SEG_CLASSES], scur[SEG_CLASSES];
    __shared__ unsigned wb[32];
    __shared__ unsigned long long wc[32];
    __shared__ unsigned long long s_nbig, s_nch;
    __shared__ unsigned long long sc0[CHUNK_ORDER_SMALL_SEGS];
    __shared__ long long sfirst[CHUNK_ORDER_SMALL_SEGS], send[CHUNK_ORDER_SMALL_SEGS];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t < SEG_CLASSES) { sc[t] = 0; scur[t] = 0; }
    __syncthreads();
    int cls[4];
    long long len[4];
    unsigned nb = 0;
    unsigned long long nc = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const long long g = (long long)t * 4 + k;
        cls[k] = -1;
        len[k] = 0;
        if (g < ng) {
            len[k] = ((g + 1 < ng) ? starts[g + 1] : total) - starts[g];
            cls[k] = seg_class(len[k]);
            atomicAdd(&sc[cls[k]], 1u);
            if (len[k] > TILE_SUM) { nb++; nc += (unsigned long long)((len[k] + TILE_SUM - 1) / TILE_SUM); }
        }
    }
    // exclusive scan of (nb, nc) over the threads
    unsigned ib = nb;
    unsigned long long ic = nc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned ob = __shfl_up_sync(0xffffffffu, ib, d);
        const unsigned long long oc = __shfl_up_sync(0xffffffffu, ic, d);
        if (lane >= d) { ib += ob; ic += oc; }
    }
    if (lane == 31) { wb[w] = ib; wc[w] = ic; }
    __syncthreads();
    if (t == 0) {
        unsigned ab = 0;
        unsigned long long ac = 0;
        for (int k = 0; k < 32; k++) {
            const unsigned b = wb[k];
            const unsigned long long c = wc[k];
            wb[k] = ab; wc[k] = ac;
            ab += b; ac += c;
        }
        s_nbig = ab;
        s_nch = ac;
        unsigned off = 0;
        for (int c = 0; c < SEG_CLASSES; c++) {
            soff[c] = off;
            off += sc[c];
            cc[c] = sc[c];
            cc[SEG_CLASSES + c] = sc[c];
            hdr[c] = sc[c];
        }
    }
    __syncthreads();
    unsigned pb = wb[w] + ib - nb;
    unsigned long long pc = wc[w] + ic - nc;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (cls[k] < 0) continue;
        const long long g = (long long)t * 4 + k;
        ids[soff[cls[k]] + atomicAdd(&scur[cls[k]], 1u)] = (unsigned)g;
        if (len[k] > TILE_SUM) {
            big[pb] = g;
            c0[pb] = pc;
            ps[pb] = (long long)pc;
            if (pb < CHUNK_ORDER_SMALL_SEGS) {
                sc0[pb] = pc;
                sfirst[pb] = starts[g];
                send[pb] = starts[g] + len[k];
            }
            pb++;
            pc += (unsigned long long)((len[k] + TILE_SUM - 1) / TILE_SUM);
        }
    }
    __syncthreads();
    const long long nbig = (long long)s_nbig;
    const unsigned long long nchunks = s_nch;
    if (t == 0) { hdr[SEG_CLASSES] = nbig; hdr[SEG_CLASSES + 1] = nchunks; }
    auto range = [&](long long k, long long& f, long long& e) {
        f = sfirst[k];
        e = send[k];
    };
    if (nbig <= CHUNK_ORDER_SMALL_SEGS)  // the long segments from shared memory
        for (long long q = t; q < (long long)nchunks; q += 1024) chunk_rank(sc0, nbig, nchunks, q, order, range);
}

static unsigned gcap(long long n, int per = 256) {
    unsigned g = grid_for(n, per);
    return g > (unsigned)g_sms * 32 ? (unsigned)g_sms * 32 : g;
}

// Segment ids by size class and the split of the segments longer than one
// tile into chunks, kept with the list: the class counts and the number of
// chunks come back in one round trip (empty classes then launch nothing),
// the rest is queued.  `rows` (the row ids behind a gather, or null) gives the
// chunks their launch order.
static I seg_plan(const long long* starts, long long ng, long long total, const long long* rows, long long nx,
                  ListInfo* li) {
    auto alloc = [li](size_t bytes) { return li->scratch ? salloc(bytes) : dalloc(bytes); };
    if (!li->cls_ids) {
        unsigned* cc = (unsigned*)alloc(2 * SEG_CLASSES * 4 + 8);
        unsigned* id = (unsigned*)alloc((size_t)ng * 4);
        if (!cc || !id) return E_DEVICE_OOM;
        unsigned long long* nch = (unsigned long long*)(cc + 2 * SEG_CLASSES);
        HG_CU(cudaMemsetAsync(cc, 0, 2 * SEG_CLASSES * 4 + 8, g_stream));
        const unsigned gb = (unsigned)((ng + 255) / 256);
        HG_LAUNCH("seg_class", gb, 256, 0, k_seg_class_count, starts, ng, total, cc, nch);
        HG_LAUNCH("seg_class_ids", gb, 256, 0, k_seg_class_ids, starts, ng, total, (const unsigned*)cc,
                  cc + SEG_CLASSES, id);
        HG_CHECK(last_launch_error());
        unsigned long long hn = 0;
        HG_CHECK(rb_queue(li->cls_host, cc, sizeof(li->cls_host)));
        HG_CHECK(rb_queue(&hn, nch, 8));
        HG_CU(stream_sync());
        li->cls_ids = id;
        li->cls_cnt = cc;
        li->cls_known = 1;
        if (!li->planned) {
            li->nbig = li->cls_host[7];
            li->nchunks = hn;
        }
    }
    if (li->planned) return 0;
    const long long nbig = li->nbig;
    if (nbig > 0) {
        long long* big = (long long*)alloc((size_t)nbig * 8);
        unsigned long long* c0 = (unsigned long long*)alloc((size_t)nbig * 8);
        long long* ps = (long long*)alloc((size_t)nbig * 8);
        if (!big || !c0 || !ps) return E_DEVICE_OOM;
        unsigned before = 0;  // ids of the classes below
        for (int c = 0; c < 7; c++) before += li->cls_host[c];
        HG_LAUNCH("big_plan", 1, 1024, 0, k_big_plan, starts, ng, total, li->cls_ids + before, nbig, big, c0, ps);
        const long long nchunks = (long long)li->nchunks;
        const unsigned cb = grid_for(nchunks, 256);
        ChunkDesc* order = (ChunkDesc*)alloc((size_t)nchunks * sizeof(ChunkDesc));
        if (!order) return E_DEVICE_OOM;
        if (rows && nbig > 1 && total >= CHUNK_ORDER_MIN_TOTAL) {
            ChunkDesc* desc = (ChunkDesc*)salloc((size_t)nchunks * sizeof(ChunkDesc));
            unsigned short* region = (unsigned short*)salloc((size_t)nchunks * 2);
            unsigned* hist = (unsigned*)salloc(CHUNK_BUCKETS * 4);
            if (!desc || !region || !hist) return E_DEVICE_OOM;
            int shift = 0;
            while ((nx >> shift) >= CHUNK_BUCKETS) shift++;
            HG_CU(cudaMemsetAsync(hist, 0, CHUNK_BUCKETS * 4, g_stream));
            HG_LAUNCH("chunk_desc", cb, 256, 0, k_chunk_desc, rows, starts, ng, total, big, c0, nbig, nchunks, shift,
                      desc, region, hist);
            HG_LAUNCH("chunk_regions", 1, 1024, 0, k_chunk_regions, hist);
            HG_LAUNCH("chunk_place", cb, 256, 0, k_chunk_place, desc, region, nchunks, hist, order);
        } else {
            HG_LAUNCH("chunk_desc", cb, 256, 0, k_chunk_desc, (const long long*)nullptr, starts, ng, total, big, c0,
                      nbig, nchunks, 0, order, (unsigned short*)nullptr, (unsigned*)nullptr);
        }
        li->corder = order;
        li->big = big;
        li->chunk0 = c0;
        li->pstarts = ps;
    }
    li->planned = 1;
    return last_launch_error();
}

I seg_plan_small(const long long* starts, long long ng, long long total, SmallPlan* p) {
    *p = SmallPlan{};
    if (ng <= 0 || ng > SEG_PLAN_SMALL) return 0;
    const size_t maxch = (size_t)(total / TILE_SUM) + (size_t)ng + 1;
    p->cc = (unsigned*)dalloc(2 * SEG_CLASSES * 4);
    p->ids = (unsigned*)dalloc((size_t)ng * 4);
    p->big = (long long*)dalloc((size_t)ng * 8);
    p->c0 = (unsigned long long*)dalloc((size_t)ng * 8);
    p->ps = (long long*)dalloc((size_t)ng * 8);
    p->order = (ChunkDesc*)dalloc(maxch * sizeof(ChunkDesc));
    unsigned long long* hd = (unsigned long long*)salloc(16 * 8);
    p->hdr = (unsigned long long*)halloc(16 * 8);
    if (p->hdr) memset(p->hdr, 0, 16 * 8);
    if (!p->cc || !p->ids || !p->big || !p->c0 || !p->ps || !p->order || !hd || !p->hdr) {
        *p = SmallPlan{};
        return E_DEVICE_OOM;
    }
    HG_LAUNCH("seg_plan_small", 1, 1024, 0, k_seg_plan_small, starts, ng, total, p->cc, p->ids, p->big, p->c0, p->ps,
              p->order, hd);
    p->hdr_dev = hd;
    return last_launch_error();
}

void seg_plan_adopt(ListInfo& li, const SmallPlan& p) {
    if (!p.hdr) return;
    li.cls_ids = p.ids;
    li.cls_cnt = p.cc;
    for (int c = 0; c < SEG_CLASSES; c++) li.cls_host[c] = (unsigned)p.hdr[c];
    li.cls_known = 1;
    li.nbig = (long long)p.hdr[SEG_CLASSES];
    li.nchunks = p.hdr[SEG_CLASSES + 1];
    li.big = p.big;
    li.chunk0 = p.c0;
    li.pstarts = p.ps;
    li.corder = p.order;
    li.planned = li.nbig <= CHUNK_ORDER_SMALL_SEGS;  // else its first aggregation orders the chunks
}

// ---- several f64 sums over the long segments of one grouping at once.
// One CTA per 4096-element chunk, as k_seg_chunk, but the chunk's row ids
// are read once and each of the ncol columns is gathered through them (all
// 16 x ncol gathers of a lane issued before the first add); each column's
// chunk partial follows the tile tree, so part[col * nchunks + c] is
// bit-identical to k_seg_chunk's for that column.
struct SegCols { const double* src[SEG_MANY]; };
template <int NCOL>
__global__ void __launch_bounds__(256, 4) k_seg_chunk_many(const __grid_constant__ SegCols cols,
                                                           const long long* __restrict__ rows, long long nx,
                                                           unsigned long long nchunks,
                                                           const ChunkDesc* __restrict__ order,
                                                           double* __restrict__ part, unsigned* derr) {
    grid_entry();
    __shared__ double ws[NCOL][256];
    const ChunkDesc d = order[blockIdx.x];
    const long long first = d.first + threadIdx.x, e = d.first + d.len;
    long long r[16];
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const long long j = first + (long long)k * 256;
        r[k] = j < e ? rows[j] : -1;
        bad |= j < e && (r[k] < 0 || r[k] >= nx);
    }
#pragma unroll 1
    for (int q = 0; q < NCOL; q++) {  // one column at a time: 16 gathers in flight, few registers
        double v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = (r[k] >= 0 && r[k] < nx) ? cols.src[q][r[k]] : 0.0;
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (first + (long long)k * 256 < e) acc = __dadd_rn(acc, v[k]);
        ws[q][threadIdx.x] = acc;
    }
    __syncthreads();
    const unsigned q = threadIdx.x >> 5;
    if (q < (unsigned)NCOL) {  // warp q folds column q
        double x[8];
#pragma unroll
        for (int v = 0; v < 8; v++) x[v] = ws[q][v * 32 + lane_id()];
        const double r = stile8<double, OP_SUM>(x);
        if (lane_id() == 0) part[(unsigned long long)q * nchunks + d.chunk] = r;
    }
    if (bad) flag_error(derr, DERR_INDEX);
}

// part[q * nchunks + c] = column q's partial of chunk c
static I seg_chunk_many(const SegCols& sc, int ncol, const long long* rows, long long nx, const ListInfo* li,
                        double* part) {
#define SEG_MANY_LAUNCH(NC)                                                                                      \
    HG_LAUNCH("seg_chunk_many", (unsigned)li->nchunks, 256, 0, k_seg_chunk_many<NC>, sc, rows, nx, li->nchunks, \
              li->corder, part, g_derr)
    if (ncol == 2) SEG_MANY_LAUNCH(2);
    else if (ncol == 3) SEG_MANY_LAUNCH(3);
    else SEG_MANY_LAUNCH(4);
#undef SEG_MANY_LAUNCH
    return last_launch_error();
}

// Reduces every segment of each of the ncol columns (io.src via rows | io.src)
// into io.out[.][ng] (device), each class of segments in one launch for all
// columns.  The plan is kept with `li` when there is one, else it serves this
// call alone.
template <typename T, typename A, int OP, bool GATHER>
static I seg_reduce(const SegIO<T, A>& io, int ncol, const long long* rows, long long nx, const long long* starts,
                    long long ng, long long total, A ident, ListInfo* li = nullptr) {
    if (ng == 0) return 0;
    ListInfo local{};
    local.scratch = 1;
    if (!li) li = &local;
    HG_CHECK(seg_plan(starts, ng, total, GATHER ? rows : nullptr, nx, li));
    const unsigned *ids = li->cls_ids, *ccnt = li->cls_cnt;
    // One warp per 32 / seg_lanes(c) small segments of class c and per mid-size one.
    // The kernels stride over the segments, so the grid decides only how many
    // run at once: with one thread per segment (8 warps per 256 segments) 64
    // plans' ~200 mid-size segments ran on 16 warps, 0.34 ms a launch against
    // 0.02 ms now.
    long long small_w = 0;
    for (int c = 0; c < 6; c++) {
        const unsigned per = 32u / seg_lanes(c);
        small_w += (li->cls_host[c] + per - 1) / per;
    }
    const long long mid_w = li->cls_host[6];
    const unsigned nc = (unsigned)ncol;
    if (small_w)
        HG_LAUNCH("seg_warps", dim3(gcap(small_w * 32), nc), 256, 0, (k_seg_warps<T, A, OP, GATHER>), io, rows, nx,
                  starts, ng, total, ids, ccnt, ident, g_derr);
    if (mid_w) {
        const unsigned g = gcap(mid_w * 32);
        const long long rest = total - (long long)(li->nchunks - li->nbig) * TILE_SUM;  // no fewer than class 6 holds
        const bool walk = mid_w > (long long)g * 8 && rest > 512 * mid_w;
        auto launch = [&](const char* name, auto kern) {
            HG_LAUNCH(name, dim3(g, nc), 256, 0, kern, io, rows, nx, starts, ng, total, ids, ccnt, ident, g_derr);
        };
        launch("seg_mid", walk ? k_seg_mid<T, A, OP, GATHER, true> : k_seg_mid<T, A, OP, GATHER, false>);
        if (walk) launch("seg_walk", k_seg_walk<T, A, OP, GATHER>);
    }
    const long long nbig = li->nbig;
    const unsigned long long nchunks = li->nchunks;
    if (nbig == 0) return last_launch_error();
    A* part = (A*)salloc((size_t)nchunks * sizeof(A) * nc);
    if (!part) return E_DEVICE_OOM;
    bool done = false;
    if constexpr (GATHER && std::is_same<T, double>::value && OP == OP_SUM) {
        if (ncol > 1) {  // the columns share one read of the row ids
            SegCols sc{};
            for (int q = 0; q < ncol; q++) sc.src[q] = io.src[q];
            HG_CHECK(seg_chunk_many(sc, ncol, rows, nx, li, part));
            done = true;
        }
    }
    if (!done)
        HG_LAUNCH("seg_chunk", dim3((unsigned)nchunks, nc), 256, 0, (k_seg_chunk<T, A, OP, GATHER>), io, rows, nx,
                  li->corder, ident, part, g_derr);
    // partials of each long segment are reduced by the same procedure: at
    // most 4096 of them per segment (certain when there are at most 4096 in
    // all) in one launch straight into out, else as segments of their own
    SegIO<A, A> pio{};
    if (nchunks <= (unsigned long long)TILE_SUM) {
        for (int q = 0; q < ncol; q++) pio.out[q] = io.out[q];
        HG_LAUNCH("seg_partials", dim3((unsigned)nbig, nc), 256, 0, (k_seg_partials<A, OP>), part, li->pstarts,
                  li->big, nbig, (long long)nchunks, ident, pio);
        return last_launch_error();
    }
    for (int q = 0; q < ncol; q++) {
        pio.src[q] = part + (size_t)q * nchunks;
        pio.out[q] = (A*)salloc((size_t)nbig * sizeof(A));
        if (!pio.out[q]) return E_DEVICE_OOM;
    }
    HG_CHECK((seg_reduce<A, A, OP, false>(pio, ncol, nullptr, 0, li->pstarts, nbig, (long long)nchunks, ident)));
    for (int q = 0; q < ncol; q++)
        HG_LAUNCH("scatter_big", gcap(nbig), 256, 0, k_scatter_big<A>, (const A*)pio.out[q], li->big, nbig, io.out[q]);
    return last_launch_error();
}

// f64 sums of ncol columns, at most SEG_MANY, over the segments of one
// grouping; sums[q] receives column q's ng sums.
template <bool GATHER>
static I seg_sum_cols(const double* const* srcs, int ncol, const long long* rows, long long nx, const long long* starts,
                      long long ng, long long total, double* const* sums, ListInfo* li) {
    SegIO<double, double> io{};
    for (int q = 0; q < ncol; q++) {
        io.src[q] = srcs[q];
        io.out[q] = sums[q];
    }
    return seg_reduce<double, double, OP_SUM, GATHER>(io, ncol, rows, nx, starts, ng, total, 0.0, li);
}

// f64 sums of several columns over segments gathered through row ids (the
// batched plans): the same kernels and order as hgpuGroupSum.
I seg_sum_f64(const double* const* srcs, int ncol, const long long* rows, long long nx, const long long* starts,
              long long ng, long long total, double* const* sums) {
    return seg_sum_cols<true>(srcs, ncol, rows, nx, starts, ng, total, sums, nullptr);
}

// ... over contiguous segments (no row indirection), same order
I seg_sum_f64_direct(const double* const* srcs, int ncol, const long long* starts, long long ng, long long total,
                     double* const* sums) {
    return seg_sum_cols<false>(srcs, ncol, nullptr, 0, starts, ng, total, sums, nullptr);
}

// ---------------------------------------------------------- finishing steps
template <typename A>
__global__ void k_avg_seg(const A* __restrict__ s, const long long* __restrict__ starts, long long ng, long long total,
                          void* __restrict__ out) {
    grid_entry();
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x) {
        long long m = ((g + 1 < ng) ? starts[g + 1] : total) - starts[g];
        if constexpr (std::is_same<A, long long>::value) ((double*)out)[g] = __ddiv_rn((double)s[g] * 1.0, (double)m);
        else if constexpr (std::is_same<A, float>::value) ((float*)out)[g] = __fdiv_rn(s[g], (float)m);
        else ((double*)out)[g] = __ddiv_rn(s[g], (double)m);
    }
}
__global__ void k_len_seg(const long long* __restrict__ starts, long long ng, long long total, long long* __restrict__ out) {
    grid_entry();
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x)
        out[g] = ((g + 1 < ng) ? starts[g + 1] : total) - starts[g];
}
// empty groups in min/max: the pfnReduce sentinel (ints become i64)
template <typename T>
__global__ void k_minmax_fix(const T* __restrict__ r, const long long* __restrict__ starts, long long ng, long long total,
                             int op, int to_long, void* __restrict__ out) {
    grid_entry();
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x) {
        long long m = ((g + 1 < ng) ? starts[g + 1] : total) - starts[g];
        if (to_long) ((long long*)out)[g] = m ? (long long)r[g] : (op == AG_MIN ? LLONG_MAX : LLONG_MIN);
        else if constexpr (std::is_same<T, float>::value) ((float*)out)[g] = m ? r[g] : (op == AG_MIN ? 3.402823466e+38f : 1.175494351e-38f);
        else if constexpr (std::is_same<T, double>::value) ((double*)out)[g] = m ? r[g] : (op == AG_MIN ? 1.7976931348623157e308 : 2.2250738585072014e-308);
        else ((T*)out)[g] = r[g];
    }
}
__global__ void k_any_empty(const long long* __restrict__ starts, long long ng, long long total, unsigned* flag) {
    grid_entry();
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x)
        if (((g + 1 < ng) ? starts[g + 1] : total) == starts[g]) atomicOr(flag, 1u);
}

// Aggregates segments of x: result vector (device) of ng values, type in *typ.
template <typename T, bool GATHER>
static I agg_typed(int ag, I xt, const T* src, const long long* rows, long long nx, const long long* starts, long long ng,
                   long long total, void** out, I* typ, ListInfo* li) {
    constexpr bool isF = std::is_same<T, float>::value, isE = std::is_same<T, double>::value;
    using SA = typename std::conditional<isF, float, typename std::conditional<isE, double, long long>::type>::type;
    if (ag == AG_LEN) {
        *typ = H_L;
        if (!*out) *out = salloc((size_t)(ng > 0 ? ng : 1) * 8);
        if (!*out) return E_DEVICE_OOM;
        if (ng > 0) HG_LAUNCH("len_seg", gcap(ng), 256, 0, k_len_seg, starts, ng, total, (long long*)*out);
        return last_launch_error();
    }
    if (ag == AG_SUM || ag == AG_AVG) {
        SA* s = (SA*)(ag == AG_SUM && *out ? *out : salloc((size_t)(ng > 0 ? ng : 1) * sizeof(SA)));
        if (!s) return E_DEVICE_OOM;
        SegIO<T, SA> io{};
        io.src[0] = src;
        io.out[0] = s;
        HG_CHECK((seg_reduce<T, SA, OP_SUM, GATHER>(io, 1, rows, nx, starts, ng, total, (SA)0, li)));
        if (ag == AG_SUM) {
            *typ = isF ? H_F : (isE ? H_E : H_L);
            *out = s;
            return 0;
        }
        *typ = isF ? H_F : H_E;
        if (!*out) *out = salloc((size_t)(ng > 0 ? ng : 1) * 8);
        if (!*out) return E_DEVICE_OOM;
        if (ng > 0) HG_LAUNCH("avg_seg", gcap(ng), 256, 0, k_avg_seg<SA>, s, starts, ng, total, *out);
        return last_launch_error();
    }
    // min / max
    T* r = (T*)salloc((size_t)(ng > 0 ? ng : 1) * sizeof(T));
    if (!r) return E_DEVICE_OOM;
    T identity;
    if (ag == AG_MIN) identity = std::numeric_limits<T>::has_infinity ? std::numeric_limits<T>::infinity() : std::numeric_limits<T>::max();
    else identity = std::numeric_limits<T>::has_infinity ? -std::numeric_limits<T>::infinity() : std::numeric_limits<T>::lowest();
    SegIO<T, T> io{};
    io.src[0] = src;
    io.out[0] = r;
    if (ag == AG_MIN) HG_CHECK((seg_reduce<T, T, OP_MIN, GATHER>(io, 1, rows, nx, starts, ng, total, identity, li)));
    else HG_CHECK((seg_reduce<T, T, OP_MAX, GATHER>(io, 1, rows, nx, starts, ng, total, identity, li)));
    unsigned h = 0;
    if (!(li && li->group_rows)) {  // @group never yields an empty group
        unsigned* fl = (unsigned*)salloc(16);
        if (!fl) return E_DEVICE_OOM;
        HG_CU(cudaMemsetAsync(fl, 0, 4, g_stream));
        if (ng > 0) HG_LAUNCH("any_empty", gcap(ng), 256, 0, k_any_empty, starts, ng, total, fl);
        HG_CHECK(rb_queue(&h, fl, 4));
        HG_CU(stream_sync());
    }
    bool to_long = h && is_int(xt);
    *typ = to_long ? H_L : xt;
    *out = salloc((size_t)(ng > 0 ? ng : 1) * (to_long ? 8 : sizeof(T)));
    if (!*out) return E_DEVICE_OOM;
    if (ng > 0) HG_LAUNCH("minmax_fix", gcap(ng), 256, 0, k_minmax_fix<T>, r, starts, ng, total, ag, to_long ? 1 : 0, *out);
    return last_launch_error();
}

template <bool GATHER>
static I agg_dispatch(int ag, I xt, const void* src, const long long* rows, long long nx, const long long* starts,
                      long long ng, long long total, void** out, I* typ, ListInfo* li) {
    switch (xt) {
    case H_B: return agg_typed<bool, GATHER>(ag, xt, (const bool*)src, rows, nx, starts, ng, total, out, typ, li);
    case H_J: return agg_typed<int8_t, GATHER>(ag, xt, (const int8_t*)src, rows, nx, starts, ng, total, out, typ, li);
    case H_H: return agg_typed<int16_t, GATHER>(ag, xt, (const int16_t*)src, rows, nx, starts, ng, total, out, typ, li);
    case H_I: return agg_typed<int32_t, GATHER>(ag, xt, (const int32_t*)src, rows, nx, starts, ng, total, out, typ, li);
    case H_L: return agg_typed<long long, GATHER>(ag, xt, (const long long*)src, rows, nx, starts, ng, total, out, typ, li);
    case H_F: return agg_typed<float, GATHER>(ag, xt, (const float*)src, rows, nx, starts, ng, total, out, typ, li);
    case H_E: return agg_typed<double, GATHER>(ag, xt, (const double*)src, rows, nx, starts, ng, total, out, typ, li);
    default: return E_DOMAIN;
    }
}

// ------------------------------------------------ lists -> contiguous segments
__global__ void k_node_lens(const V0* __restrict__ nodes, long long ng, unsigned* __restrict__ lens) {
    grid_entry();
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x)
        lens[g] = (unsigned)nodes[g].len;
}
// copies each element's payload to data + off[g] * es, one warp per element
// and one item per lane; `nodes` is a device copy of the host node array at
// host_base, so an inline element (its g points into its own host node)
// reads its item from the copy
template <typename T>
__global__ void k_node_copy(const V0* __restrict__ nodes, long long ng, unsigned long long host_base,
                            const unsigned long long* __restrict__ off, T* __restrict__ data) {
    grid_entry();
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ng; g += warps) {
        const V0 v = nodes[g];
        const unsigned long long own = host_base + (unsigned long long)g * sizeof(V0) + offsetof(V0, b);
        const T* src = ((unsigned long long)v.g == own) ? reinterpret_cast<const T*>(&nodes[g].b) : (const T*)v.g;
        for (long long b = lane_id(); b < v.len; b += 32) data[off[g] + b] = src[b];
    }
}
__global__ void k_offsets_i64(const unsigned long long* __restrict__ a, long long n, long long* __restrict__ b) {
    grid_entry();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        b[i] = (long long)a[i];
}

// Segments of a list whose elements all have type `typ`.  Lists built by this
// library are found in the registry; any other list is read through a device
// copy of its nodes.  Payloads must be device-readable.
static I list_segments(V y, I typ, const long long** starts, long long* total, const void** data,
                       ListInfo** info = nullptr) {
    long long ng = y->len;
    ListInfo* li = find_list(host_nodes(y), ng);
    if (info) *info = nullptr;
    if (li && li->kind == LIST_SEGMENTS && li->typ == typ) {
        *starts = li->starts;
        *total = li->total;
        *data = li->data;
        if (info) *info = li;
        return 0;
    }
    const V0* nodes = host_nodes(y);
    int es = esize(typ);
    for (long long g = 0; g < ng; g++) {
        if (nodes[g].typ != typ) return set_error(E_TYPE, "list element %lld has type %d, expected %d", g, nodes[g].typ, typ);
        const bool inl = nodes[g].g == (G)&nodes[g].b;
        if (nodes[g].len > 0 && !inl && !is_device_ptr(nodes[g].g))
            return set_error(E_NOT_IMPL, "list element %lld lives in pageable host memory; stage it with hgpuToDevice", g);
        if (inl && nodes[g].len > 1) return set_error(E_DOMAIN, "list element %lld: inline node with %lld items", g, nodes[g].len);
    }
    // the kernels read a device copy of the node array (one bulk copy, not
    // one host access per node)
    const unsigned long long host_base = (unsigned long long)(uintptr_t)nodes;
    V0* dn = (V0*)salloc((size_t)(ng > 0 ? ng : 1) * sizeof(V0));
    if (!dn) return E_DEVICE_OOM;
    if (ng > 0) HG_CU(cudaMemcpyAsync(dn, nodes, (size_t)ng * sizeof(V0), cudaMemcpyDefault, g_stream));
    if (!is_device_ptr(nodes)) HG_CU(stream_sync());  // pageable source: finish before returning
    nodes = dn;
    unsigned* lens = (unsigned*)salloc((size_t)(ng > 0 ? ng : 1) * 4);
    unsigned long long* off = (unsigned long long*)salloc((size_t)(ng > 0 ? ng : 1) * 8);
    long long* st = (long long*)salloc((size_t)(ng > 0 ? ng : 1) * 8);
    if (!lens || !off || !st) return E_DEVICE_OOM;
    unsigned long long tot = 0;
    if (ng > 0) {
        HG_LAUNCH("node_lens", gcap(ng), 256, 0, k_node_lens, nodes, ng, lens);
        HG_CHECK(scan_exclusive(lens, ng, off, &tot));
    }
    char* d = (char*)salloc((size_t)(tot > 0 ? tot : 1) * es);
    if (!d) return E_DEVICE_OOM;
    if (ng > 0) {
        const unsigned gr = gcap(ng * 32);
        switch (es) {
        case 1: HG_LAUNCH("node_copy", gr, 256, 0, k_node_copy<uint8_t>, nodes, ng, host_base, off, (uint8_t*)d); break;
        case 2: HG_LAUNCH("node_copy", gr, 256, 0, k_node_copy<uint16_t>, nodes, ng, host_base, off, (uint16_t*)d); break;
        case 4: HG_LAUNCH("node_copy", gr, 256, 0, k_node_copy<uint32_t>, nodes, ng, host_base, off, (uint32_t*)d); break;
        default: HG_LAUNCH("node_copy", gr, 256, 0, k_node_copy<unsigned long long>, nodes, ng, host_base, off,
                           (unsigned long long*)d); break;
        }
        HG_LAUNCH("offsets", gcap(ng), 256, 0, k_offsets_i64, off, ng, st);
    }
    *starts = st;
    *total = (long long)tot;
    *data = d;
    return last_launch_error();
}

// writes ng one-element nodes holding vals[g] (es bytes) into a device
// staging copy of the host node array at host_base (node g inline: its g
// points at its own host node)
__global__ void k_scalar_nodes(const char* __restrict__ vals, long long ng, int es, I typ, V0* __restrict__ out,
                               unsigned long long host_base) {
    grid_entry();
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x) {
        V0 v;
        v.len = 1;
        v.typ = typ;
        v.i64 = 0;
        for (int b = 0; b < es; b++) ((char*)&v.b)[b] = vals[g * es + b];
        v.g = (G)(host_base + (unsigned long long)g * sizeof(V0) + offsetof(V0, b));
        out[g] = v;
    }
}
// segment nodes over a contiguous payload (inline when one element)
__global__ void k_segment_nodes(const char* __restrict__ data, const long long* __restrict__ starts, long long ng,
                                long long total, int es, I typ, V0* __restrict__ out, unsigned long long host_base) {
    grid_entry();
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x) {
        long long s = starts[g], e = (g + 1 < ng) ? starts[g + 1] : total;
        V0 v;
        v.len = e - s;
        v.typ = typ;
        v.i64 = 0;
        if (e - s == 1) {
            for (int b = 0; b < es; b++) ((char*)&v.b)[b] = data[s * es + b];
            v.g = (G)(host_base + (unsigned long long)g * sizeof(V0) + offsetof(V0, b));
        } else {
            v.g = (G)(data + s * es);
        }
        out[g] = v;
    }
}

// An output's memory before its node is touched (which may be an input's), and
// the node once the output is computed: alloc_out in two steps.
static void* out_memory(I typ, L len) { return len > 1 ? dalloc((size_t)len * esize(typ)) : salloc(16); }
static void out_node(V z, I typ, L len, void* d) {
    z->typ = typ;
    z->len = len;
    z->g = len > 1 ? (G)d : (G)&z->b;
    if (len <= 1) z->i64 = 0;
}

static I group_agg(V z, V x, V y, int ag) {
    HG_CHECK(ensure_init());
    ScratchScope ss;
    if (y->typ != H_G) return E_DOMAIN;
    if (!is_real(x->typ)) return E_DOMAIN;
    const long long* starts;
    long long total;
    const void* rows;
    ListInfo* li;
    HG_CHECK(list_segments(y, H_L, &starts, &total, &rows, &li));
    const void* px;
    HG_CHECK(in_ptr(x, &px));
    // sums, averages and lengths, whose type is known before, are written where
    // they stay; min and max of integers widen when a group is empty
    void *res = nullptr, *dz = nullptr;
    I typ = ag == AG_LEN ? H_L : x->typ == H_F ? H_F : (x->typ == H_E || ag == AG_AVG) ? H_E : H_L;
    const L ng = y->len;
    if (ag != AG_MIN && ag != AG_MAX) {
        res = dz = out_memory(typ, ng);
        if (!dz) return E_DEVICE_OOM;
    }
    HG_CHECK(agg_dispatch<true>(ag, x->typ, px, (const long long*)rows, x->len, starts, y->len, total, &res, &typ, li));
    if (!(li && li->group_rows && x->len >= total)) HG_CHECK(check_device_errors());  // rows of @group are in range
    if (!dz) {
        dz = out_memory(typ, ng);
        if (!dz) return E_DEVICE_OOM;
        if (ng > 0) HG_CU(cudaMemcpyAsync(dz, res, (size_t)ng * esize(typ), cudaMemcpyDeviceToDevice, g_stream));
    }
    out_node(z, typ, ng, dz);
    return finish_out(z, dz);
}

}  // namespace hg

using namespace hg;

extern "C" {

I hgpuGroupSum(V z, V x, V y) { return group_agg(z, x, y, AG_SUM); }
I hgpuGroupAvg(V z, V x, V y) { return group_agg(z, x, y, AG_AVG); }
I hgpuGroupMin(V z, V x, V y) { return group_agg(z, x, y, AG_MIN); }
I hgpuGroupMax(V z, V x, V y) { return group_agg(z, x, y, AG_MAX); }
I hgpuGroupLen(V z, V x, V y) { return group_agg(z, x, y, AG_LEN); }

// z[k] = the aggregate aggs[k] (0 sum, 1 avg, 2 min, 3 max, 4 len) of x[k]
// over the grouping y, each bit for bit what hgpuGroupSum/Avg/Min/Max/Len
// returns.  The f64 sums and averages over a list this library made share
// their launches (one per size class for up to four columns), and the long
// groups' chunks read the row ids once for all of them (the common-index
// pattern applied to the segmented reductions).
I hgpuGroupAggMany(V* z, V* x, V y, const I* aggs, L n) {
    HG_CHECK(ensure_init());
    if (n < 0) return E_LENGTH;
    if (y->typ != H_G) return E_DOMAIN;
    int fused[SEG_MANY];
    int nf = 0;
    for (L k = 0; k < n; k++) {
        if (aggs[k] < AG_SUM || aggs[k] > AG_LEN || !is_real(x[k]->typ)) return E_DOMAIN;
        if ((aggs[k] == AG_SUM || aggs[k] == AG_AVG) && x[k]->typ == H_E && nf < SEG_MANY) fused[nf++] = (int)k;
    }
    bool done[64] = {false};
    if (nf >= 2 && n <= 64) {
        ScratchScope ss;
        const long long* starts;
        long long total;
        const void* rows;
        ListInfo* li;
        HG_CHECK(list_segments(y, H_L, &starts, &total, &rows, &li));
        if (li) {
            const long long ng = y->len;
            const double* srcs[SEG_MANY];
            double* sums[SEG_MANY];
            void* outs[SEG_MANY];
            long long nx = -1;
            for (int q = 0; q < nf; q++) {
                const void* px;
                HG_CHECK(in_ptr(x[fused[q]], &px));
                srcs[q] = (const double*)px;
                outs[q] = out_memory(H_E, ng);
                if (!outs[q]) return E_DEVICE_OOM;
                // a sum is reduced where it stays, an average's from scratch
                sums[q] = (double*)(aggs[fused[q]] == AG_SUM ? outs[q] : salloc((size_t)(ng > 0 ? ng : 1) * 8));
                if (!sums[q]) return E_DEVICE_OOM;
                nx = nx < 0 ? x[fused[q]]->len : (x[fused[q]]->len < nx ? x[fused[q]]->len : nx);
            }
            const bool in_range = li->group_rows && nx >= total;
            HG_CHECK(seg_sum_cols<true>(srcs, nf, (const long long*)rows, nx, starts, ng, total, sums, li));
            if (!in_range) HG_CHECK(check_device_errors());
            for (int q = 0; q < nf; q++) {
                const int k = fused[q];
                if (aggs[k] == AG_AVG) {
                    if (ng > 0) HG_LAUNCH("avg_seg", gcap(ng), 256, 0, k_avg_seg<double>, sums[q], starts, ng, total, outs[q]);
                    HG_CHECK(last_launch_error());
                }
                out_node(z[k], H_E, ng, outs[q]);
                HG_CHECK(finish_out(z[k], outs[q]));
                done[k] = true;
            }
        }
    }
    for (L k = 0; k < n; k++)
        if (!(k < 64 && done[k])) HG_CHECK(group_agg(z[k], x[k], y, aggs[k]));
    return 0;
}

// pfnEachRight: h_primitive.cc:1882-1904.  With @index over a list of i64 row
// vectors all groups are gathered in one kernel into one contiguous payload.
I pfnEachRight(V z, V x, V y, I (*foo)(V, V, V)) {
    HG_CHECK(ensure_init());
    if (y->typ != H_G) return foo(z, x, y);
    long long ng = y->len;
    if (foo == pfnIndex && is_basic(x->typ) && ng > 0) {
        bool all_long = true;
        const V0* nodes = host_nodes(y);
        const ListInfo* li = find_list(nodes, ng);
        if (!li) for (long long g = 0; g < ng && all_long; g++) all_long = nodes[g].typ == H_L;
        if (all_long) {
            ScratchScope ss;
            const long long* starts;
            long long total;
            const void* rows;
            HG_CHECK(list_segments(y, H_L, &starts, &total, &rows));
            const void* px;
            HG_CHECK(in_ptr(x, &px));
            int es = esize(x->typ);
            char* data = (char*)dalloc((size_t)(total > 0 ? total : 1) * es);
            long long* keep = (long long*)dalloc((size_t)ng * 8);
            if (!data || !keep) return E_DEVICE_OOM;
            HG_CHECK(gather_into(px, x->len, es, rows, H_L, data, total));
            HG_CHECK(check_device_errors());
            HG_CU(cudaMemcpyAsync(keep, starts, (size_t)ng * 8, cudaMemcpyDeviceToDevice, g_stream));
            HG_CHECK(init_list(z, H_G, ng));
            V0* stage = (V0*)salloc((size_t)ng * sizeof(V0));
            if (!stage) return E_DEVICE_OOM;
            HG_LAUNCH("segment_nodes", gcap(ng), 256, 0, k_segment_nodes, data, keep, ng, total, es, x->typ, stage,
                      (unsigned long long)(uintptr_t)host_nodes(z));
            HG_CU(cudaMemcpyAsync(host_nodes(z), stage, (size_t)ng * sizeof(V0), cudaMemcpyDeviceToHost, g_stream));
            HG_CHECK(last_launch_error());
            HG_CHECK(sync());
            register_list({host_nodes(z), ng, LIST_SEGMENTS, x->typ, keep, total, data, 0, 0, 0, 0, nullptr, nullptr, nullptr});
            return apply_residency(z);
        }
    }
    HG_CHECK(init_list(z, H_G, ng));
    for (long long i = 0; i < ng; i++) HG_CHECK(foo(host_nodes(z) + i, x, host_nodes(y) + i));
    return 0;
}

// pfnEach: h_primitive.cc:1818-1832.  @sum/@avg/@min/@max/@len over a list of
// vectors run as one segmented reduction; other functions are applied per element.
I pfnEach(V z, V x, I (*foo)(V, V)) {
    HG_CHECK(ensure_init());
    if (x->typ != H_G) return E_DOMAIN;
    long long ng = x->len;
    int ag = foo == pfnSum ? AG_SUM : foo == pfnAvg ? AG_AVG : foo == pfnMin ? AG_MIN : foo == pfnMax ? AG_MAX
           : foo == pfnLen ? AG_LEN : -1;
    if (ag >= 0 && ng > 0) {
        const V0* nodes = host_nodes(x);
        I t = nodes[0].typ;
        bool same = is_real(t);
        const ListInfo* li = find_list(nodes, ng);
        if (!li) for (long long g = 1; g < ng && same; g++) same = nodes[g].typ == t;
        else same = same && li->typ == t && li->kind == LIST_SEGMENTS;
        if (same) {
            ScratchScope ss;
            const long long* starts;
            long long total;
            const void* vals;
            HG_CHECK(list_segments(x, t, &starts, &total, &vals));
            void* res = nullptr;
            I typ;
            ListInfo* lk = find_list(host_nodes(x), ng);
            HG_CHECK(agg_dispatch<false>(ag, t, vals, nullptr, 0, starts, ng, total, &res, &typ, lk));
            int es = esize(typ);
            char* keep = (char*)dalloc((size_t)ng * es);
            if (!keep) return E_DEVICE_OOM;
            HG_CU(cudaMemcpyAsync(keep, res, (size_t)ng * es, cudaMemcpyDeviceToDevice, g_stream));
            HG_CHECK(init_list(z, H_G, ng));
            V0* stage = (V0*)salloc((size_t)ng * sizeof(V0));
            if (!stage) return E_DEVICE_OOM;
            HG_LAUNCH("scalar_nodes", gcap(ng), 256, 0, k_scalar_nodes, keep, ng, es, typ, stage,
                      (unsigned long long)(uintptr_t)host_nodes(z));
            HG_CU(cudaMemcpyAsync(host_nodes(z), stage, (size_t)ng * sizeof(V0), cudaMemcpyDeviceToHost, g_stream));
            HG_CHECK(last_launch_error());
            HG_CHECK(sync());
            register_list({host_nodes(z), ng, LIST_SCALARS, typ, nullptr, ng, keep, 0, 0, 0, 0, nullptr, nullptr, nullptr});
            return apply_residency(z);
        }
    }
    HG_CHECK(init_list(z, H_G, ng));
    for (long long i = 0; i < ng; i++) HG_CHECK(foo(host_nodes(z) + i, host_nodes(x) + i));
    return 0;
}

// pfnRaze: h_primitive.cc:935-955 — the elements' common type, concatenated.
I pfnRaze(V z, V x) {
    HG_CHECK(ensure_init());
    ScratchScope ss;
    if (x->typ != H_G) {
        if (is_basic(x->typ)) { *z = *x; if (is_inline(x)) z->g = (G)&z->b; return 0; }
        return E_DOMAIN;
    }
    long long ng = x->len;
    if (ng == 0) return set_error(E_RAZE_LIST, "an empty list cannot be razed");
    const V0* nodes = host_nodes(x);
    const ListInfo* li = find_list(nodes, ng);
    if (li && li->kind == LIST_SCALARS) {  // one value per element, already contiguous on the device
        void* dz;
        HG_CHECK(alloc_out(z, li->typ, ng, &dz));
        HG_CU(cudaMemcpyAsync(dz, li->data, (size_t)ng * esize(li->typ), cudaMemcpyDeviceToDevice, g_stream));
        return finish_out(z, dz);
    }
    I typ = -1;
    for (long long g = 0; g < ng; g++) {
        I t = nodes[g].typ;
        if (!is_basic(t)) return set_error(E_NOT_IMPL, "raze of nested lists");
        if (typ == -1) typ = t;
        else if (typ != t) {
            if (is_real(typ) && is_real(t)) typ = t > typ ? t : typ;
            else return E_RAZE_LIST;
        }
    }
    for (long long g = 0; g < ng; g++)
        if (nodes[g].typ != typ) return set_error(E_NOT_IMPL, "raze with type promotion across elements");
    const long long* starts;
    long long total;
    const void* data;
    HG_CHECK(list_segments(x, typ, &starts, &total, &data));
    void* dz;
    HG_CHECK(alloc_out(z, typ, total, &dz));
    if (total > 0) HG_CU(cudaMemcpyAsync(dz, data, (size_t)total * esize(typ), cudaMemcpyDeviceToDevice, g_stream));
    return finish_out(z, dz);
}

}  // extern "C"
