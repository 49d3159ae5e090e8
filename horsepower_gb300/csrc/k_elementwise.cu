// Elementwise builtins: compare, arithmetic, logic, not.
//
// Semantics (src/horseir/v3/backend/h_primitive.cc):
//   pfnCompare :1073-1170  operands promoted to MAX(type codes); f32/f64 use
//                          compareFloat (:1061) with absolute eps 1e-13, so
//                          NaN compares "greater"; ints compare exactly.
//   pfnArith   :1227-1289  result type = MAX(type codes); ints wrap; bool
//                          results are (value != 0); @div checks the divisor
//                          for zeros first (checkZero, h_system.cc:254-267).
//   pfnLogic   :1315-1332  bool only; nand/nor compute ~(x&y)/~(x|y) as bool,
//                          i.e. true for every input (h_system.cc:902-912).
//
// GB300 layout: a warp owns 512 consecutive elements.  Each of its 16-byte
// loads and stores covers 512 consecutive bytes (lane l the l-th 16), so a
// request touches four lines; with 16 consecutive elements per thread instead,
// an f64 load touched 32, and the L1's one line a cycle bound the kernels at
// 4.1-4.5 TB/s.  60M rows, kernel time: @compare f64 with a scalar 0.132 ->
// 0.082 ms (6.6 TB/s), i64 0.227 -> 0.092, i32 0.055 -> 0.046; @mul f64 0.322
// -> 0.226 ms (6.4 TB/s); @and 0.034 -> 0.027 ms.  Operands of different types
// are first converted to the common type (the reference's promoteValue), then
// the same-type kernel runs.
#include <climits>
#include <cstring>

#include "dev_common.cuh"

namespace hg {

enum { MODE_VV = 0, MODE_SV = 1, MODE_VS = 2 };  // scalar on the left / right

constexpr int EW_CHUNK = 512;  // elements of one warp's chunk, 16 per lane
// A lane's elements of a chunk, by T's vector width: pieces of 16 bytes, 512
// bytes apart.
template <typename T>
struct Lane16 {
    static constexpr int VW = 16 / (int)sizeof(T), NJ = 16 / VW;
    long long at;  // the lane's first element
    __device__ __forceinline__ Lane16(long long chunk) : at(chunk * EW_CHUNK + (long long)lane_id() * VW) {}
    __device__ __forceinline__ long long elem(int k) const { return at + (k / VW) * (32 * VW) + k % VW; }
    // `fast`: the chunk is complete and p (z) is 16-byte aligned
    __device__ __forceinline__ void load(const T* __restrict__ p, long long n, bool fast, T (&v)[16]) const {
        if (fast) {
            uint4 tmp[NJ];
#pragma unroll
            for (int j = 0; j < NJ; j++) tmp[j] = __ldcs(reinterpret_cast<const uint4*>(p + at + j * 32 * VW));
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = reinterpret_cast<const T*>(tmp)[k];
        } else {
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = elem(k) < n ? p[elem(k)] : T(0);
        }
    }
    // results of type R at the same elements, VW of them at a time
    template <typename R>
    __device__ __forceinline__ void store(R* __restrict__ z, long long n, bool fast, const R (&r)[16]) const {
        if (fast) {
            using Word = typename std::conditional<VW * sizeof(R) == 2, uint16_t,
                         typename std::conditional<VW * sizeof(R) == 4, uint32_t,
                         typename std::conditional<VW * sizeof(R) == 8, uint2, uint4>::type>::type>::type;
            static_assert(sizeof(Word) == VW * sizeof(R), "one word per piece");
#pragma unroll
            for (int j = 0; j < NJ; j++)
                *reinterpret_cast<Word*>(z + at + j * 32 * VW) = reinterpret_cast<const Word*>(r)[j];
        } else {
#pragma unroll
            for (int k = 0; k < 16; k++)
                if (elem(k) < n) z[elem(k)] = r[k];
        }
    }
};
__host__ __device__ __forceinline__ bool ew_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
// The operands of a call all begin on 16 bytes (AL of the kernels below).  When
// one does not, it is read element by element and the others and the result
// still 16 bytes at a time; that is an instance of its own, as both in one take
// the logic kernel from 32 to 39 registers and a fourth of its warps (@and 60M
// rows 33 us a call, 37).  20M rows, one column a byte off, us a call: @and 68
// with every access by element and 24 now, @lt i8 57 and 33, @mul i16 57 and 34.
static bool ew_all_aligned(const void* x, const void* y, const void* z, int mode) {
    return (mode == MODE_SV || ew_aligned(x)) && (mode == MODE_VS || ew_aligned(y)) && ew_aligned(z);
}
// Launches KERN<..., true> or KERN<..., false> by that.
#define EW_LAUNCH(name, grid, KT, KF, al, ...)                          \
    do {                                                                \
        if (al) HG_LAUNCH(name, grid, 256, 0, KT, __VA_ARGS__);         \
        else HG_LAUNCH(name, grid, 256, 0, KF, __VA_ARGS__);            \
    } while (0)
// the warps' chunks of n elements, from the warp's first one
#define EW_CHUNKS_FROM(c, first, n)                                                                      \
    for (long long c = (first), nc_ = ((n) + EW_CHUNK - 1) / EW_CHUNK,                                   \
                   st_ = ((long long)gridDim.x * blockDim.x) >> 5;                                       \
         c < nc_; c += st_)
#define EW_CHUNKS(c, n) EW_CHUNKS_FROM(c, (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5, n)

// compareFloat(x,y) (h_primitive.cc:1061), or the exact order of integers: -1, 0, 1
template <typename T>
__device__ __forceinline__ int cmp3(T a, T b) {
    if constexpr (std::is_floating_point<T>::value)
        return a < b ? ((double)(b - a) < H_EPSILON ? 0 : -1) : ((double)(a - b) < H_EPSILON ? 0 : 1);
    else return a < b ? -1 : (a > b ? 1 : 0);
}
// the ops of COMPFN (:1067-1071) as masks: bit c + 1 is the result for order c
static unsigned cmp_mask(int op) {
    switch (op) {
    case 0: return 1u;   // <
    case 1: return 3u;   // <=
    case 2: return 4u;   // >
    case 3: return 6u;   // >=
    case 4: return 2u;   // ==
    default: return 5u;  // !=
    }
}

// ARITH2 (h_primitive.cc:1225) in the promoted type.
template <typename T>
__device__ __forceinline__ T arith_op(int op, T a, T b, bool& divzero) {
    if constexpr (std::is_same<T, double>::value) {
        switch (op) {
        case 0: return __dadd_rn(a, b);
        case 1: return __dsub_rn(a, b);
        case 2: return __dmul_rn(a, b);
        default: if (b == 0.0) divzero = true; return __ddiv_rn(a, b);
        }
    } else if constexpr (std::is_same<T, float>::value) {
        switch (op) {
        case 0: return __fadd_rn(a, b);
        case 1: return __fsub_rn(a, b);
        case 2: return __fmul_rn(a, b);
        default: if (b == 0.0f) divzero = true; return __fdiv_rn(a, b);
        }
    } else if constexpr (std::is_same<T, bool>::value) {
        int x = a, y = b, r;
        switch (op) {
        case 0: r = x + y; break;
        case 1: r = x - y; break;
        case 2: r = x * y; break;
        default: if (y == 0) { divzero = true; r = 0; } else r = x / y; break;
        }
        return r != 0;
    } else if constexpr (sizeof(T) <= 2) {  // i8 / i16: computed in int, stored truncated
        int x = a, y = b, r;
        switch (op) {
        case 0: r = x + y; break;
        case 1: r = x - y; break;
        case 2: r = x * y; break;
        default: if (y == 0) { divzero = true; r = 0; } else r = x / y; break;
        }
        return (T)r;
    } else {  // i32 / i64 wrap; MIN / -1 is the wrapped negation
        using UT = typename std::make_unsigned<T>::type;
        switch (op) {
        case 0: return (T)((UT)a + (UT)b);
        case 1: return (T)((UT)a - (UT)b);
        case 2: return (T)((UT)a * (UT)b);
        default:
            if (b == 0) { divzero = true; return 0; }
            if (b == (T)-1) return (T)((UT)0 - (UT)a);
            return a / b;
        }
    }
}

// (three blocks an SM: at the 84 registers the compiler would take, f64 columns
// leave two, whose last wave costs 3 to 13% at 1.5M to 8M rows)
template <typename T, bool AL>
__global__ void __launch_bounds__(256, 3) k_compare(const T* __restrict__ x, const T* __restrict__ y,
                                                 bool* __restrict__ z, long long n, unsigned mask, int mode, T sx, T sy) {
    grid_entry();
    const bool alx = AL || ew_aligned(x), aly = AL || ew_aligned(y), alz = AL || ew_aligned(z);
    EW_CHUNKS(c, n) {
        const Lane16<T> at(c);
        const bool full = (c + 1) * EW_CHUNK <= n;
        T a[16], b[16];
        if (mode == MODE_SV) {
#pragma unroll
            for (int k = 0; k < 16; k++) a[k] = sx;
        } else at.load(x, n, full && alx, a);
        if (mode == MODE_VS) {
#pragma unroll
            for (int k = 0; k < 16; k++) b[k] = sy;
        } else at.load(y, n, full && aly, b);
        alignas(16) bool r[16];
#pragma unroll
        for (int k = 0; k < 16; k++) r[k] = (mask >> (cmp3<T>(a[k], b[k]) + 1)) & 1u;
        at.store(z, n, full && alz, r);
    }
}

// spread: consecutive chunks go to different blocks, so that what is left over
// after the warps' equal shares is shared by all SMs
template <typename T, bool AL>
__global__ void __launch_bounds__(256) k_arith(const T* __restrict__ x, const T* __restrict__ y,
                                               T* __restrict__ z, long long n, int op, int mode, T sx, T sy,
                                               int spread, unsigned* derr) {
    grid_entry();
    const bool alx = AL || ew_aligned(x), aly = AL || ew_aligned(y), alz = AL || ew_aligned(z);
    bool dz = false;
    EW_CHUNKS_FROM(c, spread ? (threadIdx.x >> 5) * (long long)gridDim.x + blockIdx.x
                             : (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5, n) {
        const Lane16<T> at(c);
        const bool full = (c + 1) * EW_CHUNK <= n;
        T a[16], b[16];
        alignas(16) T r[16];
        if (mode == MODE_SV) {
#pragma unroll
            for (int k = 0; k < 16; k++) a[k] = sx;
        } else at.load(x, n, full && alx, a);
        if (mode == MODE_VS) {
#pragma unroll
            for (int k = 0; k < 16; k++) b[k] = sy;
        } else at.load(y, n, full && aly, b);
#pragma unroll
        for (int k = 0; k < 16; k++) {
            bool d = false;
            r[k] = arith_op<T>(op, a[k], b[k], d);
            if (d && at.elem(k) < n) dz = true;
        }
        at.store(z, n, full && alz, r);
    }
    if (dz) flag_error(derr, DERR_DIVZERO);
}

// bool logic: and/or/xor act bytewise on 0/1 bytes, four at a time
__device__ __forceinline__ unsigned logic_word(int op, unsigned a, unsigned b) {
    switch (op) {
    case 0: return a & b;
    case 2: return a | b;
    case 4: return a ^ b;
    case 5: return a ^ 0x01010101u;  // not
    default: return 0x01010101u;     // nand / nor: ~(.) as bool is always true
    }
}
template <bool AL>
__global__ void __launch_bounds__(256) k_logic(const uint8_t* __restrict__ x, const uint8_t* __restrict__ y,
                                               uint8_t* __restrict__ z, long long n, int op, int mode,
                                               uint8_t sx, uint8_t sy) {
    grid_entry();
    const bool alx = AL || ew_aligned(x), aly = AL || ew_aligned(y);  // z begins a result's memory
    EW_CHUNKS(c, n) {
        const long long i0 = Lane16<uint8_t>(c).at;
        const bool full = (c + 1) * EW_CHUNK <= n;
        const unsigned ax = sx * 0x01010101u, by = sy * 0x01010101u;
        if (!full) {
            for (int k = 0; k < 16; k++)
                if (i0 + k < n)
                    z[i0 + k] = (uint8_t)logic_word(op, mode == MODE_SV ? sx : x[i0 + k], mode == MODE_VS ? sy : y[i0 + k]);
            continue;
        }
        auto load = [&](const uint8_t* p, bool al) {
            if (al) return __ldcs(reinterpret_cast<const uint4*>(p + i0));
            unsigned w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int k = 0; k < 16; k++) w[k / 4] |= (unsigned)p[i0 + k] << (8 * (k % 4));
            return make_uint4(w[0], w[1], w[2], w[3]);
        };
        uint4 a = make_uint4(ax, ax, ax, ax), b = make_uint4(by, by, by, by);
        if (mode != MODE_SV) a = load(x, alx);
        if (mode != MODE_VS) b = load(y, aly);
        *reinterpret_cast<uint4*>(z + i0) = make_uint4(logic_word(op, a.x, b.x), logic_word(op, a.y, b.y),
                                                       logic_word(op, a.z, b.z), logic_word(op, a.w, b.w));
    }
}

// promotion of a vector of type `st` to T (promoteValueWithIndex, h_system.cc:168-252)
template <typename T>
__global__ void k_convert(const void* __restrict__ src, int st, T* __restrict__ dst, long long n) {
    grid_entry();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        T v;
        switch (st) {
        case H_B: v = (T)((const bool*)src)[i]; break;
        case H_J: v = (T)((const int8_t*)src)[i]; break;
        case H_H: v = (T)((const int16_t*)src)[i]; break;
        case H_I: v = (T)((const int32_t*)src)[i]; break;
        case H_L: v = (T)((const long long*)src)[i]; break;
        case H_F: v = (T)((const float*)src)[i]; break;
        default: v = (T)((const double*)src)[i]; break;
        }
        dst[i] = v;
    }
}

static unsigned ew_grid(long long n) {
    long long chunks = (n + 15) / 16;
    long long b = (chunks + 255) / 256;
    long long cap = (long long)g_sms * 8;
    if (b > cap) b = cap;
    return (unsigned)(b < 1 ? 1 : b);
}

// Host value of element 0 of x converted to T (scalar operands are passed by value).
template <typename T>
static I scalar_as(V x, T* out) {
    uint64_t bits;
    HG_CHECK(read_elem0(x, &bits));
    switch (x->typ) {
    case H_B: *out = (T)(*(bool*)&bits); break;
    case H_J: case H_C: *out = (T)(*(int8_t*)&bits); break;
    case H_H: *out = (T)(*(int16_t*)&bits); break;
    case H_I: case H_M: case H_D: case H_U: case H_W: case H_T: *out = (T)(*(int32_t*)&bits); break;
    case H_L: case H_Z: *out = (T)(*(long long*)&bits); break;
    case H_F: *out = (T)(*(float*)&bits); break;
    case H_E: *out = (T)(*(double*)&bits); break;
    default: return E_NOT_IMPL;
    }
    return 0;
}

// Device vector of x in type T (converted into scratch when x has another type)
template <typename T>
static I vector_as(V x, I xt, const T** out) {
    const void* p;
    HG_CHECK(in_ptr(x, &p));
    if (x->typ == xt) { *out = (const T*)p; return 0; }
    T* d = (T*)salloc((size_t)x->len * sizeof(T));
    if (!d) return E_DEVICE_OOM;
    HG_LAUNCH("convert", ew_grid(x->len * 16 / 16), 256, 0, k_convert<T>, p, (int)x->typ, d, (long long)x->len);
    *out = d;
    return 0;
}

static int compare_float_host(double a, double b) {
    return a < b ? ((b - a) < H_EPSILON ? 0 : -1) : ((a - b) < H_EPSILON ? 0 : 1);
}
static double from_ord(long long o) {
    unsigned long long b = o >= 0 ? (unsigned long long)o : (0x8000000000000000ull | (unsigned long long)(-o));
    double d;
    memcpy(&d, &b, 8);
    return d;
}

F64Range f64_cmp_range(double s, bool scalar_first, int op) {
    const unsigned mask = cmp_mask(op);
    if (s != s) return F64Range{0, 0, (int)((mask >> 2) & 1u)};  // a NaN operand compares as 1 everywhere
    const long long lo = f64_ord(0xfff0000000000000ull), hi = f64_ord(0x7ff0000000000000ull) + 1;  // -inf .. +inf + 1
    auto c = [&](long long o) { return scalar_first ? compare_float_host(s, from_ord(o)) : compare_float_host(from_ord(o), s); };
    // smallest o in [lo, hi] with pred(o); o = hi stands for "no such value"
    auto first = [&](auto pred) {
        long long a = lo, b = hi;
        while (a < b) {
            long long m = a + (long long)(((unsigned long long)b - (unsigned long long)a) / 2);  // b - a can exceed 2^63
            if (pred(m)) b = m; else a = m + 1;
        }
        return a;
    };
    // the steps: order d0 below ta, 0 from ta up to tb, -d0 from tb
    const int d0 = scalar_first ? 1 : -1;
    const long long ta = first([&](long long o) { return d0 * c(o) <= 0; });
    const long long tb = first([&](long long o) { return d0 * c(o) < 0; });
    // image of the smallest value whose ord is o
    auto image = [](long long o) {
        return o > 0 ? (1ull << 63) + (unsigned long long)o : (1ull << 63) - 1 - (unsigned long long)(-o);
    };
    const unsigned long long ia = image(ta), ib = image(tb), inf = image(hi), ninf = image(lo);
    // the pieces of the circle of images, from -inf up: [-inf, ia) has order
    // d0, [ia, ib) 0, [ib, +inf] -d0, and the NaNs behind it 1.  Vector first
    // the last two agree, scalar first the NaNs agree with the first piece.
    auto bit = [&](int order) { return (mask >> (order + 1)) & 1u; };
    const unsigned ra = bit(d0), rb = bit(0), rc = bit(-d0);
    unsigned long long from, to;  // one range where the result is `one`
    unsigned one;
    bool nans = false;  // the NaNs are inside it
    if (ra == rb) { from = ib; to = scalar_first ? inf : ninf; one = rc; nans = !scalar_first; }      // rc alone differs
    else if (rb == rc) { from = scalar_first ? inf : ninf; to = ia; one = ra; nans = scalar_first; }  // ra alone
    else { from = ia; to = ib; one = rb; }                                                            // rb alone
    if (from == to && nans) return F64Range{0, 0, (int)one};  // the whole circle
    return F64Range{from, to - from, one ? 0 : 1};
}

// a double vector against a fixed double, by the range of its images
__global__ void __launch_bounds__(256) k_compare_f64_fixed(const double* __restrict__ x, bool* __restrict__ z,
                                                           long long n, F64Range range) {
    grid_entry();
    const bool alx = ew_aligned(x), alz = ew_aligned(z);
    EW_CHUNKS(c, n) {
        const Lane16<double> at(c);
        const bool full = (c + 1) * EW_CHUNK <= n;
        double a[16];
        at.load(x, n, full && alx, a);
        alignas(16) bool r[16];
#pragma unroll
        for (int k = 0; k < 16; k++) r[k] = f64_in_range(a[k], range);
        at.store(z, n, full && alz, r);
    }
}

template <typename T>
static I run_compare(V z, V x, V y, I typX, int op) {
    bool ox = x->len == 1, oy = y->len == 1;
    L n = ox ? y->len : x->len;
    int mode = ox ? MODE_SV : (oy ? MODE_VS : MODE_VV);
    T sx = 0, sy = 0;
    const T *px = nullptr, *py = nullptr;
    if (mode == MODE_SV) HG_CHECK(scalar_as<T>(x, &sx)); else HG_CHECK(vector_as<T>(x, typX, &px));
    if (mode == MODE_VS) HG_CHECK(scalar_as<T>(y, &sy)); else HG_CHECK(vector_as<T>(y, typX, &py));
    void* dz;
    HG_CHECK(alloc_out(z, H_B, n, &dz));
    if constexpr (std::is_same<T, double>::value) {
        if (mode != MODE_VV && n > 0) {  // one side fixed: a range of images instead of FP64 subtractions
            HG_LAUNCH("compare", ew_grid(n), 256, 0, k_compare_f64_fixed, mode == MODE_SV ? py : px, (bool*)dz,
                      (long long)n, f64_cmp_range(mode == MODE_SV ? sx : sy, mode == MODE_SV, op));
            HG_CHECK(last_launch_error());
            return finish_out(z, dz);
        }
    }
    if (n > 0)
        EW_LAUNCH("compare", ew_grid(n), (k_compare<T, true>), (k_compare<T, false>), ew_all_aligned(px, py, dz, mode), px,
                  py, (bool*)dz, (long long)n, cmp_mask(op), mode, sx, sy);
    HG_CHECK(last_launch_error());
    return finish_out(z, dz);
}

template <typename T>
static I run_arith(V z, V x, V y, I typ, int op) {
    bool ox = x->len == 1, oy = y->len == 1;
    L n = ox ? y->len : x->len;
    int mode = ox ? MODE_SV : (oy ? MODE_VS : MODE_VV);
    T sx = 0, sy = 0;
    const T *px = nullptr, *py = nullptr;
    if (mode == MODE_SV) HG_CHECK(scalar_as<T>(x, &sx)); else HG_CHECK(vector_as<T>(x, typ, &px));
    if (mode == MODE_VS) HG_CHECK(scalar_as<T>(y, &sy)); else HG_CHECK(vector_as<T>(y, typ, &py));
    long long mark = out_mark();
    void* dz;
    HG_CHECK(alloc_out(z, typ, n, &dz));
    // f64 columns take 103 registers, two blocks an SM, and their division is
    // bound by the FP64 unit: with one block for each 4096 rows the SMs that get
    // one more set the time (1.6M divisions 58 us a call with 16 consecutive rows
    // a thread, 63 with the warps' chunks in such blocks, 48 spread over the SMs)
    unsigned grid = ew_grid(n);
    const int spread = std::is_same<T, double>::value && op == 3 && grid > 2u * (unsigned)g_sms;
    if (spread) grid = 2u * (unsigned)g_sms;
    if (n > 0)
        EW_LAUNCH(spread ? "arith_spread" : "arith", grid, (k_arith<T, true>), (k_arith<T, false>),
                  ew_all_aligned(px, py, dz, mode), px, py, (T*)dz, (long long)n, op, mode, sx, sy, spread, g_derr);
    HG_CHECK(last_launch_error());
    if (op == 3) {  // checkZero (h_system.cc:254-267) runs before the division in the reference
        I e = check_device_errors();
        if (e) { out_rewind(mark); return e; }
    }
    return finish_out(z, dz);
}

// Device vector of x converted to basic type `typ` (promoteValue semantics).
I promote_to(V x, I typ, const void** out) {
    switch (typ) {
    case H_B: return vector_as<bool>(x, typ, (const bool**)out);
    case H_J: return vector_as<int8_t>(x, typ, (const int8_t**)out);
    case H_H: return vector_as<int16_t>(x, typ, (const int16_t**)out);
    case H_I: return vector_as<int32_t>(x, typ, (const int32_t**)out);
    case H_L: return vector_as<long long>(x, typ, (const long long**)out);
    case H_F: return vector_as<float>(x, typ, (const float**)out);
    case H_E: return vector_as<double>(x, typ, (const double**)out);
    default: return E_NOT_IMPL;
    }
}

}  // namespace hg

using namespace hg;

extern "C" {

I pfnCompare(V z, V x, V y, I op) {
    HG_CHECK(ensure_init());
    ScratchScope ss;
    if (!(is_comparable(x->typ) && is_comparable(y->typ))) return E_DOMAIN;
    if (!(x->len == 1 || y->len == 1 || x->len == y->len)) return E_LENGTH;
    if (is_real(x->typ) && is_real(y->typ)) {
        I t = x->typ > y->typ ? x->typ : y->typ;
        switch (t) {
        case H_B: return run_compare<bool>(z, x, y, t, op);
        case H_J: return run_compare<int8_t>(z, x, y, t, op);
        case H_H: return run_compare<int16_t>(z, x, y, t, op);
        case H_I: return run_compare<int32_t>(z, x, y, t, op);
        case H_L: return run_compare<long long>(z, x, y, t, op);
        case H_F: return run_compare<float>(z, x, y, t, op);
        default: return run_compare<double>(z, x, y, t, op);
        }
    }
    if (x->typ == y->typ) {
        switch (x->typ) {
        case H_C: return run_compare<int8_t>(z, x, y, H_C, op);  // signed char, as the reference's x86 build
        case H_M: case H_D: case H_U: case H_T: return run_compare<int32_t>(z, x, y, x->typ, op);
        case H_Z: return run_compare<long long>(z, x, y, H_Z, op);
        case H_Q: return compare_symbols(z, x, y, op);
        default: return set_error(E_NOT_IMPL, "compare of type %d (no case in the reference)", x->typ);
        }
    }
    return E_TYPE;
}
I pfnLt(V z, V x, V y) { return pfnCompare(z, x, y, 0); }
I pfnLeq(V z, V x, V y) { return pfnCompare(z, x, y, 1); }
I pfnGt(V z, V x, V y) { return pfnCompare(z, x, y, 2); }
I pfnGeq(V z, V x, V y) { return pfnCompare(z, x, y, 3); }
I pfnEq(V z, V x, V y) { return pfnCompare(z, x, y, 4); }
I pfnNeq(V z, V x, V y) { return pfnCompare(z, x, y, 5); }

I pfnArith(V z, V x, V y, I op) {
    HG_CHECK(ensure_init());
    ScratchScope ss;
    if (is_real(x->typ) && is_real(y->typ)) {
        if (!(x->len == 1 || y->len == 1 || x->len == y->len)) return E_LENGTH;
        I t = x->typ > y->typ ? x->typ : y->typ;
        if (op == 3 && y->len == 1) {  // scalar divisor: checkZero on the host value
            double d;
            HG_CHECK(scalar_as<double>(y, &d));
            if (d == 0.0) return E_DIV_ZERO;
        }
        switch (t) {
        case H_B: return run_arith<bool>(z, x, y, t, op);
        case H_J: return run_arith<int8_t>(z, x, y, t, op);
        case H_H: return run_arith<int16_t>(z, x, y, t, op);
        case H_I: return run_arith<int32_t>(z, x, y, t, op);
        case H_L: return run_arith<long long>(z, x, y, t, op);
        case H_F: return run_arith<float>(z, x, y, t, op);
        default: return run_arith<double>(z, x, y, t, op);
        }
    }
    if (is_dtime(x->typ) && is_dtime(y->typ)) return E_NOT_IMPL;
    return E_DOMAIN;
}
I pfnPlus(V z, V x, V y) { return pfnArith(z, x, y, 0); }
I pfnMinus(V z, V x, V y) { return pfnArith(z, x, y, 1); }
I pfnMul(V z, V x, V y) { return pfnArith(z, x, y, 2); }
I pfnDiv(V z, V x, V y) { return pfnArith(z, x, y, 3); }

static I logic(V z, V x, V y, int op) {
    HG_CHECK(ensure_init());
    ScratchScope ss;
    if (!(x->typ == H_B && y->typ == H_B)) return E_DOMAIN;
    if (!(x->len == 1 || y->len == 1 || x->len == y->len)) return E_LENGTH;
    bool ox = x->len == 1, oy = y->len == 1;
    L n = ox ? y->len : x->len;
    int mode = ox ? MODE_SV : (oy ? MODE_VS : MODE_VV);
    uint64_t bx = 0, by = 0;
    const void *px = nullptr, *py = nullptr;
    if (mode == MODE_SV) HG_CHECK(read_elem0(x, &bx)); else HG_CHECK(in_ptr(x, &px));
    if (mode == MODE_VS) HG_CHECK(read_elem0(y, &by)); else HG_CHECK(in_ptr(y, &py));
    void* dz;
    HG_CHECK(alloc_out(z, H_B, n, &dz));
    if (n > 0)
        EW_LAUNCH("logic", ew_grid(n), k_logic<true>, k_logic<false>, ew_all_aligned(px, py, dz, mode), (const uint8_t*)px,
                  (const uint8_t*)py, (uint8_t*)dz, (long long)n, op, mode, (uint8_t)(bx & 1), (uint8_t)(by & 1));
    HG_CHECK(last_launch_error());
    return finish_out(z, dz);
}
I pfnAnd(V z, V x, V y) { return logic(z, x, y, 0); }
I pfnNand(V z, V x, V y) { return logic(z, x, y, 1); }
I pfnOr(V z, V x, V y) { return logic(z, x, y, 2); }
I pfnNor(V z, V x, V y) { return logic(z, x, y, 3); }
I pfnXor(V z, V x, V y) { return logic(z, x, y, 4); }

// pfnNot: h_primitive.cc:606-615
I pfnNot(V z, V x) {
    HG_CHECK(ensure_init());
    ScratchScope ss;
    if (x->typ != H_B) return E_DOMAIN;
    const void* px;
    HG_CHECK(in_ptr(x, &px));
    void* dz;
    HG_CHECK(alloc_out(z, H_B, x->len, &dz));
    if (x->len > 0)
        EW_LAUNCH("not", ew_grid(x->len), k_logic<true>, k_logic<false>, ew_all_aligned(px, px, dz, MODE_VV), (const uint8_t*)px,
                  (const uint8_t*)px, (uint8_t*)dz, (long long)x->len, 5, MODE_VV, (uint8_t)0, (uint8_t)0);
    HG_CHECK(last_launch_error());
    return finish_out(z, dz);
}

}  // extern "C"
