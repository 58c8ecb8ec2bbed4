// digit_gemm.cu -- FP64 transforms on the tensor cores.
//
// GB300 gives FP64 about 1.2 TFLOP/s and its FP16 tensor cores about 1900, so the FP64 path's two
// contractions per direction (the row DFT and the Legendre transform) run as integer products:
// every operand is a 55-bit fixed-point number relative to its row's (table) or column's (data)
// largest value, written as seven balanced base-256 digits d in [-128, 127]; digits are exact in
// FP16, so are their products and FP32 sums up to 2^24, and the digit products of equal weight share one
// accumulator:
//     sum_k T_k x_k = sum_g 256^-g sum_{a+b=g} sum_k d_a(T_k) d_b(x_k),   g <= 6
// (products of weight 256^-7 and below are under 2^-54 of the operands' scale and are left out; the
// scheme is Ozaki, Ogita, Oishi and Rump's error-free matrix product, Numer. Algorithms 59 (2012)).
// Leading digits may take up to 256 (FP16 holds them): a data value, folds included, has 56 bits up to
// K = 256 and 54 beyond, a table value 54 to 56, as many as keep the leading group's bound K d_0 d'_0 near
// 2^22 (at most 1.5 2^22, dg_table_bits).
// Which sums stay below 2^24, and are exact, follows from the tables (the sum over a row's entries of |digit of the
// table| times the data digits' bound, its largest over all rows), for any data whatever: up to bw 256 all groups (I2
// at odd bandwidths above 200: 0 to 4), at bw 512 groups 0 to 3, at bw 511 and 1024 groups 0 and 1 and, but for I2
// (1.1 2^24), group 2.  A group passes 2^24 where the digits of data and table agree in sign over most of K, and
// then loses about two of its units for every 16 entries; in data not made for it, digits behind the first agree
// by chance only, and the sums stay tens of times smaller.  Data made for a row of the forward Legendre table of m = 0
// lose up to 1.0e-15 of sum |T x| at bw 512 (group 4) and 1.3e-12 at bw 1024 (group 3), where the FP64 kernels round at 1e-16.
//
// One MMA covers all data digits of a table digit: the data digits b = 0..6-a lie one after another
// along N, so A = table digit a times B = [x_0 | ... | x_(6-a)] adds to the accumulator groups
// a..6, which lie one after another along TMEM columns.  28 digit products take 7 MMAs per 16-deep
// K step with N = 7 NT, 6 NT, ... NT columns.
//
// Four stages share one kernel (k_dg); D[row, column] with the table on the M side:
//   F1  rows forward    row = order m        K = folded longitude    column = (field, latitude part)
//   F2  Legendre fwd    row = degree l       K = latitude            column = (field, re / im)
//   I1  Legendre inv    row = latitude j     K = degree              column = (field, re / im)
//   I2  rows inverse    row = longitude      K = order               column = (field, latitude part)
// F2 and I1 are the naive transform (naive.c:34-96) in every order, F2 but for up to three odd ones above
// bw 512 (dg_semi_orders): on the tensor cores its extra multiply-adds cost less than the DCTs of the
// seminaive form would, and it is the better conditioned of the two.  k_dg_fold turns samples into fixed point and takes the even and odd
// parts in latitude (P(m,l) has one parity) and, for even B, twice in longitude (cos and sin, m even
// and odd), so that each of F1's four tables is a quarter of the DFT matrix; k_dg_unfold undoes the
// same after I2.  Between the stages the forward keeps integers (one scale per function).  COMPLEX
// data are two real fields g + i h, combined per coefficient in F2's epilogue and split before I1.
//
#include <math.h>

#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include "s2g_common.cuh"
#include "s2g_internal.h"
#include "tc_sm103.cuh"

namespace s2g {

constexpr int kDgThreads = 896;          // warp 0 tables, 1 MMA, then from 4 the epilogue's and the data's
constexpr int kSub = 2;                   // 16-deep K steps of a stage
constexpr uint32_t kDgBRing = 86016;     // data ring: as many stages as fit
constexpr uint32_t kDgStash = 32 * 33 * 4;  // FP32 F1: an epilogue warp's results, rows by columns
constexpr int kDgMaxStagesB = 16;

// Precision of an instance.  64: FP64 transforms, seven digits each.  32: FP32 transforms: table values of
// 25 bits in three digits, data of 30 bits in four, accumulator groups 0 to 3 (nine of the twelve
// products; the rest are below 2^-28 of the result's scale).
template <int P>
struct Dg;
template <>
struct Dg<64> {
    static constexpr int DA = 7, DB = 7, G = 7, stagesA = 2, epilogue = 16, data = 8;  // warps
    using Real = double;
    using Int = long long;
    using Int2 = longlong2;
};
template <>
struct Dg<32> {
    static constexpr int DA = 3, DB = 4, G = 4, stagesA = 4, epilogue = 8, data = 16;
    using Real = float;
    using Int = int;
    using Int2 = int2;
};
template <int P>
constexpr uint32_t kDgABytes = kSub * Dg<P>::DA * 128 * 32;  // a stage of a full table tile
constexpr int kDigits = 7;
enum { kF1 = 0, kF2 = 1, kI1 = 2, kI2 = 3 };
// REAL without imaginary arrays / REAL with them / COMPLEX
enum { kReal = 0, kReal2 = 1, kCplx = 2 };

// One M tile of a table: up to 128 rows.  Blobs hold, per 16-deep K step, the seven digits' r8 x 16
// tiles in core-matrix order.
struct DgTile {
    int64_t off;      // byte offset of the first K step's blob
    int ks;           // K steps
    int k0;           // the first one with a digit that is not zero (Legendre tables: near the pole high
                      // orders vanish below the last digit, a third of all entries)
    int row0, nrows;  // rows row0 .. row0 + nrows of the panel
    int r8;           // rows stored (nrows rounded up to 8)
    int qoff;         // row scales at q[qoff + row]
    int m, t;         // F1, I2: first order, part (cos / sin); F2, I1: order, parity
    int kind;         // F1, I2: fold (0..3 two longitude folds, 4, 5 one)
    int zoff;         // F1, I2: the panel's place in a column of Z
    int vb;           // bits of a data value
    int tb;           // bits of a table value
    int pad_;
};

struct DgArgs {
    const DgTile* tiles;
    const uint8_t* tab;
    const short* q;            // table value = digits * 2^-q
    int ntiles, ncolblk, col_major;
    int B, S, N, ncols, mode;  // N functions as the caller counts them
    int BP, RL;                // latitudes of a half row of X (B, rounded up to 4); values of a column of Z
    int vbz;                   // bits of Z's samples before folds
    int tbz;                   // F2: bits of F1's table
    const void* in_r;          // I1: coefficients
    const void* in_i;
    void* out_r;               // F2: coefficients
    void* out_i;
    void* X;                   // [field, part][m][t][BP]: FP64 integers (F1 -> F2), else reals
    void* Z;                   // [field][t][j][RL]: folded samples (F1) or parts of samples (I2)
    const uint32_t* ein;       // F1: exponents of the latitude pairs; I1: of the orders; I2: of the fields
    const uint32_t* efield;    // FP64 F1, F2: exponents of the fields
    const int64_t* cmap;       // function -> coefficient offset (null: f B^2; real fields only)
    uint32_t* emax;            // F1 writes, F2 reads: X's rows (FP64 bits, FP32 exponents); I1 writes: fields
    int* err;                  // gets S2G_ERR_TIMEOUT where a bounded wait expired; device memory, or the host's
    int stall;                 // test hook: the table warp copies nothing, so that the waits run out
};

__device__ __forceinline__ uint32_t dexp(double x) { return ((uint32_t)__double2hiint(x) >> 20) & 0x7ffu; }
__device__ __forceinline__ uint32_t dexp(float x) { return (__float_as_uint(x) >> 23) & 0xffu; }

// x as an integer of unit 2^(em - 126 - vb) (|x| < 2^(em - 126), vb at most 31), rounded to nearest
__device__ __forceinline__ int dg_fix(float x, int em, int vb) {
    const uint32_t b = __float_as_uint(x);
    int e = (b >> 23) & 0xff;
    uint32_t m = b & 0x7fffffu;
    if (e) m |= 0x800000u;
    else e = 1;
    const int v = (int)((((m << 8) >> min(em - e + 31 - vb, 31)) + 1) >> 1);
    return (int)b < 0 ? -v : v;
}

// x as an integer of unit 2^(em - 1022 - vb) (|x| < 2^(em - 1022), vb at most 56), rounded to nearest
__device__ __forceinline__ long long dg_fix(double x, int em, int vb) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    int e = (hi >> 20) & 0x7ff;
    uint32_t mh = hi & 0xfffffu;
    if (e) mh |= 0x100000u;
    else e = 1;
    const unsigned long long mant = (((unsigned long long)mh << 32) | lo) << 4;
    const int rs = min(em - e + 56 - vb, 63);
    const long long v = (long long)(((mant >> rs) + 1) >> 1);
    return (int)hi < 0 ? -v : v;
}

// Digit b (0 most significant) of the biased values u0, u1 as two FP16 numbers.
template <int b>
__device__ __forceinline__ uint32_t dg_digit2(unsigned long long u0, unsigned long long u1) {
    if (b == 0) {  // the leading digit has 10 bits, biased by 512
        const uint32_t t = (__byte_perm((uint32_t)(u0 >> 32), (uint32_t)(u1 >> 32), 0x7632) & 0x03ff03ffu) | 0x64006400u;
        const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&t), __half2half2(__ushort_as_half(0x6600)));
        return *reinterpret_cast<const uint32_t*>(&d);
    }
    constexpr int i = 6 - b;  // byte
    const uint32_t w0 = i < 4 ? (uint32_t)u0 : (uint32_t)(u0 >> 32), w1 = i < 4 ? (uint32_t)u1 : (uint32_t)(u1 >> 32);
    const uint32_t t = (__byte_perm(w0, w1, (i & 3) | ((4 + (i & 3)) << 8)) & 0x00ff00ffu) | 0x64006400u;  // 1024 + byte
    const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&t), __half2half2(__ushort_as_half(0x6480)));  // - 1152
    return *reinterpret_cast<const uint32_t*>(&d);
}

// Stores the seven digits of four consecutive K entries of one column, eight bytes a digit.
template <int NT>
__device__ __forceinline__ void dg_store4(uint8_t* dst, const long long* v) {
    constexpr unsigned long long bias = 0x0200808080808080ull;
    unsigned long long u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = (unsigned long long)v[i] + bias;
    constexpr int step = NT * 32;  // bytes between digits
    *(uint2*)(dst) = make_uint2(dg_digit2<0>(u[0], u[1]), dg_digit2<0>(u[2], u[3]));
    *(uint2*)(dst + step) = make_uint2(dg_digit2<1>(u[0], u[1]), dg_digit2<1>(u[2], u[3]));
    *(uint2*)(dst + 2 * step) = make_uint2(dg_digit2<2>(u[0], u[1]), dg_digit2<2>(u[2], u[3]));
    *(uint2*)(dst + 3 * step) = make_uint2(dg_digit2<3>(u[0], u[1]), dg_digit2<3>(u[2], u[3]));
    *(uint2*)(dst + 4 * step) = make_uint2(dg_digit2<4>(u[0], u[1]), dg_digit2<4>(u[2], u[3]));
    *(uint2*)(dst + 5 * step) = make_uint2(dg_digit2<5>(u[0], u[1]), dg_digit2<5>(u[2], u[3]));
    *(uint2*)(dst + 6 * step) = make_uint2(dg_digit2<6>(u[0], u[1]), dg_digit2<6>(u[2], u[3]));
}

// Four digits of 32-bit values, all in [-128, 127].
template <int b>
__device__ __forceinline__ uint32_t dg_byte2(uint32_t u0, uint32_t u1) {
    constexpr int i = 3 - b;
    const uint32_t t = (__byte_perm(u0, u1, i | ((4 + i) << 8)) & 0x00ff00ffu) | 0x64006400u;
    const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&t), __half2half2(__ushort_as_half(0x6480)));
    return *reinterpret_cast<const uint32_t*>(&d);
}
template <int NT>
__device__ __forceinline__ void dg_store4(uint8_t* dst, const int* v) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = (uint32_t)v[i] + 0x80808080u;
    constexpr int step = NT * 32;
    *(uint2*)(dst) = make_uint2(dg_byte2<0>(u[0], u[1]), dg_byte2<0>(u[2], u[3]));
    *(uint2*)(dst + step) = make_uint2(dg_byte2<1>(u[0], u[1]), dg_byte2<1>(u[2], u[3]));
    *(uint2*)(dst + 2 * step) = make_uint2(dg_byte2<2>(u[0], u[1]), dg_byte2<2>(u[2], u[3]));
    *(uint2*)(dst + 3 * step) = make_uint2(dg_byte2<3>(u[0], u[1]), dg_byte2<3>(u[2], u[3]));
}

// Accumulator groups (exact integers) -> their sum in units of group 5.  Adding 1.5 2^23 leaves an
// integer below 2^22 in a float's low bits (full-rate adds; the conversion instruction runs at an eighth
// of their rate and set the epilogue's pace); the biases are taken off once, modulo 2^64.
__device__ __forceinline__ long long dg_sum(const uint32_t* a, int stride, uint32_t& odd) {
    constexpr float M = 12582912.0f;
    constexpr long long b = 0x4B400000ll;
    int i[kDigits];
#pragma unroll
    for (int g = 0; g < 6; ++g) i[g] = __float_as_int(__uint_as_float(a[g * stride]) + M);
    i[6] = __float_as_int(fmaf(__uint_as_float(a[6 * stride]), 0.00390625f, M));
    uint32_t x = 0;
#pragma unroll
    for (int g = 0; g < kDigits; ++g) x |= (uint32_t)i[g] ^ 0x4b000000u;
    odd |= x;
    const long long lo = (long long)i[2] * (1 << 24) + (long long)i[3] * 65536 + (long long)i[4] * 256 + (long long)i[5] + i[6];
    constexpr unsigned long long bias = ((unsigned long long)(b * 257) << 32) + (unsigned long long)(b * ((1 << 24) + 65536 + 256 + 2));
    const unsigned long long hi = (unsigned long long)(((uint32_t)i[0] << 8) + (uint32_t)i[1]) << 32;  // modulo 2^32
    return (long long)(hi + (unsigned long long)lo - bias);
}
// The same for groups of any size; dg_sum sets bits 23.. of `odd` where one is outside its range.
__device__ __noinline__ long long dg_sum_big(float a0, float a1, float a2, float a3, float a4, float a5, float a6) {
    const float a[kDigits] = {a0, a1, a2, a3, a4, a5, a6};
    long long i[kDigits];
#pragma unroll
    for (int g = 0; g < kDigits; ++g) i[g] = __float2int_rn(a[g]);
    return (i[0] * 256 + i[1]) * (1ll << 32) + i[2] * (1 << 24) + i[3] * 65536 + i[4] * 256 + i[5] + (i[6] >> 8);
}

// T 2^(eb - 1086) as a double, rounded to nearest; kDgNan in eb stands for a column that held an
// infinity or a NaN.  dg_fast is free of branches, so that several run interleaved; where it sets
// `bad` (NaN, overflow, subnormal results) dg_slow gives the value.
constexpr int kDgNan = 1 << 20;
__device__ __forceinline__ double dg_fast(long long T, int eb, bool& bad) {
    const unsigned long long m0 = T < 0 ? (unsigned long long)-T : (unsigned long long)T;
    const uint32_t mh = (uint32_t)(m0 >> 32), mw = mh ? mh : (uint32_t)m0;
    const int lz = __clz((int)mw) + (mh ? 0 : 32), e = eb - lz;
    const unsigned long long m = m0 << (lz & 63);
    bad |= (m0 != 0 && (uint32_t)(e - 1) >= 2046u) || eb >= kDgNan / 2;
    unsigned long long bits = ((unsigned long long)((uint32_t)(e - 1) << 20) << 32) + (m >> 11) + ((m >> 10) & 1);
    bits = m0 ? bits : 0;
    return __longlong_as_double((long long)(bits | ((unsigned long long)T & 0x8000000000000000ull)));
}
__device__ __noinline__ double dg_slow(long long T, int eb) {
    if (eb >= kDgNan / 2) return __longlong_as_double(0x7ff8000000000000ll);
    return T ? ldexp((double)T, eb - 1086) : 0.0;
}
// dg_fast's exponent of a column whose largest value has exponent field em
__device__ __forceinline__ int dg_eb(uint32_t em, int base) { return em == 0x7ffu ? kDgNan : base + max((int)em, 1); }

__device__ __forceinline__ void tm_ld8(uint32_t ta, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(ta));
}
__device__ __forceinline__ void tm_ld4(uint32_t ta, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(ta));
}
// Shared-memory descriptors of the digit tiles: LBO 128 B (K), SBO 256 B (rows), no swizzle; the high
// word is the same for all.
constexpr uint32_t kDescHi = (256u >> 4) | (1u << 14);
__device__ __forceinline__ uint32_t dg_desc(const void* s) { return (tc::smem_u32(s) >> 4) | ((128u >> 4) << 16); }
__device__ __forceinline__ void dg_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}\n" ::"r"(d),
        "r"(a), "r"(b), "r"(idesc), "r"(acc), "n"(kDescHi)
        : "memory");
}
__device__ __forceinline__ void tm_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Eight of I2's sums are added: each gives up its last bits.
constexpr int kDgOutShift = 2;

// FP32: unit of a column whose largest value has exponent field em, times 2^tb of the table's digits
// (groups in units of the leading one's products, 2^40 of the digits' last places).
__device__ __forceinline__ float dg_col_scale(uint32_t em, int tb, int vb) {
    return em == 0xffu ? __int_as_float(0x7fc00000) : ldexpf(1.0f, 40 - tb - vb - 126 + max((int)em, 1));
}

// Waits for a phase, for about half a second at most; another role's failure ends the wait at once.
__device__ __forceinline__ bool dg_wait(uint64_t* bar, uint32_t parity, volatile int* failed) {
    if (tc::mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!tc::mbar_try_wait(bar, parity)) {
        if (*failed) return false;
        if (clock64() - t0 > 1000000000LL) {
            *failed = 1;
            return false;
        }
    }
    return true;
}

// The same for a whole warp: every lane gets the same answer.
__device__ __forceinline__ bool dg_wait_warp(uint64_t* bar, uint32_t parity, volatile int* failed) {
    return __all_sync(0xffffffffu, dg_wait(bar, parity, failed));
}

// Both barriers at once: two lanes poll, one each.
__device__ __forceinline__ bool dg_wait_both(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb, volatile int* failed) {
    const bool second = (threadIdx.x & 31) != 0;
    uint64_t* bar = second ? b : a;
    const uint32_t parity = second ? pb : pa;
    if (!__all_sync(0xffffffffu, (threadIdx.x & 30) || tc::mbar_try_wait(bar, parity)) &&
        !dg_wait_warp(bar, parity, failed))
        return false;
    __syncwarp();  // what either lane acquired, the issuing lane sees
    return true;
}

// F2's columns keep the two fields of COMPLEX data together: column -> (field, part).
__device__ __forceinline__ int dg_f2_field(const DgArgs& p, int col) {
    if (p.mode == kReal) return col;
    const int f = col >> 2, gh = (col >> 1) & 1;
    return ((gh * p.N + f) << 1) | (col & 1);
}

// What one lane of a data warp needs of an item: its two columns (8 apart).
struct DgLane {
    const void* src[2];  // null: no such column
    int par[2];          // FP64 F2: right shift; else exponent
    int n;               // K entries there are
    int vb;
};

template <int STAGE, int P>
__device__ __forceinline__ void dg_lane(const DgArgs& p, const DgTile& tl, int col0, DgLane& L) {
    using Real = typename Dg<P>::Real;
    using Int = typename Dg<P>::Int;
    L.vb = tl.vb;
    const int B = p.B;
    if constexpr (STAGE == kF1) L.n = tl.ks * 16;
    if constexpr (STAGE == kF2) L.n = B;
    if constexpr (STAGE == kI1) L.n = (B - tl.m - tl.t + 1) / 2;
    if constexpr (STAGE == kI2) L.n = tl.kind < 4 ? (B + 1 - tl.m) / 2 : B;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int col = col0 + 8 * c;
        L.src[c] = nullptr;
        L.par[c] = 0;
        if (col >= p.ncols) continue;
        if constexpr (STAGE == kF1) {
            L.src[c] = (const Int*)p.Z + (size_t)col * p.RL + tl.zoff;
        } else if constexpr (STAGE == kF2) {
            const size_t row = (size_t)dg_f2_field(p, col) * B + tl.m;
            L.src[c] = (const Int*)p.X + row * 2 * p.BP + tl.t * p.BP;  // Int and Real have one size
            L.par[c] = P == 64 ? max((int)p.emax[row] - tl.vb, 0) : max((int)p.emax[row], 1);
        } else if constexpr (STAGE == kI1) {
            const Real* x = (const Real*)((col & 1) ? p.in_i : p.in_r);
            if (tl.m || !(col & 1))  // a real field's Im f(l, 0) is ignored
                L.src[c] = x + (p.cmap ? (size_t)p.cmap[col >> 1] : (size_t)(col >> 1) * B * B) + index_of_harmonic_coeff(tl.m, tl.m + tl.t, B);
            L.par[c] = max((int)p.ein[(size_t)col * B + tl.m], 1);
        } else {
            const int f = col / p.S, rem = col - f * p.S, t = rem >= B, j = rem - t * B;
            L.src[c] = (const Real*)p.X + ((size_t)(f * 2 + tl.t) * B + tl.m) * 2 * p.BP + t * p.BP + j;
            L.par[c] = max((int)p.ein[f], 1);
        }
    }
}

// Loads entries k .. k + 3 of column c.
template <int STAGE, int P>
__device__ __forceinline__ void dg_load(const DgArgs& p, const DgTile& tl, const DgLane& L, int c, int k,
                                        typename Dg<P>::Int* v) {
    using Int = typename Dg<P>::Int;
    using Int2 = typename Dg<P>::Int2;
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = 0;
    if (!L.src[c] || k >= L.n) return;
    if constexpr (STAGE == kF1 || STAGE == kF2) {
        const Int2* x = (const Int2*)((const Int*)L.src[c] + k);  // rows start 16-byte aligned
        if constexpr (P == 32) {
            const int4 q = *(const int4*)x;
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        } else {
            const Int2 a = x[0], b = x[1];
            v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
        }
#pragma unroll
        for (int i = 1; i < 4; ++i)
            if (k + i >= L.n) v[i] = 0;
    } else {
        const size_t step = STAGE == kI1 ? 2 : (size_t)(tl.kind < 4 ? 2 : 1) * 2 * p.BP;
        const Int* x = (const Int*)L.src[c] + step * k;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (k + i < L.n) v[i] = __ldg(x + step * i);
    }
}

// Raw entry -> integer of at most vb bits.
template <int STAGE>
__device__ __forceinline__ long long dg_conv(int par, int vb, long long v) {
    if constexpr (STAGE == kF1) return v;
    if constexpr (STAGE == kF2) return par ? ((v >> (par - 1)) + 1) >> 1 : v;
    return dg_fix(__longlong_as_double(v), par, vb);
}
template <int STAGE>
__device__ __forceinline__ int dg_conv(int par, int vb, int v) {
    if constexpr (STAGE == kF1) return v;
    return dg_fix(__int_as_float(v), par, vb);
}

template <int STAGE, int NT, int P>
__global__ void __launch_bounds__(kDgThreads, 1) k_dg(DgArgs p) {
    using Real = typename Dg<P>::Real;
    using Int2 = typename Dg<P>::Int2;
    constexpr int DA = Dg<P>::DA, DB = Dg<P>::DB, G = Dg<P>::G, kDgStagesA = Dg<P>::stagesA;
    constexpr uint32_t kABytes = kDgABytes<P>;
    extern __shared__ __align__(1024) uint8_t dsm[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)dsm + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t fullA[kDgStagesA], emptyA[kDgStagesA], fullB[kDgMaxStagesB], emptyB[kDgMaxStagesB];
    __shared__ uint64_t accFull[2], accEmpty[2], drained;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    constexpr uint32_t accCols = G * NT;              // TMEM columns of one accumulator
    constexpr int kSlots = 2 * accCols > 512 ? 1 : 2;  // accumulators
    constexpr int kEW = Dg<P>::epilogue;              // epilogue warps: groups of four cover the rows
    constexpr int kEpi = kEW / 4 / kSlots, kCols = NT / kEpi;  // groups of an accumulator, columns of each
    constexpr int kLanes = kCols > 32 ? 32 : kCols, kHalf = kCols / kLanes;
    constexpr uint32_t stepB = DB * NT * 32, stageB = kSub * stepB;  // bytes of the data digits
    constexpr int nsb = kDgBRing / stageB < kDgMaxStagesB ? kDgBRing / stageB : kDgMaxStagesB;
    constexpr int W = NT / 16;                        // data warps per K step, W kSub per stage
    constexpr int groups = Dg<P>::data / (W * kSub);
    uint8_t* ringA = smem;
    uint8_t* ringB = smem + kDgStagesA * kABytes;
    [[maybe_unused]] float* stash0 = (float*)(ringB + kDgBRing);
    const uint32_t sdA0 = dg_desc(ringA), sdB0 = dg_desc(ringB);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        failed = 0;
        for (int i = 0; i < kDgStagesA; ++i) tc::mbar_init(&fullA[i], 1), tc::mbar_init(&emptyA[i], 1);
        for (int i = 0; i < nsb; ++i) tc::mbar_init(&fullB[i], W * kSub), tc::mbar_init(&emptyB[i], 1);
        for (int i = 0; i < 2; ++i) tc::mbar_init(&accFull[i], 1), tc::mbar_init(&accEmpty[i], kEpi * 4);
        tc::mbar_init(&drained, 1);
        tc::fence_mbar_init();
    }
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int nitems = p.ntiles * p.ncolblk;
    auto decode = [&](int it, int& tile, int& cb) {
        if (p.col_major) cb = it / p.ntiles, tile = it - cb * p.ntiles;
        else tile = it / p.ncolblk, cb = it - tile * p.ncolblk;
    };

    if (warp == 0) {
        if (lane == 0) {  // table digits
            uint32_t c = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < nitems && ok && !p.stall; it += gridDim.x) {
                int tile, cb;
                decode(it, tile, cb);
                const DgTile* tl = p.tiles + tile;
                const uint32_t bytes = DA * (uint32_t)tl->r8 * 32;
                const uint8_t* src = p.tab + tl->off;
                const int n = tl->ks;
                for (int k = tl->k0; k < n; k += kSub, ++c) {
                    const uint32_t slot = c % kDgStagesA, nb = min(kSub, n - k) * bytes;
                    if (!dg_wait(&emptyA[slot], ((c / kDgStagesA) & 1) ^ 1, &failed)) {
                        ok = false;
                        break;
                    }
                    tc::mbar_arrive_expect_tx(&fullA[slot], nb);
                    tc::bulk_g2s(ringA + slot * kABytes, src + (size_t)k * bytes, nb, &fullA[slot]);
                }
            }
            if (!ok)  // own copies still in flight land before the block ends
                for (uint32_t b = c >= kDgStagesA ? c - kDgStagesA : 0; b < c; ++b)
                    tc::mbar_wait(&fullA[b % kDgStagesA], (b / kDgStagesA) & 1);
        }
    } else if (warp == 1) {
        // MMAs: the whole warp runs the loop (its values stay warp-uniform), one elected lane issues
        const bool leader = tc::elect_one();
        uint32_t sa = 0, pa = 0, sb = 0, pb = 0, use[2] = {0, 0}, nit = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x, ++nit) {
            int tile, cb;
            decode(it, tile, cb);
            const DgTile* tl = p.tiles + tile;
            const uint32_t stepA = (uint32_t)__shfl_sync(0xffffffffu, tl->r8, 0) * 2;  // descriptor units of 16 B
            const int n = __shfl_sync(0xffffffffu, tl->ks - tl->k0, 0);
            const int s0 = kSlots == 1 ? 0 : (int)(nit & 1);
            ok = dg_wait_warp(&accEmpty[s0], (use[s0]++ & 1) ^ 1, &failed);
            tc::tc_fence_after();
            const uint32_t d0 = tmem + s0 * accCols;
            for (int k = 0; k < n && ok; k += kSub) {
                ok = dg_wait_both(&fullA[sa], pa, &fullB[sb], pb, &failed);
                if (!ok) break;
                tc::tc_fence_after();
                if (leader) {
                    uint32_t da = sdA0 + sa * (kABytes >> 4), db = sdB0 + sb * (stageB >> 4);
                    const int sub = min(kSub, n - k);
#pragma unroll
                    for (int j = 0; j < kSub; ++j) {
                        if (j >= sub) break;
#pragma unroll
                        for (int a = 0; a < DA; ++a) {
                            // groups a .. G - 1; an MMA takes at most 256 columns
                            constexpr uint32_t one = 1;
                            const uint32_t acc = a > 0 || j > 0 ? one : (uint32_t)(k > 0);
                            const int n1 = (G - a < DB ? G - a : DB) * NT, parts = n1 > 256 ? 2 : 1, np = n1 / parts;
                            const uint32_t idesc = tc::idesc_f16_f32(128, np);
#pragma unroll
                            for (int h = 0; h < parts; ++h)
                                dg_mma(d0 + a * NT + h * np, da + a * stepA, db + h * np * 2, idesc, acc);
                        }
                        da += DA * stepA;
                        db += stepB >> 4;
                    }
                    tc::mma_commit(&emptyA[sa]);
                    tc::mma_commit(&emptyB[sb]);
                }
                if (++sa == kDgStagesA) sa = 0, pa ^= 1;
                if (++sb == nsb) sb = 0, pb ^= 1;
            }
            if (ok && leader) tc::mma_commit(&accFull[s0]);
        }
        if (!ok && leader) {  // MMAs already issued end before the block gives up its memory
            tc::mma_commit(&drained);
            tc::mbar_wait(&drained, 0);
        }
    } else if (warp >= 4 + kEW) {  // data digits
        const int pw = warp - 4 - kEW, g = pw / (W * kSub), wi = pw % W, sub = pw / W % kSub;
        // this group's stages: every groups-th of the block's; this warp's K step of the next one is loaded
        // before the current one is turned into digits
        struct Step {
            int par[2], vb;
            typename Dg<P>::Int v[2][4];
        };
        int it = blockIdx.x, ks = 0, tile, cb;
        uint32_t c = 0;
        DgTile tl{};
        DgLane L{};
        auto enter = [&]() {  // per-item state
            decode(it, tile, cb);
            tl = p.tiles[tile];
            dg_lane<STAGE, P>(p, tl, cb * NT + wi * 16 + (lane & 7), L);
        };
        auto skip = [&](int n) {  // n stages on; false past the last item
            ks += n * kSub;
            c += n;
            bool moved = false;
            while (it < nitems && ks >= tl.ks) {
                const int over = (ks - tl.ks) / kSub;  // stages into the next item
                it += gridDim.x;
                moved = true;
                if (it < nitems) {
                    int t2, c2;
                    decode(it, t2, c2);
                    tl.ks = p.tiles[t2].ks;
                    ks = p.tiles[t2].k0 + over * kSub;
                }
            }
            if (it >= nitems) return false;
            if (moved) enter();
            return true;
        };
        auto fetch = [&](Step& x) {
            x.vb = L.vb;
#pragma unroll
            for (int h = 0; h < 2; ++h) x.par[h] = L.par[h];
#pragma unroll
            for (int h = 0; h < 2; ++h) dg_load<STAGE, P>(p, tl, L, h, (ks + sub) * 16 + (lane >> 3) * 4, x.v[h]);
        };
        bool more = it < nitems;
        if (more) {
            enter();
            ks = tl.k0;
            more = skip(g);
        }
        Step cur{};
        if (more) fetch(cur);
        while (more) {
            const uint32_t cc = c;
            more = skip(groups);
            Step nxt{};
            if (more) fetch(nxt);
            const uint32_t slot = cc % nsb;
            if (!dg_wait_warp(&emptyB[slot], ((cc / nsb) & 1) ^ 1, &failed)) break;
            uint8_t* dst = ringB + slot * stageB + sub * stepB;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                typename Dg<P>::Int v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = dg_conv<STAGE>(cur.par[h], cur.vb, cur.v[h][i]);
                // eight columns of a core matrix by four runs of K entries: half a warp covers 128 bytes
                dg_store4<NT>(dst + (wi * 2 + h) * 256 + (lane >> 4) * 128 + (lane & 7) * 16 + ((lane >> 3) & 1) * 8, v);
            }
            tc::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&fullB[slot]);
            cur = nxt;
        }
    } else if (warp >= 4) {  // epilogue
        const int slot = kSlots == 1 ? 0 : ((warp - 4) >> 2) / kEpi, grp = ((warp - 4) >> 2) % kEpi, ew = warp & 3;
        const uint32_t lane_off = (uint32_t)(ew * 32) << 16;
        const int B = p.B, S = p.S;
        uint32_t nit = 0, use = 0;
        for (int it = blockIdx.x; it < nitems; it += gridDim.x, ++nit) {
            if (kSlots == 2 && (int)(nit & 1) != slot) continue;
            int tile, cb;
            decode(it, tile, cb);
            const DgTile tl = p.tiles[tile];
            const int r = ew * 32 + lane;
            const bool live = r < tl.nrows;
            const int row = tl.row0 + r;
            const int qrow = live ? p.q[tl.qoff + row] : 0;
            const float rscale = P == 32 && live ? ldexpf(1.0f, tl.tb - qrow) : 0.0f;
            // lane c holds what the rows need to know of column c (of 32): field, place in X, exponent or
            // shift, and for FP32 the column's unit
            int cfield_[kHalf], cpar_[kHalf];
            uint32_t coff_[kHalf];
            float cscale_[kHalf];
#pragma unroll
            for (int h = 0; h < kHalf; ++h) {
                int cfield = 0, cpar = 0;
                uint32_t coff = 0;
                float cscale = 0.0f;
                const int col = cb * NT + grp * kCols + h * 32 + lane;
                if (lane < kLanes && col < p.ncols) {
                    if constexpr (STAGE == kF1) {
                        cfield = col / S;
                        const int rem = col - cfield * S, t = rem >= B, j = rem - t * B;
                        if constexpr (P == 64) cpar = min(max((int)p.efield[cfield], 1) - max((int)p.ein[cfield * B + j], 1), 63);
                        else cscale = dg_col_scale(p.ein[cfield * B + j], tl.tb, p.vbz);
                        coff = (uint32_t)(cfield * 2 + tl.t) * B * 2 * p.BP + t * p.BP + j;
                    } else if constexpr (STAGE == kF2) {
                        const int fp = dg_f2_field(p, col);
                        if constexpr (P == 32) cscale = dg_col_scale(p.emax[(size_t)fp * B + tl.m], tl.tb, tl.vb);
                        else cpar = dg_eb(p.efield[fp >> 1], 176 - p.tbz - p.vbz + max((int)p.emax[(size_t)fp * B + tl.m] - tl.vb, 0));
                    } else if constexpr (STAGE == kI1) {
                        if constexpr (P == 32) cscale = dg_col_scale(p.ein[(size_t)col * B + tl.m], tl.tb, tl.vb);
                        else cpar = dg_eb(p.ein[(size_t)col * B + tl.m], 120 - tl.vb);
                    } else if constexpr (P == 32) {
                        cscale = dg_col_scale(p.ein[col / S], tl.tb, tl.vb);
                    }
                }
                cfield_[h] = cfield, cpar_[h] = cpar, coff_[h] = coff, cscale_[h] = cscale;
            }
            if (!dg_wait_warp(&accFull[slot], use & 1, &failed)) break;
            ++use;
            tc::tc_fence_after();
            constexpr int CH = 4;  // columns at a time
#pragma unroll
            for (int h = 0; h < kHalf; ++h) {
            const int cfield = cfield_[h], cpar = cpar_[h];
            const uint32_t coff = coff_[h];
            [[maybe_unused]] const float cscale = cscale_[h];
            const int colb = cb * NT + grp * kCols + h * 32;
            const int ncol = min(kLanes, p.ncols - colb);  // may be negative
            const uint32_t tb = tmem + lane_off + slot * accCols + grp * kCols + h * 32;
            uint32_t mx = 0;
#pragma unroll 1
            for (int c0 = 0; c0 < ncol; c0 += CH) {
                uint32_t a[G * CH];
#pragma unroll
                for (int d = 0; d < G; ++d) tm_ld4(tb + d * NT + c0, &a[d * CH]);
                tm_wait();
                Real v[CH];
                long long T[CH];
                if constexpr (P == 32) {
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        float x = __uint_as_float(a[(G - 1) * CH + c]);
#pragma unroll
                        for (int d = G - 2; d >= 0; --d) x = fmaf(x, 0.00390625f, __uint_as_float(a[d * CH + c]));
                        v[c] = x * __shfl_sync(0xffffffffu, cscale, (c0 + c) & 31) * rscale;
                    }
                } else {
                    uint32_t odd = 0;
#pragma unroll
                    for (int c = 0; c < CH; ++c) T[c] = dg_sum(&a[c], CH, odd);
                    if (odd & 0xff800000u) {
#pragma unroll
                        for (int c = 0; c < CH; ++c)
                            T[c] = dg_sum_big(__uint_as_float(a[c]), __uint_as_float(a[CH + c]), __uint_as_float(a[2 * CH + c]),
                                              __uint_as_float(a[3 * CH + c]), __uint_as_float(a[4 * CH + c]),
                                              __uint_as_float(a[5 * CH + c]), __uint_as_float(a[6 * CH + c]));
                    }
                    if constexpr (STAGE == kF2 || STAGE == kI1) {
                        bool bad = false;
                        int eb[CH];
#pragma unroll
                        for (int c = 0; c < CH; ++c) {
                            eb[c] = __shfl_sync(0xffffffffu, cpar, (c0 + c) & 31) - qrow;
                            v[c] = dg_fast(T[c], eb[c], bad);
                        }
                        if (bad)
#pragma unroll
                            for (int c = 0; c < CH; ++c) v[c] = dg_slow(T[c], eb[c]);
                    }
                }
                const int col0 = colb + c0, nc = ncol - c0;  // columns of this chunk: min(CH, nc)
                if constexpr (STAGE == kF1) {
                    // FP64: integers in the scale of the function
                    const int m = (tl.kind < 4 ? 2 : 1) * row + tl.m;
                    const size_t xm = (size_t)m * 2 * p.BP;
                    const int fa = __shfl_sync(0xffffffffu, cfield, c0 & 31);
                    const int fb = __shfl_sync(0xffffffffu, cfield, (c0 + min(CH - 1, nc - 1)) & 31);
                    uint32_t x[CH], o[CH];  // sizes for the row's largest, places
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        o[c] = __shfl_sync(0xffffffffu, coff, (c0 + c) & 31);
                        if constexpr (P == 64) {
                            T[c] >>= __shfl_sync(0xffffffffu, cpar, (c0 + c) & 31);
                            x[c] = 64u - (uint32_t)__clzll(T[c] < 0 ? -T[c] : T[c]);
                        } else {
                            x[c] = dexp(v[c]);
                        }
                        if (c >= nc) x[c] = 0;
                    }
                    if constexpr (P == 64) {
                        long long* X = (long long*)p.X + xm;
                        if ((B & 1) == 0) {
#pragma unroll
                            for (int c = 0; c < CH; c += 2)
                                if (live && c < nc) *(longlong2*)(X + o[c]) = make_longlong2(T[c], T[c + 1]);
                        } else {
#pragma unroll
                            for (int c = 0; c < CH; ++c)
                                if (live && c < nc) X[o[c]] = T[c];
                        }
                    } else if ((B & 3) == 0) {
                        if (live) *(float4*)((float*)p.X + xm + o[0]) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
                        float* stash = stash0 + (warp - 4) * (kDgStash / 4) + lane * 33 + c0;
#pragma unroll
                        for (int c = 0; c < CH; ++c) stash[c] = v[c];
                    }
                    if (fa == fb) {
#pragma unroll
                        for (int c = 0; c < CH; ++c) mx = max(mx, x[c]);
                        const int fn = c0 + CH < ncol ? __shfl_sync(0xffffffffu, cfield, (c0 + CH) & 31) : -1;
                        if (fn != fa) {
                            if (live) atomicMax(p.emax + (size_t)(fa * 2 + tl.t) * B + m, mx);
                            mx = 0;
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < CH; ++c) {
                            const int f = __shfl_sync(0xffffffffu, cfield, (c0 + c) & 31);
                            mx = max(mx, x[c]);
                            if (live && c < nc) atomicMax(p.emax + (size_t)(f * 2 + tl.t) * B + m, mx);
                            const int fn = __shfl_sync(0xffffffffu, cfield, (c0 + c + 1) & 31);
                            if (fn != f) mx = 0;
                        }
                    }
                } else if constexpr (STAGE == kF2) {
                    const int m = tl.m, l = m + tl.t + 2 * row;
                    const bool modd = (m & 1) != 0;
                    const int i0 = index_of_harmonic_coeff(m, l, B), i1 = index_of_harmonic_coeff(-m, l, B);
                    if (p.mode == kReal) {
#pragma unroll
                        for (int c = 0; c < CH; c += 2) {
                            const int f = (col0 + c) >> 1;
                            if (live && c < nc) {
                                const size_t fb = p.cmap ? (size_t)p.cmap[f] : (size_t)f * B * B;
                                Real* qr = (Real*)p.out_r + fb;
                                Real* qi = (Real*)p.out_i + fb;
                                qr[i0] = v[c];
                                qi[i0] = v[c + 1];
                                if (m) {
                                    qr[i1] = modd ? -v[c] : v[c];
                                    qi[i1] = modd ? v[c + 1] : -v[c + 1];
                                }
                            }
                        }
                    } else {
                        Real* qr = (Real*)p.out_r + (size_t)(col0 >> 2) * B * B;
                        Real* qi = (Real*)p.out_i + (size_t)(col0 >> 2) * B * B;
#pragma unroll
                        for (int c = 0; c < CH; c += 4) {
                            const Real gr = v[c], gi = v[c + 1], hr = v[c + 2], hi = v[c + 3];
                            if (live && c < nc) {
                                const Real vr = gr - hi, vi = gi + hr;
                                qr[i0] = vr;
                                qi[i0] = vi;
                                if (m) {
                                    const Real nr = p.mode == kCplx ? gr + hi : vr;
                                    const Real ni = p.mode == kCplx ? hr - gi : -vi;
                                    qr[i1] = modd ? -nr : nr;
                                    qi[i1] = modd ? -ni : ni;
                                }
                            }
                            qr += B * B;
                            qi += B * B;
                        }
                    }
                } else if constexpr (STAGE == kI1) {
                    Real* X = (Real*)p.X + ((size_t)col0 * B + tl.m) * 2 * p.BP + tl.t * p.BP + row;
                    const size_t step = (size_t)B * 2 * p.BP;
                    uint32_t x[CH];
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        if (live && c < nc) X[c * step] = v[c];
                        x[c] = live ? dexp(v[c]) : 0;
                    }
                    // exponent of the field: lane c / 2 ends with that of columns c, c + 1
#pragma unroll
                    for (int c = 0; c < CH; c += 2) {
                        const uint32_t y = __reduce_max_sync(0xffffffffu, max(x[c], x[c + 1]));
                        if (lane == c / 2) mx = y;
                    }
                    if (lane < CH / 2 && 2 * lane < nc) atomicMax(p.emax + (col0 >> 1) + lane, mx);
                } else {
                    const size_t z = (size_t)col0 * p.RL + tl.zoff + row;
#pragma unroll
                    for (int c = 0; c < CH; ++c)
                        if (live && c < nc) {
                            if constexpr (P == 32) ((float*)p.Z)[z + (size_t)c * p.RL] = v[c];
                            else ((long long*)p.Z)[z + (size_t)c * p.RL] = (T[c] + 2) >> kDgOutShift;
                        }
                }
            }
            if (P == 32 && STAGE == kF1 && (B & 3) != 0) {
                // rows that no float4 fits: a row's columns are consecutive latitudes, stored as whole lines
                // (bw 255, 64 functions: 144 us with a thread's scalar stores, 107 so)
                __syncwarp();
                const float* stash = stash0 + (warp - 4) * (kDgStash / 4) + lane;
                const int rows = min(32, tl.nrows - ew * 32), row0 = tl.row0 + ew * 32;
                float* X = (float*)p.X + coff;
#pragma unroll 4
                for (int i = 0; i < rows; ++i)
                    if (lane < ncol) X[(size_t)((tl.kind < 4 ? 2 : 1) * (row0 + i) + tl.m) * 2 * p.BP] = stash[i * 33];
                __syncwarp();
            }
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&accEmpty[slot]);
        }
    }
    __syncwarp();
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
        if (lane == 0 && failed) *(volatile int*)p.err = S2G_ERR_TIMEOUT;
    }
}

// ------------------------------------------------------------------------------------
// Folded longitudes: where value k of fold kd lies in a column, and the column's length.
struct DgFold {
    int n[6], off[6], len;  // entries, place and total (padded to the K steps)
};
// Rows of 2B samples fold twice where B is even and from 128 on: four tables of B/2 orders, a quarter of the DFT
// matrix.  Below, one tile of 128 rows holds all orders, or all B + 1 longitudes of a fold, and a second fold
// would halve the rows a tile uses along with its K, at twice the epilogues and a pass more (bw 100, 1024
// functions, FP32: once F1 179 us, I2 168; twice 263, 228 and k_dg_mid 15).
static bool dg_twice(int B) { return B % 2 == 0 && B >= 128; }
static DgFold dg_fold_layout(int B, bool inv) {
    DgFold f{};
    const int h = B / 2;
    auto put = [&](int kd, int n) {
        f.n[kd] = n;
        f.off[kd] = f.len;
        f.len += (n + 15) & ~15;
    };
    if (dg_twice(B)) {
        // inverse: the cosines of even orders at longitude index B/2 come from k_dg_mid
        put(0, inv ? h : h + 1);
        for (int kd = 1; kd < 4; ++kd) put(kd, h);
    } else {
        put(4, B + 1);
        put(5, B - 1);
    }
    return f;
}

// Latitudes j and 2B-1-j of one field -> fixed point (|x| < 2^vb, scale in e[field][j]) -> even and odd
// latitude parts of the folded rows, Z[field][t][j][..].  One block per (j, field), a thread for every kDgFoldV
// samples: they are all loaded before the first is used and stay in registers until the scale is known (with a
// loop over shared memory instead, loads waited for one another: bw 256, 64 functions 67 us against 52, bw 1024, 16
// functions 406 against 204, bw 255, 64 functions in FP32 54 against 39).
constexpr int kDgFoldV = 8;
static int dg_fold_threads(int S) { return std::max(64, ((2 * S + kDgFoldV - 1) / kDgFoldV + 31) & ~31); }  // 512 at bw 1024
template <int P>
__global__ void __launch_bounds__(512) k_dg_fold(const typename Dg<P>::Real* __restrict__ r,
                                                 const typename Dg<P>::Real* __restrict__ im, int B, int N, int vb,
                                                 DgFold fl, const int64_t* __restrict__ gmap, typename Dg<P>::Int* Z,
                                                 uint32_t* e, uint32_t* ef) {
    using Real = typename Dg<P>::Real;
    using Int = typename Dg<P>::Int;
    extern __shared__ __align__(16) uint8_t fold_sm[];  // [2][S]
    Int* rows = reinterpret_cast<Int*>(fold_sm);
    __shared__ uint32_t red[16];
    const int S = 2 * B, j = blockIdx.x, ff = blockIdx.y;
    const Real* g = gmap ? r + gmap[ff] : ff < N ? r + (size_t)ff * S * S : im + (size_t)(ff - N) * S * S;
    const Real *x0 = g + (size_t)j * S, *x1 = g + (size_t)(S - 1 - j) * S - S;
    uint32_t mx = 0;
    Real v[kDgFoldV];
#pragma unroll
    for (int u = 0; u < kDgFoldV; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        v[u] = i < 2 * S ? (i < S ? x0 : x1)[i] : Real(0);
    }
#pragma unroll
    for (int u = 0; u < kDgFoldV; ++u) mx = max(mx, dexp(v[u]));
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = red[0];
    for (int q = 1; q < (int)blockDim.x >> 5; ++q) mx = max(mx, red[q]);
    if (threadIdx.x == 0) {
        e[ff * B + j] = mx;
        atomicMax(ef + ff, mx);
    }
    const int em = max((int)mx, 1);
#pragma unroll
    for (int u = 0; u < kDgFoldV; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        if (i < 2 * S) rows[i] = dg_fix(v[u], em, vb);
    }
    __syncthreads();
    Int* z0 = Z + ((size_t)ff * S + j) * fl.len;
    Int* z1 = z0 + (size_t)B * fl.len;
    const Int* a = rows;
    const Int* b = rows + S;
    auto both = [&](int at, Int u, Int w) {
        z0[at] = u + w;
        z1[at] = u - w;
    };
    if (fl.n[0]) {
        const int h = B / 2, pad = ((h + 1 + 15) & ~15);
        for (int k = threadIdx.x; k < pad; k += blockDim.x) {
            Int c[2][4] = {};
            if (k <= h) {
                const int ks = k ? S - k : 0;
                const Int* row[2] = {a, b};
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const Int p0 = row[q][k], p1 = row[q][ks], p2 = row[q][B - k], p3 = row[q][B + k];
                    c[q][0] = (p0 + p1) + (p2 + p3);
                    c[q][1] = (p0 + p1) - (p2 + p3);
                    c[q][2] = (p0 - p1) - (p2 - p3);
                    c[q][3] = (p0 - p1) + (p2 - p3);
                }
            }
            const int hp = (h + 15) & ~15;
            both(fl.off[0] + k, c[0][0], c[1][0]);
            if (k < hp) {
                const bool in = k < h;
                both(fl.off[1] + k, in ? c[0][1] : 0, in ? c[1][1] : 0);
                both(fl.off[2] + k, in ? c[0][2] : 0, in ? c[1][2] : 0);
            }
            // the sines of odd orders run over k = 1 .. h; their padding follows
            if (k >= 1 && k <= h) both(fl.off[3] + k - 1, c[0][3], c[1][3]);
            if (k >= h && k < hp) both(fl.off[3] + k, 0, 0);
        }
    } else {
        const int pad = ((B + 1 + 15) & ~15), sp = ((B - 1 + 15) & ~15);
        for (int k = threadIdx.x; k < pad; k += blockDim.x) {
            Int u0 = 0, u1 = 0, w0 = 0, w1 = 0;
            if (k <= B) {
                const int ks = k ? S - k : 0;
                u0 = a[k] + a[ks];
                w0 = b[k] + b[ks];
                u1 = a[k] - a[ks];
                w1 = b[k] - b[ks];
            }
            both(fl.off[4] + k, u0, w0);
            if (k >= 1 && k < B) both(fl.off[5] + k - 1, u1, w1);
            if (k >= B - 1 && k < sp) both(fl.off[5] + k, 0, 0);
        }
    }
}

// Inverse, even B: sum over the even orders of c_m (-1)^(m/2) Re F_m, the cosine part at longitude index
// B/2, for every column of I2.
template <class Real>
__global__ void __launch_bounds__(256) k_dg_mid(const Real* __restrict__ X, int B, int ncols, Real* mid) {
    __shared__ Real part[8][33];
    const int col = blockIdx.x * 32 + threadIdx.x, S = 2 * B;  // 32 columns, eight runs of orders
    const int nb = (B + 3) / 4, per = (nb + 7) / 8;
    Real s = 0;
    if (col < ncols) {
        const int f = col / S, rem = col - f * S;
        const int BP = (B + 3) & ~3, t = rem >= B;
        const Real* x = X + (size_t)(f * 2) * B * 2 * BP + t * BP + (rem - t * B);
        const int b1 = min(nb, (int)(threadIdx.y + 1) * per);
#pragma unroll 4
        for (int b = threadIdx.y * per; b < b1; ++b) {
            const int m = 4 * b;
            s += x[(size_t)m * 2 * BP] - (m + 2 < B ? x[(size_t)(m + 2) * 2 * BP] : Real(0));
        }
    }
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && col < ncols) {
        for (int q = 1; q < 8; ++q) s += part[q][threadIdx.x];
        const int f = col / S, rem = col - f * S, BP = (B + 3) & ~3, t = rem >= B;
        mid[col] = (2 * s - X[(size_t)(f * 2) * B * 2 * BP + t * BP + (rem - t * B)]) * Real(0.39894228040143267794);
    }
}

// Parts of I2 -> samples of latitudes j and 2B-1-j.  One block per (j, field).
template <int P>
__global__ void __launch_bounds__(128, P == 64 ? 10 : 16) k_dg_unfold(const void* __restrict__ Zv, const typename Dg<P>::Real* __restrict__ mid,
                                                   const uint32_t* __restrict__ ef, int B, int N, int qv, DgFold fl,
                                                   const int64_t* __restrict__ gmap, typename Dg<P>::Real* r, typename Dg<P>::Real* im) {
    using Real = typename Dg<P>::Real;
    using Part = std::conditional_t<P == 64, long long, float>;
    const Part* Z = (const Part*)Zv;
    const int S = 2 * B, j = blockIdx.x, ff = blockIdx.y;
    Real* g = gmap ? r + gmap[ff] : ff < N ? r + (size_t)ff * S * S : im + (size_t)(ff - N) * S * S;
    Real* out[2] = {g + (size_t)j * S, g + (size_t)(S - 1 - j) * S};
    const Part* z0 = Z + ((size_t)ff * S + j) * fl.len;
    const Part* z1 = z0 + (size_t)B * fl.len;
    [[maybe_unused]] const int eb = P == 64 ? dg_eb(ef[ff], 120 + kDgOutShift - qv) : 0;  // qv: bits of table and data values
    auto value = [&](Part T) -> Real {
        if constexpr (P == 32) {
            return T;
        } else {
            bool bad = false;
            const double v = dg_fast(T, eb, bad);
            return bad ? dg_slow(T, eb) : v;
        }
    };
    auto put = [&](int k, Part u, Part w) {  // even and odd latitude parts
        out[0][k] = value(u + w);
        out[1][k] = value(u - w);
    };
    if (fl.n[0]) {
        const int h = B / 2;
        for (int k = threadIdx.x; k < h; k += blockDim.x) {
            Part c[2], d[2], s[2], q[2];
            const Part* z[2] = {z0, z1};
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const Part ce = z[t][fl.off[0] + k], co = z[t][fl.off[1] + k];
                const Part se = k ? z[t][fl.off[2] + k] : 0, so = k ? z[t][fl.off[3] + k - 1] : 0;
                c[t] = ce + co;
                d[t] = ce - co;
                s[t] = se + so;
                q[t] = so - se;
            }
            put(k, c[0] + s[0], c[1] + s[1]);
            put(B + k, d[0] - q[0], d[1] - q[1]);
            if (k) {
                put(S - k, c[0] - s[0], c[1] - s[1]);
                put(B - k, d[0] + q[0], d[1] + q[1]);
            }
        }
        if (threadIdx.x < 2) {  // k = B/2 and 3B/2
            const Real sg = threadIdx.x ? -1 : 1;
            const Real m0 = mid[(size_t)ff * S + j], m1 = mid[(size_t)ff * S + B + j];
            const Real s0 = value(z0[fl.off[3] + h - 1]), s1 = value(z1[fl.off[3] + h - 1]);
            const int k = threadIdx.x ? B + h : h;
            out[0][k] = (m0 + m1) + sg * (s0 + s1);
            out[1][k] = (m0 - m1) + sg * (s0 - s1);
        }
    } else {
        for (int k = threadIdx.x; k <= B; k += blockDim.x) {
            const Part c0 = z0[fl.off[4] + k], c1 = z1[fl.off[4] + k];
            const bool in = k >= 1 && k < B;
            const Part s0 = in ? z0[fl.off[5] + k - 1] : 0, s1 = in ? z1[fl.off[5] + k - 1] : 0;
            put(k, c0 + s0, c1 + s1);
            if (in) put(S - k, c0 - s0, c1 - s1);
        }
    }
}

// Largest exponent of every order's coefficients (I1), e[field, part][m]; COMPLEX data, and REAL data with an
// imaginary output, are first split into two real fields' coefficients (cr, ci, orders m >= 0):
//   g = (a + s conj b) / 2, h = (a - s conj b) / 2i with a = f(l,m), b = f(l,-m), s = (-1)^m.
// One warp per (function, order).
template <class Real>
__global__ void k_dg_coefmax(const Real* __restrict__ rc, const Real* __restrict__ ic, int B, int N, int mode,
                             const int64_t* __restrict__ cmap, Real* cr, Real* ci, uint32_t* e) {
    const int id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (id >= N * B) return;
    const int f = id / B, m = id - f * B;
    const size_t cb = cmap ? (size_t)cmap[f] : (size_t)f * B * B, hb = (size_t)(N + f) * B * B;
    uint32_t mx[4] = {0, 0, 0, 0};
    for (int l = m + lane; l < B; l += 32) {
        const int i = index_of_harmonic_coeff(m, l, B);
        const Real ar = rc[cb + i], ai = ic[cb + i];
        if (mode == kReal) {
            mx[0] = max(mx[0], dexp(ar));
            if (m) mx[1] = max(mx[1], dexp(ai));
            continue;
        }
        Real v[4] = {ar, m ? ai : Real(0), m ? Real(0) : ai, 0};  // Im f(l, 0) is the second field's
        if (mode == kCplx && m) {
            const int k = index_of_harmonic_coeff(-m, l, B);
            const Real s = (m & 1) ? -1 : 1, br = s * rc[cb + k], bi = s * ic[cb + k];
            v[0] = Real(0.5) * ar + Real(0.5) * br;
            v[1] = Real(0.5) * ai - Real(0.5) * bi;
            v[2] = Real(0.5) * ai + Real(0.5) * bi;
            v[3] = Real(0.5) * br - Real(0.5) * ar;
        }
        cr[cb + i] = v[0];
        ci[cb + i] = v[1];
        cr[hb + i] = v[2];
        ci[hb + i] = v[3];
#pragma unroll
        for (int q = 0; q < 4; ++q) mx[q] = max(mx[q], dexp(v[q]));
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) mx[q] = __reduce_max_sync(0xffffffffu, mx[q]);
    if (lane) return;
    e[(size_t)(2 * f) * B + m] = mx[0];
    e[(size_t)(2 * f + 1) * B + m] = mx[1];
    if (mode != kReal) {
        e[(size_t)(2 * (N + f)) * B + m] = mx[2];
        e[(size_t)(2 * (N + f) + 1) * B + m] = mx[3];
    }
}

// ------------------------------------------------------------------------------------
// Tables.  P(m,l)(x_j) by the three-term recurrence in double-double arithmetic, rounded to
// double once, so that the digits carry the table to its last place.
struct dd {
    double h, l;
};
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
    const double p = a.h * b.h;
    const double e = fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h);
    const double s = p + e;
    return {s, e - (s - p)};
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
    const double s = a.h + b.h, t = s - a.h;
    const double e = (a.h - (s - t)) + (b.h - t) + (a.l + b.l);
    const double r = s + e;
    return {r, e - (r - s)};
}
// sqrt(n / d) for integers n, d held exactly
__device__ __forceinline__ dd dd_sqrt_ratio(double n, double d) {
    if (n == 0.0) return {0.0, 0.0};
    const double q = n / d, q1 = fma(-q, d, n) / d;
    const double s = sqrt(q), e = (fma(-s, s, q) + q1) / (2.0 * s);
    const double r = s + e;
    return {r, e - (r - s)};
}

// One block per order m0 + blockIdx.x: rows l - m of P at the B northern nodes into tmp + off[blockIdx.x].
__global__ void k_dg_legendre(int B, int m0, const double2* __restrict__ cosn, const double2* __restrict__ sinn,
                              const double2* __restrict__ seed, double* tmp, const int64_t* __restrict__ off) {
    extern __shared__ double2 ac[];  // [B] a, [B] c
    const int m = m0 + blockIdx.x;
    for (int l = m + threadIdx.x; l < B; l += blockDim.x) {
        const double d = (l + 1.0 - m) * (l + 1.0 + m);
        const dd a = dd_sqrt_ratio((2.0 * l + 3.0) * (2.0 * l + 1.0), d);
        dd c{0.0, 0.0};
        if (l > m) c = dd_sqrt_ratio((2.0 * l + 3.0) * (double)(l - m) * (l + m), (2.0 * l - 1.0) * d);
        ac[l] = make_double2(a.h, a.l);
        ac[B + l] = make_double2(-c.h, -c.l);
    }
    __syncthreads();
    double* out = tmp + off[blockIdx.x];
    for (int j = threadIdx.x; j < B; j += blockDim.x) {
        const dd x{cosn[j].x, cosn[j].y};
        dd cur{seed[m].x, seed[m].y}, prev{0.0, 0.0}, b{sinn[j].x, sinn[j].y};
        for (int e = m; e; e >>= 1) {  // sin^m
            if (e & 1) cur = dd_mul(cur, b);
            b = dd_mul(b, b);
        }
        for (int l = m; l < B; ++l) {
            out[(size_t)(l - m) * B + j] = cur.h;
            const dd a{ac[l].x, ac[l].y}, c{ac[B + l].x, ac[B + l].y};
            const dd nx = dd_add(dd_mul(a, dd_mul(x, cur)), dd_mul(c, prev));
            prev = cur;
            cur = nx;
        }
    }
}

// Rows of an odd order m as the forward seminaive transform applies them (seminaive.c:170-197): the
// order's cosine series (cospml.c:161-242), evaluated at the nodes and times sin.  One block per degree.
__global__ void k_dg_seminaive(int B, int m, const double* __restrict__ T, const double2* __restrict__ tw4S,
                               double* out) {
    const int S = 2 * B, l = m + blockIdx.x, t = (l - m) & 1, n = row_size(m, l);
    const double* row = T + table_offset(m, l);
    const double nrm = 2.0 / sqrt(2.0 * S);
    for (int j = threadIdx.x; j < B; j += blockDim.x) {
        dd acc{0.0, 0.0};
        int r = (int)((long long)t * (2 * j + 1) % (4 * S));  // angle k (2j + 1) pi / 2S, k = t, t + 2, ..
        const int step = (4 * j + 2) % (4 * S);
        for (int i = 0; i < n; ++i) {
            const double a = row[i] * ((2 * i + t) ? nrm : nrm * 0.70710678118654752440), c = tw4S[r].x;
            const double q = a * c;
            acc = dd_add(acc, {q, fma(a, c, -q)});
            r += step;
            if (r >= 4 * S) r -= 4 * S;
        }
        out[(size_t)(l - m) * B + j] = acc.h * sinpi((2.0 * j + 1.0) / (2.0 * S));
    }
}

// Scale of a row whose largest value is mx: 2^(tb-1) <= mx 2^q < 2^tb.
__device__ __forceinline__ int dg_scale(double mx, int tb) {
    if (!(mx > 0.0)) return 0;
    int e;
    frexp(mx, &e);
    return tb - e;
}

// Digits of one 8-row group; 128 threads = 8 rows x 16 K entries per step.  val(row, k): the table value.
template <int P, class Val>
__device__ __forceinline__ int dg_pack_rows(Val val, int q, uint8_t* blob, int r8, int ks, int rg) {
    const int r = threadIdx.x >> 4, kk = threadIdx.x & 15;
    constexpr int DA = Dg<P>::DA;
    const uint32_t bytes = DA * (uint32_t)r8 * 32;
    int first = ks;  // this thread's first step with a nonzero value
    for (int s = 0; s < ks; ++s) {
        const double x = val(r, s * 16 + kk);
        const long long v = __double2ll_rn(scalbn(x, q));
        if (v && first == ks) first = s;
        const unsigned long long u = (unsigned long long)v + (P == 64 ? 0x0200808080808080ull : 0x02008080ull);
        uint8_t* d = blob + (size_t)s * bytes + rg * 256 + (kk >> 3) * 128 + r * 16 + (kk & 7) * 2;
#pragma unroll
        for (int a = 0; a < DA; ++a)
            *(__half*)(d + (size_t)a * r8 * 32) =
                __int2half_rn(a ? (int)((u >> (8 * (DA - 1 - a))) & 255) - 128 : (int)(u >> (8 * DA - 8)) - 512);
    }
    return first;
}

// A node's row of the inverse that is below this anywhere (2^-64 of the order's largest values) is zero.
constexpr double kDgTiny = 5.4e-20;

// Legendre tables of the orders m0 ..: one block per (tile, 8-row group); tiles of kind F2 (rows degrees,
// weighted) or I1 (rows nodes).
template <int P>
__global__ void __launch_bounds__(128) k_dg_pack_leg(int B, int fwd, const DgTile* __restrict__ tiles, int m0,
                                                     const double* __restrict__ tmp, const int64_t* __restrict__ off,
                                                     const double* __restrict__ w, double wscale, uint8_t* tab,
                                                     short* qs, int* first) {
    __shared__ double red[8][17];
    const DgTile tl = tiles[blockIdx.x];
    const int rg = blockIdx.y;
    if (rg * 8 >= tl.r8) return;
    const double* leg = tmp + off[tl.m - m0];
    const int nl = (B - tl.m - tl.t + 1) / 2;  // degrees of this parity
    auto val = [&](int r, int k) -> double {
        const int row = tl.row0 + rg * 8 + r;
        if (rg * 8 + r >= tl.nrows) return 0.0;
        if (fwd) return k < B ? leg[(size_t)(tl.t + 2 * row) * B + k] * (w[k] * wscale) : 0.0;
        return k < nl ? leg[(size_t)(tl.t + 2 * k) * B + row] : 0.0;
    };
    const int r = threadIdx.x >> 4, kk = threadIdx.x & 15;
    double mx = 0.0;
    for (int s = 0; s < tl.ks; ++s) mx = fmax(mx, fabs(val(r, s * 16 + kk)));
    red[r][kk] = mx;
    __syncthreads();
    for (int q = 0; q < 16; ++q) mx = fmax(mx, red[r][q]);
    const bool tiny = !fwd && mx < kDgTiny;
    const int q = tiny ? 0 : dg_scale(mx, tl.tb);
    if (kk == 0 && rg * 8 + r < tl.nrows) qs[tl.qoff + tl.row0 + rg * 8 + r] = (short)q;
    const int f = dg_pack_rows<P>([&](int a, int k) { return tiny ? 0.0 : val(a, k); }, q, tab + tl.off, tl.r8, tl.ks, rg);
    atomicMin(first + blockIdx.x, f);
}

// On-the-fly family: the same tables, a chunk of orders at a time in scratch, from what a plan keeps per
// (order, degree) and (order, node): the recurrence's coefficients ac and the first row P(m,m).
__global__ void k_dg_fly_init(int B, const double2* __restrict__ sinn, const double2* __restrict__ seed, double2* ac,
                              double* first) {
    const int m = blockIdx.x;
    for (int l = threadIdx.x; l < B; l += blockDim.x) {
        ac[(size_t)m * B + l] = l < m ? make_double2(0.0, 0.0) : make_double2(l2_an(m, l), l2_cn(m, l));
        first[(size_t)m * B + l] = seed[m].x * pow(sinn[l].x, (double)m);
    }
}

// Rows l - m of P (times the weight of the node where w is given) by the FP64 recurrence: one thread per
// node, an x off the chain, so that a degree costs one dependent multiply-add.  Near the pole the rounding
// of x would be the largest error (d theta = dx / sin theta), so the warps there add its low part.
// FP64-bound, three or four operations a value; one-warp blocks keep the SMs evenly loaded (bw 256: 56 us a
// chunk of 64 MB with four-warp blocks).
__global__ void __launch_bounds__(32) k_dg_legendre64(int B, int m0, const double2* __restrict__ cosn,
                                                      const double2* __restrict__ ac, const double* __restrict__ first,
                                                      const double* __restrict__ w, double wscale, double* tmp,
                                                      const int64_t* __restrict__ off) {
    const int m = m0 + blockIdx.x, j = min(blockIdx.y * 32 + threadIdx.x, (unsigned)B - 1);
    const double x = cosn[j].x, xl = cosn[j].y;
    double pc = first[(size_t)m * B + j], pp = 0.0;
    if (w) pc *= w[j] * wscale;  // the recurrence is linear: once
    const double2* c = ac + (size_t)m * B;
    double* out = tmp + off[m] + j;
    if (__any_sync(0xffffffffu, x > 0.8)) {
#pragma unroll 4
        for (int l = m; l < B; ++l, out += B) {
            *out = pc;
            const double2 k = c[l];
            const double nx = fma(fma(k.x, x, k.x * xl), pc, k.y * pp);
            pp = pc;
            pc = nx;
        }
    } else {
#pragma unroll 4
        for (int l = m; l < B; ++l, out += B) {
            *out = pc;
            const double2 k = c[l];
            const double nx = fma(k.x * x, pc, k.y * pp);
            pp = pc;
            pc = nx;
        }
    }
}

// Digits of those rows (degrees, or nodes for the inverse).  One block per (tile, 8-row group): eight rows
// by sixteen runs of eight K entries.
__global__ void __launch_bounds__(128) k_dg_pack_fly(int B, int fwd, const DgTile* __restrict__ tiles,
                                                     const double* __restrict__ tmp, const int64_t* __restrict__ off,
                                                     uint8_t* tab, short* qs, int* first) {
    __shared__ uint32_t red[8][17];
    const DgTile tl = tiles[blockIdx.x];
    const int rg = blockIdx.y;
    if (rg * 8 >= tl.r8) return;
    const int r = threadIdx.x & 7, kc = threadIdx.x >> 3;
    const bool live = rg * 8 + r < tl.nrows;
    const int row = tl.row0 + rg * 8 + r, nl = (B - tl.m - tl.t + 1) / 2;
    const int n = live ? (fwd ? B : nl) : 0;
    const double* src = tmp + off[tl.m] + (fwd ? (size_t)(tl.t + 2 * row) * B : (size_t)tl.t * B + row);
    const size_t step = fwd ? 1 : 2 * (size_t)B;
    uint32_t mx = 0;
    for (int k = kc * 8; k < n; k += 128)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (k + i < n) mx = max(mx, dexp(src[step * (k + i)]));
    red[r][kc] = mx;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) mx = max(mx, red[r][i]);
    const bool tiny = !fwd && mx < 1022 - 63;  // below 2^-64, as kDgTiny
    const int em = max((int)mx, 1);
    int zero = tl.ks;  // first: null, or where the tile's first step with a nonzero digit goes
    if (kc == 0 && live) qs[tl.qoff + row] = (short)(tl.tb + 1022 - em);
    const uint32_t bytes = kDigits * (uint32_t)tl.r8 * 32;
    for (int k = kc * 8; k < tl.ks * 16; k += 128) {
        unsigned long long u[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            u[i] = (unsigned long long)(k + i < n && !tiny ? dg_fix(src[step * (k + i)], em, tl.tb) : 0) + 0x0200808080808080ull;
        if (first && zero == tl.ks) {
            bool any = false;
#pragma unroll
            for (int i = 0; i < 8; ++i) any |= u[i] != 0x0200808080808080ull;
            if (any) zero = k >> 4;
        }
        if (!first && (k >> 4) < tl.k0) continue;
        uint8_t* d = tab + tl.off + (size_t)(k >> 4) * bytes + rg * 256 + ((k >> 3) & 1) * 128 + r * 16;
        const size_t ds = (size_t)tl.r8 * 32;
#define S2G_DG_PUT(a)                                                                                       \
    *(uint4*)(d + a * ds) = make_uint4(dg_digit2<a>(u[0], u[1]), dg_digit2<a>(u[2], u[3]), dg_digit2<a>(u[4], u[5]), \
                                       dg_digit2<a>(u[6], u[7]))
        S2G_DG_PUT(0);
        S2G_DG_PUT(1);
        S2G_DG_PUT(2);
        S2G_DG_PUT(3);
        S2G_DG_PUT(4);
        S2G_DG_PUT(5);
        S2G_DG_PUT(6);
#undef S2G_DG_PUT
    }
    if (first) atomicMin(first + blockIdx.x, zero);
}

// DFT tables: F1 (rows orders, K longitudes) and I2 (rows longitudes, K orders), folds as k_dg_fold.
template <int P>
__global__ void __launch_bounds__(128) k_dg_pack_dft(int B, int inv, const DgTile* __restrict__ tiles, uint8_t* tab,
                                                     short* qs) {
    const DgTile tl = tiles[blockIdx.x];
    const int rg = blockIdx.y, S = 2 * B;
    if (rg * 8 >= tl.r8) return;
    const int kd = tl.kind, k0 = (kd == 3 || kd == 5) ? 1 : 0, mstep = kd < 4 ? 2 : 1;
    const int nlon = kd < 4 ? B / 2 + (kd == 0 ? 1 : 0) : (kd == 5 ? B - 1 : B + 1);
    auto val = [&](int r, int k) -> double {
        const int row = tl.row0 + rg * 8 + r;
        if (rg * 8 + r >= tl.nrows) return 0.0;
        const int m = (inv ? k : row) * mstep + tl.m, lon = (inv ? row : k) + k0;
        if (m >= B || (!inv && k >= nlon)) return 0.0;
        // forward: the folds count the samples at their fixed points twice; inverse: orders m and -m,
        // 1/sqrt(2 pi) (FST_semi_memo.c:344-348)
        double f = (lon == 0 || (kd < 4 ? 2 * lon == B : lon == B)) ? 0.5 : 1.0;
        if (inv) f = (m ? 2.0 : 1.0) * 0.39894228040143267794;
        const double a = 2.0 * (double)((long long)m * lon % S) / (double)S;  // angle / pi
        return tl.t ? -f * sinpi(a) : f * cospi(a);
    };
    dg_pack_rows<P>(val, tl.tb, tab + tl.off, tl.r8, tl.ks, rg);
    const int r = threadIdx.x >> 4;
    if ((threadIdx.x & 15) == 0 && rg * 8 + r < tl.nrows) qs[tl.qoff + tl.row0 + rg * 8 + r] = (short)tl.tb;
}

// ------------------------------------------------------------------------------------
struct DgTable {
    std::vector<DgTile> h;
    DgTile* tiles = nullptr;
    uint8_t* tab = nullptr;
    short* q = nullptr;
    int64_t bytes = 0;
    int rows = 0;
    void release() {
        cudaFree(tiles);
        cudaFree(tab);
        cudaFree(q);
        tiles = nullptr;
        tab = nullptr;
        q = nullptr;
    }
};

// A run of orders whose tables lie in scratch together (on-the-fly family).
struct DgChunk {
    int m0, m1;
    size_t t0, t1;  // tiles
};

struct DgTabs {
    int device = -1, bw = 0, refs = 0, prec = 64;
    bool fly = false;  // no Legendre tables: chunks, nodes and offsets instead
    int semi = 0;      // orders of F2 in seminaive form (dg_semi_orders)
    DgTable t[4];
    std::vector<DgChunk> chunks[4];
    size_t tmp_bytes[4] = {0, 0, 0, 0}, tab_bytes[4] = {0, 0, 0, 0};
    double2* nodes = nullptr;          // cos, sin, seeds: B each; recurrence coefficients: B x B
    double* first = nullptr;           // P(m,m) at the nodes: B x B
    int64_t* off[4] = {nullptr, nullptr, nullptr, nullptr};
};

static std::mutex g_dg_mu;
static std::atomic<int> g_dg_test{0};  // see s2g_test_digits
enum { kDgStall = 1, kDgNoTables = 2, kDgNoScratch = 3 };
static int dg_test() { return g_dg_test.load(std::memory_order_relaxed); }
constexpr int kDgSkip = 63;  // calls that do not try again what did not fit
static std::map<std::tuple<int, int, int, bool, int>, DgTabs*> g_dg;  // device, bw, prec, fly, semi

static void dg_free(DgTabs* d) {
    for (auto& t : d->t) t.release();
    for (auto* o : d->off) cudaFree(o);
    cudaFree(d->nodes);
    cudaFree(d->first);
    delete d;
}

void dg_put(void* h) {
    DgTabs* d = (DgTabs*)h;
    if (!d) return;
    std::lock_guard<std::mutex> lk(g_dg_mu);
    if (--d->refs == 0) {
        g_dg.erase(std::make_tuple(d->device, d->bw, d->prec, d->fly, d->semi));
        dg_free(d);
    }
}

// Bits of a sample: eight (rows folded once: four) of them add up to a data value.
static int dg_vbz(int bw, int prec) {
    const bool two = dg_twice(bw);
    if (prec == 32) return two ? 27 : 28;
    return (two ? 51 : 52) + (dg_fold_layout(bw, false).n[two ? 0 : 4] <= 272 ? 2 : 0);
}

// Bits of a table value: the leading group, at most K 2^(vb - 48) 2^(tb - 48), stays below 1.5 2^22, so that the
// sum in units of 2^8 of the last group's has 63 bits.  I2 (values up to 2/sqrt(2 pi), eight sums of
// which each gives up kDgOutShift bits) keeps strictly below 2^22.
static int dg_table_bits(int K, int vb, bool inv_rows) {
    int kb = 0;
    while ((inv_rows ? 2 : 3) << kb < 2 * K) ++kb;
    return 48 + std::min(8, 22 - kb - (vb - 48));
}

static void dg_tiles(DgTable& t, int stage, int B, int prec) {
    auto add = [&](int rows, int k, int m, int par, int kind, int zoff) {
        const int q0 = t.rows;
        for (int r0 = 0; r0 < rows; r0 += 128) {
            DgTile tl{};
            tl.row0 = r0;
            tl.nrows = std::min(128, rows - r0);
            tl.r8 = (tl.nrows + 7) & ~7;
            tl.qoff = q0;
            tl.m = m;
            tl.t = par;
            tl.kind = kind;
            tl.zoff = zoff;
            tl.ks = std::max(1, (k + 15) / 16);  // no degree of a parity: one zero step
            // F1's data have vbz bits and folds; I2's sums of eight parts stay below 2^63
            tl.vb = stage == kI2 ? (k <= 128 ? 55 : k <= 256 ? 54 : 53) : (stage == kI1 ? (k <= 256 ? 55 : 54) : (k <= 256 ? 56 : 54));
            // the panels of F1 share one scale
            if (stage == kF1) tl.tb = dg_table_bits(dg_twice(B) ? B / 2 + 1 : B + 1, dg_vbz(B, 64) >= 53 ? 56 : 54, false);
            else tl.tb = dg_table_bits(k, tl.vb, stage == kI2);
            if (prec == 32) {
                tl.vb = 30;
                tl.tb = k <= 257 ? 25 : 24;
                if (stage == kF1) tl.tb = B <= 512 ? 25 : 24;
            }
            tl.off = t.bytes;
            t.bytes += (int64_t)tl.ks * (prec == 32 ? Dg<32>::DA : Dg<64>::DA) * tl.r8 * 32;
            t.h.push_back(tl);
        }
        t.rows += rows;
    };
    if (stage == kF1 || stage == kI2) {
        const DgFold f = dg_fold_layout(B, stage == kI2);
        for (int kd = dg_twice(B) ? 0 : 4; kd < (dg_twice(B) ? 4 : 6); ++kd) {
            const int m0 = kd < 4 ? kd & 1 : 0, part = kd < 4 ? kd >> 1 : kd - 4, nm = kd < 4 ? B / 2 : B;
            if (stage == kF1) add(nm, f.n[kd], m0, part, kd, f.off[kd]);
            else add(f.n[kd], nm, m0, part, kd, f.off[kd]);
        }
        return;
    }
    for (int m = 0; m < B; ++m)
        for (int par = 0; par < 2; ++par) {
            const int nl = (B - m - par + 1) / 2;
            if (stage == kI1) add(B, nl, m, par, 0, 0);
            else if (nl > 0) add(nl, B, m, par, 0, 0);
        }
}

static int dg_upload(DgTable& t, int stage, int B, int prec, cudaStream_t st) {
    dg_tiles(t, stage, B, prec);
    S2G_CUDA(cudaMalloc(&t.tiles, sizeof(DgTile) * t.h.size()));
    S2G_CUDA(cudaMalloc(&t.tab, (size_t)t.bytes + 4096));
    S2G_CUDA(cudaMalloc(&t.q, sizeof(short) * t.rows));
    S2G_CUDA(cudaMemcpyAsync(t.tiles, t.h.data(), sizeof(DgTile) * t.h.size(), cudaMemcpyHostToDevice, st));
    return S2G_OK;
}

// Above this bandwidth the forward's orders 1, 3 and 5 take their rows from the cosine series, where they are
// seminaive (below the cutoff).  The series of G = P / sin have large coefficients there, and their FP64
// rounding is part of the reference's results: on samples that are not band-limited (noise), at bw 1024, the
// exact transform is 4.1e-11 of the order's largest coefficient away from them at order 1, 6e-12 at order 3 and
// 4.5e-12 at order 5, while the FP64 path keeps to the reference within 1e-11.  From the cutoff on the reference
// is naive, and within 1e-13 of the exact transform.
constexpr int kDgNaiveBw = 512;
// How many of these orders a table has: tables are shared by all cutoffs but for this.
static int dg_semi_orders(int B, int cutoff, int prec, bool fly) {
    return B > kDgNaiveBw && prec == 64 && !fly ? std::min(cutoff, 6) / 2 : 0;
}
static int dg_low_orders(int B, int semi, double* tmp, const std::vector<int64_t>& off, int m1, cudaStream_t st) {
    const int S = 2 * B;
    m1 = std::min(m1, 2 * semi);
    struct Buf {
        void* p[3] = {nullptr, nullptr, nullptr};
        ~Buf() {
            for (void* q : p) cudaFree(q);
        }
    } b;
    int64_t most = 0;
    for (int m = 1; m < m1; m += 2) most = std::max(most, table_size(m, B));
    const std::vector<int64_t> zero(8, 0);  // each order's table alone, at the buffer's start
    S2G_CUDA(cudaMalloc(&b.p[0], sizeof(double) * (size_t)most));
    S2G_CUDA(cudaMalloc(&b.p[1], sizeof(double2) * 4 * S));
    S2G_CUDA(cudaMalloc(&b.p[2], sizeof(int64_t) * zero.size()));
    S2G_CUDA(cudaMemcpyAsync(b.p[2], zero.data(), sizeof(int64_t) * zero.size(), cudaMemcpyHostToDevice, st));
    S2G_TRY(twiddles_device(4 * S, (double2*)b.p[1], nullptr, st));
    for (int m = 1; m < m1; m += 2) {
        S2G_TRY(generate_cos_pml_device(B, m, m + 1, (double*)b.p[0], (const int64_t*)b.p[2], st));
        ProfScope ps_("dg_seminaive", st);
        k_dg_seminaive<<<B - m, 256, 0, st>>>(B, m, (const double*)b.p[0], (const double2*)b.p[1], tmp + off[m]);
        S2G_CUDA(cudaGetLastError());
    }
    S2G_CUDA(cudaStreamSynchronize(st));
    return S2G_OK;
}

// The tiles' first steps with nonzero digits: an array for the pack kernels, then into the tiles.
static int dg_first_alloc(const DgTable& t, void** mem, int** first, cudaStream_t st) {
    S2G_CUDA(cudaMalloc(mem, sizeof(int) * t.h.size()));
    S2G_CUDA(cudaMemsetAsync(*mem, 0x7f, sizeof(int) * t.h.size(), st));
    *first = (int*)*mem;
    return S2G_OK;
}
static int dg_first_read(DgTable& t, const int* first, cudaStream_t st) {
    std::vector<int> f(t.h.size());
    S2G_CUDA(cudaMemcpyAsync(f.data(), first, sizeof(int) * f.size(), cudaMemcpyDeviceToHost, st));
    S2G_CUDA(cudaStreamSynchronize(st));
    for (size_t i = 0; i < f.size(); ++i) t.h[i].k0 = std::min(f[i], t.h[i].ks - 1);
    S2G_CUDA(cudaMemcpyAsync(t.tiles, t.h.data(), sizeof(DgTile) * t.h.size(), cudaMemcpyHostToDevice, st));
    S2G_CUDA(cudaStreamSynchronize(st));
    return S2G_OK;
}

// Digits in scratch at a time, on-the-fly family: enough orders to fill the GPU.
static int64_t dg_fly_budget(int bw) { return (int64_t)(bw <= 256 ? 64 : bw <= 512 ? 128 : 384) << 20; }

// Tables of one chunk of orders in scratch; first: see dg_first_alloc.
static int dg_fly_tables(const DgTabs* d, int stage, const DgChunk& c, const double* weights, double* tmp, uint8_t* tab,
                         short* q, int* first, cudaStream_t st) {
    const int B = d->bw;
    const DgTable& t = d->t[stage];
    {
        ProfScope ps_("dg_fly_legendre", st);
        k_dg_legendre64<<<dim3(c.m1 - c.m0, (B + 31) / 32), 32, 0, st>>>(
            B, c.m0, d->nodes, d->nodes + 3 * (size_t)B, d->first, stage == kF2 ? weights : nullptr,
            sqrt(2.0 * 3.14159265358979323846) / (2 * B), tmp, d->off[stage]);
    }
    S2G_CUDA(cudaGetLastError());
    {
        ProfScope ps_("dg_fly_pack", st);
        k_dg_pack_fly<<<dim3((unsigned)(c.t1 - c.t0), 16), 128, 0, st>>>(B, stage == kF2, t.tiles + c.t0, tmp,
                                                                        d->off[stage], tab, q, first);
    }
    S2G_CUDA(cudaGetLastError());
    return S2G_OK;
}

// Tiles of F2 or I1 in chunks of orders, their offsets counted from the chunk's start; off[m]: doubles of the recurrence
// before order m in its chunk; the chunks' largest sizes.  Host only.
static void dg_fly_layout(int s, int B, DgTable& t, std::vector<DgChunk>& chunks, std::vector<int64_t>& off,
                          size_t& tmp_bytes, size_t& tab_bytes) {
    dg_tiles(t, s, B, 64);
    off.resize(B);
    int64_t base = 0, at = 0;
    size_t k = 0;
    DgChunk c{0, 0, 0, 0};
    for (int m = 0; m < B; ++m) {
        size_t e = k;
        while (e < t.h.size() && t.h[e].m == m) ++e;
        const int64_t end = e < t.h.size() ? t.h[e].off : t.bytes;
        if (m > c.m0 && end - base > dg_fly_budget(B)) {
            chunks.push_back(c);
            c = DgChunk{m, m, k, k};
            base = t.h[k].off;
            at = 0;
        }
        for (; k < e; ++k) t.h[k].off -= base;
        c.m1 = m + 1;
        c.t1 = e;
        off[m] = at;
        at += (int64_t)(B - m) * B;
        tab_bytes = std::max(tab_bytes, (size_t)(end - base));
        tmp_bytes = std::max(tmp_bytes, (size_t)at * sizeof(double));
    }
    chunks.push_back(c);
}

static int dg_fly_chunks(DgTabs* d, const double* weights, cudaStream_t st) {
    const int B = d->bw;
    for (int s = kF2; s <= kI1; ++s) {
        DgTable& t = d->t[s];
        std::vector<int64_t> off;
        dg_fly_layout(s, B, t, d->chunks[s], off, d->tmp_bytes[s], d->tab_bytes[s]);
        S2G_CUDA(cudaMalloc(&t.tiles, sizeof(DgTile) * t.h.size()));
        S2G_CUDA(cudaMemcpyAsync(t.tiles, t.h.data(), sizeof(DgTile) * t.h.size(), cudaMemcpyHostToDevice, st));
        S2G_CUDA(cudaMalloc(&d->off[s], sizeof(int64_t) * B));
        S2G_CUDA(cudaMemcpyAsync(d->off[s], off.data(), sizeof(int64_t) * B, cudaMemcpyHostToDevice, st));
        // generated once here, for the tiles' first steps
        struct Buf {
            void* p[4] = {nullptr, nullptr, nullptr, nullptr};
            ~Buf() {
                for (void* q : p) cudaFree(q);
            }
        } b;
        int* first = nullptr;
        S2G_TRY(dg_first_alloc(t, &b.p[0], &first, st));
        S2G_CUDA(cudaMalloc(&b.p[1], d->tmp_bytes[s]));
        S2G_CUDA(cudaMalloc(&b.p[2], d->tab_bytes[s]));
        S2G_CUDA(cudaMalloc(&b.p[3], sizeof(short) * t.rows));
        for (const DgChunk& q : d->chunks[s])
            S2G_TRY(dg_fly_tables(d, s, q, s == kF2 ? weights : nullptr, (double*)b.p[1], (uint8_t*)b.p[2], (short*)b.p[3],
                                  first + q.t0, st));
        S2G_TRY(dg_first_read(t, first, st));
    }
    return S2G_OK;
}

static int dg_build(DgTabs* d, const double* weights, cudaStream_t st) {
    const int B = d->bw, S = 2 * B;
    for (int s = 0; s < 4; ++s)
        if (!d->fly || s == kF1 || s == kI2) S2G_TRY(dg_upload(d->t[s], s, B, d->prec, st));
    for (int s = kF1; s <= kI2; s += kI2 - kF1) {
        const DgTable& t = d->t[s];
        ProfScope ps_("dg_pack_dft", st);
        const dim3 grid((unsigned)t.h.size(), 16);
        if (d->prec == 32) k_dg_pack_dft<32><<<grid, 128, 0, st>>>(B, s == kI2, t.tiles, t.tab, t.q);
        else k_dg_pack_dft<64><<<grid, 128, 0, st>>>(B, s == kI2, t.tiles, t.tab, t.q);
        S2G_CUDA(cudaGetLastError());
    }
    // nodes, seeds P(m,m) = seed_m sin^m: long double, split in two doubles
    std::vector<double2> h(3 * (size_t)B);
    auto put = [](long double v) {
        const double a = (double)v;
        return make_double2(a, (double)(v - (long double)a));
    };
    const long double pi = 3.141592653589793238462643383279502884L;
    long double c = sqrtl(0.5L);
    for (int j = 0; j < B; ++j) {
        const long double a = pi * (2 * j + 1) / (2 * (long double)S);
        h[j] = put(cosl(a));
        h[B + j] = put(sinl(a));
        if (j) c *= -sqrtl((2 * j + 1) / (2 * (long double)j));
        h[2 * (size_t)B + j] = put(c);
    }
    if (d->fly) {
        S2G_CUDA(cudaMalloc(&d->nodes, sizeof(double2) * (h.size() + (size_t)B * B)));
        S2G_CUDA(cudaMalloc(&d->first, sizeof(double) * (size_t)B * B));
        S2G_CUDA(cudaMemcpyAsync(d->nodes, h.data(), sizeof(double2) * h.size(), cudaMemcpyHostToDevice, st));
        {
            ProfScope ps_("dg_fly_init", st);
            k_dg_fly_init<<<B, 128, 0, st>>>(B, d->nodes + B, d->nodes + 2 * (size_t)B, d->nodes + h.size(), d->first);
        }
        S2G_CUDA(cudaGetLastError());
        return dg_fly_chunks(d, weights, st);
    }
    struct Tmp {
        void* p[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
        ~Tmp() {
            for (void* q : p) cudaFree(q);
        }
    } tmp;
    S2G_CUDA(cudaMalloc(&tmp.p[0], sizeof(double2) * h.size()));
    S2G_CUDA(cudaMemcpyAsync(tmp.p[0], h.data(), sizeof(double2) * h.size(), cudaMemcpyHostToDevice, st));
    // orders in chunks of at most 1 GiB of table values; off[m]: doubles before order m in its chunk
    const int64_t most = std::max<int64_t>((int64_t)B * B, (int64_t)1 << 27);
    std::vector<int64_t> off(B);
    int64_t at = 0, need = 0;
    for (int m = 0; m < B; ++m) {
        const int64_t n = (int64_t)(B - m) * B;
        if (at + n > most) at = 0;
        off[m] = at;
        at += n;
        need = std::max(need, at);
    }
    S2G_CUDA(cudaMalloc(&tmp.p[1], sizeof(double) * (size_t)need));
    S2G_CUDA(cudaMalloc(&tmp.p[2], sizeof(int64_t) * B));
    S2G_CUDA(cudaMemcpyAsync(tmp.p[2], off.data(), sizeof(int64_t) * B, cudaMemcpyHostToDevice, st));
    const double2* nodes = (const double2*)tmp.p[0];
    int* first[4] = {nullptr, nullptr, nullptr, nullptr};
    for (int s = kF2; s <= kI1; ++s) S2G_TRY(dg_first_alloc(d->t[s], &tmp.p[s + 2], &first[s], st));
    const size_t smem = sizeof(double2) * 2 * (size_t)B;
    S2G_TRY(set_smem((const void*)k_dg_legendre, smem));
    for (int m0 = 0; m0 < B;) {
        int m1 = m0 + 1;
        while (m1 < B && off[m1] != 0) ++m1;
        {
            ProfScope ps_("dg_legendre", st);
            k_dg_legendre<<<m1 - m0, std::min(1024, (B + 31) & ~31), smem, st>>>(
                B, m0, nodes, nodes + B, nodes + 2 * (size_t)B, (double*)tmp.p[1], (const int64_t*)tmp.p[2] + m0);
        }
        S2G_CUDA(cudaGetLastError());
        for (int s = kI1; s >= kF2; --s) {
            if (s == kF2 && d->semi && m0 <= 1) S2G_TRY(dg_low_orders(B, d->semi, (double*)tmp.p[1], off, m1, st));
            const DgTable& t = d->t[s];
            size_t a = 0, b = t.h.size();
            while (a < b && t.h[a].m < m0) ++a;
            while (b > a && t.h[b - 1].m >= m1) --b;
            ProfScope ps_("dg_pack_leg", st);
            const auto pack = d->prec == 32 ? k_dg_pack_leg<32> : k_dg_pack_leg<64>;
            pack<<<dim3((unsigned)(b - a), 16), 128, 0, st>>>(
                B, s == kF2, t.tiles + a, m0, (const double*)tmp.p[1], (const int64_t*)tmp.p[2] + m0, weights,
                sqrt(2.0 * 3.14159265358979323846) / S, t.tab, t.q, first[s] + a);
            S2G_CUDA(cudaGetLastError());
        }
        m0 = m1;
    }
    for (int s = kF2; s <= kI1; ++s) S2G_TRY(dg_first_read(d->t[s], first[s], st));
    return S2G_OK;
}

// Digit tables of bandwidth bw on the current device, shared by every plan; the caller holds a reference.
static int dg_get(int bw, int prec, bool fly, int semi, const double* weights, DgTabs** out) {
    int dev = 0;
    S2G_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_dg_mu);
    const auto key = std::make_tuple(dev, bw, prec, fly, semi);
    auto it = g_dg.find(key);
    if (it != g_dg.end()) {
        ++it->second->refs;
        *out = it->second;
        return S2G_OK;
    }
    const RelaxCapture relax;  // the first call that takes this path may not be the plan's first
    DgTabs* d = new DgTabs();
    d->device = dev;
    d->bw = bw;
    d->prec = prec;
    d->fly = fly;
    d->semi = semi;
    cudaStream_t st;
    S2G_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    const int r = dg_build(d, weights, st);
    cudaStreamDestroy(st);
    if (r != S2G_OK) {
        dg_free(d);
        return r;
    }
    d->refs = 1;
    g_dg[key] = d;
    *out = d;
    return S2G_OK;
}

template <int STAGE, int NT, int P>
static int launch_dg_nt(const DgArgs& p, int sms, cudaStream_t st) {
    static const char* names[8] = {"dg_rows_fwd", "dg_leg_fwd", "dg_leg_inv", "dg_rows_inv",
                                   "dg_rows_fwd_f32", "dg_leg_fwd_f32", "dg_leg_inv_f32", "dg_rows_inv_f32"};
    const size_t smem = 1024 + Dg<P>::stagesA * kDgABytes<P> + kDgBRing +
                        (P == 32 && STAGE == kF1 ? Dg<P>::epilogue * kDgStash : 0);
    S2G_TRY(set_smem((const void*)k_dg<STAGE, NT, P>, smem));
    const int64_t items = (int64_t)p.ntiles * p.ncolblk;
    {
        ProfScope ps_(names[STAGE + (P == 32 ? 4 : 0)], st);
        k_dg<STAGE, NT, P><<<(unsigned)std::min<int64_t>(items, sms), kDgThreads, smem, st>>>(p);
    }
    S2G_CUDA(cudaGetLastError());
    return S2G_OK;
}

// Columns per item.  While one wave of blocks holds them all, more and smaller items are faster (bw 64, one
// function: F1 16.4 us at 64 columns, 11.2 at 16); and up to 64 columns in all are one item a tile even beyond one
// wave.  (For 33 to 64 columns of F2 and I1 that is the better choice for the fewest, 17 fields at bw 512: I1 280 us,
// 307 at 32; not for the most: 32 fields at bw 101, F2 30.6 and 24.5, at bw 256 75.7 and 69.6, I1 75.7 and 71.6.)
// More than 64 columns beyond one wave, FP64: 64 columns take one accumulator (7 x 64
// TMEM columns) whose epilogue the next item's MMAs wait for (F1 at bw 256: 44% of the time), 32 take two by
// turns, but seven dependent MMAs of about 115 cycles for each 16-deep K step where 64 take ten for twice the
// columns.  So 64 is for the long K
// ranges: I1 (K = the degrees of a parity) never, F2 (K = bw) above bw 256 (bw 256, 256 functions: 478 us at
// 64, 463 at 32; bw 512, 64 functions: 519 and 601), F1 above 300 (bw 256, 64 functions: 165 and 156; bw 512:
// 897 and 998), I2 (whose epilogue is the shortest) above 112 orders (bw 192, 64 functions: 97 and 79; bw 256:
// 118 and 126).  FP32 (G = 4) has two accumulators at 64 columns.
// Items of F1 and I2 go column by column (their tables, 1 MB at bw 256, stay in L2), those of F2 and I1 table
// by table (117 MB each at bw 256).
// At bw 256, 64 functions: F1 156 us, F2 116, I1 123, I2 118, k_dg_fold 52, k_dg_unfold 53, k_dg_mid 17;
// forward and inverse together 0.64 ms against 4.59 ms on the FP64 units (DFMA-bound there).  The tensor
// pipe alone would take 47 us for each of the four; MMA issue and the waits around it make up the rest.
template <int STAGE>
static int dg_columns(const DgTabs* d, const DgArgs& p, int sms) {
    auto items = [&](int n) { return (int64_t)p.ntiles * ((p.ncols + n - 1) / n); };
    for (int n : {16, 32, 64})
        if (p.ncols <= n || items(n) <= sms) return n;
    if (d->prec == 32) return 64;
    if (STAGE == kI1) return 32;
    if (STAGE == kF2) return d->bw <= 256 ? 32 : 64;
    if (STAGE == kF1) return d->bw <= 300 ? 32 : 64;
    return d->t[kI2].h[0].ks <= 7 ? 32 : 64;
}
template <int STAGE>
static int launch_dg_tiles(const DgTabs* d, DgArgs p, cudaStream_t st) {
    p.col_major = STAGE == kF1 || STAGE == kI2;
    p.stall = dg_test() == kDgStall;
    int dev = 0, sms = 0;
    S2G_CUDA(cudaGetDevice(&dev));
    S2G_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int per = dg_columns<STAGE>(d, p, sms);
    p.ncolblk = (p.ncols + per - 1) / per;
    if (d->prec == 32) {
        if (per == 16) return launch_dg_nt<STAGE, 16, 32>(p, sms, st);
        if (per == 32) return launch_dg_nt<STAGE, 32, 32>(p, sms, st);
        return launch_dg_nt<STAGE, 64, 32>(p, sms, st);
    }
    if (per == 16) return launch_dg_nt<STAGE, 16, 64>(p, sms, st);
    if (per == 32) return launch_dg_nt<STAGE, 32, 64>(p, sms, st);
    return launch_dg_nt<STAGE, 64, 64>(p, sms, st);
}

// A stage over its whole table; on the fly, F2 and I1 generate theirs chunk by chunk in `scratch`.
template <int STAGE>
static int launch_dg(const DgTabs* d, DgArgs p, const double* weights, char* scratch, cudaStream_t st) {
    const DgTable& t = d->t[STAGE];
    p.tiles = t.tiles;
    p.tab = t.tab;
    p.q = t.q;
    p.ntiles = (int)t.h.size();
    if (!d->fly || STAGE == kF1 || STAGE == kI2) return launch_dg_tiles<STAGE>(d, p, st);
    double* tmp = (double*)scratch;
    uint8_t* tab = (uint8_t*)scratch + ((d->tmp_bytes[STAGE] + 255) & ~(size_t)255);
    short* q = (short*)(tab + ((d->tab_bytes[STAGE] + 4096 + 255) & ~(size_t)255));
    for (const DgChunk& c : d->chunks[STAGE]) {
        S2G_TRY(dg_fly_tables(d, STAGE, c, weights, tmp, tab, q, nullptr, st));
        p.tiles = t.tiles + c.t0;
        p.ntiles = (int)(c.t1 - c.t0);
        p.tab = tab;
        p.q = q;
        S2G_TRY(launch_dg_tiles<STAGE>(d, p, st));
    }
    return S2G_OK;
}

static int dg_fields(int mode) { return mode == kReal ? 1 : 2; }
static int dg_mode(const void* imag, int fmt) { return fmt == COMPLEX ? kCplx : (imag ? kReal2 : kReal); }

// Functions transformed at a time (es: bytes of a value).
int dg_chunk(int bw, int batch, int es) {
    const int64_t per = 2 * es * 4 * (int64_t)bw * bw;
    return (int)std::min<int64_t>(batch, std::min<int64_t>(16384, std::max<int64_t>(64, ((int64_t)256 << 20) / per)));
}

struct DgWork {
    void *X, *Z;
    uint32_t *ej, *ef, *ex;
    void *mid, *cr, *ci;
    size_t bytes;
};
static DgWork dg_work(char* w, int bw, int n, bool two, int es) {
    const size_t ff = (size_t)n * (two ? 2 : 1), S = 2 * (size_t)bw, BP = (bw + 3) & ~3;
    const size_t len = std::max(dg_fold_layout(bw, false).len, dg_fold_layout(bw, true).len);
    size_t at = 0;
    auto take = [&](size_t bytes) {
        char* q = w + at;
        at += (bytes + 255) & ~(size_t)255;
        return (void*)q;
    };
    DgWork k{};
    k.X = take(ff * 2 * bw * 2 * BP * es);
    k.Z = take(ff * S * len * es);
    k.ej = (uint32_t*)take(ff * bw * 4);
    k.ef = (uint32_t*)take(ff * 4);
    k.ex = (uint32_t*)take(ff * 2 * bw * 4);
    k.mid = take(ff * S * es);
    k.cr = take(two ? ff * bw * bw * es : 0);
    k.ci = take(two ? ff * bw * bw * es : 0);
    k.bytes = at;
    return k;
}

// Scratch of a stage's generated tables: recurrence, digits, scales (launch_dg).
static size_t dg_fly_stage(size_t tmp_bytes, size_t tab_bytes, int rows) {
    return tmp_bytes + tab_bytes + 2 * (size_t)rows + 4096 + 1024;
}
size_t dg_fly_bytes(const Tables* t, int batch, bool two) {
    const DgTabs* d = (const DgTabs*)t->dg;
    size_t need = 0;
    for (int s = kF2; s <= kI1; ++s) need = std::max(need, dg_fly_stage(d->tmp_bytes[s], d->tab_bytes[s], d->t[s].rows));
    return dg_work_bytes(t->bw, batch, two) + need;
}
size_t dg_fly_bytes(int bw, int batch, bool two) {
    size_t need = 0;
    for (int s = kF2; s <= kI1; ++s) {
        DgTable t;
        std::vector<DgChunk> chunks;
        std::vector<int64_t> off;
        size_t tmp = 0, tab = 0;
        dg_fly_layout(s, bw, t, chunks, off, tmp, tab);
        need = std::max(need, dg_fly_stage(tmp, tab, t.rows));
    }
    return dg_work_bytes(bw, batch, two) + need;
}

size_t dg_work_bytes(int bw, int batch, bool two) {
    return dg_work(nullptr, bw, dg_chunk(bw, batch, 8), two, 8).bytes;
}
size_t dg32_work_bytes(int bw, int batch, bool two) {
    return dg_work(nullptr, bw, dg_chunk(bw, batch, 4), two, 4).bytes;
}

// Bandwidths of the digit path: up to 1024 (its Legendre tables take 14 bw^3 bytes: 15 GB there).  Below 32
// its five or six launches cost more than the FP64 kernels' two where those have a radix-2 FFT (one
// function at bw 16: 24 and 33 us against 24 and 25), but not where they take Bluestein's (bw 12: 25 and
// 34 us against 87 and 87).
bool dg_takes(int bw) { return bw <= 1024 && (bw >= 32 || (bw > 8 && (bw & (bw - 1)))); }

bool dg_fly_takes(int bw, int fields) { return dg_takes(bw) && bw >= 64 && fields >= (bw > 512 ? 4 : 2); }

// Builds (or finds) the digit tables of t's bandwidth; *yes where they are there.  Where the stream is being
// captured, or they do not fit in device memory, t stays without them and the other kernels run; what did not
// fit is tried again by every 64th call that asks (an attempt costs the allocations before the one that fails).
static int prepare(Tables* t, int prec, void** slot, int* skip, cudaStream_t st, bool* yes) {
    *yes = false;
    if (dg_test() == kDgNoTables) return S2G_OK;
    if (!__atomic_load_n(slot, __ATOMIC_ACQUIRE)) {
        if (__atomic_load_n(skip, __ATOMIC_RELAXED) > 0) {
            __atomic_fetch_sub(skip, 1, __ATOMIC_RELAXED);
            return S2G_OK;
        }
        if (capturing(st)) return S2G_OK;
        DgTabs* d;
        const bool fly = t->cutoff == 0;
        const int r = dg_get(t->bw, prec, fly, dg_semi_orders(t->bw, t->cutoff, prec, fly), t->weights, &d);
        if (r == S2G_ERR_NOMEM) {
            cudaGetLastError();
            __atomic_store_n(skip, kDgSkip, __ATOMIC_RELAXED);
            return S2G_OK;
        }
        if (r != S2G_OK) return r;
        void* none = nullptr;
        if (!__atomic_compare_exchange_n(slot, &none, (void*)d, false, __ATOMIC_ACQ_REL, __ATOMIC_ACQUIRE)) dg_put(d);
    }
    *yes = true;
    return S2G_OK;
}
int dg_prepare(Tables* t, cudaStream_t st, bool* yes) {
    *yes = false;
    return dg_takes(t->bw) ? prepare(t, 64, &t->dg, &t->dg_skip, st, yes) : S2G_OK;
}
// Bandwidths whose FP32 transforms take the digit path: chirp-z ones, where its matrix products beat the two
// FFTs of each chirp-z stage (forward 1.1 to 1.6 times as fast over bw 65 .. 255 and batches of 1 to 1024,
// inverse 1.1 to 1.8; bw 255, 256 functions: 798 us against 880 and 703 against 912).  Below 64 they do not for large batches (bw 33, 4096 functions: 498 us against
// 452), nor where a warp FFT takes the length (bw 256, 64 functions: 187 us against 96).
bool dg32_takes(int bw) { return bw >= 64 && split_czt(bw); }
int dg32_prepare(Tables* t, cudaStream_t st, bool* yes) {
    *yes = false;
    return dg32_takes(t->bw) ? prepare(t, 32, &t->dg32, &t->dg32_skip, st, yes) : S2G_OK;
}

bool dg_no_scratch() { return dg_test() == kDgNoScratch; }
int dg_scratch(Scratch& s, size_t need, cudaStream_t st, bool* yes) {
    *yes = false;
    if (dg_no_scratch()) return S2G_OK;
    if (need > s.bytes) {
        if (need >= s.nofit && s.skip > 0) {
            --s.skip;
            return S2G_OK;
        }
        if (capturing(st)) return S2G_OK;
    }
    const RelaxCapture relax;
    const int r = s.ensure(need, st);
    if (r == S2G_ERR_NOMEM) {
        cudaGetLastError();
        s.nofit = need;
        s.skip = kDgSkip;
        return S2G_OK;
    }
    *yes = r == S2G_OK;
    return r;
}

template <int P>
static int dg_fst(const DgTabs* d, const double* weights, const typename Dg<P>::Real* rdata,
                  const typename Dg<P>::Real* idata, typename Dg<P>::Real* rc, typename Dg<P>::Real* ic, int batch, int fmt,
                  void* work, cudaStream_t st, int* err, const int64_t* gmap = nullptr, const int64_t* cmap = nullptr) {
    using Real = typename Dg<P>::Real;
    const int B = d->bw, S = 2 * B, mode = dg_mode(idata, fmt), chunk = dg_chunk(B, batch, sizeof(Real));
    const DgFold fl = dg_fold_layout(B, false);
    const DgWork w = dg_work((char*)work, B, chunk, mode != kReal, sizeof(Real));
    char* scratch = (char*)work + w.bytes;  // on the fly: tables
    S2G_TRY(set_smem((const void*)k_dg_fold<P>, 2 * (size_t)S * sizeof(Real)));
    for (int f0 = 0; f0 < batch; f0 += chunk) {
        const int n = std::min(chunk, batch - f0), ff = n * dg_fields(mode);
        const size_t g0 = gmap ? 0 : (size_t)f0 * S * S, c0 = cmap ? 0 : (size_t)f0 * B * B;
        const int64_t *gm = gmap ? gmap + f0 : nullptr, *cm = cmap ? cmap + f0 : nullptr;
        S2G_CUDA(cudaMemsetAsync(w.ef, 0, (size_t)((char*)(w.ex + (size_t)ff * 2 * B) - (char*)w.ef), st));
        DgArgs p{};
        p.B = B;
        p.S = S;
        p.N = n;
        p.mode = mode;
        p.cmap = cm;
        p.err = err;
        p.BP = (B + 3) & ~3;
        p.RL = fl.len;
        p.vbz = dg_vbz(B, P);
        p.tbz = d->t[kF1].h[0].tb;
        p.X = w.X;
        p.Z = w.Z;
        {
            ProfScope ps_(P == 32 ? "dg_fold_f32" : "dg_fold", st);
            k_dg_fold<P><<<dim3(B, ff), dg_fold_threads(S), 2 * (size_t)S * sizeof(Real), st>>>(
                rdata + g0, idata ? idata + g0 : nullptr, B, n, p.vbz, fl, gm, (typename Dg<P>::Int*)w.Z, w.ej, w.ef);
        }
        S2G_CUDA(cudaGetLastError());
        p.ncols = ff * S;
        p.ein = w.ej;
        p.efield = w.ef;
        p.emax = w.ex;
        S2G_TRY(launch_dg<kF1>(d, p, weights, scratch, st));
        p.ncols = ff * 2;
        p.out_r = rc + c0;
        p.out_i = ic + c0;
        S2G_TRY(launch_dg<kF2>(d, p, weights, scratch, st));
    }
    return S2G_OK;
}

template <int P>
static int dg_inv_fst(const DgTabs* d, const double* weights, const typename Dg<P>::Real* rc,
                      const typename Dg<P>::Real* ic, typename Dg<P>::Real* rdata, typename Dg<P>::Real* idata, int batch,
                      int fmt, void* work, cudaStream_t st, int* err, const int64_t* gmap = nullptr,
                      const int64_t* cmap = nullptr) {
    using Real = typename Dg<P>::Real;
    const int B = d->bw, S = 2 * B, mode = dg_mode(idata, fmt), chunk = dg_chunk(B, batch, sizeof(Real));
    const DgFold fl = dg_fold_layout(B, true);
    const DgWork w = dg_work((char*)work, B, chunk, mode != kReal, sizeof(Real));
    char* scratch = (char*)work + w.bytes;  // on the fly: tables
    for (int f0 = 0; f0 < batch; f0 += chunk) {
        const int n = std::min(chunk, batch - f0), ff = n * dg_fields(mode);
        const size_t g0 = gmap ? 0 : (size_t)f0 * S * S, c0 = cmap ? 0 : (size_t)f0 * B * B;
        const int64_t *gm = gmap ? gmap + f0 : nullptr, *cm = cmap ? cmap + f0 : nullptr;
        S2G_CUDA(cudaMemsetAsync(w.ef, 0, (size_t)ff * 4, st));
        {
            ProfScope ps_(P == 32 ? "dg_coefmax_f32" : "dg_coefmax", st);
            k_dg_coefmax<Real><<<(n * B + 7) / 8, 256, 0, st>>>(rc + c0, ic + c0, B, n, mode, cm, (Real*)w.cr, (Real*)w.ci, w.ex);
        }
        S2G_CUDA(cudaGetLastError());
        DgArgs p{};
        p.B = B;
        p.S = S;
        p.N = n;
        p.mode = mode;
        p.cmap = cm;
        p.err = err;
        p.BP = (B + 3) & ~3;
        p.RL = fl.len;
        p.X = w.X;
        p.Z = w.Z;
        p.ncols = ff * 2;
        p.in_r = mode == kReal ? (const void*)(rc + c0) : w.cr;
        p.in_i = mode == kReal ? (const void*)(ic + c0) : w.ci;
        p.ein = w.ex;
        p.emax = w.ef;
        S2G_TRY(launch_dg<kI1>(d, p, weights, scratch, st));
        p.ncols = ff * S;
        p.ein = w.ef;
        S2G_TRY(launch_dg<kI2>(d, p, weights, scratch, st));
        if (fl.n[0]) {
            ProfScope ps_(P == 32 ? "dg_mid_f32" : "dg_mid", st);
            k_dg_mid<Real><<<(ff * S + 31) / 32, dim3(32, 8), 0, st>>>((const Real*)w.X, B, ff * S, (Real*)w.mid);
            S2G_CUDA(cudaGetLastError());
        }
        {
            ProfScope ps_(P == 32 ? "dg_unfold_f32" : "dg_unfold", st);
            k_dg_unfold<P><<<dim3(B, ff), 128, 0, st>>>(w.Z, (const Real*)w.mid, w.ef, B, n,
                                                        d->t[kI2].h[0].vb + d->t[kI2].h[0].tb, fl, gm, rdata + g0,
                                                        idata ? idata + g0 : nullptr);
        }
        S2G_CUDA(cudaGetLastError());
    }
    return S2G_OK;
}

int fst_f64_dg(const Tables* t, const double* rdata, const double* idata, double* rc, double* ic, int batch, int fmt,
               void* work, cudaStream_t st, int* err) {
    return dg_fst<64>((const DgTabs*)t->dg, t->weights, rdata, idata, rc, ic, batch, fmt, work, st, err);
}
int inv_fst_f64_dg(const Tables* t, const double* rc, const double* ic, double* rdata, double* idata, int batch, int fmt,
                   void* work, cudaStream_t st, int* err) {
    return dg_inv_fst<64>((const DgTabs*)t->dg, t->weights, rc, ic, rdata, idata, batch, fmt, work, st, err);
}
int fst_dg32(const Tables* t, const float* rgrid, const float* igrid, float* rc, float* ic, int batch, void* work,
             cudaStream_t st, int* err, const int64_t* gmap, const int64_t* cmap) {
    return dg_fst<32>((const DgTabs*)t->dg32, t->weights, rgrid, igrid, rc, ic, batch, igrid ? COMPLEX : REAL, work, st,
                      err, gmap, cmap);
}
int inv_fst_dg32(const Tables* t, const float* rc, const float* ic, float* rgrid, float* igrid, int batch, void* work,
                 cudaStream_t st, int* err, const int64_t* gmap, const int64_t* cmap) {
    return dg_inv_fst<32>((const DgTabs*)t->dg32, t->weights, rc, ic, rgrid, igrid, batch, igrid ? COMPLEX : REAL, work, st,
                          err, gmap, cmap);
}

int dg_status(int* err) {
    int v = 0;
    S2G_CUDA(cudaMemcpy(&v, err, sizeof(int), cudaMemcpyDeviceToHost));
    if (v) S2G_CUDA(cudaMemset(err, 0, sizeof(int)));
    return v ? dg_expired(v) : S2G_OK;
}
int dg_expired(int code) { return fail(code, "a bounded wait in the digit-product kernel expired"); }

}  // namespace s2g

extern "C" int s2g_test_digits(int what) {
    if (what < 0 || what > s2g::kDgNoScratch) return s2g::fail(S2G_ERR_ARG, "s2g_test_digits(%d)", what);
    s2g::g_dg_test = what;
    return S2G_OK;
}
