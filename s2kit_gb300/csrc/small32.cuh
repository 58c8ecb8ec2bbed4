// small32.cuh -- FP32 real-field transforms of small bandwidths, one kernel each way.
//
// A function of bandwidth 16 to 31 is 4 to 15 KB: a block holds a few whole functions in shared memory
// and takes them from samples to coefficients (or back) by direct sums on the FP32 units, where the staged
// path writes and reads the intermediates twice and gives the contraction tiles that are mostly padding.
// Per function and direction (B = bw, S = 2B, everything folded about the equator, so that a latitude j < B
// stands for two, an even and an odd part):
//   forward  Z[k][(part, j)]   rows folded in longitude, x_k +- x_(S-k), for even B again about S/4   (fold)
//            G[m][part][c][j]  = sum_k Z[k] cos / -sin (2 pi k m / S)          2 B^3 multiply-adds (odd B: 4 B^3)
//            coefficient (l,m) = sum_j P(l,m,j) w_j G[m][(l+m) odd][c][j]      B^2 (B+1)
//   inverse  Y[m][(part, j)]   = sum_l P(l,m,j) f(l,m), O[k] = sum_m c_m Y cos / -sin, unfold
// Both sums are 4 x 4 register tiles: a thread reads four values of either operand as one float4 (a table's
// from L1 or L2, the data's from shared memory), a warp's 8 x 4 tiles share them.  Every output is one
// thread's sum in one order, so a function's result does not depend on the batch or the launch it is in.
// Bound by the FP32 units and shared memory; the figures are at small_takes.
#pragma once
#include <string.h>

#include <algorithm>
#include <vector>

#include "s2g_common.cuh"
#include "s2g_internal.h"

namespace s2g {

constexpr int kSmallT = 256;

// Functions of a block, N in all: enough rows for its threads (bw 16: four, above: two), fewer as long as every
// block has its SM (bw 20, four functions: 12.8 and 11.1 us with two a block, 9.9 and 8.8 with one).
inline int small_nf(int B, int N, int sms) {
    int nf = B <= 16 ? 4 : 2;
    while (nf > 1 && (N + nf / 2 - 1) / (nf / 2) <= sms) nf /= 2;
    return nf;
}
__host__ __device__ constexpr int small_pad(int n) { return (n + 3) & ~3; }
// Row of Z, Y, O: 2B entries for each function, an odd number of 16-byte units.
__host__ __device__ constexpr int small_pitch(int B, int nf) { return 4 * ((nf * 2 * B + 3) / 4 | 1); }

// The row DFT's parts (odd B: cosines, sines; even B: each for even and odd orders): rows of Z and O, orders.
struct SmallKind {
    int start, n;       // rows: longitudes k0 ..
    int k0, part, m0;   // first longitude, 0 cosines or 1 sines, first order
};
__host__ __device__ constexpr bool small_twice(int B) { return B % 2 == 0; }
__host__ __device__ constexpr int small_kinds(int B) { return small_twice(B) ? 4 : 2; }
__host__ __device__ constexpr int small_orders(int B) { return small_twice(B) ? B / 2 : B; }      // of a kind
__host__ __device__ constexpr int small_longs(int B) { return (small_twice(B) ? B / 2 : B) + 1; }  // at most
__host__ __device__ inline SmallKind small_kind(int B, int kd) {
    const int h = B / 2;
    if (!small_twice(B)) return kd ? SmallKind{B + 1, B - 1, 1, 1, 0} : SmallKind{0, B + 1, 0, 0, 0};
    return kd == 0   ? SmallKind{0, h + 1, 0, 0, 0}
           : kd == 1 ? SmallKind{h + 1, h, 0, 0, 1}
           : kd == 2 ? SmallKind{2 * h + 1, h - 1, 1, 1, 0} : SmallKind{3 * h, h, 1, 1, 1};
}

struct SmallTab {  // device, per bandwidth
    const float* ft;    // forward rows [row of Z][order of its kind, padded to 4]: cosines or minus sines
    const float* it;    // inverse rows [kind][order][longitude, padded]: the same times 1 or 2 over sqrt(2 pi)
    const float* pf;    // P(l,m,j) w_j sqrt(2 pi) / S, [tile / 32][j / 4][4 degrees][tile % 32][4 j]
    const float* pi;    // P(l,m,j), [(m, l)][j padded to 4]
    const int* tiles;   // of pf: up to four degrees of one parity of an order: m, first l, count in 8 bits each
    int ntiles;         // a multiple of 32
};

struct SmallArgs {
    int B, N, nf;       // B 0: not a small class; nf: functions of a block (small_nf)
    SmallTab t;
    const float* in;    // grid (forward)
    float* out;         // grid (inverse)
    float *rc, *ic;     // coefficients, read by the inverse
    const int64_t *gmap, *cmap;  // function -> offset of its samples, coefficients (null: back to back)
};

inline size_t small_smem(int B, int nf, bool fwd) {
    const size_t z = (size_t)2 * B * small_pitch(B, nf);
    return sizeof(float) * (fwd ? z + (size_t)2 * B * (2 * nf * small_pad(B) + 4) : 2 * z);
}

__device__ __forceinline__ void small_fma(float (&a)[4][4], const float4& x, const float4& y) {
    const float u[4] = {x.x, x.y, x.z, x.w}, v[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) a[i][j] = fmaf(u[i], v[j], a[i][j]);
}

// acc = sum over i < n of x(i) y(i), the even and the odd terms apart: half the roundings of one chain (error
// of the inverse at bw 16: 0.93e-7 against 1.03e-7)
template <class X, class Y>
__device__ __forceinline__ void small_sum(float (&acc)[4][4], int n, X x, Y y) {
    float odd[4][4] = {};
#pragma unroll 2
    for (int i = 0; i + 1 < n; i += 2) {
        small_fma(acc, x(i), y(i));
        small_fma(odd, x(i + 1), y(i + 1));
    }
    if (n & 1) small_fma(acc, x(n - 1), y(n - 1));
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += odd[i][j];
}

__device__ __forceinline__ float4 small_ld(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 small_ldg(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// Brings a table to L1 while the data come in; a launch starts with nothing there.
__device__ __forceinline__ void small_prefetch(const float* p, int n) {
    for (int i = threadIdx.x * 32; i < n; i += kSmallT * 32) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + i));
}

__device__ __forceinline__ void small_fwd_body(const SmallArgs& p, int blk, float* sm) {
    const int B = p.B, S = 2 * B, NF = p.nf, RP = small_pitch(B, NF), BP = small_pad(B), GS = 2 * NF * BP + 4;
    const int f0 = blk * NF, nf = min(NF, p.N - f0), R = nf * S;
    float *Z = sm, *G = sm + S * RP;
    small_prefetch(p.t.ft, S * small_pad(small_orders(B)));
    if (B <= 20 || NF == 1) small_prefetch(p.t.pf, p.t.ntiles * 4 * BP);
    // fold: eight longitudes by four latitudes a warp (whole sectors in, no bank conflicts out)
    {
        const int lane = threadIdx.x & 31, nj = (B + 3) / 4, KX = small_longs(B), nk = (KX + 7) / 8, h = B / 2;
        for (int w = threadIdx.x >> 5; w < nf * nj * nk; w += kSmallT / 32) {
            const int k = w % nk * 8 + (lane >> 2), j = w / nk % nj * 4 + (lane & 3), f = w / (nk * nj);
            if (k >= KX || j >= B) continue;
            const float* g = p.in + (p.gmap ? p.gmap[f0 + f] : (int64_t)(f0 + f) * S * S);
            const float *a = g + j * S, *b = g + (S - 1 - j) * S;
            float* z = Z + k * RP + f * S + j;
            auto both = [&](int row, float u, float v) {
                z[row * RP] = u + v;
                z[row * RP + B] = u - v;
            };
            if (!small_twice(B)) {
                const bool two = k > 0 && k < B;
                const float a0 = a[k], b0 = b[k], a1 = two ? a[S - k] : 0.f, b1 = two ? b[S - k] : 0.f;
                both(0, a0 + a1, b0 + b1);
                if (two) both(B, a0 - a1, b0 - b1);
            } else {
                // k = 0 stands for 0 and S/2 only, k = h for h and S - h
                const float a0 = a[k], b0 = b[k], a1 = k ? a[S - k] : 0.f, b1 = k ? b[S - k] : 0.f;
                const float a2 = k < h ? a[B - k] : 0.f, b2 = k < h ? b[B - k] : 0.f;
                const float a3 = k && k < h ? a[B + k] : 0.f, b3 = k && k < h ? b[B + k] : 0.f;
                both(0, (a0 + a1) + (a2 + a3), (b0 + b1) + (b2 + b3));
                if (k < h) both(h + 1, (a0 + a1) - (a2 + a3), (b0 + b1) - (b2 + b3));
                if (k && k < h) both(2 * h, (a0 - a1) - (a2 - a3), (b0 - b1) - (b2 - b3));
                if (k) both(3 * h - 1, (a0 - a1) + (a2 - a3), (b0 - b1) + (b2 - b3));
            }
        }
        if (BP != B)
            for (int i = threadIdx.x; i < S * 2 * NF; i += kSmallT)
                for (int j = B; j < BP; ++j) G[i / (2 * NF) * GS + i % (2 * NF) * BP + j] = 0.f;
    }
    __syncthreads();
    const int M = small_orders(B), MP = small_pad(M), MT = MP / 4, RT = (R + 3) / 4, ms = small_twice(B) ? 2 : 1;
    const int rb = (RT + 7) / 8, mb = (MT + 3) / 4;
    for (int q = threadIdx.x; q < small_kinds(B) * rb * mb * 32; q += kSmallT) {  // a warp: 8 x 4 tiles
        const int w = q >> 5, rt = w % rb * 8 + (q & 7), mt = w / rb % mb * 4 + (q >> 3 & 3);
        if (rt >= RT || mt >= MT) continue;
        const SmallKind kd = small_kind(B, w / (rb * mb));
        const int part = kd.part;
        const float *z = Z + kd.start * RP + 4 * rt, *t = p.t.ft + kd.start * MP + 4 * mt;
        float acc[4][4] = {};
        small_sum(acc, kd.n, [&](int k) { return small_ldg(t + k * MP); }, [&](int k) { return small_ld(z + k * RP); });
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int m = ms * (4 * mt + i) + kd.m0;
            if (4 * mt + i >= M) break;
            if ((B & 3) == 0) {
                const int r = 4 * rt, f = r / S, rem = r - f * S, par = rem >= B;
                *reinterpret_cast<float4*>(G + (m * 2 + par) * GS + (2 * f + part) * BP + rem - par * B) =
                    make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int r = 4 * rt + c, f = r / S, rem = r - f * S, par = rem >= B;
                    if (r < R) G[(m * 2 + par) * GS + (2 * f + part) * BP + rem - par * B] = acc[i][c];
                }
            }
        }
    }
    __syncthreads();
    const int cg = (2 * nf + 3) / 4;
    float* out = Z;  // [function][re, im][B B]
    for (int q = threadIdx.x; q < p.t.ntiles * cg; q += kSmallT) {
        const int ti = q % p.t.ntiles, c0 = q / p.t.ntiles * 4, t = __ldg(p.t.tiles + ti);
        const int m = t & 255, l0 = t >> 8 & 255, n = t >> 16, par = (l0 + m) & 1;
        const int at = m * B - m * (m - 1) / 2 - m;  // place of (m, l) less l
        const float* g = G + (m * 2 + par) * GS;
        const float* P = p.t.pf + (ti >> 5) * (BP * 128) + (ti & 31) * 4;
        const float* g4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) g4[i] = g + min(c0 + i, 2 * nf - 1) * BP;
        float acc[4][4] = {}, odd[4][4] = {};
#pragma unroll 2
        for (int j = 0; j < BP; j += 4) {
            float4 y[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) y[c] = small_ld(g4[c] + j);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 x = small_ldg(P + (j + i) * 128);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    acc[i][c] = fmaf(x.x, y[c].x, acc[i][c]);
                    odd[i][c] = fmaf(x.y, y[c].y, odd[i][c]);
                    acc[i][c] = fmaf(x.z, y[c].z, acc[i][c]);
                    odd[i][c] = fmaf(x.w, y[c].w, odd[i][c]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= n) break;
            const int l = l0 + 2 * i, neg = index_of_harmonic_coeff(-m, l, B);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (c0 + c >= 2 * nf) break;
                float* o = out + (c0 + c) * B * B;
                const float v = acc[i][c] + odd[i][c];
                o[at + l] = v;
                if (m) o[neg] = ((m + c) & 1) ? -v : v;  // (-1)^m conj; c0 is even
            }
        }
    }
    __syncthreads();
    for (int f = 0; f < nf; ++f) {
        const int64_t o = p.cmap ? p.cmap[f0 + f] : (int64_t)(f0 + f) * B * B;
        for (int i = threadIdx.x; i < B * B; i += kSmallT) {
            p.rc[o + i] = out[2 * f * B * B + i];
            p.ic[o + i] = out[(2 * f + 1) * B * B + i];
        }
    }
}

__device__ __forceinline__ void small_inv_body(const SmallArgs& p, int blk, float* sm) {
    const int B = p.B, S = 2 * B, NF = p.nf, RP = small_pitch(B, NF), BP = small_pad(B), KP = small_pad(small_longs(B));
    const int f0 = blk * NF, nf = min(NF, p.N - f0), R = nf * S, NC = (2 * NF + 3) & ~3, np = B * (B + 1) / 2;
    float *Y = sm, *O = sm + S * RP, *C = O;  // the coefficients' place is the sums' later
    small_prefetch(p.t.pi, NF == 1 ? np * BP : min(np * BP, 8192));
    small_prefetch(p.t.it, small_kinds(B) * small_orders(B) * KP);
    for (int f = 0; f < nf; ++f) {
        const int64_t o = p.cmap ? p.cmap[f0 + f] : (int64_t)(f0 + f) * B * B;
#pragma unroll 2
        for (int i = threadIdx.x; i < np; i += kSmallT) {
            C[i * NC + 2 * f] = p.rc[o + i];
            C[i * NC + 2 * f + 1] = p.ic[o + i];
        }
    }
    __syncthreads();
    const int JT = BP / 4, cg = (2 * nf + 3) / 4;
    for (int q = threadIdx.x; q < B * 2 * cg * JT; q += kSmallT) {
        const int jt = q % JT, c0 = q / JT % cg * 4, par = q / (JT * cg) & 1, m = q / (JT * cg) >> 1;
        const int at = m * B - m * (m - 1) / 2 + par, n = (B - m - par + 1) / 2;
        const float *P = p.t.pi + at * BP + 4 * jt, *c = C + at * NC + c0;
        float acc[4][4] = {};
        small_sum(acc, n, [&](int i) { return small_ld(c + 2 * i * NC); }, [&](int i) { return small_ldg(P + 2 * i * BP); });
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int col = c0 + i;
            if (col >= 2 * nf) break;
            float* y = Y + ((col & 1) * B + m) * RP + (col >> 1) * S + par * B + 4 * jt;
            if ((B & 3) == 0) {
                *reinterpret_cast<float4*>(y) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (4 * jt + j < B) y[j] = acc[i][j];
            }
        }
    }
    __syncthreads();
    const int M = small_orders(B), ms = small_twice(B) ? 2 : 1, KT = KP / 4, RT = (R + 3) / 4;
    const int rb = (RT + 7) / 8, kb = (KT + 3) / 4;
    for (int q = threadIdx.x; q < small_kinds(B) * rb * kb * 32; q += kSmallT) {  // a warp: 8 x 4 tiles
        const int w = q >> 5, rt = w % rb * 8 + (q & 7), kt = w / rb % kb * 4 + (q >> 3 & 3), ki = w / (rb * kb);
        if (rt >= RT || kt >= KT) continue;
        const SmallKind kd = small_kind(B, ki);
        const float *y = Y + (kd.part * B + kd.m0) * RP + 4 * rt, *t = p.t.it + ki * M * KP + 4 * kt;
        float acc[4][4] = {};
        small_sum(acc, M, [&](int a) { return small_ldg(t + a * KP); }, [&](int a) { return small_ld(y + ms * a * RP); });
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = 4 * kt + i - kd.k0;
            if (k >= 0 && k < kd.n)
                *reinterpret_cast<float4*>(O + (kd.start + k) * RP + 4 * rt) =
                    make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, nj = (B + 3) / 4, KX = small_longs(B), nk = (KX + 7) / 8, h = B / 2;
    for (int w = threadIdx.x >> 5; w < nf * nj * nk; w += kSmallT / 32) {
        const int k = w % nk * 8 + (lane >> 2), j = w / nk % nj * 4 + (lane & 3), f = w / (nk * nj);
        if (k >= KX || j >= B) continue;
        float* g = p.out + (p.gmap ? p.gmap[f0 + f] : (int64_t)(f0 + f) * S * S);
        float *a = g + j * S, *b = g + (S - 1 - j) * S;
        const float* o = O + k * RP + f * S + j;
        auto put = [&](int x, float e, float d) {  // even and odd latitude parts
            a[x] = e + d;
            b[x] = e - d;
        };
        if (!small_twice(B)) {
            const bool two = k > 0 && k < B;
            const float ce = o[0], co = o[B], se = two ? o[B * RP] : 0.f, so = two ? o[B * RP + B] : 0.f;
            put(k, ce + se, co + so);
            if (two) put(S - k, ce - se, co - so);
        } else {
            const bool in = k && k < h;
            float c[2], d[2], s[2], t[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float c0 = o[q * B], c1 = k < h ? o[(h + 1) * RP + q * B] : 0.f;
                const float s0 = in ? o[2 * h * RP + q * B] : 0.f, s1 = k ? o[(3 * h - 1) * RP + q * B] : 0.f;
                c[q] = c0 + c1, d[q] = c0 - c1, s[q] = s0 + s1, t[q] = s1 - s0;
            }
            put(k, c[0] + s[0], c[1] + s[1]);
            if (k) put(S - k, c[0] - s[0], c[1] - s[1]);
            if (k < h) put(B - k, d[0] + t[0], d[1] + t[1]);
            if (in) put(B + k, d[0] - t[0], d[1] - t[1]);
        }
    }
}

// OCC: blocks an SM's registers are shared out for.
template <bool FWD, int OCC>
__global__ void __launch_bounds__(kSmallT, OCC) k_small(const __grid_constant__ SmallArgs p) {
    extern __shared__ __align__(16) float small_sm[];
    if constexpr (FWD) small_fwd_body(p, blockIdx.x, small_sm);
    else small_inv_body(p, blockIdx.x, small_sm);
}

// Tables of bandwidth B as one array: forward rows, inverse rows, pf, pi, then the forward's tiles as ints.
// weights: the quadrature weights of the 2B latitudes.
inline std::vector<float> small_tables(int B, const double* weights, size_t (&off)[4], size_t& tiles, int& ntiles) {
    const int S = 2 * B, BP = small_pad(B), KP = small_pad(small_longs(B)), M = small_orders(B), MP = small_pad(M);
    const int ms = small_twice(B) ? 2 : 1;
    const long double pi = 3.141592653589793238462643383279502884L;
    std::vector<float> v;
    auto term = [&](const SmallKind& kd, int k, int m) -> long double {  // exact zeros of the sines stay zero
        const int q = k * m % S;
        const long double a = 2 * pi * q / S;
        return kd.part ? (q % B ? -sinl(a) : 0.0L) : cosl(a);
    };
    off[0] = 0;
    for (int ki = 0; ki < small_kinds(B); ++ki) {
        const SmallKind kd = small_kind(B, ki);
        for (int r = 0; r < kd.n; ++r)
            for (int a = 0; a < MP; ++a) v.push_back(a < M ? (float)term(kd, kd.k0 + r, ms * a + kd.m0) : 0.f);
    }
    off[1] = v.size();
    for (int ki = 0; ki < small_kinds(B); ++ki) {
        const SmallKind kd = small_kind(B, ki);
        for (int a = 0; a < M; ++a)
            for (int k = 0; k < KP; ++k) {
                const int m = ms * a + kd.m0;
                v.push_back(k < small_longs(B) ? (float)((m ? 2 : 1) / sqrtl(2 * pi) * term(kd, k, m)) : 0.f);
            }
    }
    const size_t np = (size_t)B * (B + 1) / 2;
    std::vector<int> tile, place(np), row(np);  // tiles; tile and row of each (m, l)
    for (int m = 0; m < B; ++m)
        for (int par = 0; par < 2; ++par)
            for (int l = m + par; l < B; l += 8) {
                const int n = std::min(4, (B - l + 1) / 2);
                for (int i = 0; i < n; ++i) {
                    const int at = m * B - m * (m - 1) / 2 + l + 2 * i - m;
                    place[at] = (int)tile.size();
                    row[at] = i;
                }
                tile.push_back(m | l << 8 | n << 16);
            }
    while (tile.size() % 32) tile.push_back(0);
    ntiles = (int)tile.size();
    off[2] = v.size();
    off[3] = off[2] + (size_t)ntiles * 4 * BP;
    v.resize(off[3] + np * BP, 0.f);
    for (int j = 0; j < B; ++j) {
        const long double a = pi * (2 * j + 1) / (2 * (long double)S), x = cosl(a), s = sinl(a);
        const long double w = (long double)weights[j] * sqrtl(2 * pi) / S;
        long double top = sqrtl(0.5L);
        size_t at = 0;
        for (int m = 0; m < B; ++m) {
            if (m) top *= -sqrtl((2 * m + 1) / (2 * (long double)m)) * s;
            long double cur = top, prev = 0;
            for (int l = m; l < B; ++l, ++at) {
                v[off[2] + ((size_t)(place[at] / 32) * BP + j / 4 * 4 + row[at]) * 128 + place[at] % 32 * 4 + j % 4] =
                    (float)(cur * w);
                v[off[3] + at * BP + j] = (float)cur;
                const long double d = (l + 1.0L - m) * (l + 1.0L + m);
                const long double nx = sqrtl((2 * l + 3.0L) * (2 * l + 1.0L) / d) * x * cur -
                                       (l > m ? sqrtl((2 * l + 3.0L) * (l - m) * (l + m) / ((2 * l - 1.0L) * d)) * prev : 0.0L);
                prev = cur;
                cur = nx;
            }
        }
    }
    tiles = v.size();
    for (int t : tile) {
        float f;
        memcpy(&f, &t, sizeof f);
        v.push_back(f);
    }
    return v;
}

}  // namespace s2g
