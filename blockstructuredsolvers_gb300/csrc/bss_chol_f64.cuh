// FP64 Cholesky + inverse of an NB x NB SPD tile in shared memory, laid out
// for GB300's FP64 pipe.
//
// What bounds it: an FP64 warp-instruction (FMA, add, multiply alike, however
// few lanes are active) holds its scheduler's FP64 port for 64 cycles, and
// the SM retires one per 19 cycles over its four schedulers (measured); the
// dependent latency of one FMA is the same 64 cycles.  An IEEE square root
// is 810 cycles and a division 550.  So the serial part, the pivots, should
// issue few instructions from one warp, and everything else should fill its
// lanes and spread over all four schedulers.
//
//   * pivot tiles (16 x 16, one warp): in-place Gauss-Jordan on [S | I], so
//     the tile's factor and its inverse come out of one sweep with all 16
//     column slots always in use: S = L D L^T, V = L^-T D^-1/2.  A pivot
//     costs 1 + (rows below) / 2 FP64 warp-instructions; its reciprocal is an
//     FP32 seed and one third-order correction in integers (below) instead of
//     a square root and a division, runs under the FMAs of the rows that do
//     not hold the next pivot, and the 16 square roots are taken together.
//   * row panels U(K, J) = V_KK^T S(K, J), trailing updates and V's
//     off-diagonal columns: one output per lane, rows grouped so that the
//     triangular contractions of a warp have (almost) one length.
//   * V's block column K - 1 is formed by the warps of the other three
//     schedulers while warp 0 factors pivot tile K.
//
// Measured against the form before it (IEEE square root and division per
// pivot, one-warp back substitution per tile, inverse in stages): plain FP64
// factor + solve of N = 16384, n = 64: 42.1 -> 35.6 ms, N = 1531, n = 37:
// 7.55 -> 6.42 ms, N = 100, n = 32: 936 -> 679 us, N = 2048, n = 128: 63.9 ->
// 61.5 ms (the rest is the chain step's products).
//
// Reciprocal: y = FP32 reciprocal of the pivot's mantissa (|e| <= 2^-21 for
// e = 1 - p y), 1/p = y (1 + e + e^2) / (1 - e^3), so y (1 + e + e^2) is off by
// |e|^3 < 2^-62; reciprocal square root: y (1 + e/2 + 3 e^2 / 8) with
// e = 1 - p y^2, off by (5/16) |e|^3 (Newton-Householder iterations of third
// order).  The seed is a function of 23 mantissa bits, and every one of them
// is tried (bss_diag_pivot_selftest): no seed of a reciprocal is below 1/2,
// and the results are within one unit of the last place of 1 / p and two of
// 1 / sqrt(p) (itself rounded twice).  Pivots with a biased exponent outside
// [24, 2022] take IEEE divide and square root.
#pragma once

namespace bss {

// y 2^-shift as FP64, for a normal FP32 y: exponent arithmetic on the bits
__device__ __forceinline__ double f64_from_seed(float y, int shift)
{
    const unsigned b = __float_as_uint(y);
    return __hiloint2double((int)((((b >> 23) + 896u - (unsigned)shift) << 20) | ((b & 0x7FFFFFu) >> 3)),
                            (int)(b << 29));
}

__device__ __forceinline__ bool f64_pivot_ordinary(double p)
{
    return (unsigned)(__double2hiint(p) - (24 << 20)) < (unsigned)(1999 << 20);
}

// 1/p for an ordinary p, in integer arithmetic (the FP64 port stays free):
// p = M 2^(E - 1075), the FP32 seed y = Y 2^-24 of the mantissa m = M 2^-52;
// e = 1 - m y = D 2^-76 with D = -(M Y mod 2^64), then y (1 + e + e^2) in units
// of 2^-56, rounded once
__device__ __forceinline__ double f64_rcp(double p)
{
    const unsigned hi = (unsigned)__double2hiint(p), lo = (unsigned)__double2loint(p);
    const unsigned mh = (hi & 0xFFFFFu) | 0x100000u;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3F800000u | ((hi & 0xFFFFFu) << 3) | (lo >> 29))));
    const unsigned yb = __float_as_uint(y);
    const unsigned Y = ((yb & 0x7FFFFFu) | 0x800000u) << ((yb >> 23) - 126u);  // y in (1/2, 1]
    const unsigned long long MY = (unsigned long long)lo * Y + ((unsigned long long)(mh * Y) << 32);
    const long long D = (long long)(0ull - MY);
    const int es = (int)(D >> 32);
    const long long t = (D >> 20) + __mulhi(es, es);  // e + e^2 in units of 2^-56
    const long long Yt = (long long)((unsigned long long)(unsigned)t * Y + ((unsigned long long)((unsigned)(t >> 32) * Y) << 32));
    const unsigned long long R = ((unsigned long long)Y << 32) + (unsigned long long)(Yt >> 24);
    return __longlong_as_double((long long)(((R + 4) >> 3) + ((unsigned long long)(1021u + 1023u - (hi >> 20)) << 52)));
}

// 1/sqrt(p), p > 0
__device__ __forceinline__ double f64_rsqrt(double p)
{
    if (!f64_pivot_ordinary(p)) return 1.0 / sqrt(p);
    const unsigned hi = (unsigned)__double2hiint(p), lo = (unsigned)__double2loint(p);
    const int e2 = (int)(hi >> 20) - 1023, k = e2 >> 1;  // p = m 4^k, m in [1, 4)
    const float m = __uint_as_float(((unsigned)(127 + (e2 & 1)) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29));
    const double y = f64_from_seed(rsqrtf(m), k);
    const double e = fma(-(p * y), y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// one warp: V_KK of the pivot tile at (o, o) of sS (upper triangle read),
// written to sV with zeros below the diagonal; nonzero if a pivot failed.
// Lane = column slot c (lane % 16) and row parity h (lane / 16); v[q] is row
// 2 q + h.  Slot c of a row r holds S(r, c) until column c is eliminated and
// the inverse's L^-1(r, c) from then on.
// Out of line: 40 KB of straight code that every panel shares (one copy per
// panel ran 1.5 times as long, on instruction fetches).
template <int LD>
__device__ __noinline__ int f64_pivot_tile(const double *sS, double *sV, int o, int lane)
{
    constexpr unsigned ALL = 0xFFFFFFFFu;
    const int c = lane & 15, h = lane >> 4;
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int r = 2 * q + h;
        v[q] = r <= c ? sS[(o + r) + (o + c) * LD] : 0.0;
    }
    int bad = 0;
    double dj = 1.0;
    double piv = __shfl_sync(ALL, v[0], 0);
    double row = __shfl_sync(ALL, v[0], c);  // row j: S right of the pivot, L^-1 left of it
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int hj = j & 1, qj = j >> 1;
        if (c == j) row = 1.0;
        double s[8];  // S(j, row q of this lane)
#pragma unroll
        for (int q = (j + 1) >> 1; q < 8; ++q) s[q] = __shfl_sync(ALL, v[qj], 2 * q + h + 16 * hj);
        double m;  // row / pivot
        if (f64_pivot_ordinary(piv)) {
            m = row * f64_rcp(piv);
        } else {
            if (!(piv > 0.0 && piv < INFINITY)) {
                bad = 1;
                piv = 1.0;
            }
            m = row / piv;
        }
        if (c == j) dj = piv;
        // row j + 1 first: the next pivot's broadcasts and reciprocal run under the other rows' FMAs
#pragma unroll
        for (int q = (j + 1) >> 1; q < 8; ++q) {
            const double base = c == j ? 0.0 : v[q];
            const double x = fma(-s[q], m, base);
            if (2 * q > j || h == 1) v[q] = x;  // the first q of an even j also holds the pivot row (h = 0)
            if (q == (j + 1) >> 1) {
                piv = __shfl_sync(ALL, v[q], (j + 1) + 16 * (hj ^ 1));
                row = __shfl_sync(ALL, v[q], c + 16 * (hj ^ 1));
            }
        }
    }
    const double rs = f64_rsqrt(dj);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int r = 2 * q + h;
        const double rr = __shfl_sync(ALL, rs, r);
        sV[(o + c) + (o + r) * LD] = c < r ? v[q] * rr : (c == r ? rr : 0.0);
    }
    return bad;
}

// units of a half-warp (16 lanes): unit u = (row a, group g of 16 columns)
// with a = u / G, so that the two units of a warp differ by one row at most
// and the triangular sums of a warp have nearly one length

// row panel of pivot tile K, in place: U(o + a, c) = sum_{p <= a} V(o + p, o + a) S(o + p, c)
// for the G tiles right of it.  All warps; ends with a barrier.
template <int LD, int NW, int G>
__device__ __forceinline__ void f64_row_panel(double *sS, const double *sV, int o, int warp, int lane)
{
    constexpr int IT = (8 * G + NW - 1) / NW;
    double out[IT];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        // rounds alternate direction: every warp gets about the same share of long rows
        const int x = it * NW + ((it & 1) ? NW - 1 - warp : warp);
        out[it] = 0.0;
        if (x < 8 * G) {
            const int u = 2 * x + (lane >> 4), a = u / G, g = u - a * G;
            const double *vc = sV + o + (o + a) * LD;
            const double *sc = sS + o + (o + 16 + 16 * g + (lane & 15)) * LD;
            double s0 = 0.0, s1 = 0.0;
            for (int p = 0; p <= a; p += 2) {  // V(p, a) = 0 for p > a
                const double2 vv = *reinterpret_cast<const double2 *>(vc + p);
                const double2 ss = *reinterpret_cast<const double2 *>(sc + p);
                s0 = fma(vv.x, ss.x, s0);
                s1 = fma(vv.y, ss.y, s1);
            }
            out[it] = s0 + s1;
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int x = it * NW + ((it & 1) ? NW - 1 - warp : warp);
        if (x < 8 * G) {
            const int u = 2 * x + (lane >> 4), a = u / G, g = u - a * G;
            sS[(o + a) + (o + 16 + 16 * g + (lane & 15)) * LD] = out[it];
        }
    }
    __syncthreads();
}

// trailing update of pivot tile K: S(a, b) -= sum_p U(o + p, a) U(o + p, b)
// for a <= b in the M x M block right of and below it, one packed
// upper-triangle element per thread and round
template <int LD, int THREADS, int M>
__device__ __forceinline__ void f64_trailing(double *sS, int o, int tid)
{
    constexpr int COUNT = M * (M + 1) / 2;
    for (int e = tid; e < COUNT; e += THREADS) {
        int b = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
        if (b * (b + 1) / 2 > e) --b;
        if ((b + 1) * (b + 2) / 2 <= e) ++b;
        const int a = e - b * (b + 1) / 2;
        const double *pa = sS + o + (o + 16 + a) * LD, *pb = sS + o + (o + 16 + b) * LD;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int p = 0; p < 16; p += 2) {
            const double2 x = *reinterpret_cast<const double2 *>(pa + p);
            const double2 y = *reinterpret_cast<const double2 *>(pb + p);
            s0 = fma(x.x, y.x, s0);
            s1 = fma(x.y, y.y, s1);
        }
        sS[(o + 16 + a) + (o + 16 + b) * LD] -= s0 + s1;
    }
}

// block column J of V above its pivot tile, from V U = I:
//   T(r, c) = sum_{q = r .. 16 J - 1} V(r, q) U(q, 16 J + c)    (kept in the scratch lower tiles of row J of sS)
//   V(r, 16 J + b) = -sum_{c <= b} T(r, c) V(16 J + c, 16 J + b)
// by NWX warps (this one is number wx of them); `bar` joins exactly those
// (0: the whole CTA).
template <int LD, int NWX, int J>
__device__ __forceinline__ void f64_inv_column(double *sS, double *sV, int wx, int lane, int bar)
{
    const int half = lane >> 4, c = lane & 15;
    for (int x = wx; x < 8 * J; x += NWX) {
        const int r = 2 * x + half;
        const double *uc = sS + (16 * J + c) * LD;
        double s0 = 0.0, s1 = 0.0;
        for (int q = 2 * x; q < 16 * J; q += 2) {  // V(r, q) = 0 for q < r
            const double2 u = *reinterpret_cast<const double2 *>(uc + q);
            s0 = fma(sV[r + q * LD], u.x, s0);
            s1 = fma(sV[r + (q + 1) * LD], u.y, s1);
        }
        sS[(16 * J + c) + r * LD] = s0 + s1;
    }
    if (bar == 0)
        __syncthreads();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * NWX) : "memory");
    for (int x = wx; x < 8 * J; x += NWX) {
        const int u = 2 * x + half, b = u / J, g = u - b * J, r = 16 * g + c;
        const double *tc = sS + 16 * J + r * LD;                 // T(r, .)
        const double *vc = sV + 16 * J + (16 * J + b) * LD;      // V(16 J + ., 16 J + b)
        double s0 = 0.0, s1 = 0.0;
        for (int q = 0; q <= b; q += 2) {
            const double2 t = *reinterpret_cast<const double2 *>(tc + q);
            const double2 v = *reinterpret_cast<const double2 *>(vc + q);
            s0 = fma(t.x, v.x, s0);
            s1 = fma(t.y, v.y, s1);
        }
        sV[r + (16 * J + b) * LD] = -(s0 + s1);
    }
}

// the warps that form V's block columns while warp 0 factors a pivot tile:
// those of the other three schedulers
template <int NW>
__device__ __forceinline__ constexpr int f64_aside()
{
    return NW - (NW + 3) / 4;
}

// `aside(K)` runs on the warps other than warp 0 while that factors pivot tile
// K: the caller's own work, which must not write sS or sV.
struct F64NoAside {
    __device__ __forceinline__ void operator()(int) const {}
};

template <int LD, int NW, int NB, int K, class Aside>
__device__ __forceinline__ void f64_chol_panel(double *sS, double *sV, int *sflag, int warp, int lane, Aside &aside)
{
    constexpr int KP = NB / 16, o = 16 * K;
    constexpr int NA = f64_aside<NW>();
    if (warp == 0) {
        const int bad = f64_pivot_tile<LD>(sS, sV, o, lane);
        if (bad && lane == 0) *sflag = 1;
    } else {
        aside(K);
        if constexpr (K >= 2) {
            if (warp % 4 != 0) f64_inv_column<LD, NA, K - 1>(sS, sV, warp - 1 - warp / 4, lane, 1);
        }
    }
    __syncthreads();
    if constexpr (K + 1 < KP) {
        f64_row_panel<LD, NW, KP - 1 - K>(sS, sV, o, warp, lane);
        f64_trailing<LD, 32 * NW, NB - o - 16>(sS, o, 32 * warp + lane);
        __syncthreads();
        f64_chol_panel<LD, NW, NB, K + 1>(sS, sV, sflag, warp, lane, aside);
    } else if constexpr (KP > 1) {
        f64_inv_column<LD, NW, KP - 1>(sS, sV, warp, lane, 0);
        __syncthreads();
    }
}

// the whole tile (contract of chol_inv_blocked; sS keeps no factor)
template <int NB, int THREADS, class Aside>
__device__ __forceinline__ int f64_chol_inv_i(double *sS, double *sV, int *sflag, int tid, Aside &aside)
{
    if (tid == 0) *sflag = 0;  // (set by the same thread: no barrier needed before it)
    f64_chol_panel<Geo<double, NB>::LD, THREADS / 32, NB, 0>(sS, sV, sflag, tid >> 5, tid & 31, aside);
    return *sflag;
}
template <int NB, int THREADS>
__device__ __noinline__ int f64_chol_inv(double *sS, double *sV, int *sflag, int tid)
{
    F64NoAside none;
    return f64_chol_inv_i<NB, THREADS>(sS, sV, sflag, tid, none);
}

}  // namespace bss
