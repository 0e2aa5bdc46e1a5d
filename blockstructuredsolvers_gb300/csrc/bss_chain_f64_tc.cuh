// Chain factor kernel for FP64 factors of 17..64-wide blocks with the chain
// step's products on the 5th-generation tensor cores: the same recursion and
// outputs as chain_factor_body (V_i, W_i, Y_i, S_LL / S_RR / S_LR; also the
// sequential coarsest chain), one CTA per partition.
//
// What bounds it: GB300's FP64 pipe retires 1.7 FMA per clock and SM, so the
// five n^3 products of a 64-wide step took ~460K of its ~560K cycles.  FP16
// MMAs run 2400 times faster, and an FP64 product can be put together from
// FP16 products exactly (error-free splitting: Ozaki, Ogita, Oishi, Rump,
// Numer. Algorithms 59, 2012): every operand row is scaled by a power of two
// to |x| < 1 and cut into seven 8-bit digits,
//     x = sum_{s=0..6} d_s 2^-(6 + 8 s),   d_s an integer, |d_0| <= 64, |d_s| <= 128,
// which are exact in FP16; the products of digits s and t with s + t = l
// form level l, whose 64-term sums are integers below 2^23 and so exact in
// the FP32 accumulator of the MMA.  Levels 0..7 (34 digit products; level 8 is
// 2^-59 of the largest term) are put together in 64-bit integers and rounded
// to FP64 once.  Error: the digits hold 54 bits below the power of two above
// the row's largest element, so a product is off by ~2^-54 of the product of
// its two rows' largest elements.  That is an FP64 Cholesky's own error
// (2^-53 sqrt(S_aa S_bb)) as long as the contraction index has one scale.  In
// W^T W, Y^T W and Y^T Y it has: row r of W and Y is in units of the r-th
// pivot's root.  In Z^T V and B^T V it has not: where T = D T0 D, row k of Z and
// B goes with D_k and row k of V with 1 / D_k, and a row cut as it stands would
// lose log2(max D / min D) bits.  There index k is first balanced by the power
// of two h_k ~ sqrt(S_kk): 2^h_k V(k, .) and 2^-h_k Z(k, .), which cancel in the
// product, are two operands of one scale (S balanced has diagonal [1, 4)); it
// is an integer added to the exponents that the cut works with, and a result
// does not depend on a D of powers of two at all.  D in 2^+-40, 19 blocks: 0.2
// off without the balance, within 1e-12 with it, in the same time (N = 16384,
// n = 64: 10.1 ms; the step's asides are spread better as well).  What an FMA
// chain keeps and digits do not: terms of one balanced row that are smaller
// than 2^-54 of its largest.  Rows with an infinity or NaN give NaN.
//
// A step of the chain (NB = 64 or 32, the block padded with the identity):
//   P1 = [W_{i-1} | Y_{i-1}]^T W_{i-1}   -> S = A_i - W^T W (slot 0 rows), Z_i^T = -Y^T W (slot 1 rows)
//   PL = [W_{i-1} | Y_{i-1}]^T Y_{i-1}   -> S_LL += Y^T Y (slot 1 rows), during the first pivot tile
//   Cholesky + inverse V_i on the FP64 pipe (f64_chol_inv), Z_i and B_i cut into digits beside it
//   P2 = [Z_i | B_i]^T V_i               -> Y_i^T (slot 0 rows), W_i^T (slot 1 rows)
//
// Operand layout (FP16, K-major, no swizzle, core matrices of 8 rows x 16
// bytes, those of an 8-row group adjacent along K): digit s of slot j's row
// group g is at ((s NB/8 + g) 2 + j) GRP with GRP = 16 NB bytes.  As the A
// operand the groups of both slots follow one another (stride GRP: 128 MMA
// rows, slots alternating every 8); as the B operand one slot's groups of
// all digits do (stride 2 GRP), so one MMA with N = 64 J multiplies a digit of
// A with J digits of B and its J results land in J consecutive levels'
// accumulator columns.  The 34 digit products of a K-step are 12 MMAs instead
// of 34 and 64-column MMAs at a third of the rate are avoided.
//
// TMEM: 8 levels x NB columns (all 512 for NB = 64).  Shared memory: 214 KB
// (NB = 64, one CTA per SM), 58 KB (NB = 32; 128 registers allow two CTAs).
//
// Measured (the digit products of one operand pair: 4.7K cycles for NB = 64,
// 1.4K for NB = 32, against 131K and 16K for one product on the FP64 pipe):
// plain FP64 factor + solve of N = 16384, n = 64: 35.6 -> 11.3 ms; N = 1531,
// n = 37, k = 3: 6.42 -> 2.68 ms; N = 100, n = 32: 679 -> 435 us (10.1 ms, 2.1 ms
// and 372 us with the sweeps as they are now).  A 64-wide step takes ~145K cycles:
// 49K in the four pivot tiles, 46K in the Cholesky's other FP64 products, 31K
// cutting and putting together digits, 15K in MMAs.
#pragma once

namespace bss {

constexpr int SL_DIGITS = 7, SL_LEVELS = 8, SL_THREADS = 256;
constexpr int SL_NAN = 1 << 20;  // row exponent of a row with an infinity or a NaN

template <int NB>
struct SlGeo {
    static constexpr int LD = Geo<double, NB>::LD;
    static constexpr uint32_t GRP = 16u * NB;                    // 8 rows x NB digits
    static constexpr uint32_t SLICE = 2u * (NB / 8) * GRP;       // one digit of both slots
    static constexpr uint32_t VSLICE = (NB / 8) * GRP;           // one digit of the V operand
    static constexpr uint32_t TILE = (uint32_t)Geo<double, NB>::SLOT * 8u;  // sS, X, sV
    static constexpr uint32_t OFF_S = SL_DIGITS * SLICE;         // sS; after the Cholesky sS and X hold the V operand
    static constexpr uint32_t OFF_X = OFF_S + TILE;              // Z in FP64; after P2 (sS, sX) hold W and Y in FP64
    static constexpr uint32_t OFF_V = OFF_X + TILE;              // sV
    static constexpr uint32_t OFF_EX = OFF_V + TILE;             // row exponents: slot 0 (W, Z), Y, B (slot 1), V; hV, hB, none
    static constexpr uint32_t OFF_CTL = OFF_EX + 7u * 64u * 4u;
    static constexpr uint32_t BYTES = OFF_CTL + 64u;
    static constexpr uint32_t TMEM = SL_LEVELS * NB;
    static_assert(SL_DIGITS * VSLICE <= 2 * TILE, "the V operand overlays sS and X");
};

__device__ __forceinline__ uint64_t sl_desc(uint32_t saddr, uint32_t sbo)
{
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(128u >> 4) << 16;  // leading byte offset: next core matrix along K
    d |= (uint64_t)(sbo >> 4) << 32;   // stride byte offset: next 8-row group
    d |= (uint64_t)1 << 46;            // descriptor version of the sm_100 family
    return d;
}

// kind::f16, D = F32, A = B = F16, both K-major, M = 128
__host__ __device__ constexpr uint32_t sl_idesc(int N)
{
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void sl_mma1(uint32_t tm, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tm),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}

// every digit product of levels 0..7: A = both slots' rows at a, B = the NB
// rows per digit at b with 8-row groups bsbo bytes apart; one thread
template <int NB>
__device__ __forceinline__ void sl_mma(uint32_t tm, uint32_t a, uint32_t b, uint32_t bsbo)
{
    using G = SlGeo<NB>;
    constexpr int JMAX = 256 / NB;  // digits of B per MMA
    const uint32_t bslice = (NB / 8) * bsbo;
#pragma unroll 1
    for (int kk = 0; kk < NB / 16; ++kk) {
#pragma unroll
        for (int s = 0; s < SL_DIGITS; ++s) {
            const uint64_t da = sl_desc(a + s * G::SLICE + kk * 256u, G::GRP);
            const int J = SL_LEVELS - s < SL_DIGITS ? SL_LEVELS - s : SL_DIGITS;
            // digit 0 of A opens levels 0..6, digit 1 opens level 7 (with digit 6 of B)
            const int split = s == 1 ? J - 1 : J;
#pragma unroll
            for (int j = 0; j < J;) {
                const int end = j < split ? split : J;
                const int cnt = end - j < JMAX ? end - j : JMAX;
                const bool opens = s == 0 || (s == 1 && j == split);
                sl_mma1(tm + (uint32_t)((s + j) * NB), da, sl_desc(b + j * bslice + kk * 256u, bsbo),
                        sl_idesc(cnt * NB), (opens && kk == 0) ? 0u : 1u);
                j += cnt;
            }
        }
    }
}

// value v 2^e as FP64, in full: subnormal and infinite results, NaN for the
// marked exponents
static __device__ __noinline__ double sl_to_f64_rare(long long v, int e)
{
    if (e >= SL_NAN / 2) return __longlong_as_double(0x7FF8000000000000ll);
    const unsigned long long u0 = (unsigned long long)(v < 0 ? ~v : v);
    unsigned long long bits = 0;
    if (u0 != 0) {
        const int lz = __clzll((long long)u0), be = e + 63 - lz + 1023;
        const unsigned long long u = u0 << lz;
        if (be >= 2047)
            bits = 0x7FF0000000000000ull;
        else if (be > 0)
            bits = ((unsigned long long)(be - 1) << 52) + (u >> 11) + ((u >> 10) & 1ull);
        else if (be > -52)
            bits = (u >> (12 - be)) + ((u >> (11 - be)) & 1ull);
    }
    return __longlong_as_double((long long)(bits | (v < 0 ? 0x8000000000000000ull : 0ull)));
}
// the same for ordinary results, one rounding to nearest (|v| of a negative v
// is taken one unit, 2^-56 of the scale, small); sets `rare` where the above
// has to be asked instead.  32-bit operations spelled out (64-bit shifts by a
// variable compile to three times as many) and no branch, so that a thread's
// elements overlap: integer instructions run at half rate here and this is
// what a readout spends its time on.
__device__ __forceinline__ double sl_to_f64(long long v, int e, bool &rare)
{
    const unsigned vh = (unsigned)((unsigned long long)v >> 32), sg = (unsigned)((int)vh >> 31);
    const unsigned uh = vh ^ sg, ul = (unsigned)v ^ sg;
    const bool low = uh == 0;
    const unsigned h = low ? ul : uh, l = low ? 0u : ul;
    const int lz = __clz((int)h);
    const unsigned mh = __funnelshift_l(l, h, lz), ml = l << (lz & 31);  // bit 31 of mh set (h != 0)
    const int be1 = e + 63 + 1022 - lz - (low ? 32 : 0);                 // biased exponent - 1
    rare |= (unsigned)be1 > 2045u;  // (zeros too where the exponents are far down or marked)
    const unsigned ql = __funnelshift_r(ml, mh, 11), r = (ml >> 10) & 1u;
    unsigned lo, hi;
    asm("add.cc.u32 %0, %2, %3;\n addc.u32 %1, %4, %5;" : "=r"(lo), "=r"(hi) : "r"(ql), "r"(r), "r"(mh >> 11), "r"((unsigned)be1 << 20));
    lo = h ? lo : 0u;
    hi = h ? (hi | (sg & 0x80000000u)) : 0u;
    return __hiloint2double((int)hi, (int)lo);
}

// eight accumulator columns of this thread's TMEM lane, all levels -> FP64:
// row exponent er, column exponents ec[0..7]
template <int NB>
__device__ __forceinline__ void sl_read8(uint32_t addr, int er, const int *ec, double (&out)[8])
{
    uint32_t r[SL_LEVELS][8];
#pragma unroll
    for (int l = 0; l < SL_LEVELS; ++l)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[l][0]), "=r"(r[l][1]), "=r"(r[l][2]), "=r"(r[l][3]), "=r"(r[l][4]), "=r"(r[l][5]),
                       "=r"(r[l][6]), "=r"(r[l][7])
                     : "r"(addr + (uint32_t)(l * NB)));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    // FP32 integers to int32 through the bits of f + 1.5 2^23 (|f| <= 2^22: levels
    // 0..4, by 64 (|d_0| 128 2 + 128 128 (pairs - 2))); levels 5..7 reach 6 2^20:
    // 5 in two parts, 6 and 7 halved (their last bit is 2^-60 and less).  The
    // conversion instruction takes ~30 cycles of a scheduler, an add one.
    constexpr float C23 = 12582912.f, C24 = 25165824.f;
    constexpr unsigned B23 = 0x4B400000u, B24 = 0x4BC00000u;
    bool rare = false;
    long long vs[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        unsigned b[SL_LEVELS];
#pragma unroll
        for (int l = 0; l < 5; ++l) b[l] = __float_as_uint(__uint_as_float(r[l][q]) + C23);
        {
            const float f = __uint_as_float(r[5][q]), f2 = f + C24;  // f2: f to even
            const float rest = f - (f2 - C24);
            b[5] = 2u * __float_as_uint(f2) + __float_as_uint(rest + C23);
        }
#pragma unroll
        for (int l = 6; l < 8; ++l) b[l] = __float_as_uint(fmaf(__uint_as_float(r[l][q]), 0.5f, C23));
        // two levels each, |t| < 2^31
        const int t0 = (int)(b[0] * 256u + b[1] - (B23 * 256u + B23));
        const int t1 = (int)(b[2] * 256u + b[3] - (B23 * 256u + B23));
        const int t2 = (int)(b[4] * 256u + b[5] - (B23 * 256u + 2u * B24 + B23));
        const int t3 = (int)(b[6] * 256u + b[7] - (B23 * 256u + B23));  // halved
        // unit 2^-56 (level l has unit 2^-(12 + 8 l)); |v| <= 2^62
        vs[q] = (long long)((unsigned long long)(long long)t0 << 36) + (long long)t1 * (1 << 20) + (long long)t2 * 16 + (t3 >> 11);
        out[q] = sl_to_f64(vs[q], er + ec[q] - 56, rare);
    }
    if (rare) {
#pragma unroll
        for (int q = 0; q < 8; ++q) out[q] = sl_to_f64_rare(vs[q], er + ec[q] - 56);
    }
}

// The balance of contraction index k: h_k, half the exponent of a diagonal
// element of S (0 where it is no pivot), as what is added to the high words
// of V's row k (hV) and of B's and Z's (hB): +-h_k in the exponent field's
// place, less SL_BIAS, which keeps the sums of a field and h_k inside 32 bits.
constexpr int SL_BIAS = 1 << 30;
__device__ __forceinline__ void sl_balance(double s, int *hV, int *hB)
{
    const int E = __double2hiint(s) >> 20, h = (unsigned)E < 2047u ? (E - 1023) >> 1 : 0;
    *hV = h * (1 << 20) - SL_BIAS;
    *hB = -h * (1 << 20) - SL_BIAS;
}

// eight consecutive K values of one operand row as digits: 16 bytes per
// digit at dst + s * stride.  fe: the values' exponent fields (at least 1) as
// balanced, emax: the row's largest.
__device__ __forceinline__ void sl_put8(unsigned char *dst, uint32_t stride, const double (&x)[8], const int (&fe)[8],
                                        int emax)
{
    uint32_t lo[8], hi[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const unsigned xh = (unsigned)__double2hiint(x[q]), xl = (unsigned)__double2loint(x[q]);
        const unsigned mh = (xh & 0xFFFFFu) | ((xh & 0x7FF00000u) ? 0x100000u : 0u);
        int sh = emax - fe[q];  // (negative only for a zero)
        // |x| 2^54 / 2^(row exponent), rounded: ((M << 2) >> sh) + 1 >> 1
        const unsigned h0 = __funnelshift_l(xl, mh, 2), l0 = xl << 2;
        const bool far = sh >= 32;
        sh = min(sh, 63);
        unsigned h = far ? 0u : h0, l = far ? h0 : l0;
        l = __funnelshift_r(l, h, sh);  // (by sh % 32; h0 < 2^23, so a shift by 31 leaves nothing of it)
        h >>= (sh & 31);
        unsigned r0, r1;
        asm("add.cc.u32 %0, %2, 1;\n addc.u32 %1, %3, 0;" : "=r"(r0), "=r"(r1) : "r"(l), "r"(h));
        r0 = __funnelshift_r(r0, r1, 1);
        r1 >>= 1;
        const unsigned sg = (unsigned)((int)xh >> 31);
        // byte 6 - s = digit s + 128: (|x| ^ sg) - sg + 0x0080808080808080
        asm("add.cc.u32 %0, %2, %4;\n addc.u32 %1, %3, %5;"
            : "=r"(lo[q]), "=r"(hi[q])
            : "r"(r0 ^ sg), "r"(r1 ^ sg), "r"(0x80808080u - sg), "r"(0x00808080u));
    }
#pragma unroll
    for (int s = 0; s < SL_DIGITS; ++s) {
        const int byte = 6 - s;
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t a = byte < 4 ? lo[2 * u] : hi[2 * u], c = byte < 4 ? lo[2 * u + 1] : hi[2 * u + 1];
            const unsigned k = (unsigned)(byte & 3);
            // two FP16 numbers 1024 + byte, less 1024 + 128
            const uint32_t p = (__byte_perm(a, c, k | ((4u + k) << 8)) & 0x00FF00FFu) | 0x64006400u;
            asm("add.f16x2 %0, %1, %2;" : "=r"(w[u]) : "r"(p), "r"(0xE480E480u));
        }
        *reinterpret_cast<uint4 *>(dst + s * stride) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// one warp cuts eight operand rows into digits (lane: row lane % 8, quarter
// lane / 8 of K) at dst (the row group's first core matrix of digit 0), their
// exponents to exps[0..7].  row: the lane's row, its K values kstride apart,
// zero from kvalid on; value k is taken times 2^(+-h_k), h: hV or hB of
// sl_balance (h_k = 0: -SL_BIAS).  Out of line, in one copy: five callers, and
// the step's code should stay in the instruction cache.
template <int NB>
__device__ __noinline__ void sl_cut_group(unsigned char *dst, uint32_t stride, int *exps, const double *row,
                                          long long kstride, int kvalid, const int *h)
{
    constexpr int KE = NB / 4;
    const int lane = threadIdx.x & 31, k0 = (lane >> 3) * KE;
    double x[KE];
    int fe[KE];
#pragma unroll
    for (int q = 0; q < KE; ++q) x[q] = k0 + q < kvalid ? row[(k0 + q) * kstride] : 0.0;
    // the row's largest high word (a field of at least 1) as balanced, zeros left out
    constexpr int NAN_ROW = 0x7FFFFFFF;
    int top = 0, emax = -NAN_ROW;
#pragma unroll
    for (int q = 0; q < KE; ++q) {
        const int mag = __double2hiint(x[q]) & 0x7FFFFFFF;
        top = max(top, mag);
        fe[q] = max(mag, 1 << 20) + h[k0 + q];
        if ((mag | __double2loint(x[q])) != 0) emax = max(emax, fe[q]);
        fe[q] >>= 20;
    }
    if (top >= 0x7FF00000) emax = NAN_ROW;
    emax = max(emax, __shfl_xor_sync(0xFFFFFFFFu, emax, 8));
    emax = max(emax, __shfl_xor_sync(0xFFFFFFFFu, emax, 16));
    if (lane < 8) exps[lane] = emax == NAN_ROW ? SL_NAN : (emax >> 20) + (SL_BIAS >> 20) - 1022;
    emax >>= 20;
#pragma unroll
    for (int q = 0; q < KE; q += 8) {
        const double x8[8] = {x[q], x[q + 1], x[q + 2], x[q + 3], x[q + 4], x[q + 5], x[q + 6], x[q + 7]};
        const int f8[8] = {fe[q], fe[q + 1], fe[q + 2], fe[q + 3], fe[q + 4], fe[q + 5], fe[q + 6], fe[q + 7]};
        sl_put8(dst + (uint32_t)((k0 + q) / 8) * 128u + (uint32_t)(lane & 7) * 16u, stride, x8, f8, emax);
    }
    fence_async_smem();
}

// accumulator columns qa .. qb - 1 of this thread's row (m of a slot with row
// exponents ex, columns the same slot's) to C, added where `add`; C null: none
// of its own.  Out of line: three callers (see sl_cut_group).
template <int NB>
__device__ __noinline__ void sl_add(uint32_t tl, const int *ex, double *C, int m, int n, bool add, int qa, int qb)
{
    tc_fence_after();
    const int er = ex[m];
#pragma unroll 1
    for (int q0 = qa; q0 < qb; q0 += 8) {
        double v[8];
        sl_read8<NB>(tl + (uint32_t)q0, er, ex + q0, v);
        if (C) {
            double c[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) c[q] = add && q0 + q < n ? __ldcg(C + (long long)(q0 + q) * n) : 0.0;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q0 + q < n) __stcg(C + (long long)(q0 + q) * n, c[q] + v[q]);
        }
    }
    tc_fence_before();
}

struct SlCtx {
    uint32_t tm;      // TMEM base
    C64Bar bM, bL;    // P1 / P2 (thread 0 waits), PL (thread 128 waits)
    int *abort;
};

// one partition's chain (or the whole sequential chain when g.seq)
template <int NB>
__device__ __forceinline__ void chain_f64_tc_body(const ChainFactorArgs<double, double> &g, const long long p, SlCtx &cx)
{
    using G = SlGeo<NB>;
    constexpr int LD = G::LD, HC = NB / 2, NW = SL_THREADS / 32;
    extern __shared__ __align__(128) unsigned char smem_sl[];
    unsigned char *OP = smem_sl;                                   // the operand slots
    double *sS = reinterpret_cast<double *>(smem_sl + G::OFF_S);
    double *sX = reinterpret_cast<double *>(smem_sl + G::OFF_X);
    double *sV = reinterpret_cast<double *>(smem_sl + G::OFF_V);
    unsigned char *OV = smem_sl + G::OFF_S;                        // the V operand
    int *ex0 = reinterpret_cast<int *>(smem_sl + G::OFF_EX), *ex1 = ex0 + 64, *exB = ex1 + 64, *exV = exB + 64;
    int *hV = exV + 64, *hB = hV + 64, *hN = hB + 64;
    int *sflag = reinterpret_cast<int *>(smem_sl + G::OFF_CTL);
    const uint32_t aOP = smem_u32(OP), aOV = smem_u32(OV);

    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int L = 32 * (w & 3) + lane;               // accumulator row
    const bool live = L < 2 * NB;                    // (warp-uniform: NB = 32 uses rows 0-63)
    const int slot = (L >> 3) & 1, m = (L >> 4) * 8 + (L & 7);  // its operand slot and row there
    const int c0 = HC * (w >> 2);                    // its first accumulator column
    const uint32_t tl = cx.tm + ((uint32_t)(32 * (w & 3)) << 16);
    const int n = g.n;
    const long long nn = (long long)n * n;
    const bool seq = g.seq != 0;
    long long first, last, sL = 0;
    if (seq) {
        first = 0;
        last = g.N - 1;
    } else {
        sL = (p * (g.N - 1)) / g.Q;
        const long long sR = ((p + 1) * (g.N - 1)) / g.Q;
        first = sL + 1;
        last = sR - 1;
    }
    double *Cp = seq ? nullptr : g.C + p * 3 * nn;
    for (int e = tid; e < Geo<double, NB>::SLOT; e += SL_THREADS) sV[e] = 0.0;  // V's strictly lower tiles stay zero
    if (tid < NB) hN[tid] = -SL_BIAS;
    __syncthreads();

    // S_LL (+)= Y^T Y from the PL accumulator: its columns qa .. qb - 1, by warps 4-7
    auto wait_pl = [&]() {  // warps 1-7
        if (tid == 128) c64_wait1(cx.bL, cx.abort);
        asm volatile("bar.sync 3, 224;" ::: "memory");
    };
    auto add_sll = [&](bool add, int qa, int qb) {
        if (!*cx.abort && live) sl_add<NB>(tl, ex1, slot == 1 && m < n ? Cp + m : nullptr, m, n, add, qa, qb);
    };
    auto issue_pl = [&]() {
        if (tid == 128) {  // (not warp 0: an MMA holds its issuing thread for its duration)
            tc_fence_after();
            sl_mma<NB>(cx.tm, aOP, aOP + G::GRP, 2 * G::GRP);
            tc_commit(cx.bL.addr);
            cx.bL.pending = true;
        }
    };

    // A_i into sS (identity outside n x n), asynchronously, by warps 1-7
    auto fetch_a = [&](long long i) {
        const double *Ag = g.A_in + i * nn;
        if (w == 0) return;
        if (n == NB && ((uintptr_t)Ag & 15u) == 0) {
            for (int e = tid - 32; e < NB * NB / 2; e += SL_THREADS - 32)
                cp_async16(sS + 2 * (e % (NB / 2)) + (e / (NB / 2)) * LD, Ag + 2 * e);
        } else {
            for (int e = tid - 32; e < NB * NB; e += SL_THREADS - 32) {
                const int r = e % NB, c = e / NB;
                if (r < n && c < n)
                    cp_async8(sS + r + c * LD, Ag + r + (long long)c * n);
                else
                    sS[r + c * LD] = r == c ? 1.0 : 0.0;
            }
        }
        cp_async_commit();
    };
    fetch_a(first);
    for (long long i = first; i <= last; ++i) {
        const long long t = i - first;
        const bool has_next = !seq || (i < g.N - 1);
        if (t > 0 && tid == 0) c64_wait1(cx.bM, cx.abort);
        cp_async_wait_all();
        __syncthreads();
        if (*cx.abort) break;
        // ---- S = A_i - W^T W in sS (its upper triangle) by the slot 0 rows, Z_i into sX by the slot 1 rows
        if (t > 0) {
            tc_fence_after();
            if (live) {
                const int er = slot == 0 ? ex0[m] : ex1[m];
                const int rmax = 16 * (w & 3) + 15;  // the last column of S in this warp
#pragma unroll 1
                for (int q0 = c0; q0 < c0 + HC; q0 += 8) {
                    if (seq && q0 > rmax) break;
                    double v[8];
                    sl_read8<NB>(tl + (uint32_t)q0, er, ex0 + q0, v);
                    if (slot == 0) {
                        if (q0 <= rmax) {
                            double2 *s = reinterpret_cast<double2 *>(sS + q0 + m * LD);
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                double2 x = s[q];
                                x.x -= v[2 * q];
                                x.y -= v[2 * q + 1];
                                s[q] = x;
                            }
                        }
                    } else if (!seq) {
                        double2 *z = reinterpret_cast<double2 *>(sX + q0 + m * LD);
#pragma unroll
                        for (int q = 0; q < 4; ++q) z[q] = make_double2(-v[2 * q], -v[2 * q + 1]);
                    }
                }
            }
            tc_fence_before();
            __syncthreads();
            if (!seq) issue_pl();
        }
        // ---- Cholesky + inverse; beside the pivot tiles S_LL (warps 4-7) and the digits of
        // B_i (slot 1) and Z_i (slot 0; first block: B_sL^T) (warps 1-3).  A 64-wide block's
        // are spread so that they end with the pivot tile they run beside (14K cycles, 4K of the
        // first one's spent waiting for PL; 8 columns of S_LL take 3K, a group of 8 rows 3K to 5K).
        auto aside = [&](int K) {
            const bool pl = t > 0 && !seq;
            if (K == 0) {  // the balance of B_i, Z_i and V_i, before the pivots change S's diagonal
                if (w <= 3 && tid - 32 < NB) sl_balance(sS[(tid - 32) * (LD + 1)], hV + tid - 32, hB + tid - 32);
                if (pl) wait_pl();
                else if (w <= 3) asm volatile("bar.sync 4, 96;" ::: "memory");
            }
            constexpr int NG = NB / 8;
            constexpr int S1 = 24, S2 = NB == 64 ? 56 : NB;                // columns of S_LL
            constexpr int B1 = NB == 64 ? 6 : NG, B2 = NB == 64 ? 7 : NG;  // row groups of B_i
            if (w >= 4) {
                const int qa = K == 0 ? 0 : K == 1 ? S1 : S2, qb = K == 0 ? S1 : K == 1 ? S2 : K == 2 ? NB : S2;
                if (pl && qa < qb) add_sll(t > 1, qa, qb);
            } else {
                const int ua = K == 0 ? 0 : !pl ? NG : K == 1 ? B1 : K == 2 ? B2 : NG;
                const int ub = !pl ? NG : K == 0 ? B1 : K == 1 ? B2 : NG;
                for (int u = ua + w - 1; u < ub + (K == 1 ? NG : 0); u += 3) {
                    const bool isB = u < ub;
                    if (isB ? !has_next : seq) continue;
                    const int gi = isB ? u : u - ub, r = 8 * gi + (lane & 7);
                    const double *row = isB ? g.B_in + i * nn + (long long)r * n : pl ? sX + r * LD : g.B_in + sL * nn + r;
                    sl_cut_group<NB>(OP + (uint32_t)(2 * gi + (isB ? 1 : 0)) * G::GRP, G::SLICE,
                                           (isB ? exB : ex0) + 8 * gi, row, isB || pl ? 1 : n,
                                           !isB && pl ? NB : r < n ? n : 0, hB);
                }
            }
        };
        const int bad = f64_chol_inv_i<NB, SL_THREADS>(sS, sV, sflag, tid, aside);
        if (bad && tid == 0) record_bad_pivot(g.st, g.level, i);
        if (*cx.abort) break;
        // ---- V_i's digits over sS and sX, V_i to global memory while P2 = [Z_i | B_i]^T V_i runs
        if (has_next) {
            if (w < NB / 8) sl_cut_group<NB>(OV + (uint32_t)w * G::GRP, G::VSLICE, exV + 8 * w, sV + (8 * w + (lane & 7)) * LD, 1, NB, hV);
            tc_fence_before();
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
                sl_mma<NB>(cx.tm, aOP, aOV, G::GRP);
                tc_commit(cx.bM.addr);
                cx.bM.pending = true;
            }
        }
        if (w > 0 || !has_next) {
            double *dst = g.A_f + i * nn;
            const int nn32 = n * n;
            for (int e = has_next ? tid - 32 : tid; e < nn32; e += has_next ? SL_THREADS - 32 : SL_THREADS) {
                const int c = e / n, r = e - c * n;
                dst[e] = sV[r + c * LD];
            }
        }
        if (!has_next) break;  // the last block of the sequential chain
        if (tid == 0) c64_wait1(cx.bM, cx.abort);
        __syncthreads();
        if (*cx.abort) break;
        tc_fence_after();
        // ---- Y_i (slot 0 rows) and W_i (slot 1 rows) in FP64 over sX and sS
        if (live) {
            const int er = slot == 0 ? ex0[m] : exB[m];
            double *o = (slot == 0 ? sX : sS) + m * LD;
#pragma unroll 1
            for (int q0 = c0; q0 < c0 + HC; q0 += 8) {
                double v[8];
                sl_read8<NB>(tl + (uint32_t)q0, er, exV + q0, v);
#pragma unroll
                for (int q = 0; q < 8; q += 2) *reinterpret_cast<double2 *>(o + q0 + q) = make_double2(v[q], v[q + 1]);
            }
        }
        tc_fence_before();
        __syncthreads();
        // ---- their digits into the slots as [W_i | Y_i]; P1 of the next step (or of the chain end)
        for (int u = w; u < 2 * (NB / 8); u += NW) {
            const int gi = u >> 1, row = 8 * gi + (lane & 7);
            unsigned char *dst = OP + (uint32_t)(2 * gi + (u & 1)) * G::GRP;
            if (u & 1) {
                if (!seq) sl_cut_group<NB>(dst, G::SLICE, ex1 + 8 * gi, sX + row * LD, 1, NB, hN);
            } else {
                sl_cut_group<NB>(dst, G::SLICE, ex0 + 8 * gi, sS + row * LD, 1, NB, hN);
            }
        }
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            sl_mma<NB>(cx.tm, aOP, aOP, 2 * G::GRP);
            tc_commit(cx.bM.addr);
            cx.bM.pending = true;
        } else if (w > 0) {  // meanwhile Y_i and W_i to global memory
            double *dW = g.B_f + i * nn, *dY = seq ? nullptr : g.Y + i * nn;
            const int nn32 = n * n;
            for (int e = tid - 32; e < nn32; e += SL_THREADS - 32) {
                const int c = e / n, r = e - c * n;
                dW[e] = sS[r + c * LD];
                if (!seq) dY[e] = sX[r + c * LD];
            }
            asm volatile("bar.sync 2, 224;" ::: "memory");  // sS is read (warp 0 only issues P1)
            if (i < last) fetch_a(i + 1);
        }
    }

    // ---- chain end: S_RR = W^T W, S_LR = Y^T W, the last S_LL term
    if (!seq && !*cx.abort) {
        if (tid == 0) c64_wait1(cx.bM, cx.abort);
        __syncthreads();
        if (!*cx.abort) {
            tc_fence_after();
            if (live) {
                const int er = slot == 0 ? ex0[m] : ex1[m];
                double *dst = Cp + (slot == 0 ? nn : 2 * nn);
#pragma unroll 1
                for (int q0 = c0; q0 < c0 + HC; q0 += 8) {
                    double v[8];
                    sl_read8<NB>(tl + (uint32_t)q0, er, ex0 + q0, v);
                    if (m < n) {
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            if (q0 + q < n) dst[m + (long long)(q0 + q) * n] = v[q];
                    }
                }
            }
            tc_fence_before();
            __syncthreads();
            issue_pl();
            if (w > 0) wait_pl();
            if (w >= 4) add_sll(last > first, 0, NB);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*cx.abort) {
        // a wait gave up: wait (bounded) for the MMAs still in flight before
        // shared memory and TMEM are released
        int ignored = 0;
        if (tid == 0) {
            c64_wait1(cx.bM, &ignored);
            if (g.st) atomicExch(&g.st->tc_timeout, 1);
        } else if (tid == 128) {
            c64_wait1(cx.bL, &ignored);
        }
        __syncthreads();
    }
}

// TMEM columns and mbarriers of a CTA; ctl: 64 bytes (the first word is the
// Cholesky's flag)
__device__ __forceinline__ void sl_begin(SlCtx &cx, unsigned char *ctl, uint32_t cols)
{
    uint32_t *tslot = reinterpret_cast<uint32_t *>(ctl + 4);
    cx.abort = reinterpret_cast<int *>(ctl + 8);
    uint64_t *mbars = reinterpret_cast<uint64_t *>(ctl + 16);
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbars[q])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *cx.abort = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    cx.tm = *tslot;
    cx.bM = C64Bar{smem_u32(&mbars[0]), 0u, false};
    cx.bL = C64Bar{smem_u32(&mbars[1]), 0u, false};
}

__device__ __forceinline__ void sl_end(const SlCtx &cx, uint32_t cols)
{
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(cx.tm), "r"(cols)
                     : "memory");
    }
}

template <int NB>
__global__ void __launch_bounds__(SL_THREADS, NB == 64 ? 1 : 2) chain_f64_tc_kernel(ChainFactorArgs<double, double> g)
{
    extern __shared__ __align__(128) unsigned char smem_sl[];
    SlCtx cx;
    sl_begin(cx, smem_sl + SlGeo<NB>::OFF_CTL, SlGeo<NB>::TMEM);
    chain_f64_tc_body<NB>(g, blockIdx.x, cx);
    sl_end(cx, SlGeo<NB>::TMEM);
}

}  // namespace bss
