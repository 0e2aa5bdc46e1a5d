// Chain factor kernel for FP64 factors of 65..128-wide blocks: the chain step
// of wide_chain_factor_body (every n x n matrix of the chain in global memory,
// a partition's few blocks in L2) with its 64-wide tile products on the tensor
// cores by exact digit products (bss_chain_f64_tc.cuh), two row tiles per MMA.
//
// What bounds it: the 36 tile products of a step took ~5.1M of its ~5.4M
// cycles on the FP64 pipe (156K each).  Here a product of 128 rows x 64
// columns x 64 is 4.7K cycles of MMAs, 6.5K of readout and 3K per tile cut
// into digits; a step has 20 of them and 4 of 64 rows (the blocked Cholesky),
// and two 64-wide Cholesky factorizations on the FP64 pipe (~75K each).  Both
// operand tiles of a contraction index K stay in the slots while they meet
// every column tile, and a slot is its own B operand in W^T W and Y^T Y.
//
// Shared memory: the two operand slots (112 KB; during a factorization sS and
// sV), two B operands (56 KB each).  TMEM: all 512 columns.  One CTA per SM.
//
// Measured: plain FP64 factor + solve of N = 2048, n = 128, k = 4:
// 61.5 -> 15.0 ms (13.4 ms with the sweeps as they are now).
#pragma once

namespace bss {

struct WlGeo {
    using G = SlGeo<64>;
    static constexpr uint32_t OFF_B = G::OFF_S;                               // two B operands
    static constexpr uint32_t B_BYTES = SL_DIGITS * G::VSLICE;
    static constexpr uint32_t OFF_EX = OFF_B + 2u * B_BYTES;                  // row exponents: slots 0, 1, B operands 0, 1
    static constexpr uint32_t OFF_H = OFF_EX + 4u * 64u * 4u;                  // hV, hB of the block's 128 rows; none (64)
    static constexpr uint32_t OFF_CTL = OFF_H + 5u * 64u * 4u;
    static constexpr uint32_t BYTES = OFF_CTL + 64u;
    static_assert(2 * G::TILE <= SL_DIGITS * G::SLICE, "sS and sV overlay the slots");
};

// tile of a column-major matrix with leading dimension n as an operand: row
// r of the operand is column r of the tile (or its row r, `rows`)
struct WlTile {
    const double *p;  // the tile's first element; null: leave the operand alone
    int nk, nr;       // elements along K, operand rows (zero beyond)
    bool rows;
    const int *h;     // the contraction index's balance (sl_balance)
};

__device__ __forceinline__ void wl_cut(unsigned char *dst, uint32_t group, uint32_t slice, int *exps, const WlTile &t,
                                       int n, int gi)
{
    const int r = 8 * gi + (threadIdx.x & 7);
    sl_cut_group<64>(dst + (uint32_t)gi * group, slice, exps + 8 * gi, t.p + (t.rows ? (long long)r : (long long)r * n),
                     t.rows ? n : 1, r < t.nr ? t.nk : 0, t.h);
}

// the accumulator, times sign, plus base, to a column tile of global memory:
// slot j's rows to dst[j] (a tile's first element; null: dropped), base[j] added
// (null: none; may be dst[j]).  nr[j], nc: rows and columns inside the block.
static __device__ __noinline__ void wl_emit(uint32_t tm, const int *ex, const int *ecol, double *dst0, double *dst1,
                                     const double *base0, const double *base1, int nr0, int nr1, int nc, int n,
                                     double sign)
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int L = 32 * (w & 3) + lane, slot = (L >> 3) & 1, m = (L >> 4) * 8 + (L & 7), c0 = 32 * (w >> 2);
    const uint32_t tl = tm + ((uint32_t)(32 * (w & 3)) << 16);
    double *dst = slot ? dst1 : dst0;
    const double *base = slot ? base1 : base0;
    const bool mine = dst != nullptr && m < (slot ? nr1 : nr0);
    const int er = ex[64 * slot + m];
    const bool add = mine && base != nullptr;
    const long long flip = sign < 0.0 ? (long long)0x8000000000000000ull : 0;
    tc_fence_after();
    double c[8];  // base, fetched one chunk ahead
#pragma unroll
    for (int q = 0; q < 8; ++q) c[q] = add && c0 + q < nc ? __ldcg(base + m + (long long)(c0 + q) * n) : 0.0;
#pragma unroll 1
    for (int q0 = c0; q0 < c0 + 32 && q0 < nc; q0 += 8) {
        double v[8], cn[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            cn[q] = add && q0 + 8 < c0 + 32 && q0 + 8 + q < nc ? __ldcg(base + m + (long long)(q0 + 8 + q) * n) : 0.0;
        sl_read8<64>(tl + (uint32_t)q0, er, ecol + q0, v);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = __longlong_as_double(__double_as_longlong(v[q]) ^ flip);
        if (__any_sync(0xFFFFFFFFu, add)) {  // (an FP64 add costs a warp 64 cycles)
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = add ? v[q] + c[q] : v[q];
        }
        if (mine) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q0 + q < nc) dst[m + (long long)(q0 + q) * n] = v[q];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q] = cn[q];
    }
    tc_fence_before();
}

// one partition's chain (or the whole sequential chain when g.seq)
__device__ __forceinline__ void chain128_f64_tc_body(const ChainFactorArgs<double, double> &g, const long long p, SlCtx &cx)
{
    using G = SlGeo<64>;
    constexpr int LD = G::LD;
    extern __shared__ __align__(128) unsigned char smem_sl[];
    unsigned char *OP = smem_sl, *OB = smem_sl + WlGeo::OFF_B;
    double *sS = reinterpret_cast<double *>(smem_sl), *sV = sS + Geo<double, 64>::SLOT;
    int *ex = reinterpret_cast<int *>(smem_sl + WlGeo::OFF_EX);
    int *hV = reinterpret_cast<int *>(smem_sl + WlGeo::OFF_H), *hB = hV + 128, *hN = hB + 128;
    int *sflag = reinterpret_cast<int *>(smem_sl + WlGeo::OFF_CTL);
    const uint32_t aOP = smem_u32(OP), aOB = smem_u32(OB);
    const int tid = threadIdx.x, w = tid >> 5;
    const int n = g.n, n1 = n - 64;  // n1: size of the second tile
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
    // tile (I, J) of a matrix; h: hV or hB where the contraction index is a row of the block
    auto at = [&](auto *M, int I, int J) { return M + 64 * I + (long long)64 * J * n; };
    auto tile = [&](const double *M, int I, int J, bool rows = false, const int *h = nullptr) {
        const int a = I ? n1 : 64, b = J ? n1 : 64;
        return WlTile{at(M, I, J), rows ? b : a, rows ? a : b, rows, h ? h + 64 * (rows ? J : I) : hN};
    };
    // cut x0, x1 into the slots and b0, b1 into the B operands (p null: left alone); ends with a barrier
    auto cut = [&](const WlTile &x0, const WlTile &x1, const WlTile &b0, const WlTile &b1) {
        if (x0.p) wl_cut(OP, 2 * G::GRP, G::SLICE, ex, x0, n, w);
        if (x1.p) wl_cut(OP + G::GRP, 2 * G::GRP, G::SLICE, ex + 64, x1, n, w);
        if (b0.p) wl_cut(OB, G::GRP, G::VSLICE, ex + 128, b0, n, w);
        if (b1.p) wl_cut(OB + WlGeo::B_BYTES, G::GRP, G::VSLICE, ex + 192, b1, n, w);
        tc_fence_before();
        __syncthreads();
    };
    const WlTile none{nullptr, 0, 0, false, hN};
    // [slot 0 | slot 1]^T times operand b (0, 1: a slot; 2, 3: a B operand); false when the wait expired
    auto product = [&](int b) {
        if (tid == 0) {
            tc_fence_after();
            sl_mma<64>(cx.tm, aOP, b < 2 ? aOP + b * G::GRP : aOB + (b - 2) * WlGeo::B_BYTES, b < 2 ? 2 * G::GRP : G::GRP);
            tc_commit(cx.bM.addr);
            cx.bM.pending = true;
            c64_wait1(cx.bM, cx.abort);
        }
        __syncthreads();
        return *cx.abort == 0;
    };
    // column tile J of D = sign [slots]^T (operand b), its top and / or bottom row
    // tile, plus that of b0 (top) and b1 (bottom); false when a wait expired
    auto emit = [&](int b, double *D, const double *b0, const double *b1, int J, bool top, bool bottom, double sign) {
        if (!product(b)) return false;
        wl_emit(cx.tm, ex, ex + 64 * b, top ? at(D, 0, J) : nullptr, bottom ? at(D, 1, J) : nullptr,
                b0 ? at(b0, 0, J) : nullptr, b1 ? at(b1, 1, J) : nullptr, 64, n1, J ? n1 : 64, n, sign);
        __syncthreads();
        return true;
    };
    // Cholesky + inverse of diagonal tile K of D in place
    auto factor = [&](double *D, int K, long long i) {
        const int a = K ? n1 : 64;
        double *t = at(D, K, K);
        for (int e = tid; e < 64 * 64; e += SL_THREADS) {
            const int r = e & 63, c = e >> 6;
            sS[r + c * LD] = r < a && c < a ? __ldcg(t + r + (long long)c * n) : (r == c ? 1.0 : 0.0);
            sV[r + c * LD] = 0.0;  // V's strictly lower tiles
        }
        __syncthreads();
        const int bad = f64_chol_inv<64, SL_THREADS>(sS, sV, sflag, tid);
        if (bad && tid == 0) record_bad_pivot(g.st, g.level, i);
        for (int e = tid; e < 64 * 64; e += SL_THREADS) {
            const int r = e & 63, c = e >> 6;
            if (r < a && c < a) t[r + (long long)c * n] = sV[r + c * LD];
        }
        __syncthreads();
    };

    if (tid < 64) hN[tid] = -SL_BIAS;  // (read after factor's barriers)
    double *Cp = seq ? nullptr : g.C + p * 3 * nn;
    bool ok = true;
    for (long long i = first; i <= last && ok; ++i) {
        const long long t = i - first;
        const bool has_next = !seq || (i < g.N - 1);
        double *V = g.A_f + i * nn, *Z = seq ? nullptr : g.Y + i * nn;
        const double *A = g.A_in + i * nn, *Wp = g.B_f + (i - 1) * nn, *Yp = seq ? nullptr : g.Y + (i - 1) * nn;
        // ---- S = A_i - W^T W (upper tiles, into V_i's slot), Z = -W^T Y (into Y_i's; first block: B_sL^T)
        if (t > 0) {
            for (int K = 0; K < 2 && ok; ++K) {
                const double *from = K ? V : A;
                cut(tile(Wp, K, 0), tile(Wp, K, 1), seq ? none : tile(Yp, K, 0), seq ? none : tile(Yp, K, 1));
                ok = emit(0, V, from, from, 0, true, false, -1.0) && emit(1, V, from, from, 1, true, true, -1.0);
                const double *z = K ? Z : nullptr;
                for (int J = 0; J < 2 && ok && !seq; ++J) ok = emit(2 + J, Z, z, z, J, true, true, -1.0);
            }
            if (!ok) break;
        } else {
            for (long long e = tid; e < nn; e += SL_THREADS) V[e] = A[e];
            if (!seq) {
                const double *Bs = g.B_in + sL * nn;
                for (long long e = tid; e < nn; e += SL_THREADS) {
                    const long long r = e % n, c = e / n;
                    Z[e] = Bs[c + r * n];
                }
            }
            __syncthreads();
        }
        // ---- blocked Cholesky and V_i = U^-1 in its slot
        if (tid < 128) sl_balance(tid < n ? __ldcg(V + (long long)tid * (n + 1)) : 1.0, hV + tid, hB + tid);
        factor(V, 0, i);
        cut(tile(V, 0, 0, false, hV), none, tile(V, 0, 1, false, hB), none);
        if (!(ok = emit(2, V, nullptr, nullptr, 1, true, false, 1.0))) break;  // U01 = V00^T S01
        cut(tile(V, 0, 1), none, tile(V, 0, 1), none);
        if (!(ok = product(2))) break;  // S11 -= U01^T U01
        wl_emit(cx.tm, ex, ex + 128, at(V, 1, 1), nullptr, at(V, 1, 1), nullptr, n1, 0, n1, n, -1.0);
        __syncthreads();
        factor(V, 1, i);
        cut(tile(V, 0, 0, true), none, none, tile(V, 1, 1, false, hV));  // (B operand 0 still holds U01)
        if (!(ok = emit(2, V, nullptr, nullptr, 1, true, false, 1.0))) break;  // T = V00 U01
        cut(tile(V, 0, 1, true, hB), none, none, none);
        if (!(ok = emit(3, V, nullptr, nullptr, 1, true, false, -1.0))) break;  // V01 = -T V11
        for (int e = tid; e < 64 * n1; e += SL_THREADS) at(V, 1, 0)[e % n1 + (long long)(e / n1) * n] = 0.0;
        // ---- Y_i = V^T Z, W_i = V^T B_i in place: the bottom row tiles of the inputs
        // first, then the top ones (rows of tile K are overwritten after they are cut;
        // the bottom tile of the result gets its second part with K = 0)
        for (int K = 1; K >= 0 && ok; --K) {
            const WlTile x0 = K ? none : tile(V, 0, 0, false, hV), x1 = tile(V, K, 1, false, hV);
            if (!seq) {
                cut(x0, x1, tile(Z, K, 0, false, hB), tile(Z, K, 1, false, hB));
                for (int J = 0; J < 2 && ok; ++J) ok = emit(2 + J, Z, nullptr, K ? nullptr : Z, J, K == 0, true, 1.0);
            }
            if (has_next && ok) {
                const double *B = g.B_in + i * nn;
                double *W = g.B_f + i * nn;
                cut(seq ? x0 : none, seq ? x1 : none, tile(B, K, 0, false, hB), tile(B, K, 1, false, hB));
                for (int J = 0; J < 2 && ok; ++J) ok = emit(2 + J, W, nullptr, K ? nullptr : W, J, K == 0, true, 1.0);
            }
        }
        // ---- S_LL += Y^T Y
        if (!seq)
            for (int K = 0; K < 2 && ok; ++K) {
                cut(tile(Z, K, 0), tile(Z, K, 1), none, none);
                const double *from = t > 0 || K ? Cp : nullptr;
                ok = emit(0, Cp, from, from, 0, true, true, 1.0) && emit(1, Cp, from, from, 1, true, true, 1.0);
            }
    }
    // ---- chain end: S_RR = W^T W, S_LR = Y^T W
    if (!seq && ok) {
        const double *W = g.B_f + last * nn, *Y = g.Y + last * nn;
        double *RR = Cp + nn, *LR = Cp + 2 * nn;
        for (int K = 0; K < 2 && ok; ++K) {
            const double *rr = K ? RR : nullptr, *lr = K ? LR : nullptr;
            cut(tile(W, K, 0), tile(W, K, 1), tile(W, K, 0), tile(W, K, 1));
            for (int J = 0; J < 2 && ok; ++J) ok = emit(J, RR, rr, rr, J, true, true, 1.0);
            if (!ok) break;
            cut(tile(Y, K, 0), tile(Y, K, 1), none, none);  // (the B operands still hold W)
            for (int J = 0; J < 2 && ok; ++J) ok = emit(2 + J, LR, lr, lr, J, true, true, 1.0);
        }
    }
    if (*cx.abort && tid == 0) {
        int ignored = 0;
        c64_wait1(cx.bM, &ignored);  // the MMAs still in flight, bounded, before shared memory and TMEM are released
        if (g.st) atomicExch(&g.st->tc_timeout, 1);
    }
}

template <class T>  // (a template: the header is in several translation units)
__global__ void __launch_bounds__(SL_THREADS, 1) chain128_f64_tc_kernel(ChainFactorArgs<T, T> g)
{
    extern __shared__ __align__(128) unsigned char smem_sl[];
    SlCtx cx;
    sl_begin(cx, smem_sl + WlGeo::OFF_CTL, SlGeo<64>::TMEM);
    chain128_f64_tc_body(g, blockIdx.x, cx);
    sl_end(cx, SlGeo<64>::TMEM);
}

}  // namespace bss
