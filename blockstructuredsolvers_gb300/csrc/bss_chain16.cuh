// Chain factor kernel for blocks up to 16 wide, FP32 and FP64: the recursion
// and outputs of chain_factor_body, one 128-thread CTA per partition.
//
// What bounds it: the latency of one step, since a step's five products are
// 32 FMAs a thread each.  The step is therefore cut to four phases with a CTA
// barrier between them:
//   A  S = A_i - W^T W                              all warps
//   B  V_i = U^-1 by one warp (in-place Gauss-Jordan, as f64_pivot_tile);
//      beside it, on the other three schedulers, Z_i = -W^T Y and S_LL += Y^T Y
//   C  Y_i = V^T Z, W_i = V^T B_i                   all warps
//   D  V_i, W_i, Y_i to global memory, in A's shadow of the next step
// A_i and B_i are fetched into registers a step ahead.  In phase C a warp's
// lanes share one row of V^T (two neighbouring rows), so the triangular sums
// have one length per warp and half the FP64 instructions are saved.
//
// Measured (one chain step, 20 partitions): FP32 19.1 -> 1.5 us, FP64 43.7 ->
// 8.9 us against the general kernel with 16 x 16 tiles, whose step was slower
// than that of 32-wide blocks (8.2 us).
#pragma once

namespace bss {

constexpr int C16_THREADS = 128;

template <class T>
struct C16Geo {
    static constexpr int LD = 16 + 16 / (int)sizeof(T);
    static constexpr int SLOT = 16 * LD;
    static constexpr size_t BYTES = (size_t)6 * SLOT * sizeof(T) + 16;
};

// f64_pivot_tile's sweep in FP32: V = U^-1 of the tile in sS (upper triangle read) to sV
template <int LD>
__device__ __forceinline__ int f32_pivot_tile(const float *sS, float *sV, int lane)
{
    constexpr unsigned ALL = 0xFFFFFFFFu;
    const int c = lane & 15, h = lane >> 4;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int r = 2 * q + h;
        v[q] = r <= c ? sS[r + c * LD] : 0.f;
    }
    int bad = 0;
    float dj = 1.f;
    float piv = __shfl_sync(ALL, v[0], 0), row = __shfl_sync(ALL, v[0], c);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int hj = j & 1, qj = j >> 1;
        if (c == j) row = 1.f;
        float s[8];
#pragma unroll
        for (int q = (j + 1) >> 1; q < 8; ++q) s[q] = __shfl_sync(ALL, v[qj], 2 * q + h + 16 * hj);
        float m;
        if (piv > 1e-30f && piv < 1e30f) {
            float y;
            asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(piv));
            m = row * y;
        } else {
            if (!(piv > 0.f && piv < INFINITY)) {
                bad = 1;
                piv = 1.f;
            }
            m = row / piv;
        }
        if (c == j) dj = piv;
#pragma unroll
        for (int q = (j + 1) >> 1; q < 8; ++q) {
            const float x = fmaf(-s[q], m, c == j ? 0.f : v[q]);
            if (2 * q > j || h == 1) v[q] = x;
            if (q == (j + 1) >> 1) {
                piv = __shfl_sync(ALL, v[q], (j + 1) + 16 * (hj ^ 1));
                row = __shfl_sync(ALL, v[q], c + 16 * (hj ^ 1));
            }
        }
    }
    const float rs = rsqrtf(dj);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int r = 2 * q + h;
        const float rr = __shfl_sync(ALL, rs, r);
        sV[c + r * LD] = c < r ? v[q] * rr : (c == r ? rr : 0.f);
    }
    return bad;
}
template <int LD>
__device__ __forceinline__ int pivot_tile16(const float *sS, float *sV, int lane)
{
    return f32_pivot_tile<LD>(sS, sV, lane);
}
template <int LD>
__device__ __forceinline__ int pivot_tile16(const double *sS, double *sV, int lane)
{
    return f64_pivot_tile<LD>(sS, sV, 0, lane);
}

// sum_k X(k, i) Y(k, j) over k = 0 .. 16 - 1 (or up to and including kmax,
// rounded up to a vector), columns in shared memory
template <class T>
__device__ __forceinline__ T c16_dot(const T *x, const T *y, int kmax = 15)
{
    using V = typename Vec<T>::type;
    constexpr int W = Vec<T>::W;
    T s0 = T(0), s1 = T(0);
#pragma unroll
    for (int k = 0; k < 16; k += 2 * W) {
        if (k <= kmax) fma_vec(s0, *reinterpret_cast<const V *>(x + k), *reinterpret_cast<const V *>(y + k));
        if (k + W <= kmax) fma_vec(s1, *reinterpret_cast<const V *>(x + k + W), *reinterpret_cast<const V *>(y + k + W));
    }
    return s0 + s1;
}

template <class Tin, class T>
__device__ __forceinline__ void chain16_body(const ChainFactorArgs<Tin, T> &g, const long long p)
{
    constexpr int LD = C16Geo<T>::LD, SLOT = C16Geo<T>::SLOT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *sS = reinterpret_cast<T *>(smem_raw), *sV = sS + SLOT, *sW = sV + SLOT, *sY = sW + SLOT, *sZ = sY + SLOT, *sB = sZ + SLOT;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
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
    // elements of a tile: this thread's are (er, ec) and (er, ec + 8)
    const int er = tid & 15, ec = tid >> 4;
    const bool in0 = er < n && ec < n, in1 = er < n && ec + 8 < n;
    const int o0 = er + ec * LD, o1 = o0 + 8 * LD, g0 = er + ec * n, g1 = g0 + 8 * n;
    const T id0 = er == ec ? T(1) : T(0), id1 = er == ec + 8 ? T(1) : T(0);
    // phase B beside the pivots: thread u of 96 has elements u, u + 96, u + 192
    const int u = tid - 32;
    T ll[3] = {T(0), T(0), T(0)};
    // phase C: rows 2 x, 2 x + 1 for x = w and 7 - w, column lane % 16
    const int cc = lane & 15, ch = lane >> 4;

    T a0, a1, b0, b1;
    auto fetch = [&](long long i) {
        const Tin *A = g.A_in + i * nn, *B = g.B_in + i * nn;
        const bool has = !seq || i < g.N - 1;
        a0 = in0 ? (T)A[g0] : id0;
        a1 = in1 ? (T)A[g1] : id1;
        b0 = in0 && has ? (T)B[g0] : T(0);
        b1 = in1 && has ? (T)B[g1] : T(0);
    };
    fetch(first);
    if (!seq) {  // the first block's Z = B_sL^T
        const Tin *Bs = g.B_in + sL * nn;
        sZ[o0] = in0 ? (T)Bs[ec + er * n] : T(0);
        sZ[o1] = in1 ? (T)Bs[ec + 8 + er * n] : T(0);
    }
    for (long long i = first; i <= last; ++i) {
        const bool chained = i > first;
        const bool has_next = !seq || i < g.N - 1;
        // ---- A
        {
            T s0 = a0, s1 = a1;
            if (chained) {
                s0 -= c16_dot(sW + er * LD, sW + ec * LD);
                s1 -= c16_dot(sW + er * LD, sW + (ec + 8) * LD);
            }
            sS[o0] = s0;
            sS[o1] = s1;
            sB[o0] = b0;
            sB[o1] = b1;
        }
        if (i < last) fetch(i + 1);
        __syncthreads();
        // ---- B
        if (w == 0) {
            const int bad = pivot_tile16<LD>(sS, sV, lane);
            if (bad && lane == 0) record_bad_pivot(g.st, g.level, i);
        } else if (chained && !seq) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int e = u + 96 * q, r = e & 15, c = e >> 4;
                if (e < 256) {
                    sZ[r + c * LD] = -c16_dot(sW + r * LD, sY + c * LD);
                    ll[q] += c16_dot(sY + r * LD, sY + c * LD);
                }
            }
        }
        __syncthreads();
        // ---- C
        if (has_next) {
            T y[2], x[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r2 = 2 * (q ? 7 - w : w), r = r2 + ch;
                y[q] = seq ? T(0) : c16_dot(sV + r * LD, sZ + cc * LD, r2 + 1);
                x[q] = c16_dot(sV + r * LD, sB + cc * LD, r2 + 1);
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = 2 * (q ? 7 - w : w) + ch;
                sW[r + cc * LD] = x[q];
                if (!seq) sY[r + cc * LD] = y[q];
            }
        }
        __syncthreads();
        // ---- D
        {
            T *V = g.A_f + i * nn, *W = g.B_f + i * nn;
            if (in0) V[g0] = sV[o0];
            if (in1) V[g1] = sV[o1];
            if (has_next) {
                if (in0) W[g0] = sW[o0];
                if (in1) W[g1] = sW[o1];
            }
            if (!seq) {
                T *Y = g.Y + i * nn;
                if (in0) Y[g0] = sY[o0];
                if (in1) Y[g1] = sY[o1];
            }
        }
    }
    if (!seq) {
        T *C = g.C + p * 3 * nn;
        if (in0) {
            C[nn + g0] = c16_dot(sW + er * LD, sW + ec * LD);
            C[2 * nn + g0] = c16_dot(sY + er * LD, sW + ec * LD);
        }
        if (in1) {
            C[nn + g1] = c16_dot(sW + er * LD, sW + (ec + 8) * LD);
            C[2 * nn + g1] = c16_dot(sY + er * LD, sW + (ec + 8) * LD);
        }
        if (w > 0) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int e = u + 96 * q, r = e & 15, c = e >> 4;
                if (e < 256 && r < n && c < n) C[r + c * n] = ll[q] + c16_dot(sY + r * LD, sY + c * LD);
            }
        }
    }
}

template <class Tin, class T>
__global__ void __launch_bounds__(C16_THREADS) chain16_kernel(ChainFactorArgs<Tin, T> g)
{
    chain16_body<Tin, T>(g, blockIdx.x);
}

// persistent form for many systems (see chain_factor_queue_kernel)
template <class Tin, class T>
__global__ void __launch_bounds__(C16_THREADS)
    chain16_queue_kernel(const ChainFactorArgs<Tin, T> *__restrict__ descs, const WorkItem *__restrict__ items,
                         int nitems, int *head)
{
    __shared__ int cur;
    for (;;) {
        if (threadIdx.x == 0) cur = atomicAdd(head, 1);
        __syncthreads();
        const int it = cur;
        __syncthreads();
        if (it >= nitems) break;
        const WorkItem item = items[it];
        const ChainFactorArgs<Tin, T> g = descs[item.desc];
        chain16_body<Tin, T>(g, item.p);
        __syncthreads();
    }
}

}  // namespace bss
