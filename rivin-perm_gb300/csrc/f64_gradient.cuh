// FP64-accurate gradient of the Glynn permanent, real matrices of order 2..32.
//
//   d per / d a_ij = 2^(1-n) sum_g (-1)^g d_j(g) E_i(g),
//   E_i(g) = prod_{l != i} s_l(g)                     (no reference counterpart)
//
// Row sums are kept on fixed FP32 grids as in the forward kernel
// (f64_forward.cuh): three additions per row and Gray step, no drift.  P
// lanes (1, 2 or 4) walk one Gray range together, each with RW = ceil(N / P)
// rows.  Per state a lane forms the prefix products of its rows, the lanes
// exchange their products (log2 P shuffles), and a suffix pass that starts
// from the other lanes' product yields E_i: 3 products per row, no division,
// so zero row sums need no second path.
//
// Gradient columns by a pairwise tree over the Gray range.  With w = (-1)^g
// E_i(g), two neighbouring blocks A, B of 2^t states have opposite signs of
// column t, so
//   sum over both of w       = S_A + S_B,
//   sum over both of d_t w   = +-(S_A - S_B),
// and column t takes one double-float addition of the difference per 2^(t+1)
// states: 3 additions per row and state for the first four columns together
// (1 + M = 5 when every state adds to each).  Columns 4..R-1 take the
// 16-state sums, the columns above the range's 2^R states its total.  The
// tree's waiting sums and the accumulators of columns 1..R-1 live in shared
// memory ([slot][row][thread]: no bank conflicts).  After each range the warp
// adds its walkers' sums (shuffles, double-float) and folds them into the
// warp's FP64 Kahan sums in global memory.
//
// Where a warp's walkers cover a whole matrix in one range each (orders up to
// GRAD_WHOLE_N) a thread block is one warp, takes one matrix and writes its
// gradient itself: no slots and no reduction.  Four warps on one matrix left
// three of them idle and cost slots that were zeroed and reduced: 65536
// matrices 5x5 3.72 -> 0.76 ms, 8x8 7.86 -> 1.38, 14x14 48.1 -> 17.9 (a lane
// per row: 0.73, 1.96, 97.9), 16 of order 4 95 -> 73 us (77).
//
// About 46 FP32 operations per row and state; two warps a scheduler wait on
// dependent ones (issue 62 %, FMA pipe 46 %).  16 x 26x26 with the forward
// walk: 114.3 -> 36.1 ms against a lane per row with a shuffle
// butterfly for the product and a double-float division per row for E_i;
// error against 64 bits 9.5e-12 -> 5.5e-13.
#pragma once

#include "f64_forward.cuh"

namespace pg {

struct GradArgs {
    const double *A;           // [batch][n][n] row-major, device
    int batch;
    int blocks_per;            // thread blocks per matrix
    int log_range;             // 2^R states of a walker's range, R <= GradShape::RMAX
    double *slots;             // [batch][blocks_per][GRAD_WARPS][grad_slot(n)], zeroed
    double *grad, *grad_abs;   // results of the one-warp blocks (grad_abs may be null)
    volatile const int *abort_flag;
    int *status;
    int resident;              // blocks of the first wave, at most
};

constexpr int GRAD_WARPS = 4;  // warps of a thread block
constexpr int GRAD_TREE = 4;   // levels of the pairwise tree
constexpr int GRAD_WHOLE_N = 14;   // largest order whose matrices a warp can take whole
constexpr int GRAD_SPLIT_N = 11;   // smallest order with more than one range a walker

// per-warp slot: per entry the Kahan sum and its compensation, then the
// rows' sums of |E|
__host__ __device__ constexpr int grad_slot(int n) { return 2 * n * n + n; }

template <int N>
struct GradShape {
    static constexpr int LP = N <= 8 ? 0 : N <= 16 ? 1 : 2;    // log2 of a walker's lanes
    // log2 of a warp's walkers, each with two states or more (fewer than 32
    // lanes work below order 7)
    static constexpr int P = 1 << LP, LW = N - 2 < 5 - LP ? N - 2 : 5 - LP, WK = 1 << LW;
    static constexpr int RW = (N + P - 1) / P;
    static constexpr int RP = (RW + 3) & ~3;
    static constexpr int COL = P * 3 * RP;                     // floats of a column
    // two blocks of 128 threads per SM: (RMAX + waiting slots) rows of 8
    // bytes per thread and the table in 113 KB
    static constexpr int RCAP = RW == 8 ? 8 : 10;
    static constexpr int RMAX = N - 1 - LW < RCAP ? N - 1 - LW : RCAP;
    static constexpr int WAIT = LW + 1 > GRAD_TREE - 1 ? LW + 1 : GRAD_TREE - 1;
    static constexpr int SLOTS = RMAX + WAIT;
    static constexpr size_t smem(int warps) {
        return sizeof(float) * (size_t)N * COL + (size_t)SLOTS * RW * 32 * warps * sizeof(float2);
    }
};

// sum += f x, f = +-1
__device__ __forceinline__ void df_accumulate(df &sum, float f, df x) {
    const float t = fmaf(f, x.hi, sum.hi);
    const float b = t - sum.hi;
    sum.lo += (sum.hi - (t - b)) + fmaf(f, x.hi, -b);
    sum.lo = fmaf(f, x.lo, sum.lo);
    sum.hi = t;
}
// a + f b, unnormalised low word
__device__ __forceinline__ df df_sum(df a, float f, df b) {
    df_accumulate(a, f, b);
    return a;
}

// Two FP32 values in a register pair: one issue slot does both (the FP32
// pipes take the same time, but two warps per scheduler cannot issue enough
// single operations to fill them).
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float x, float y) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(f2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 f2_neg(f2 a) { return a ^ 0x8000000080000000ull; }
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) { return f2_fma(b, f2_pack(-1.f, -1.f), a); }

struct df2 { f2 hi, lo; };       // two double-floats
__device__ __forceinline__ void df2_chain(df2 &p, df2 s) {
    const f2 q = f2_mul(p.hi, s.hi);
    f2 e = f2_fma(p.hi, s.hi, f2_neg(q));
    e = f2_fma(p.hi, s.lo, e);
    p.lo = f2_fma(p.lo, s.hi, e);
    p.hi = q;
}
__device__ __forceinline__ df2 df2_renorm(df2 a) {
    const f2 h = f2_add(a.hi, a.lo);
    return df2{h, f2_sub(a.lo, f2_sub(h, a.hi))};
}
__device__ __forceinline__ f2 f2_shfl_xor(f2 a, int off) {
    const float2 v = f2_unpack(a);
    return f2_pack(__shfl_xor_sync(0xffffffffu, v.x, off), __shfl_xor_sync(0xffffffffu, v.y, off));
}
__device__ __forceinline__ df2 df2_shfl_xor(df2 a, int off) {
    return df2{f2_shfl_xor(a.hi, off), f2_shfl_xor(a.lo, off)};
}

// WARPS = GRAD_WARPS: slots for the reduction; 1: a matrix a block, the result
template <int N, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 8 / WARPS) glynn_gradient_kernel(GradArgs a) {
    using S = GradShape<N>;
    constexpr bool WHOLE = WARPS == 1;
    constexpr int P = S::P, RW = S::RW, RP = S::RP, COL = S::COL, WK = S::WK, LW = S::LW;
    constexpr int BL = fwd_bound_log(false), BT = 32 * WARPS;
    extern __shared__ float4 grad_smem[];
    float *tab = reinterpret_cast<float *>(grad_smem);   // [N][P][3][RP]; column N-1: all-plus sums
    __shared__ int row_exp[N];
    __shared__ bool stop;
    if (threadIdx.x == 0) stop = f64_stopped(a);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p = lane & (P - 1), w = lane >> S::LP;
    // this thread's column of the slots: slot t, row r at [(t RW + r) BT]
    float2 *mine = reinterpret_cast<float2 *>(tab + N * COL) + threadIdx.x;
    const float2 *warp0 = mine - lane;
    const int b = WHOLE ? blockIdx.x : blockIdx.x / a.blocks_per;
    const int part = WHOLE ? 0 : blockIdx.x - b * a.blocks_per;
    const double *A = a.A + (size_t)b * N * N;
    for (int r = threadIdx.x; r < N; r += BT) row_exp[r] = fwd_row_exponent(A + r * N, nullptr, N, BL);
    __syncthreads();
    if (stop) return;
    for (int idx = threadIdx.x; idx < N * P * RP; idx += BT) {
        const int j = idx / (P * RP), q = idx - j * (P * RP), lp = q / RP, r = q - lp * RP;
        float *t = tab + j * COL + lp * 3 * RP + r;
        const int row = lp * RW + r;
        if (r < RW && row < N) {
            fwd_split(ldexp(A[row * N + j], row_exp[row]), BL, t, RP);
        } else {
            // rows beyond N: s = 1
            t[0] = j == N - 1 && r < RW ? 1.f : 0.f;
            t[RP] = t[2 * RP] = 0.f;
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < COL; idx += BT) {
        float sum = tab[(N - 1) * COL + idx];
        for (int j = 0; j < N - 1; j++) {
            const float v = tab[j * COL + idx];
            sum += v;
            tab[j * COL + idx] = 2.f * v;
        }
        tab[(N - 1) * COL + idx] = sum;
    }
    __syncthreads();

    const int R = a.log_range, M = R < GRAD_TREE ? R : GRAD_TREE;
    const bool active = w < WK;
    const uint64_t tasks = 1ull << (N - 1 - R - LW);
    double *slot = WHOLE ? nullptr : a.slots + ((size_t)blockIdx.x * WARPS + warp) * grad_slot(N);
    int exps = 0;              // of all rows; E_i was formed from the rows l != i
    if (WHOLE)
        for (int r = 0; r < N; r++) exps += row_exp[r];
    auto unscaled = [&](double v, int row) { return ldexp(v, row_exp[row] - exps - (N - 1)); };
    const float *own = tab + p * 3 * RP;
    double gabs[RW];
#pragma unroll
    for (int r = 0; r < RW; r++) gabs[r] = 0.0;
    bool aborted = false;
    const uint64_t first = (uint64_t)part * WARPS + warp;
    for (uint64_t k = first; k < (WHOLE ? 1 : tasks); k += (uint64_t)a.blocks_per * WARPS) {
        // voted: the lanes must leave the loop together
        if (k != first && __any_sync(0xffffffffu, *a.abort_flag != 0)) { aborted = true; break; }
        const uint64_t g0 = active ? ((k << LW) + w) << R : 0;
        // row sums of two states: u (column 0 plus) and v (column 0 minus)
        f2 s[3][RW];
        auto column = [&](int j, float (&x)[3][RW]) {
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int v = 0; v < RP / 4; v++) {
                    const float4 q = reinterpret_cast<const float4 *>(own + j * COL + c * RP)[v];
                    x[c][4 * v] = q.x;
                    if (4 * v + 1 < RW) x[c][4 * v + 1] = q.y;
                    if (4 * v + 2 < RW) x[c][4 * v + 2] = q.z;
                    if (4 * v + 3 < RW) x[c][4 * v + 3] = q.w;
                }
        };
        auto step = [&](int j, float f) {
            float x[3][RW];
            column(j, x);
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int r = 0; r < RW; r++) {
                    const float2 t = f2_unpack(s[c][r]);
                    s[c][r] = f2_pack(fmaf(f, x[c][r], t.x), fmaf(f, x[c][r], t.y));
                }
        };
        {
            float x[3][RW], y[3][RW];
            column(N - 1, x);
            column(0, y);
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int r = 0; r < RW; r++) s[c][r] = f2_pack(x[c][r], x[c][r] - y[c][r]);
        }
        const uint64_t gr = g0 ^ (g0 >> 1);
        for (int j = 1; j < N - 1; j++)
            if (__any_sync(0xffffffffu, (gr >> j) & 1)) step(j, ((gr >> j) & 1) ? -1.f : 0.f);

        df V0[RW], WT[RW];
        float ga[RW];
#pragma unroll
        for (int r = 0; r < RW; r++) {
            V0[r] = WT[r] = df{0.f, 0.f};
            ga[r] = 0.f;
        }
        for (int t = 1; t < R; t++)
#pragma unroll
            for (int r = 0; r < RW; r++) mine[(t * RW + r) * BT] = make_float2(0.f, 0.f);

        // states g0 + i and g0 + i + 1 together: u and v share every sign but
        // column 0's, which costs no update
        for (uint32_t i = 0; i < (1u << R); i += 2) {
            const uint64_t g = g0 + i;
            if (i) {
                const int j = __ffs(i) - 1;
                step(j, ((g >> (j + 1)) & 1) ? 1.f : -1.f);
            }
            // E_r of both: prefix products, the other lanes' product, suffix pass
            df2 x[RW], pre[RW];
#pragma unroll
            for (int r = 0; r < RW; r++) {
                const f2 h = f2_add(s[0][r], s[1][r]);
                x[r] = df2{h, f2_add(f2_sub(s[1][r], f2_sub(h, s[0][r])), s[2][r])};
                pre[r] = x[r];
                if (r > 0) {
                    pre[r] = pre[r - 1];
                    df2_chain(pre[r], x[r]);
                }
            }
            df2 q = x[RW - 1];
            if constexpr (P > 1) {
                df2 mine2 = df2_renorm(pre[RW - 1]);
                q = df2_shfl_xor(mine2, 1);
                if constexpr (P > 2) {
                    df2_chain(mine2, q);
                    df2_chain(q, df2_shfl_xor(df2_renorm(mine2), 2));
                    q = df2_renorm(q);
                }
            }
            // with p = (-1)^(minus signs but column 0's): w is p E_u and -p E_v,
            // so column 0 takes p (E_u + E_v); T = E_u - E_v goes up the tree
            const float p0 = ((g >> 1) & 1) ? -1.f : 1.f;
            df T[RW];
#pragma unroll
            for (int r = RW - 1; r >= 0; r--) {
                df2 E;
                if (r == 0) {
                    E = q;
                } else if (P == 1 && r == RW - 1) {
                    E = pre[r - 1];
                } else {
                    E = pre[r - 1];
                    df2_chain(E, q);
                    df2_chain(q, x[r]);
                }
                const float2 h = f2_unpack(E.hi), l = f2_unpack(E.lo);
                const df u = df{h.x, l.x}, v = df{h.y, l.y};
                ga[r] += fabsf(u.hi) + fabsf(v.hi);
                df_accumulate(V0[r], p0, df_sum(u, 1.f, v));
                T[r] = df_sum(u, -1.f, v);
            }
            // Join T with the waiting sums.  On the first level the two pairs
            // have opposite p (the earlier one +), above it sums are signed.
            int t = 1;
            for (; t < M && ((i >> t) & 1); t++) {
                const float f = ((g >> (t + 1)) & 1) ? -1.f : 1.f, e = t == 1 ? -1.f : 1.f;
#pragma unroll
                for (int r = 0; r < RW; r++) {
                    const float2 hv = mine[((S::RMAX + t - 1) * RW + r) * BT];
                    float2 &vv = mine[(t * RW + r) * BT];
                    const df h = df{hv.x, hv.y};
                    df v = df{vv.x, vv.y};
                    df_accumulate(v, f, df_sum(h, -e, T[r]));
                    vv = make_float2(v.hi, v.lo);
                    T[r] = df_sum(h, e, T[r]);
                }
            }
            if (t < M) {
#pragma unroll
                for (int r = 0; r < RW; r++)
                    mine[((S::RMAX + t - 1) * RW + r) * BT] = make_float2(T[r].hi, T[r].lo);
            } else {
#pragma unroll
                for (int r = 0; r < RW; r++) df_accumulate(WT[r], M == 1 ? p0 : 1.f, T[r]);
                const uint64_t gm = g ^ (g >> 1);
                for (t = M; t < R; t++) {
                    const float f = ((gm >> t) & 1) ? -1.f : 1.f;
#pragma unroll
                    for (int r = 0; r < RW; r++) {
                        float2 &vv = mine[(t * RW + r) * BT];
                        df v = df{vv.x, vv.y};
                        df_accumulate(v, f, T[r]);
                        vv = make_float2(v.hi, v.lo);
                    }
                }
            }
        }

        // The walkers' sums, added over the warp; lanes of walker 0 leave
        // them in their slots: columns 0..R-1, then the total W signed by
        // each of the LW columns that differ between walkers, then W.  Those
        // come by pairs, as in the tree: two walkers of a pair (halves of a
        // pair of pairs, ...) have opposite signs of the level's column.
        if (!active) {
#pragma unroll
            for (int r = 0; r < RW; r++) V0[r] = WT[r] = df{0.f, 0.f};
        }
#pragma unroll
        for (int r = 0; r < RW; r++) {
            for (int t = 0; t < R; t++) {
                float2 &vv = mine[(t * RW + r) * BT];
                df v = t == 0 ? V0[r] : df{vv.x, vv.y};
#pragma unroll
                for (int l = 0; l < LW; l++) v = df_add(v, df_shfl_xor(v, P << l));
                if (w == 0) vv = make_float2(v.hi, v.lo);
            }
            df d[LW > 0 ? LW : 1], v = WT[r];
#pragma unroll
            for (int l = 0; l < LW; l++) {
#pragma unroll
                for (int t = 0; t < l; t++) d[t] = df_add(d[t], df_shfl_xor(d[t], P << l));
                const df o = df_shfl_xor(v, P << l);
                // column R + l is minus where the bits of g at it and above differ
                const bool neg = (((g0 >> (R + l)) ^ (g0 >> (R + l + 1))) & 1) != 0;
                d[l] = df_add(neg ? df_neg(v) : v, neg ? o : df_neg(o));
                v = df_add(v, o);
            }
            if (w == 0) {
#pragma unroll
                for (int t = 0; t < LW; t++)
                    mine[((S::RMAX + t) * RW + r) * BT] = make_float2(d[t].hi, d[t].lo);
                mine[((S::RMAX + LW) * RW + r) * BT] = make_float2(v.hi, v.lo);
            }
        }
        __syncwarp();
        const uint64_t gt = (k << LW) << R, gtm = gt ^ (gt >> 1);
        for (int e = lane; e < N * N; e += 32) {
            const int i = e / N, j = e - i * N, rr = i % RW, ln = i / RW;
            const int t = j == N - 1 || j >= R + LW ? S::RMAX + LW : j < R ? j : S::RMAX + j - R;
            const float2 v = warp0[(t * RW + rr) * BT + ln];
            double x = (double)v.x + (double)v.y;
            if (j < N - 1 && j >= R + LW && ((gtm >> j) & 1)) x = -x;
            if constexpr (WHOLE) {
                a.grad[(size_t)b * N * N + e] = unscaled(x, i);
                continue;
            }
            double sm = slot[e], cp = slot[N * N + e];
            kahan(sm, cp, x);
            slot[e] = sm;
            slot[N * N + e] = cp;
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < RW; r++) gabs[r] += active ? (double)ga[r] : 0.0;
    }
#pragma unroll
    for (int o = P; o < P << LW; o <<= 1)
#pragma unroll
        for (int r = 0; r < RW; r++) gabs[r] += __shfl_xor_sync(0xffffffffu, gabs[r], o);
    if (lane == 0 && aborted) atomicExch(a.status, 1);
    if (w != 0) return;
#pragma unroll
    for (int r = 0; r < RW; r++) {
        const int row = p * RW + r;
        if (row >= N) continue;
        if constexpr (!WHOLE) slot[2 * N * N + row] = gabs[r];
        else if (a.grad_abs) a.grad_abs[(size_t)b * N + row] = unscaled(gabs[r], row);
    }
}

template <int N, int WARPS>
cudaError_t launch_glynn_gradient_warps(const GradArgs &a, cudaStream_t s) {
    constexpr size_t smem = GradShape<N>::smem(WARPS);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(glynn_gradient_kernel<N, WARPS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    glynn_gradient_kernel<N, WARPS>
        <<<(unsigned)(a.batch * a.blocks_per), 32 * WARPS, smem, s>>>(a);
    return cudaGetLastError();
}
// a.slots null: one-warp blocks, which need one range a walker at most
template <int N>
cudaError_t launch_glynn_gradient(const GradArgs &a, cudaStream_t s) {
    if constexpr (N <= GRAD_WHOLE_N) {
        if (!a.slots) return launch_glynn_gradient_warps<N, 1>(a, s);
    }
    if constexpr (N >= GRAD_SPLIT_N) {
        if (a.slots) return launch_glynn_gradient_warps<N, GRAD_WARPS>(a, s);
    }
    return cudaErrorInvalidValue;
}

// log2 of a warp's walkers and of the longest range at order n
void gradient_shape(int n, int *log_walkers, int *log_range_max);

// Instantiated in f64_grad_{lo,mid,hi}.cu: orders 2..16, 17..24, 25..32.
cudaError_t launch_gradient_lo(int n, const GradArgs &a, cudaStream_t s);
cudaError_t launch_gradient_mid(int n, const GradArgs &a, cudaStream_t s);
cudaError_t launch_gradient_hi(int n, const GradArgs &a, cudaStream_t s);

}  // namespace pg
