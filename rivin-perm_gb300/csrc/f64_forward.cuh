// FP64-accurate Glynn permanent (forward) of real or complex matrices of
// order 2..32: one thread per Gray range, exact row sums on fixed grids.
//
//   per(A) = 2^(1-n) sum_g (-1)^g prod_i s_i(g),   s_i(g) = sum_j d_j(g) a_ij
// (rivin-perm permanent_glynn_kernel, perm_parallel_cuda.cu:68-209).
//
// FP64 issues at 1/70 of FP32 on this part, so the walk runs on the FP32
// pipes.  Rows are scaled by powers of two and every scaled entry is split
// once into three FP32 parts on fixed grids,
//   a = h + m + l,  h a multiple of 2^GH, m a multiple of 2^GM, l the rest,
// chosen so that any signed sum of 32 entries' h parts (and of their m
// parts) has at most 24 bits: a Gray step is then three FP32 additions per
// row with no rounding in h and m (l's rounding is below 2^-61 of the row
// bound), against the 11 of a double-float addition, and nothing drifts, so
// the sums are never recomputed.  Per state a row is renormalised to a
// double-float (fast two-sum, four operations) and multiplied into one of
// four product chains (double-float products whose error word is left
// unnormalised inside the chain: four operations instead of seven).
//
// A thread walks 2^R consecutive states, aligned, so every lane of a warp
// toggles the same column and reads it by broadcast from the block's shared
// table.  Each warp takes aligned blocks of 2^log_block states of the
// block's matrix.  A lane-per-row layout (32 lanes form one state's product
// by a shuffle butterfly) spends 5 products and 10 shuffles per lane where
// this one spends n - 1 products per 32 states.  64 x 28x28 real: 824 -> 106
// ms; 32 x 21x21 complex: 12.5 -> 1.67 ms, error against 64 bits 1.9e-12 ->
// 2e-13.
//
// A real matrix that one warp covers (orders up to 9, to 13 in large batches)
// gets a thread block of that warp, which writes the result itself: 65536
// matrices 8x8 0.65 -> 0.35 ms, 13x13 2.33 -> 1.81, against four warps, slots and a
// reduction.
//
// abs_sum: real |terms| are summed per thread.  Complex |terms| are summed
// in FP32 in Gray order over each block of 2^12 states, as the error scale
// has always been, so a warp keeps its block's magnitudes in shared memory
// and adds them in order afterwards (4 % of the walk).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "df_arith.cuh"

namespace pg {

struct FwdArgs {
    const double *Are, *Aim;   // [batch][n][n] row-major, device; Aim null when real
    int batch;
    int blocks_per;            // thread blocks per matrix
    int log_block;             // states of a warp's block: 2^log_block <= 2^(n-1)
    double *slots;             // [batch][blocks_per][FWD_WARPS][FWD_SLOT]; null: one-warp blocks,
    double *re, *abs_sum;      // a matrix each, that write the results (abs_sum may be null)
    volatile const int *abort_flag;
    int *status;
    int resident;              // blocks of the first wave, at most
};

// Blocks beyond the first wave ask before they start (a batch of small
// matrices is one range a warp, which polls only between ranges): every 64th
// reads the host-mapped word and passes it on through the status.
template <class Args>
__device__ __forceinline__ bool f64_stopped(const Args &a) {
    if ((int)blockIdx.x < a.resident) return false;
    if (*(volatile const int *)a.status) return true;
    if ((blockIdx.x & 63) || !*a.abort_flag) return false;
    atomicExch(a.status, 1);
    return true;
}

constexpr int FWD_WARPS = 4;       // warps of a thread block
constexpr int FWD_SLOT = 3;        // re, im, sum |term|
constexpr int FWD_LOG_BLOCK = 12;  // largest block of a warp
constexpr int FWD_WHOLE_N = 13;    // largest order whose real matrices a warp can take whole
constexpr int FWD_SPLIT_N = 10;    // smallest order with more than one block of states

// Power-of-two scaling: row bounds (sum |re| + |im|) in [2^(b-1), 2^b).
// Real products of 32 rows then stay within 2^64 and typical ones near 1;
// the complex walk keeps bounds below 1.
__host__ __device__ constexpr int fwd_bound_log(bool cplx) { return cplx ? 0 : 2; }

// exponent e with 2^e * bound in [2^(b-1), 2^b); 0 for a zero row
__device__ __forceinline__ int fwd_row_exponent(const double *re, const double *im, int n, int b) {
    double sum = 0.0;
    for (int j = 0; j < n; j++) sum += fabs(re[j]) + (im ? fabs(im[j]) : 0.0);
    int e = 0;
    if (sum > 0.0) {
        frexp(sum, &e);
        e = b - e;
    }
    return e;
}

// x = parts[0] + parts[stride] + parts[2 stride]: multiples of 2^(b - 23),
// of 2^(b - 43), and the rest.  |x| <= 2^b: 32 h parts sum to at most
// 2^b + 2^(b-19) < 2^24 grid steps, 32 m parts (each at most 2^(b-24)) to
// 2^(b-19) = 2^24 grid steps.
__device__ __forceinline__ void fwd_split(double x, int b, float *parts, int stride) {
    const double ch = ldexp(1.5, 52 + b - 23), cm = ldexp(1.5, 52 + b - 43);
    const double h = (x + ch) - ch, r = x - h, m = (r + cm) - cm;
    parts[0] = (float)h;
    parts[stride] = (float)m;
    parts[2 * stride] = (float)(r - m);
}

// (p, e) *= s without renormalising e (|e| stays within a few ulps of p)
__device__ __forceinline__ void df_chain(df &p, df s) {
    const float q = p.hi * s.hi;
    float e = fmaf(p.hi, s.hi, -q);
    e = fmaf(p.hi, s.lo, e);
    p.lo = fmaf(p.lo, s.hi, e);
    p.hi = q;
}
__device__ __forceinline__ df df_renorm(df a) {
    const float h = a.hi + a.lo;
    return df{h, a.lo - (h - a.hi)};
}
// sum += x (two-sum; the low word collects the errors unnormalised)
__device__ __forceinline__ void df_accumulate(df &sum, df x) {
    const float t = sum.hi + x.hi;
    const float b = t - sum.hi;
    sum.lo += ((sum.hi - (t - b)) + (x.hi - b)) + x.lo;
    sum.hi = t;
}
// a b - c d, error word unnormalised
__device__ __forceinline__ df df_det(df a, df b, df c, df d) {
    const float p = a.hi * b.hi, q = c.hi * d.hi;
    const float pe = fmaf(a.hi, b.hi, -p), qe = fmaf(c.hi, d.hi, -q);
    const float x = p - q, t = p - x;
    float e = ((p - (x + t)) + (t - q)) + (pe - qe);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    e = fmaf(-c.hi, d.lo, e);
    e = fmaf(-c.lo, d.hi, e);
    return df{x, e};
}
__device__ __forceinline__ dc dc_chain(dc p, dc s) {
    return dc{df_det(p.re, s.re, p.im, s.im), df_det(p.re, s.im, df_neg(p.im), s.re)};
}
__device__ __forceinline__ dc dc_renorm(dc a) { return dc{df_renorm(a.re), df_renorm(a.im)}; }

template <int N, bool CPLX>
struct FwdShape {
    static constexpr int NP = (N + 3) & ~3;
    static constexpr int C = CPLX ? 6 : 3;             // parts of an entry
    static constexpr int COL = C * NP;                 // floats of a column
    static constexpr int LB = N - 1 < FWD_LOG_BLOCK ? N - 1 : FWD_LOG_BLOCK;
    static constexpr size_t smem = sizeof(float) * ((size_t)N * COL +
                                                    (CPLX ? (size_t)FWD_WARPS << LB : 0));
};

// WARPS = FWD_WARPS: slots for the reduction; 1: a matrix a block, the results
template <int N, bool CPLX, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) glynn_forward_kernel(FwdArgs a) {
    using S = FwdShape<N, CPLX>;
    constexpr bool WHOLE = WARPS == 1;
    constexpr int BT = 32 * WARPS;
    constexpr int NP = S::NP, C = S::C, COL = S::COL, BL = fwd_bound_log(CPLX);
    extern __shared__ float4 fwd_smem[];
    // columns 0..N-2 hold 2 a'_ij, column N-1 the all-plus row sums
    float *tab = reinterpret_cast<float *>(fwd_smem);
    __shared__ int row_exp[N];
    __shared__ bool stop;
    if (threadIdx.x == 0) stop = f64_stopped(a);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = blockIdx.x / a.blocks_per, part = blockIdx.x - b * a.blocks_per;
    const double *Ar = a.Are + (size_t)b * N * N;
    const double *Ai = CPLX ? a.Aim + (size_t)b * N * N : nullptr;
    for (int r = threadIdx.x; r < N; r += BT)
        row_exp[r] = fwd_row_exponent(Ar + r * N, CPLX ? Ai + r * N : nullptr, N, BL);
    __syncthreads();
    if (stop) return;
    for (int idx = threadIdx.x; idx < N * NP; idx += BT) {
        const int j = idx / NP, r = idx - j * NP;
        float *t = tab + j * COL + r;
        if (r < N) {
            fwd_split(ldexp(Ar[r * N + j], row_exp[r]), BL, t, NP);
            if (CPLX) fwd_split(ldexp(Ai[r * N + j], row_exp[r]), BL, t + 3 * NP, NP);
        } else {
            for (int c = 0; c < C; c++) t[c * NP] = 0.f;
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

    float *mags = tab + N * COL + ((size_t)warp << S::LB);    // complex only
    const int lanes_log = a.log_block < 5 ? a.log_block : 5, R = a.log_block - lanes_log;
    const bool active = lane < (1 << lanes_log);
    const uint64_t blocks = (1ull << (N - 1)) >> a.log_block;
    double sre = 0.0, cre = 0.0, sim = 0.0, cim = 0.0, asum = 0.0;
    bool aborted = false;
    const uint64_t first = (uint64_t)part * WARPS + warp;
    for (uint64_t k = first; k < blocks; k += (uint64_t)a.blocks_per * WARPS) {
        // voted: the lanes must leave the loop together
        if (k != first && __any_sync(0xffffffffu, *a.abort_flag != 0)) { aborted = true; break; }
        const uint64_t g0 = (k << a.log_block) + ((uint64_t)(active ? lane : 0) << R);
        float s[C][N];
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
            for (int v = 0; v < NP / 4; v++) {
                const float4 x = reinterpret_cast<const float4 *>(tab + (N - 1) * COL + c * NP)[v];
                s[c][4 * v] = x.x;
                if (4 * v + 1 < N) s[c][4 * v + 1] = x.y;
                if (4 * v + 2 < N) s[c][4 * v + 2] = x.z;
                if (4 * v + 3 < N) s[c][4 * v + 3] = x.w;
            }
        auto step = [&](int j, float sgn) {
#pragma unroll
            for (int c = 0; c < C; c++)
#pragma unroll
                for (int v = 0; v < NP / 4; v++) {
                    const float4 x = reinterpret_cast<const float4 *>(tab + j * COL + c * NP)[v];
                    s[c][4 * v] = fmaf(sgn, x.x, s[c][4 * v]);
                    if (4 * v + 1 < N) s[c][4 * v + 1] = fmaf(sgn, x.y, s[c][4 * v + 1]);
                    if (4 * v + 2 < N) s[c][4 * v + 2] = fmaf(sgn, x.z, s[c][4 * v + 2]);
                    if (4 * v + 3 < N) s[c][4 * v + 3] = fmaf(sgn, x.w, s[c][4 * v + 3]);
                }
        };
        const uint64_t gr = g0 ^ (g0 >> 1);
        for (int j = 0; j < N - 1; j++)
            if (__any_sync(0xffffffffu, (gr >> j) & 1)) step(j, ((gr >> j) & 1) ? -1.f : 0.f);

        df bre = df{0.f, 0.f}, bim = df{0.f, 0.f};
        float babs = 0.f;
        for (uint32_t i = 0;;) {
            // double-float row sums (h dominates m unless the sum nearly vanishes)
            auto row = [&](int c, int r) {
                const float h = s[c][r] + s[c + 1][r];
                return df{h, (s[c + 1][r] - (h - s[c][r])) + s[c + 2][r]};
            };
            constexpr int CH = N < 4 ? N : 4;
            if constexpr (CPLX) {
                dc P[CH];
#pragma unroll
                for (int r = 0; r < N; r++) {
                    const dc x = dc{row(0, r), row(3, r)};
                    if (r < CH) P[r] = x;
                    else P[r % CH] = dc_renorm(dc_chain(P[r % CH], x));
                }
                dc T = P[0];
                if (CH == 4) T = dc_renorm(dc_chain(dc_renorm(dc_chain(P[0], P[1])),
                                                    dc_renorm(dc_chain(P[2], P[3 % CH]))));
                else
                    for (int r = 1; r < CH; r++) T = dc_renorm(dc_chain(T, P[r]));
                if (i & 1) T = dc{df_neg(T.re), df_neg(T.im)};
                df_accumulate(bre, T.re);
                df_accumulate(bim, T.im);
                const float mag = hypotf(T.re.hi, T.im.hi);
                // [lane][i], groups of four permuted by lane against bank conflicts
                if (active)
                    mags[R < 5 ? ((uint32_t)lane << R) + i
                               : ((uint32_t)lane << R) + ((((i >> 2) ^ (uint32_t)lane) & 7u) << 2) +
                                     (i & ~31u) + (i & 3u)] = mag;
            } else {
                df P[CH];
#pragma unroll
                for (int r = 0; r < N; r++) {
                    const df x = row(0, r);
                    if (r < CH) P[r] = x;
                    else df_chain(P[r % CH], x);
                }
                df T;
                if (CH == 4) {
                    df U = df_renorm(P[0]), V = df_renorm(P[2]);
                    df_chain(U, df_renorm(P[1]));
                    df_chain(V, df_renorm(P[3 % CH]));
                    T = df_renorm(U);
                    df_chain(T, df_renorm(V));
                } else {
                    T = P[0];
#pragma unroll
                    for (int r = 1; r < CH; r++) df_chain(T, P[r]);
                }
                T = df_renorm(T);
                babs += fabsf(T.hi);
                df_accumulate(bre, (i & 1) ? df_neg(T) : T);
            }
            if (++i >> R) break;
            const int j = __ffs(i) - 1;
            step(j, (((g0 + i) >> (j + 1)) & 1) ? 1.f : -1.f);
        }
        // ranges start at even states unless they are single ones
        if (R == 0 && (g0 & 1)) {
            bre = df_neg(bre);
            bim = df_neg(bim);
        }
        kahan(sre, cre, active ? df_to(bre) : 0.0);
        if constexpr (CPLX) {
            kahan(sim, cim, active ? df_to(bim) : 0.0);
            __syncwarp();
            float t = 0.f;
            if (R >= 5) {
                for (uint32_t l = 0; l < 32; l++)
#pragma unroll 8
                    for (uint32_t q = 0; q < (1u << R) >> 2; q++) {
                        const float4 x = reinterpret_cast<const float4 *>(
                            mags + (l << R))[(q & ~7u) | ((q ^ l) & 7u)];
                        t += x.x;
                        t += x.y;
                        t += x.z;
                        t += x.w;
                    }
            } else {
                for (uint32_t q = 0; q < (1u << a.log_block); q++) t += mags[q];
            }
            asum += (double)t;
            __syncwarp();
        } else {
            asum += active ? (double)babs : 0.0;
        }
    }
    // warp sums in a fixed order
    sre -= cre;
    sim -= cim;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sre += __shfl_xor_sync(0xffffffffu, sre, o);
        if (CPLX) sim += __shfl_xor_sync(0xffffffffu, sim, o);
        if (!CPLX) asum += __shfl_xor_sync(0xffffffffu, asum, o);
    }
    if (lane != 0) return;
    if constexpr (WHOLE) {
        int e = N - 1;
        for (int r = 0; r < N; r++) e += row_exp[r];
        a.re[b] = ldexp(sre + 0.0, -e);          // + 0.0: no negative zero, as from the reduction
        if (a.abs_sum) a.abs_sum[b] = ldexp(asum, -e);
    } else {
        double *slot = a.slots + ((size_t)blockIdx.x * WARPS + warp) * FWD_SLOT;
        slot[0] = sre;
        slot[1] = sim;
        slot[2] = asum;
        if (aborted) atomicExch(a.status, 1);
    }
}

template <int N, bool CPLX, int WARPS>
cudaError_t launch_glynn_forward_warps(const FwdArgs &a, cudaStream_t s) {
    constexpr size_t smem = FwdShape<N, CPLX>::smem;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(glynn_forward_kernel<N, CPLX, WARPS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    glynn_forward_kernel<N, CPLX, WARPS>
        <<<(unsigned)(a.batch * a.blocks_per), 32 * WARPS, smem, s>>>(a);
    return cudaGetLastError();
}
template <int N, bool CPLX>
cudaError_t launch_glynn_forward(const FwdArgs &a, cudaStream_t s) {
    if constexpr (!CPLX && N <= FWD_WHOLE_N) {
        if (!a.slots) return launch_glynn_forward_warps<N, CPLX, 1>(a, s);
    }
    if constexpr (CPLX || N >= FWD_SPLIT_N) {
        if (a.slots) return launch_glynn_forward_warps<N, CPLX, FWD_WARPS>(a, s);
    }
    return cudaErrorInvalidValue;
}

// Instantiated in f64_fwd_{real,cplx_lo,cplx_hi}.cu: orders 2..32.
cudaError_t launch_forward_real(int n, const FwdArgs &a, cudaStream_t s);
cudaError_t launch_forward_cplx_lo(int n, const FwdArgs &a, cudaStream_t s);
cudaError_t launch_forward_cplx_hi(int n, const FwdArgs &a, cudaStream_t s);

}  // namespace pg
