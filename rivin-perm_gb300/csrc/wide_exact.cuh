// Exact Glynn kernel for integer matrices whose row sums need more than 32
// bits: 64-bit row sums, one traversal, no moduli.
//
//   S = sum_g (-1)^g prod_i s_i(g),  per(A) = S / 2^(n-1)
// (rivin-perm perm.matrix_permanent, perm.py:1076-1212, reduces such matrices
// modulo dozens of primes and lifts).  Row sums below 2^B (B up to 48) are
// kept as exact 64-bit integers; their magnitudes are multiplied as unsigned
// multi-word integers in a tree over each half of the rows, X = prod of the
// first half and Y = prod of the second, and X Y is added into a per-thread
// accumulator.  Word counts are compile-time constants from B and the number
// of rows.  A residue walk pays 24 Montgomery products of five issue slots
// for each of 34 primes at order 25 and entries of 38 bits; here a state takes
// about 650 32 x 32 products, each one multiply-add with carry.
//
// Products: schoolbook with two accumulators, even and odd word pairs, so
// that every partial product is a mad.lo.cc / madc.hi.cc pair on one carry
// chain per multiplier word.
//
// Sign: with the term's sign as a mask m, X ^ m is X or 2^(32 KX) - 1 - X, so
//   sum (X ^ m) Y = S + (2^(32 KX) - 1) sum_{m} Y;
// the accumulator stays unsigned and the masked Y are summed beside it.
//
// A thread walks 2^R consecutive states, aligned, so the toggled column is
// common to the block and read by broadcast; row sums live in shared memory
// ([row][thread]).  Multiply-add bound.  25 x 25, entries up to 2^38, the whole
// call: 8.8 ms by 34 residues and the CRT lift (7.3 with full waves of blocks,
// 2.4 of it prime search and lift on the host), 1.68 ms here.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace pg {

constexpr int WX_THREADS = 128;

struct WideExactArgs {
    const int64_t *tab;        // [n-1][2][N]: +2 a_ij, -2 a_ij; then [N] zeros
    const int64_t *init;       // [N] all-plus row sums (1 beyond n)
    int n, log_range;          // 2^log_range states a thread
    int resident;              // blocks of the first wave (later ones read the abort word)
    unsigned long long *part;  // [words][gridDim] per-block sums
    int *status;
    volatile const int *abort_flag;
};

__host__ __device__ constexpr int wx_words(int rows, int B) { return (rows * B + 31) / 32; }

template <int N, int B>
struct WideShape {
    static constexpr int RX = N / 2, RY = N - RX;
    static constexpr int KX = wx_words(RX, B), KY = wx_words(RY, B), K = KX + KY;
    static constexpr int WORDS = K + 1 + KY + 1;       // accumulator, then the masked Y
    static constexpr size_t smem = ((size_t)(2 * N - 1) * N + (size_t)N * WX_THREADS) * 8;
};

__device__ __forceinline__ void wx_mad_lo_cc(uint32_t &d, uint32_t a, uint32_t b) {
    asm volatile("mad.lo.cc.u32 %0, %1, %2, %0;" : "+r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void wx_madc_lo_cc(uint32_t &d, uint32_t a, uint32_t b) {
    asm volatile("madc.lo.cc.u32 %0, %1, %2, %0;" : "+r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void wx_madc_hi_cc(uint32_t &d, uint32_t a, uint32_t b) {
    asm volatile("madc.hi.cc.u32 %0, %1, %2, %0;" : "+r"(d) : "r"(a), "r"(b));
}
__device__ __forceinline__ void wx_add_cc(uint32_t &d, uint32_t a) {
    asm volatile("add.cc.u32 %0, %0, %1;" : "+r"(d) : "r"(a));
}
__device__ __forceinline__ void wx_addc_cc(uint32_t &d, uint32_t a) {
    asm volatile("addc.cc.u32 %0, %0, %1;" : "+r"(d) : "r"(a));
}
__device__ __forceinline__ void wx_addc(uint32_t &d, uint32_t a) {
    asm volatile("addc.u32 %0, %0, %1;" : "+r"(d) : "r"(a));
}

// acc (pairs starting at even or odd words) += a[first], a[first + 2], ...
// times b, the products at word offset `at`; the carry goes to the next word.
template <int KA, int first, int at, int LEN>
__device__ __forceinline__ void wx_row(uint32_t *acc, const uint32_t *a, uint32_t b) {
#pragma unroll
    for (int i = first; i < KA; i += 2) {
        if (i == first) wx_mad_lo_cc(acc[at + i], a[i], b);
        else wx_madc_lo_cc(acc[at + i], a[i], b);
        wx_madc_hi_cc(acc[at + i + 1], a[i], b);
    }
    constexpr int last = first + (KA - 1 - first) / 2 * 2;       // largest i
    if constexpr (at + last + 2 < LEN) wx_addc(acc[at + last + 2], 0u);
}
template <int KA, int KB, int j>
__device__ __forceinline__ void wx_rows(uint32_t *even, uint32_t *odd, const uint32_t *a,
                                        const uint32_t *b) {
    if constexpr (j < KB) {
        // a[i] b[j] starts at word i + j
        wx_row<KA, 0, j, KA + KB>((j & 1) ? odd : even, a, b[j]);
        if constexpr (KA > 1) wx_row<KA, 1, j, KA + KB>((j & 1) ? even : odd, a, b[j]);
        wx_rows<KA, KB, j + 1>(even, odd, a, b);
    }
}
// even + odd = a b, both of KA + KB words
template <int KA, int KB>
__device__ __forceinline__ void wx_mul(uint32_t *even, uint32_t *odd, const uint32_t *a,
                                       const uint32_t *b) {
#pragma unroll
    for (int i = 0; i < KA + KB; i++) even[i] = odd[i] = 0;
    wx_rows<KA, KB, 0>(even, odd, a, b);
}

// x += y + carry words, LX >= LY
template <int LX, int LY>
__device__ __forceinline__ void wx_add(uint32_t *x, const uint32_t *y) {
#pragma unroll
    for (int i = 0; i < LX; i++) {
        const uint32_t v = i < LY ? y[i] : 0u;
        if (i == 0) wx_add_cc(x[0], v);
        else if (i < LX - 1) wx_addc_cc(x[i], v);
        else wx_addc(x[i], v);
    }
}

// The rows' walk state: moves row r by one Gray step and returns its magnitude.
struct WideRows {
    uint64_t *sums;            // this thread's column of [N][WX_THREADS]
    const int64_t *delta;      // the toggled column
    uint32_t sign;             // XOR of the high words
};

// out[wx_words(M, B)] = |s_r| ... |s_{r + M - 1}|
template <int B, int M>
struct WideProduct {
    static constexpr int K = wx_words(M, B);
    static __device__ __forceinline__ void run(uint32_t *out, WideRows &w, int r) {
        constexpr int ML = M / 2, MR = M - ML;
        constexpr int KL = wx_words(ML, B), KR = wx_words(MR, B);
        uint32_t a[KL], b[KR], even[KL + KR], odd[KL + KR];
        WideProduct<B, ML>::run(a, w, r);
        WideProduct<B, MR>::run(b, w, r + ML);
        wx_mul<KL, KR>(even, odd, a, b);
        wx_add<K, K>(even, odd);
#pragma unroll
        for (int i = 0; i < K; i++) out[i] = even[i];
    }
};
template <int B>
struct WideProduct<B, 1> {
    static __device__ __forceinline__ void run(uint32_t *out, WideRows &w, int r) {
        const int64_t s = (int64_t)w.sums[r * WX_THREADS] + w.delta[r];
        w.sums[r * WX_THREADS] = (uint64_t)s;
        w.sign ^= (uint32_t)((uint64_t)s >> 32);
        const uint64_t m = s < 0 ? 0 - (uint64_t)s : (uint64_t)s;
        out[0] = (uint32_t)m;
        out[1] = (uint32_t)(m >> 32);
    }
};

template <int N, int B>
__global__ void __launch_bounds__(WX_THREADS, 2) wide_exact_kernel(WideExactArgs a) {
    using S = WideShape<N, B>;
    static_assert(B > 32 && B <= 48, "two words a row sum");
    constexpr int KX = S::KX, KY = S::KY, K = S::K, TAB = (2 * N - 1) * N;
    extern __shared__ int64_t wx_smem[];
    int64_t *tab = wx_smem;                       // [N-1][2][N], zeros [N]
    uint64_t *sums = reinterpret_cast<uint64_t *>(wx_smem + TAB) + threadIdx.x;
    __shared__ int stop;
    if (threadIdx.x == 0) stop = (int)blockIdx.x >= a.resident && *a.abort_flag != 0;
    // columns n - 1 .. N - 2 of the compiled order are never toggled
    for (int i = threadIdx.x; i < 2 * (a.n - 1) * N; i += WX_THREADS) tab[i] = a.tab[i];
    for (int i = threadIdx.x; i < N; i += WX_THREADS) tab[2 * (N - 1) * N + i] = 0;
    __syncthreads();
    uint32_t acc[K + 1], ysum[KY + 1];
#pragma unroll
    for (int i = 0; i <= K; i++) acc[i] = 0;
#pragma unroll
    for (int i = 0; i <= KY; i++) ysum[i] = 0;
    const uint64_t tid = (uint64_t)blockIdx.x * WX_THREADS + threadIdx.x;
    const uint64_t g0 = tid << a.log_range;
    if (!stop && g0 >> (a.n - 1) == 0) {
        const uint64_t gr = g0 ^ (g0 >> 1);
        for (int r = 0; r < N; r++) {
            int64_t s = a.init[r];
            for (int j = 0; j < a.n - 1; j++) s += ((gr >> j) & 1) ? tab[(2 * j + 1) * N + r] : 0;
            sums[r * WX_THREADS] = (uint64_t)s;
        }
        for (uint32_t i = 0; i < (1u << a.log_range); i++) {
            WideRows w;
            w.sums = sums;
            w.sign = i << 31;                     // Glynn sign (-1)^g, ranges start even
            w.delta = tab + 2 * (N - 1) * N;
            if (i) {
                const int j = __ffs(i) - 1;
                // lanes differ only in the sign of the range's top column
                w.delta = tab + (2 * j + ((((g0 + i) >> (j + 1)) & 1) ? 0 : 1)) * N;
            }
            uint32_t x[KX], y[KY];
            WideProduct<B, S::RX>::run(x, w, 0);
            WideProduct<B, S::RY>::run(y, w, S::RX);
            const uint32_t m = (uint32_t)((int32_t)w.sign >> 31);
#pragma unroll
            for (int k = 0; k < KX; k++) x[k] ^= m;
            {
                uint32_t even[K], odd[K];
                wx_mul<KX, KY>(even, odd, x, y);
                wx_add<K + 1, K>(acc, even);
                wx_add<K + 1, K>(acc, odd);
            }
#pragma unroll
            for (int k = 0; k < KY; k++) y[k] &= m;
            wx_add<KY + 1, KY>(ysum, y);
        }
    }
    // block sums of every word, as 64-bit integers
    __shared__ unsigned long long red[WX_THREADS / 32][S::WORDS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto reduce = [&](uint32_t x, int l) {
        unsigned long long v = x;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][l] = v;
    };
#pragma unroll
    for (int i = 0; i <= K; i++) reduce(acc[i], i);
#pragma unroll
    for (int i = 0; i <= KY; i++) reduce(ysum[i], K + 1 + i);
    __syncthreads();
    for (int l = threadIdx.x; l < S::WORDS; l += WX_THREADS) {
        unsigned long long t = 0;
        for (int w = 0; w < WX_THREADS / 32; w++) t += red[w][l];
        a.part[(size_t)l * gridDim.x + blockIdx.x] = t;
    }
    if (threadIdx.x == 0 && stop) atomicExch(a.status, 1);
}

// Compiled shapes (wide_exact_*.cu, one file for each B).
struct WideEntry {
    int N, B, kx, ky, words;
    size_t smem;
    cudaError_t (*launch)(const WideExactArgs &, int, cudaStream_t);
};
template <int N, int B>
cudaError_t launch_wide_exact(const WideExactArgs &a, int blocks, cudaStream_t s) {
    using S = WideShape<N, B>;
    cudaError_t e = cudaFuncSetAttribute(wide_exact_kernel<N, B>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem);
    if (e != cudaSuccess) return e;
    wide_exact_kernel<N, B><<<blocks, WX_THREADS, S::smem, s>>>(a);
    return cudaGetLastError();
}
template <int N, int B>
bool wide_entry(int n, WideEntry *out) {
    using S = WideShape<N, B>;
    if (n > N) return false;
    *out = WideEntry{N, B, S::KX, S::KY, S::WORDS, S::smem, launch_wide_exact<N, B>};
    return true;
}
// The smallest compiled order that holds n for row sums below 2^B.
bool wide_entry_36(int n, WideEntry *out);
bool wide_entry_40(int n, WideEntry *out);
bool wide_entry_44(int n, WideEntry *out);
bool wide_entry_48(int n, WideEntry *out);

}  // namespace pg
