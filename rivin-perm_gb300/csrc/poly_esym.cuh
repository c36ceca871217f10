// Exact polynomial Glynn for a constant matrix C = gamma J and a matrix L of
// small row sums (the rook polynomials: per(J + x A), perm_polynomial.py:
// 1288-1411), with no moduli.
//
// With m the number of minus signs, every row's constant part is
// c = gamma (n - 2 m), so
//   sum_d (prod d) prod_i (c + x l_i(d))
//     = sum_k x^k sum_m (-1)^m (gamma (n - 2 m))^(n-k) T[m][k],
//   T[m][k] = sum over the d with m minus signs of e_k(l_1(d), ..., l_n(d)).
// The kernel sums the exact integers T[m][k]; the host combines them modulo
// every requested modulus.
//
// e_k: the recurrence E[d] += l_r E[d-1] on integers in radix 2^26, digits
// 0..2^26 - 1 under a signed top digit.  |l_r| <= 31 keeps
// l E_j + F_j + carry in 32 bits, so a digit costs one 32-bit multiply-add,
// one addition, one shift and one mask, and the coefficients start as single
// digits: the digit count of every (row, d) is a compile-time constant from
// the bound C(r, d) LMAX^d.  At order 25 a state takes about 2100
// instructions; the modular recurrence (pg_poly_uniform.cu) takes 433
// Montgomery products for each of five moduli, about 15000.
//
// Walk: the low six columns run through all 64 sign sets in order of their
// weight, so that m is constant while a class is summed; the other columns'
// signs differ between lanes, the lanes of a warp holding 32 sets of one
// weight (unranked combinations), so m is common to the warp.  Row sums are
// bytes 128 + l, four rows to a word: a sign change is one addition per word.
// At the end of a class the warp adds its digits (redux) and adds them to the
// bins of m with 64-bit atomics.
//
// Bound by the integer pipes (2.2 instructions per clock; shifts and masks on
// one pipe, multiply-adds on another).  Five moduli at order 25: 13.7 ms with
// the modular kernel, 1.95 ms here; 25x25 rook polynomial with its host work
// 9.9 -> 2.4 ms; order 28: 141 -> 18.6 ms.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace pg {

constexpr int ESYM_LOW = 6;            // columns walked inside a thread
constexpr int ESYM_RADIX = 26;
constexpr int ESYM_MIN_N = 14, ESYM_MAX_N = 31, ESYM_MAX_L = 31;

// Digit counts: nd[r][d] digits hold every |E_r[d]| <= C(r, d) LMAX^d, the
// top one below 2^26 in magnitude.
template <int N, int LMAX>
struct EsymTable {
    int nd[N + 1][N + 1] = {};
    constexpr EsymTable() {
        uint64_t b[N + 1][8] = {};     // bounds of the current row, 32 bits a word
        b[0][0] = 1;
        nd[0][0] = 1;
        for (int r = 1; r <= N; r++) {
            for (int d = r; d >= 1; d--) {
                uint64_t carry = 0;
                for (int w = 0; w < 8; w++) {
                    const uint64_t t = b[d][w] + LMAX * b[d - 1][w] + carry;
                    b[d][w] = t & 0xffffffffull;
                    carry = t >> 32;
                }
            }
            nd[r][0] = 1;
            for (int d = 1; d <= r; d++) {
                int bits = 0;
                for (int w = 0; w < 8; w++)
                    for (int k = 0; k < 32; k++)
                        if ((b[d][w] >> k) & 1) bits = 32 * w + k + 1;
                nd[r][d] = (bits + ESYM_RADIX - 1) / ESYM_RADIX;
            }
        }
    }
};

template <int N, int LMAX>
struct EsymShape {
    static constexpr EsymTable<N, LMAX> T{};
    static constexpr int nd(int r, int d) { return d < 0 || d > r ? 0 : T.nd[r][d]; }
    // digits of E[1..N], coefficient-major, and of the sums (one more each)
    static constexpr int off(int d) {
        int s = 0;
        for (int k = 1; k < d; k++) s += T.nd[N][k];
        return s;
    }
    static constexpr int DIGITS = off(N + 1);
    static constexpr int sum_off(int d) { return off(d) + d - 1; }
    static constexpr int SUMS = DIGITS + N;
    // Sums in registers, eight warps, while E and they fit (order 25: 1.87 ms
    // against 2.03 with the sums in shared memory and twelve warps); else in
    // shared memory with the warps that fit (order 28: 18.5 ms with twelve,
    // 20.2 with eight).
    static constexpr bool REG = DIGITS <= 90;
    static constexpr int THREADS = REG || SUMS * 320 * 4 > 220 * 1024 ? 256
                                   : SUMS * 384 * 4 > 220 * 1024 ? 320 : 384;
    static constexpr int NW = (N + 3) / 4, NWP = (NW + 3) & ~3;
    static constexpr size_t smem = REG ? 0 : (size_t)SUMS * THREADS * 4;
};

struct EsymArgs {
    const uint32_t *cols;      // [n-1][NWP] packed 2 a_ij (integer sums over the bytes)
    const uint32_t *init;      // [NWP] packed 128 + row sums
    const uint32_t *binom;     // [32][32] C(i, k)
    const uint32_t *first;     // [high + 2] first warp task of every weight of the high columns
    const uint8_t *sets;       // [64] low sign sets by weight
    int n, high;               // high = n - 1 - ESYM_LOW
    long long *bins;           // [n][SUMS], zeroed
    int *status;
    volatile const int *abort_flag;
};

// E[d] += l E[d-1] at row r (1-based)
template <class S, int r, int d>
__device__ __forceinline__ void esym_coef(int32_t *E, int32_t l) {
    constexpr int K = S::nd(r, d), KE = S::nd(r - 1, d - 1), KF = S::nd(r - 1, d);
    constexpr int M = (1 << ESYM_RADIX) - 1;
    int32_t carry = 0;
#pragma unroll
    for (int j = 0; j < K; j++) {
        int32_t t = carry;
        if (j < KF) t += E[S::off(d) + j];
        if constexpr (d == 1) {
            if (j == 0) t += l;
        } else {
            if (j < KE) t += l * E[S::off(d - 1) + j];
        }
        if (j < K - 1) {
            carry = t >> ESYM_RADIX;
            t &= M;
        }
        E[S::off(d) + j] = t;
    }
}
template <class S, int r, int... I>
__device__ __forceinline__ void esym_row(int32_t *E, int32_t l, std::integer_sequence<int, I...>) {
    (esym_coef<S, r, r - I>(E, l), ...);       // d = r, r - 1, ..., 1
}
template <class S, int NN, int... I>
__device__ __forceinline__ void esym_rows(int32_t *E, const int32_t *l, int n,
                                          std::integer_sequence<int, I...>) {
    ((I < n ? esym_row<S, I + 1>(E, l[I], std::make_integer_sequence<int, I + 1>{}) : (void)0), ...);
}

template <int K>
__device__ __forceinline__ int32_t esym_byte(uint32_t x) {
    int32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "n"(0x8880 + 0x1111 * K));
    return r;
}

// sums[digit] += E (registers or this thread's column of shared memory)
template <class S, int N, int d>
__device__ __forceinline__ void esym_add(const int32_t *E, int32_t *acc, int32_t *sm) {
#pragma unroll
    for (int j = 0; j < S::nd(N, d); j++) {
        if constexpr (S::REG) acc[S::sum_off(d) + j] += E[S::off(d) + j];
        else sm[(S::sum_off(d) + j) * S::THREADS] += E[S::off(d) + j];
    }
}
template <class S, int N, int... I>
__device__ __forceinline__ void esym_add_all(const int32_t *E, int32_t *acc, int32_t *sm,
                                             std::integer_sequence<int, I...>) {
    (esym_add<S, N, I + 1>(E, acc, sm), ...);
}

// Carries coefficient d's sums (a class adds at most 20 digits below 2^26, so
// they fit 32 bits), adds them over the warp and leaves digit i in lane
// i mod 32's `hold`; every 32 digits go to the bins.
template <class S, int N, int d>
__device__ __forceinline__ void esym_flush(int32_t *acc, int32_t *sm, bool active, int lane,
                                           int32_t &hold, long long *bin) {
    constexpr int K = S::nd(N, d), M = (1 << ESYM_RADIX) - 1;
    int32_t carry = 0;
#pragma unroll
    for (int j = 0; j <= K; j++) {
        constexpr int base = S::sum_off(d);
        int32_t v = carry;
        if constexpr (S::REG) {
            v += acc[base + j];
            acc[base + j] = 0;
        } else {
            v += sm[(base + j) * S::THREADS];
            sm[(base + j) * S::THREADS] = 0;
        }
        if (j < K) {
            carry = v >> ESYM_RADIX;
            v &= M;
        }
        const int32_t t = __reduce_add_sync(0xffffffffu, active ? v : 0);
        const int i = base + j;
        if (lane == (i & 31)) hold = t;
        if ((i & 31) == 31 || i == S::SUMS - 1) {
            if (lane <= (i & 31))
                atomicAdd((unsigned long long *)(bin + (i & ~31) + lane),
                          (unsigned long long)(long long)hold);
        }
    }
}
template <class S, int N, int... I>
__device__ __forceinline__ void esym_flush_all(int32_t *acc, int32_t *sm, bool active, int lane,
                                               long long *bin, std::integer_sequence<int, I...>) {
    int32_t hold = 0;
    (esym_flush<S, N, I + 1>(acc, sm, active, lane, hold, bin), ...);
}

template <int N, int LMAX>
__global__ void __launch_bounds__(EsymShape<N, LMAX>::THREADS, 1) poly_esym_kernel(EsymArgs a) {
    using S = EsymShape<N, LMAX>;
    constexpr int NW = S::NW, NWP = S::NWP;
    extern __shared__ int32_t esym_smem[];
    __shared__ uint4 cols_s[(ESYM_MAX_N - 1) * NWP / 4];
    __shared__ uint32_t binom_s[32 * 32], first_s[32];
    __shared__ uint8_t sets_s[64];
    const int lane = threadIdx.x & 31, n = a.n;
    for (int i = threadIdx.x; i < (n - 1) * NWP / 4; i += S::THREADS)
        cols_s[i] = reinterpret_cast<const uint4 *>(a.cols)[i];
    for (int i = threadIdx.x; i < 32 * 32; i += S::THREADS) binom_s[i] = a.binom[i];
    if (threadIdx.x < 64) sets_s[threadIdx.x] = a.sets[threadIdx.x];
    if (threadIdx.x < a.high + 2) first_s[threadIdx.x] = a.first[threadIdx.x];
    int32_t acc[S::REG ? S::SUMS : 1];
    int32_t *sm = esym_smem + threadIdx.x;
    if constexpr (S::REG) {
#pragma unroll
        for (int i = 0; i < S::SUMS; i++) acc[i] = 0;
    } else {
        for (int i = 0; i < S::SUMS; i++) sm[i * S::THREADS] = 0;
    }
    __syncthreads();

    uint32_t u[NW];
    auto turn = [&](int j, bool minus) {
        uint32_t c[NWP];
#pragma unroll
        for (int v = 0; v < NWP / 4; v++) {
            const uint4 x = cols_s[j * (NWP / 4) + v];
            c[4 * v] = x.x;
            c[4 * v + 1] = x.y;
            c[4 * v + 2] = x.z;
            c[4 * v + 3] = x.w;
        }
#pragma unroll
        for (int v = 0; v < NW; v++) u[v] += minus ? 0u - c[v] : c[v];
    };
    // The block's warps take neighbouring tasks and run in step (a barrier per
    // state): a state is thousands of straight-line instructions, which the
    // warps then fetch together.
    constexpr uint32_t PER = S::THREADS / 32;
    const uint32_t tasks = first_s[a.high + 1];
    bool aborted = false;
    for (uint32_t t0 = blockIdx.x * PER; t0 < tasks; t0 += gridDim.x * PER) {
        if (t0 != blockIdx.x * PER && __syncthreads_or(*a.abort_flag != 0)) {
            aborted = true;
            break;
        }
        const uint32_t task = t0 + (threadIdx.x >> 5);
        int p = 0;                      // minus signs among the high columns
        while (p < a.high && first_s[p + 1] <= task) p++;
        uint32_t q = (task - first_s[p]) * 32 + lane;
        const bool active = q < binom_s[a.high * 32 + p];
        if (!active) q = 0;
#pragma unroll
        for (int v = 0; v < NW; v++) u[v] = a.init[v];
        for (int i = a.high - 1, k = p; i >= 0; i--) {
            const uint32_t c = binom_s[i * 32 + k];
            const bool in = k > 0 && q >= c;         // the q-th set of k among the low i + 1
            if (in) {
                q -= c;
                k--;
                turn(ESYM_LOW + i, true);
            }
        }
        uint32_t set = 0;
        for (int i = 0; i < 64; i++) {
            const uint32_t next = sets_s[i];
            for (uint32_t diff = set ^ next; diff; diff &= diff - 1) {
                const int j = __ffs(diff) - 1;
                turn(j, (next >> j) & 1);
            }
            const int w = __popc(next);
            if (w != __popc(set))
                esym_flush_all<S, N>(acc, sm, active, lane, a.bins + (size_t)(p + w - 1) * S::SUMS,
                                     std::make_integer_sequence<int, N>{});
            set = next;
            __syncthreads();
            int32_t l[4 * NW];
#pragma unroll
            for (int v = 0; v < NW; v++) {
                const uint32_t x = u[v] ^ 0x80808080u;
                l[4 * v] = esym_byte<0>(x);
                l[4 * v + 1] = esym_byte<1>(x);
                l[4 * v + 2] = esym_byte<2>(x);
                l[4 * v + 3] = esym_byte<3>(x);
            }
            int32_t E[S::DIGITS];
#pragma unroll
            for (int k = 0; k < S::DIGITS; k++) E[k] = 0;
            esym_rows<S, N>(E, l, n, std::make_integer_sequence<int, N>{});
            esym_add_all<S, N>(E, acc, sm, std::make_integer_sequence<int, N>{});
        }
        esym_flush_all<S, N>(acc, sm, active, lane, a.bins + (size_t)(p + ESYM_LOW) * S::SUMS,
                             std::make_integer_sequence<int, N>{});
    }
    if (aborted && lane == 0) atomicExch(a.status, 1);
}

// Layout of a compiled shape for the host.
struct EsymLayout {
    int n_max, l_max, sums, words;      // words: NWP
    int digits[ESYM_MAX_N + 1], sum_off[ESYM_MAX_N + 1];
};

template <int N, int LMAX>
EsymLayout esym_layout() {
    using S = EsymShape<N, LMAX>;
    EsymLayout o = {};
    o.n_max = N;
    o.l_max = LMAX;
    o.sums = S::SUMS;
    o.words = S::NWP;
    for (int d = 1; d <= N; d++) {
        o.digits[d] = S::T.nd[N][d] + 1;
        o.sum_off[d] = S::sum_off(d);
    }
    return o;
}

template <int N, int LMAX>
cudaError_t launch_esym(const EsymArgs &a, int sm_count, uint32_t tasks, cudaStream_t s) {
    using S = EsymShape<N, LMAX>;
    cudaError_t e = cudaFuncSetAttribute(poly_esym_kernel<N, LMAX>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem);
    if (e != cudaSuccess) return e;
    const uint32_t per = S::THREADS / 32;
    const uint32_t most = (tasks + per - 1) / per;
    poly_esym_kernel<N, LMAX>
        <<<most < (uint32_t)sm_count ? most : sm_count, S::THREADS, S::smem, s>>>(a);
    return cudaGetLastError();
}

// Compiled shapes, smallest first (poly_esym_*.cu): the entry that takes
// order n and row sums up to lmax; false when there is none.  Orders rise by a
// quarter (16, 20, 25, 31), with 28 between the last two, where a call takes
// longest; rows beyond n are skipped, so that padding only costs the last
// coefficients' sums.  Finer steps gain little or lose: a shape for 18 takes 9 %
// off orders 17 and 18, one for 22 adds 10 % to 21 and 22 (222 -> 246 us), and
// each costs seconds of every build.
struct EsymEntry {
    EsymLayout layout;
    cudaError_t (*launch)(const EsymArgs &, int, uint32_t, cudaStream_t);
};
bool esym_entry_15(int n, EsymEntry *out);
bool esym_entry_20(int n, EsymEntry *out);
bool esym_entry_31(int n, EsymEntry *out);

}  // namespace pg
