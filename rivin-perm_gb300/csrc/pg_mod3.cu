// Permanent modulo 3 by Glynn's formula with table lookups over 2048 states.
//
//   per(A) = 2^(1-n) sum_d (prod_k d_k) prod_i s_i(d)   over F_3,
// s_i(d) = sum_j d_j a_ij, last sign fixed: 2^(n-1) sign vectors (2 is a unit
// modulo 3, 2^(1-n) = (-1)^(n-1)), half of the 2^n subsets of the Ryser walk
// of rivin-perm perm_mod3.py:143-228, perm_mod3_omp.c and
// perm_mod3_cuda.cu:52-131.  An element of F_3 is two bits (magnitude, sign):
// 0 = (0, either), 1 = (1,0), 2 = (1,1); adding or subtracting a canonical
// element is a few bitwise operations (the bipedal formulas of
// arXiv:2407.20205; their truth table over every row-sum encoding and
// canonical column is checked on the host in the tests).
//
// A term counts only when no row sum is zero, about (2/3)^n of the states
// for random entries, so the walk is a search for states without a zero row.
// The low eleven columns' signs are spread over a warp: bit k of word h of
// lane l is the state with low signs (k | l << 5 | h << 10).  The high
// columns are common to the warp, so row i's sum is h_i + low_i(lane, h, bit),
// and "row i is nonzero" is a pair of words that depends only on the lane and
// on h_i in {0, 1, 2}.  For the first six groups of four rows (five above
// order 52) the 81 AND-ed pairs per lane sit in shared memory
// ([81][32] pairs, lane-minor: no bank conflicts): one high state (2048 sign
// vectors) is six 8-byte loads and ANDs for the first 24 rows.  (2/3)^24 of
// the states, in one of eight high states, go on row by row, and only states
// with every row nonzero read the rows' sign words.  The 32 lanes hold the
// high row sums of 32 consecutive high states (row-sliced, one column update
// per 32 of them) and publish their table offsets through shared memory.
//
// Bound by shared-memory loads (95 % of their rate): 17 wavefronts per 2048
// states.  35 x 35 random, a call: 22.9 ms with the row-sliced Ryser walk
// (17.5 instructions per subset, ALU pipe 91 % busy), 0.67 ms with single
// words and tables for every row group, 0.66 with five groups, 0.51 now.  A
// matrix whose states all survive (equal rows) reads every row's words for
// every high state, ~14 instructions per row and 2048 states, still well below
// the row-sliced walk, so no other path is kept.
#include "pg_internal.h"

#include <algorithm>
#include <cstring>

namespace pg {

constexpr int MOD3_THREADS = 1024;   // one block per SM: the tables take up to 224 KB
constexpr int MOD3_LOW = 11;         // columns over word bits (5), lanes (5) and words (1)
constexpr int MOD3_DIGITS = 81;      // states of a group of four rows' high sums

constexpr unsigned long long MOD3_ABORTED = ~0ull;
struct Mod3Args {
    uint64_t mags[64], sgns[64];   // the columns' magnitude and sign words
    int n;
    uint64_t batches;         // 32 high states each (without tables: one)
    // [gridDim], pinned host memory: each block's count (each warp's
    // modulo 3), or MOD3_ABORTED
    volatile unsigned long long *part;
    volatile const int *abort_flag;
};

// row groups with tables, from order 25 on (MOD3_SHORT): six (24 rows) where
// memory allows, else five
__host__ __device__ constexpr int mod3_tables(int n) { return n <= 52 ? 6 : 5; }
// per-row words [n][3][32] pairs; the lists hold six offsets a high state
__host__ __device__ constexpr size_t mod3_row_bytes(int n) { return (size_t)n * 3 * 32 * 8; }
// Few high states (up to 2^12, order 24): no tables, a high state a warp, every
// row read in turn; building the tables took longer than the walk.  A call of
// order 4..16 30 -> 15-18 us, 17..19 43 -> 19, 20..23 35 -> 21, about 10 of
// them by passing the columns as arguments and leaving out both copies (the
// row-sliced walk's: 20-23 us to order 19, 32 to 23).
constexpr int MOD3_SHORT = 12;
__host__ __device__ constexpr int mod3_threads(int GT) { return GT ? MOD3_THREADS : 256; }
__host__ __device__ constexpr size_t mod3_smem(int n) {
    return (size_t)mod3_tables(n) * MOD3_DIGITS * 256 + 2 * mod3_row_bytes(n) + MOD3_THREADS * 24;
}

// row sums (m, s) += or -= column (cm, cs) over F_3, bitwise per row
template <typename W>
__device__ __forceinline__ void f3_add(W &m, W &s, W cm, W cs) {
    const W t = m ^ s ^ cs;
    const W mo = (cm & t) | (m ^ cm);
    s = (cm & t) ^ s;
    m = mo;
}
template <typename W>
__device__ __forceinline__ void f3_sub(W &m, W &s, W cm, W cs) {
    const W t = s ^ cs;
    const W mo = (m & t) | (m ^ cm);
    s = (m & t) ^ (cm ^ cs);
    m = mo;
}

// word of the states k = 0..31 whose bit j is set
__device__ __forceinline__ uint32_t mod3_pattern(int j) {
    return j == 0 ? 0xaaaaaaaau : j == 1 ? 0xccccccccu : j == 2 ? 0xf0f0f0f0u
         : j == 3 ? 0xff00ff00u : 0xffff0000u;
}

template <typename W, int GT>
__global__ void __launch_bounds__(mod3_threads(GT), 1) mod3_kernel(const __grid_constant__ Mod3Args a) {
    constexpr int THREADS = mod3_threads(GT);
    extern __shared__ uint4 mod3_shared[];
    const int n = a.n;
    uint2 *gtab = reinterpret_cast<uint2 *>(mod3_shared);            // [GT][81][32]
    uint2 *rsgn = gtab + GT * MOD3_DIGITS * 32;              // [n][3][32]
    uint2 *rmag = rsgn + (size_t)n * 96;                             // [n][3][32]
    uint4 *lists = reinterpret_cast<uint4 *>(rmag + (size_t)n * 96); // [warps][32]
    uint2 *lists2 = reinterpret_cast<uint2 *>(lists + MOD3_THREADS);
    __shared__ uint16_t dmap[256];      // (magnitudes | signs << 4) -> byte offset in a group
    __shared__ uint64_t cm_s[64], cs_s[64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = THREADS / 32;
    for (int j = threadIdx.x; j < n; j += THREADS) {
        cm_s[j] = a.mags[j];
        cs_s[j] = a.sgns[j];
    }
    if (GT > 0 && threadIdx.x < 256) {
        int idx = 0, p3 = 1;
        for (int t = 0; t < 4; t++, p3 *= 3)
            if ((threadIdx.x >> t) & 1) idx += p3 * (1 + ((threadIdx.x >> (t + 4)) & 1));
        dmap[threadIdx.x] = (uint16_t)(idx * 256);
    }
    __syncthreads();
    const int low = n - 1 < MOD3_LOW ? n - 1 : MOD3_LOW;
    for (int r = warp; r < n; r += warps) {
        uint32_t m = 0, s = 0;
        for (int j = 0; j < low && j < 10; j++) {
            if (!((cm_s[j] >> r) & 1)) continue;
            const uint32_t minus = j < 5 ? mod3_pattern(j) : 0u - ((lane >> (j - 5)) & 1u);
            f3_add(m, s, 0xffffffffu, ((cs_s[j] >> r) & 1) ? ~minus : minus);
        }
        // word 0: column 10 plus, word 1: minus
        const uint32_t cm = low > 10 && ((cm_s[10] >> r) & 1) ? 0xffffffffu : 0u;
        const uint32_t cs = cm && ((cs_s[10] >> r) & 1) ? 0xffffffffu : 0u;
        uint32_t m1 = m, s1 = s;
        f3_add(m, s, cm, cs);
        f3_sub(m1, s1, cm, cs);
        for (int d = 0; d < 3; d++) {
            uint32_t a0 = m, b0 = s, a1 = m1, b1 = s1;
            if (d) {
                f3_add(a0, b0, 0xffffffffu, d == 2 ? 0xffffffffu : 0u);
                f3_add(a1, b1, 0xffffffffu, d == 2 ? 0xffffffffu : 0u);
            }
            rmag[(r * 3 + d) * 32 + lane] = make_uint2(a0, a1);
            rsgn[(r * 3 + d) * 32 + lane] = make_uint2(b0, b1);
        }
    }
    __syncthreads();
    for (int e = warp; e < GT * MOD3_DIGITS; e += warps) {
        const int g = e / MOD3_DIGITS;
        int d = e - g * MOD3_DIGITS;
        uint2 w = make_uint2(0xffffffffu, 0xffffffffu);
        for (int t = 0; t < 4; t++, d /= 3) {
            const int r = 4 * g + t;
            if (r >= n) continue;
            const uint2 x = rmag[(r * 3 + d % 3) * 32 + lane];
            w.x &= x.x;
            w.y &= x.y;
        }
        gtab[e * 32 + lane] = w;
    }
    __syncthreads();

    // low states that exist (n - 1 < 11: fewer words, lanes or word bits) and
    // those with an odd number of minus signs in word 0
    const uint32_t exist = low < 5 ? (lane == 0 ? (1u << (1 << low)) - 1u : 0u)
                           : low < 10 ? (lane < (1 << (low - 5)) ? 0xffffffffu : 0u) : 0xffffffffu;
    const uint32_t exist1 = low > 10 ? 0xffffffffu : 0u;
    const uint32_t odd = 0x96696996u ^ (0u - (__popc(lane) & 1u));

    // one contiguous, balanced range of batches per warp
    const uint64_t TW = (uint64_t)gridDim.x * warps;
    const uint64_t wid = (uint64_t)blockIdx.x * warps + warp;
    const uint64_t b_begin = wid * a.batches / TW, b_end = (wid + 1) * a.batches / TW;
    const char *tab = reinterpret_cast<const char *>(gtab + lane);
    constexpr int GB = MOD3_DIGITS * 256;
    uint4 *list = lists + warp * 32;
    uint2 *list2 = lists2 + warp * 32;
    unsigned long long count = 0;   // sum of 1 (term +1) or 2 (term -1)
    bool aborted = false;
    // high signs of lane l in batch b: l | gray(b) << 5, bit t the sign of
    // column 11 + t; the last column's sign is +
    W m = 0, s = 0;
    if (b_begin < b_end) {
        m = (W)cm_s[n - 1];
        s = (W)cs_s[n - 1];
        // (without tables a batch is the one high state with the signs b)
        const uint64_t minus = GT == 0 ? b_begin : (uint64_t)lane | ((b_begin ^ (b_begin >> 1)) << 5);
        for (int j = MOD3_LOW; j < n - 1; j++) {
            if ((minus >> (j - MOD3_LOW)) & 1) f3_sub(m, s, (W)cm_s[j], (W)cs_s[j]);
            else f3_add(m, s, (W)cm_s[j], (W)cs_s[j]);
        }
    }

    // The states `alive` of high state k after the tables' rows: the other
    // rows, then the signs.  Everything but the words is warp-uniform.
    auto finish = [&](int k, uint2 alive, uint32_t flip) {
        const W km = __shfl_sync(0xffffffffu, m, k), ks = __shfl_sync(0xffffffffu, s, k);
        const auto digit = [&](int r) { return ((km >> r) & 1) ? 1 + (int)((ks >> r) & 1) : 0; };
        for (int r = 4 * GT; r < n; r += 2) {
            const int q = r + 1 < n ? r + 1 : r;
            const uint2 x = rmag[(r * 3 + digit(r)) * 32 + lane], y = rmag[(q * 3 + digit(q)) * 32 + lane];
            alive.x &= x.x & y.x;
            alive.y &= x.y & y.y;
            if (!__any_sync(0xffffffffu, (alive.x | alive.y) != 0)) return;
        }
        uint2 neg;
        neg.x = odd ^ flip ^ (0u - (__popc(k) & 1u));
        neg.y = ~neg.x;
        for (int r = 0; r < n; r++) {
            const uint2 x = rsgn[(r * 3 + digit(r)) * 32 + lane];
            neg.x ^= x.x;
            neg.y ^= x.y;
        }
        count += (unsigned long long)(__popc(alive.x) + __popc(alive.x & neg.x) + __popc(alive.y) +
                                      __popc(alive.y & neg.y));
    };

    if constexpr (GT == 0) {
        if (b_begin < b_end)
            finish(0, make_uint2(exist, exist1), 0u - (uint32_t)(__popcll(b_begin) & 1));
    } else
    for (uint64_t b = b_begin; b < b_end; b++) {
        if (b != b_begin) {
            // the host-mapped abort word is read once per 2^12 batches, from
            // the warp's second period on
            if (((b - b_begin) & 4095) == 0 && __any_sync(0xffffffffu, *a.abort_flag != 0)) {
                aborted = true;
                break;
            }
            // column j turns minus: -2 a = a is added, else 2 a = -a
            const int z = __ffsll((long long)b) - 1, j = MOD3_LOW + 5 + z;
            if (((b >> (z + 1)) & 1) == 0) f3_add(m, s, (W)cm_s[j], (W)cs_s[j]);
            else f3_sub(m, s, (W)cm_s[j], (W)cs_s[j]);
        }
        uint32_t off[GT];
#pragma unroll
        for (int g = 0; g < GT; g++)
            off[g] = dmap[(uint32_t)((m >> (4 * g)) & 15) | (uint32_t)((s >> (4 * g)) & 15) << 4];
        list[lane] = make_uint4(off[0], off[1] + GB, off[2] + 2 * GB, off[3] + 3 * GB);
        list2[lane] = make_uint2(off[4] + 4 * GB, GT > 5 ? off[GT - 1] + (GT - 1) * GB : 0);
        __syncwarp();
        const uint32_t flip = 0u - (uint32_t)(b & 1);     // parity of gray(b)
        for (int k0 = 0; k0 < 32; k0 += 4) {
            uint2 alive[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint4 o = list[k0 + t];
                const auto at = [&](uint32_t off) { return *reinterpret_cast<const uint2 *>(tab + off); };
                const uint2 z0 = at(o.x), z1 = at(o.y), z2 = at(o.z), z3 = at(o.w);
                const uint2 p = list2[k0 + t], z4 = at(p.x);
                alive[t].x = z0.x & z1.x & z2.x & z3.x & z4.x & exist;
                alive[t].y = z0.y & z1.y & z2.y & z3.y & z4.y & exist1;
                if constexpr (GT > 5) {
                    const uint2 z5 = at(p.y);
                    alive[t].x &= z5.x;
                    alive[t].y &= z5.y;
                }
            }
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (__any_sync(0xffffffffu, (alive[t].x | alive[t].y) != 0))
                    finish(k0 + t, alive[t], flip);
        }
        __syncwarp();
    }
    count %= 3;
    __shared__ unsigned long long red[THREADS / 32];
    __shared__ int any_abort;
    if (threadIdx.x == 0) any_abort = 0;
    __syncthreads();
    if (aborted) any_abort = 1;
    for (int o = 16; o > 0; o >>= 1) count += __shfl_down_sync(0xffffffffu, count, o);
    if (lane == 0) red[warp] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < warps; w++) t += red[w];
        a.part[blockIdx.x] = any_abort ? MOD3_ABORTED : t;
    }
}

template <typename W, int GT>
static cudaError_t launch_mod3(const Mod3Args &a, int blocks, cudaStream_t s) {
    const size_t smem = GT ? mod3_smem(a.n) : 2 * mod3_row_bytes(a.n);
    cudaError_t e = cudaFuncSetAttribute(mod3_kernel<W, GT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    mod3_kernel<W, GT><<<(unsigned)blocks, mod3_threads(GT), smem, s>>>(a);
    return cudaGetLastError();
}

// perm(A) mod 3 from the F_3 column encodings (n >= 3).  One launch and no
// copies: the columns are kernel arguments, the blocks' counts go to pinned
// host memory.
static int mod3_impl(const uint64_t *mags, const uint64_t *sgns, int n, int *out) {
    DeviceInfo dev;
    int st = device_info(&dev);
    if (st != PG_OK) return st;
    volatile int *abort_dev;
    st = abort_flag_device(&abort_dev);
    if (st != PG_OK) return st;
    const int high = n - 1 - MOD3_LOW;          // columns common to a warp
    const bool tables = high > MOD3_SHORT;
    Mod3Args a;
    std::memcpy(a.mags, mags, (size_t)n * 8);
    std::memcpy(a.sgns, sgns, (size_t)n * 8);
    a.n = n;
    // (without tables a batch is one high state)
    a.batches = high <= 0 ? 1 : tables ? 1ull << (high - 5) : 1ull << high;
    const uint64_t warps = mod3_threads(tables) / 32;
    const uint64_t most = tables ? (uint64_t)dev.sm_count : a.batches;
    const int blocks = (int)std::min((a.batches + (tables ? 1 : warps) - 1) / (tables ? 1 : warps), most);
    Workspace *ws;
    st = workspace(&ws, 0, (size_t)blocks * 8);
    if (st != PG_OK) return st;
    void *part;
    PG_CUDA(cudaHostGetDevicePointer(&part, ws->host, 0));
    a.part = (volatile unsigned long long *)part;
    a.abort_flag = abort_dev;
    const bool six = mod3_tables(n) == 6;
    if (!tables) PG_CUDA((launch_mod3<uint32_t, 0>(a, blocks, ws->stream)));
    else if (n <= 32) PG_CUDA((launch_mod3<uint32_t, 6>(a, blocks, ws->stream)));
    else if (six) PG_CUDA((launch_mod3<uint64_t, 6>(a, blocks, ws->stream)));
    else PG_CUDA((launch_mod3<uint64_t, 5>(a, blocks, ws->stream)));
    PG_CUDA(cudaStreamSynchronize(ws->stream));
    unsigned long long total = 0;
    for (int i = 0; i < blocks; i++) {
        const unsigned long long v = ((const unsigned long long *)ws->host)[i];
        if (v == MOD3_ABORTED) return fail(PG_EABORT, "launch aborted by pg_abort()");
        total += v;
    }
    // 2^(1-n) = (-1)^(n-1) modulo 3
    *out = (int)((n & 1) ? total % 3 : (3 - total % 3) % 3);
    return PG_OK;
}

}  // namespace pg

extern "C" int pg_permanent_mod3_cols(const uint64_t *col_mags, const uint64_t *col_sgns,
                                      int n, int *out) {
    using namespace pg;
    if (!out) return fail(PG_EINVAL, "null argument");
    if (n < 0 || n >= 64) return fail(PG_ERANGE, "n must satisfy 0 <= n < 64");
    if (n == 0) { *out = 1; return PG_OK; }
    if (!col_mags || !col_sgns) return fail(PG_EINVAL, "column encodings must not be NULL");
    const uint64_t mask = (1ull << n) - 1;
    for (int j = 0; j < n; j++)
        if ((col_mags[j] & ~mask) || (col_sgns[j] & ~col_mags[j]))
            return fail(PG_EINVAL, "column encodings out of range (sign bit without magnitude "
                                   "or row >= n)");
    if (n <= 2) {
        // per = a00 (n = 1) or a00 a11 + a01 a10 (n = 2), elements of F_3
        auto el = [&](int i, int j) -> int {
            if (!((col_mags[j] >> i) & 1)) return 0;
            return ((col_sgns[j] >> i) & 1) ? 2 : 1;
        };
        *out = n == 1 ? el(0, 0) : (el(0, 0) * el(1, 1) + el(0, 1) * el(1, 0)) % 3;
        return PG_OK;
    }
    return mod3_impl(col_mags, col_sgns, n, out);
}

extern "C" int pg_permanent_mod3(const int64_t *A, int n, int *out) {
    using namespace pg;
    if (!out) return fail(PG_EINVAL, "null argument");
    if (n < 0 || n >= 64) return fail(PG_ERANGE, "n must satisfy 0 <= n < 64");
    if (n == 0) { *out = 1; return PG_OK; }
    if (!A) return fail(PG_EINVAL, "matrix must not be NULL");
    uint64_t mags[64] = {0}, sgns[64] = {0};
    for (int j = 0; j < n; j++)
        for (int i = 0; i < n; i++) {
            const int64_t r = A[(size_t)i * n + j] % 3;
            const int v = (int)(r < 0 ? r + 3 : r);
            if (v) mags[j] |= 1ull << i;
            if (v == 2) sgns[j] |= 1ull << i;
        }
    return pg_permanent_mod3_cols(mags, sgns, n, out);
}
