// Host side of the 64-bit exact engine (wide_exact.cuh): bound check, tables,
// launch shape and the multi-word result.
#include "pg_internal.h"
#include "wide_exact.cuh"

#include <cmath>
#include <cstring>
#include <vector>

namespace pg {

// out[word] = the word's sum over the blocks; the last block moves the status
__global__ void __launch_bounds__(256) wide_exact_finish(const unsigned long long *part, int blocks,
                                                         const int *status,
                                                         unsigned long long *out) {
    unsigned long long t = 0;
    for (int b = threadIdx.x; b < blocks; b += 256) t += part[(size_t)blockIdx.x * blocks + b];
    __shared__ unsigned long long red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        t = 0;
        for (int w = 0; w < 8; w++) t += red[w];
        out[blockIdx.x] = t;
        if (blockIdx.x == gridDim.x - 1) out[gridDim.x] = (unsigned long long)(unsigned)*status;
    }
}

static size_t wx_align(size_t v) { return (v + 255) / 256 * 256; }

// S += f 2^(32 pos) v for a 64-bit word v, f = +-1 (two's complement)
static void wx_add_at(std::vector<uint32_t> &S, size_t pos, uint64_t v, bool negative) {
    uint64_t carry = negative ? 1 : 0;
    for (size_t i = pos, k = 0; i < S.size(); i++, k++) {
        uint32_t add = k == 0 ? (uint32_t)v : k == 1 ? (uint32_t)(v >> 32) : 0u;
        if (negative) add = ~add;
        const uint64_t t = (uint64_t)S[i] + add + carry;
        S[i] = (uint32_t)t;
        carry = t >> 32;
    }
}

// Smallest compiled class for row bounds below 2^bits, false beyond 48.
static bool wide_entry(int n, int bits, WideEntry *out) {
    return bits <= 36   ? wide_entry_36(n, out)
           : bits <= 40 ? wide_entry_40(n, out)
           : bits <= 44 ? wide_entry_44(n, out)
                        : bits <= 48 && wide_entry_48(n, out);
}

}  // namespace pg

extern "C" int pg_exact_wide(const int64_t *A, int n, uint32_t *out, int limbs) {
    using namespace pg;
    if (n < 2 || n > 32) return fail(PG_ERANGE, "the 64-bit exact engine takes 2 <= n <= 32");
    if (!A || !out || limbs < 1) return fail(PG_EINVAL, "null argument");
    int bits = 0;
    double need = 2.0;                     // bits of the result, sign and rounding margin
    for (int i = 0; i < n; i++) {
        unsigned __int128 s = 0;
        for (int j = 0; j < n; j++) {
            const int64_t v = A[(size_t)i * n + j];
            s += v < 0 ? (unsigned __int128)(-(__int128)v) : (unsigned __int128)v;
        }
        if (s >> 48) return fail(PG_EOVERFLOW, "row-sum bound exceeds 48 bits");
        const uint64_t b = (uint64_t)s;
        while (bits < 64 && (b >> bits)) bits++;
        need += std::log2(b < 1 ? 1.0 : (double)b);
    }
    if (32.0 * limbs < need) return fail(PG_ERANGE, "output limb count too small for the permanent bound");
    WideEntry e;
    if (!wide_entry(n, bits, &e)) return fail(PG_EOVERFLOW, "no compiled shape");
    DeviceInfo dev;
    int st = device_info(&dev);
    if (st != PG_OK) return st;
    volatile int *abort_dev;
    st = abort_flag_device(&abort_dev);
    if (st != PG_OK) return st;
    // at least eight waves of two blocks per SM, so that the last one costs
    // little, while a thread keeps four states
    const uint64_t resident = 2 * (uint64_t)dev.sm_count;
    int R = n - 1;
    while (R > 2 && ((1ull << (n - 1 - R)) + WX_THREADS - 1) / WX_THREADS < 8 * resident) R--;
    if (R > n - 1) R = n - 1;
    const int blocks = (int)(((1ull << (n - 1 - R)) + WX_THREADS - 1) / WX_THREADS);
    const int N = e.N;
    const size_t off_init = wx_align((size_t)(n - 1) * 2 * N * 8);
    const size_t off_status = wx_align(off_init + (size_t)N * 8);
    const size_t off_out = off_status + 256;
    const size_t off_part = wx_align(off_out + (size_t)(e.words + 1) * 8);
    const size_t total = off_part + (size_t)blocks * e.words * 8;
    Workspace *ws;
    st = workspace(&ws, total, off_part);
    if (st != PG_OK) return st;
    char *h = (char *)ws->host, *d = (char *)ws->dev;
    std::memset(h, 0, off_part);
    int64_t *tab = (int64_t *)h, *init = (int64_t *)(h + off_init);
    for (int i = 0; i < n; i++) {
        int64_t sum = 0;
        for (int j = 0; j < n; j++) {
            const int64_t v = A[(size_t)i * n + j];
            sum += v;
            if (j < n - 1) {
                tab[(size_t)(2 * j) * N + i] = 2 * v;
                tab[(size_t)(2 * j + 1) * N + i] = -2 * v;
            }
        }
        init[i] = sum;
    }
    for (int i = n; i < N; i++) init[i] = 1;
    WideExactArgs a;
    a.tab = (const int64_t *)d;
    a.init = (const int64_t *)(d + off_init);
    a.n = n;
    a.log_range = R;
    a.resident = (int)resident;
    a.part = (unsigned long long *)(d + off_part);
    a.status = (int *)(d + off_status);
    a.abort_flag = abort_dev;
    cudaStream_t s = ws->stream;
    PG_CUDA(cudaMemcpyAsync(d, h, off_out, cudaMemcpyHostToDevice, s));
    PG_CUDA(e.launch(a, blocks, s));
    wide_exact_finish<<<e.words, 256, 0, s>>>(a.part, blocks, a.status,
                                              (unsigned long long *)(d + off_out));
    PG_CUDA(cudaGetLastError());
    PG_CUDA(cudaMemcpyAsync(h + off_out, d + off_out, (size_t)(e.words + 1) * 8,
                            cudaMemcpyDeviceToHost, s));
    PG_CUDA(cudaStreamSynchronize(s));
    const unsigned long long *w = (const unsigned long long *)(h + off_out);
    if (w[e.words]) return fail(PG_EABORT, "exact launch aborted by pg_abort()");
    // S = sum (X ^ m) Y - (2^(32 KX) - 1) sum_m Y
    const int K = e.kx + e.ky;
    std::vector<uint32_t> S((size_t)K + 5, 0);
    for (int l = 0; l <= K; l++) wx_add_at(S, l, w[l], false);
    for (int l = 0; l <= e.ky; l++) {
        wx_add_at(S, l, w[K + 1 + l], false);
        wx_add_at(S, (size_t)e.kx + l, w[K + 1 + l], true);
    }
    const int sh = n - 1;
    for (int b = 0; b < sh; b++)
        if ((S[b >> 5] >> (b & 31)) & 1) return fail(PG_EINTERNAL, "Glynn sum not divisible by 2^(n-1)");
    const uint32_t ext = (S.back() >> 31) ? 0xffffffffu : 0u;
    for (int i = 0; i < limbs; i++) {
        const size_t wi = (size_t)(32 * i + sh) >> 5;
        const int bo = (32 * i + sh) & 31;
        const uint32_t lo = wi < S.size() ? S[wi] : ext, hi = wi + 1 < S.size() ? S[wi + 1] : ext;
        out[i] = bo ? (lo >> bo) | (hi << (32 - bo)) : lo;
    }
    return PG_OK;
}
