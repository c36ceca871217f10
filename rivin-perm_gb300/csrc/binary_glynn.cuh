// Exact Glynn kernel for 0/1 matrices: zero-row lookup over 1024 states and
// warp-compacted exact evaluation of the states that survive it.
//
// For a 0/1 matrix the Glynn row sum of state d is s_r = deg_r - 2 m_r,
// where m_r counts the row's ones in columns whose sign is minus.  A term
// is zero as soon as one row sum is zero, which needs an even degree and
// m_r = deg_r / 2; for the benchmark matrices that is most states
// (40 x 40 Bernoulli(1/2): ~92 %; the 4x4x5 grid: ~99.9 %).  The reference
// keeps int16 row sums, a zero counter and a ratio-updated product mod p
// for every state (perm_binary_omp.c:236-347, perm_binary_cuda.cu:111-205);
// this kernel only searches for the states without a zero row.
//
// Search.  A chunk is the 1024 states of one setting of the high columns'
// signs: bit k of lane l's word is the state whose low ten signs are
// k | l << 5 (aligned 2^10-state Gray windows, in another order).  The high
// columns are common to the warp, so an even-degree row is zero exactly
// where the low columns hold x = deg_r / 2 - (ones in high minus columns)
// more, a word that depends only on the lane and on x in 0..dlow_r (any
// other x: never zero).  Rows are packed into groups whose table of AND-ed
// "no zero" words, one per combination of the rows' x, fits in shared
// memory ([entry][32 lanes]: no bank conflicts); a chunk costs one load and
// one AND per group, with a vote after every four groups.  The 32 lanes
// prepare the table entries of 32 consecutive chunks (popcounts of the high
// signs) and publish them through shared memory.
//
// Evaluation.  Surviving states are appended to a per-warp queue; whenever
// 32 are queued every lane evaluates one exactly.  The row sums come as
// bytes: base bytes of the chunk minus low-column bytes of the state (two
// shared tables, four rows per 32-bit subtraction) and one byte permute per
// row, then the exact multi-word term of exact_glynn.cuh (row groups, signed
// running product, 64-bit column accumulators).  Counting the signs by
// popcount took 40 issues of the quarter-rate pipe per 32 states, two thirds
// of the evaluation.
//
// Rows are padded to NPAD (pad rows: degree 1, no toggled column, s = 1) so
// that one instantiation serves a range of orders; the walk itself runs the
// true order's 2^(n-1) states.  Accumulation, the block reduction and the
// per-block result slots are those of the exact kernel.
//
// Issue bound (82 % of the issue slots; 6 % quarter-rate pipe).  Whole calls
// against the bit-sliced tracker that updated one state per lane and step
// and evaluated by popcount: 4x4x5 grid (40 x 40, 0.08 % survive) 446 -> 59
// ms, 36 x 36 Bernoulli(1/2) (6-13 % survive) 68 -> 32 ms.
#pragma once

#include "exact_glynn.cuh"

namespace pg {

constexpr int BIN_LOW = 10;        // columns spread over word bits (5) and lanes (5)
constexpr int BIN_QCAP = 320;      // queue entries per warp (31 pending + 32 lanes x 8 bits)
constexpr size_t BIN_SMEM = 222 * 1024;   // dynamic shared memory of a block, at most

// One even-degree row, in table-group order.
struct BinTrack {
    uint64_t high;      // the row's ones in toggled columns 10, 11, ... (bit 0: column 10)
    uint16_t low;       // the row's ones in columns 0..9
    uint8_t half;       // deg / 2
    uint8_t cap;        // ones in columns 0..9, plus 1: the entry of "never zero"
    uint16_t stride;    // entries per unit of this row's x in its group's table
    uint16_t base;      // the group's first entry on its first row, else 0xffff
};

struct BinaryArgs {
    const uint64_t *rmask;     // [NPAD] toggled-column bits of each row (group order)
    const int32_t *deg;        // [NPAD] row degrees (pad rows 1)
    const BinTrack *trk;       // [ntracked]
    int ntracked;              // even-degree rows, 1..48
    int entries;               // table entries (entry 0: no row is zero)
    int list_words;            // words of a chunk's list: the byte offset of each group's
                               // entry, padded with entry 0 to a multiple of four
    int sparse;                // few states survive
    int warps;                 // warps of a block
    unsigned long long *acc;   // [NL] per-word sums (exact kernel layout)
    int *status;
    unsigned long long *part;  // [NL][gridDim] per-block slots (exact_epilogue), or nullptr
    unsigned long long *next;  // work units taken beyond each warp's first: zero at launch,
                               // re-zeroed by the finishing kernel
    volatile const int *abort_flag;
    uint64_t state_lo, state_hi;   // Gray states to walk
    int log_steps;             // chunks of a batch (<= 5)
    int log_unit;              // batches of a work unit
};

#ifndef BIN_T32
#define BIN_T32 768
#endif
#ifndef BIN_T40
#define BIN_T40 768
#endif
#ifndef BIN_T48
#define BIN_T48 512
#endif
// threads of a block, at most: as many warps as the registers allow
// (fewer when the tables leave no room for their lists)
__host__ __device__ constexpr int binary_max_threads(int NPAD) {
    return NPAD > 40 ? BIN_T48 : NPAD > 32 ? BIN_T40 : BIN_T32;
}
// words of a state's row bytes, padded for 16-byte loads
__host__ __device__ constexpr int binary_row_words(int NPAD) { return (NPAD / 4 + 3) & ~3; }
__host__ __device__ constexpr size_t binary_warp_bytes(int NPAD, int list_words) {
    return (size_t)32 * binary_row_words(NPAD) * 4 + (size_t)32 * list_words * 4 + BIN_QCAP * 2;
}
__host__ __device__ constexpr size_t binary_smem(int NPAD, int entries, int list_words, int warps) {
    return (size_t)entries * 128 + (size_t)1024 * binary_row_words(NPAD) * 4 +
           warps * binary_warp_bytes(NPAD, list_words);
}

// byte K of x, sign-extended
template <int K>
__device__ __forceinline__ int32_t binary_byte(uint32_t x) {
    int32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "n"(0x8880 + 0x1111 * K));
    return r;
}

template <int NPAD, int G>
__global__ void __launch_bounds__(binary_max_threads(NPAD), 1) binary_glynn_kernel(BinaryArgs a) {
    using S = ExactShape<NPAD, G>;
    constexpr int NL = S::NL, NR = S::NR;
    constexpr int FOLD = 1 << EXACT_LOGU;   // terms the 64-bit columns hold between folds
    constexpr int NW = NPAD / 4, LS = binary_row_words(NPAD);
    extern __shared__ uint4 bin_shared[];
    uint32_t *ztab = reinterpret_cast<uint32_t *>(bin_shared);     // [entries][32]
    uint32_t *ltab = ztab + (size_t)a.entries * 32;                 // [1024][LS]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    char *mine = reinterpret_cast<char *>(ltab + 1024 * LS) + warp * binary_warp_bytes(NPAD, a.list_words);
    uint32_t *base = reinterpret_cast<uint32_t *>(mine);            // [32][LS]
    uint32_t *list = base + 32 * LS;                                // [32][list_words]
    uint16_t *q = reinterpret_cast<uint16_t *>(list + 32 * a.list_words);
    __shared__ BinTrack s_trk[48];
    __shared__ uint64_t s_rm[NPAD];
    __shared__ int32_t s_deg[NPAD];
    __shared__ uint32_t s_eq[32][6];    // [mask][v]: the k in 0..31 with popc(k & mask) == v
    exact_allow_dependents();
    for (int i = threadIdx.x; i < NPAD; i += blockDim.x) {
        s_rm[i] = a.rmask[i];
        s_deg[i] = a.deg[i];
    }
    for (int i = threadIdx.x; i < a.ntracked; i += blockDim.x) s_trk[i] = a.trk[i];
    for (int i = threadIdx.x; i < 32 * 6; i += blockDim.x) {
        uint32_t w = 0;
        for (int k = 0; k < 32; k++) w |= (uint32_t)(__popc(k & (i / 6)) == i % 6) << k;
        s_eq[i / 6][i % 6] = w;
    }
    __syncthreads();
    if (warp == 0) ztab[lane] = 0xffffffffu;
    for (int e0 = 0; e0 < a.ntracked;) {            // table groups
        int e1 = e0 + 1, size = s_trk[e0].cap + 1;
        for (; e1 < a.ntracked && s_trk[e1].base == 0xffff; e1++) size *= s_trk[e1].cap + 1;
        for (int idx = warp; idx < size; idx += warps) {
            uint32_t w = 0xffffffffu;
            for (int e = e0, rem = idx; e < e1; e++) {
                const int cap = s_trk[e].cap, low = s_trk[e].low;
                const int x = rem % (cap + 1), v = x - __popc((low >> 5) & lane);
                rem /= cap + 1;
                if (x < cap && v >= 0 && v <= 5) w &= ~s_eq[low & 31][v];
            }
            ztab[(s_trk[e0].base + idx) * 32 + lane] = w;
        }
        e0 = e1;
    }
    for (int i = threadIdx.x; i < 1024 * NW; i += blockDim.x) {
        const int w = i & 1023, r = (i >> 10) * 4;
        uint32_t b = 0;
#pragma unroll
        for (int t = 0; t < 4; t++)
            b |= (uint32_t)(2 * __popc((uint32_t)s_rm[r + t] & (uint32_t)w)) << (8 * t);
        ltab[w * LS + (i >> 10)] = b;
    }
    __syncthreads();

    uint32_t acc[NL];
#pragma unroll
    for (int l = 0; l < NL; l++) acc[l] = 0;
    uint64_t col[NR > 1 ? NR - 1 : 1];
    int64_t colt = 0;
    int terms = 0;       // terms in the columns since the last fold (warp-uniform)
    int qn = 0;          // queued states (warp-uniform)
    uint32_t c_odd = 0;  // parity of the batch's first chunk

    // evaluates the last `count` (<= 32) queued states
    auto evaluate = [&](int count) {
        __syncwarp();
        qn -= count;
        const bool live = lane < count;
        const uint32_t e = live ? q[qn + lane] : 0, w = e & 1023u, k = e >> 10;
        uint32_t d[LS];
#pragma unroll
        for (int v = 0; v < LS / 4; v++) {
            const uint4 x = reinterpret_cast<const uint4 *>(base + k * LS)[v];
            const uint4 y = reinterpret_cast<const uint4 *>(ltab + w * LS)[v];
            // bytes 128 + s_r, no borrow between them; then two's complement
            d[4 * v + 0] = (x.x - y.x) ^ 0x80808080u;
            d[4 * v + 1] = (x.y - y.y) ^ 0x80808080u;
            d[4 * v + 2] = (x.z - y.z) ^ 0x80808080u;
            d[4 * v + 3] = (x.w - y.w) ^ 0x80808080u;
        }
        int32_t s[NPAD];
#pragma unroll
        for (int v = 0; v < NW; v++) {
            s[4 * v + 0] = binary_byte<0>(d[v]);
            s[4 * v + 1] = binary_byte<1>(d[v]);
            s[4 * v + 2] = binary_byte<2>(d[v]);
            s[4 * v + 3] = binary_byte<3>(d[v]);
        }
        if (!live) s[0] = 0;
        exact_term_col<NPAD, G, 0>(s, col, colt, (__popc(w) ^ k ^ c_odd) & 1u, terms == 0);
        if (++terms == FOLD) {
            FoldCols<NR, NL>::apply(acc, col, colt);
            terms = 0;
        }
        __syncwarp();
    };

    // appends the states `part` of chunk k at queue positions given by a scan
    // over the lanes (inc: inclusive count), then evaluates full rounds
    auto push = [&](uint32_t part, int k, int inc, int total) {
        int pos = qn + inc - __popc(part);
        while (part) {
            const uint32_t rest = part & (part - 1);
            q[pos++] = (uint16_t)((k << 10) | (lane << 5) | __popc((part ^ rest) - 1));
            part = rest;
        }
        qn += total;
        while (qn >= 32) evaluate(32);
    };
    auto scan = [&](uint32_t part) {
        int inc = __popc(part);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        return inc;
    };
    auto append = [&](uint32_t alive, int k) {
        if (a.sparse) {                              // one state of each lane at a time
            for (uint32_t mask = __ballot_sync(0xffffffffu, alive != 0); mask;
                 mask = __ballot_sync(0xffffffffu, alive != 0)) {
                if (alive) {
                    const uint32_t rest = alive & (alive - 1);
                    q[qn + __popc(mask & ((1u << lane) - 1u))] =
                        (uint16_t)((k << 10) | (lane << 5) | __popc((alive ^ rest) - 1));
                    alive = rest;
                }
                qn += __popc(mask);
                if (qn >= 32) evaluate(32);
            }
            return;
        }
        const int inc = scan(alive), total = __shfl_sync(0xffffffffu, inc, 31);
        if (qn + total <= BIN_QCAP) {
            push(alive, k, inc, total);
        } else {                                     // at most 256 states at a time
            for (int o = 0; o < 32; o += 8) {
                const uint32_t part = alive & (0xffu << o);
                const int pi = scan(part);
                push(part, k, pi, __shfl_sync(0xffffffffu, pi, 31));
            }
        }
    };

    // Work units go to warps from a counter (the share of surviving states
    // varies strongly along the walk with the signs of the columns), one
    // ahead, so that the atomic's round trip overlaps the work.
    const uint64_t chunk0 = a.state_lo >> BIN_LOW;
    const uint64_t chunks = ((a.state_hi + (1u << BIN_LOW) - 1) >> BIN_LOW) - chunk0;
    const uint64_t units = (chunks + (1ull << (a.log_steps + a.log_unit)) - 1) >> (a.log_steps + a.log_unit);
    const char *zl = reinterpret_cast<const char *>(ztab + lane);
    bool aborted = false;
    uint32_t polls = 0;
    for (uint64_t unit = (uint64_t)warp * gridDim.x + blockIdx.x; unit < units && !aborted;) {
        unsigned long long nx = 0;
        if (lane == 0) nx = (uint64_t)gridDim.x * warps + atomicAdd(a.next, 1ull);
        for (uint32_t bb = 0; bb < (1u << a.log_unit); bb++) {
            const uint64_t ci = ((unit << a.log_unit) + bb) << a.log_steps;
            if (ci >= chunks) break;
            // the host-mapped abort word is read once per 128 batches, from
            // the warp's second period on
            if ((++polls & 127) == 0 && __any_sync(0xffffffffu, *a.abort_flag != 0)) {
                aborted = true;
                break;
            }
            const int steps = chunks - ci < (1ull << a.log_steps) ? (int)(chunks - ci) : 1 << a.log_steps;
            const uint64_t c0 = chunk0 + ci;
            c_odd = (uint32_t)c0;
            // this lane's chunk: row bytes and table entries of its high signs
            const uint64_t hw = (c0 + lane) ^ ((c0 + lane) >> 1);
            auto ones = [&](uint64_t m) {
                return NPAD > 40 ? __popcll(m & hw) : __popc((uint32_t)m & (uint32_t)hw);
            };
            if (lane < steps) {
#pragma unroll
                for (int v = 0; v < NW; v++) {
                    uint32_t b = 0;
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        b |= (uint32_t)(128 + s_deg[4 * v + t] - 2 * ones(s_rm[4 * v + t] >> BIN_LOW))
                             << (8 * t);
                    base[lane * LS + v] = b;
                }
            }
            {
                uint32_t *ll = list + lane * a.list_words;
                int g = -1;
                uint32_t off = 0;
                for (int e = 0; e < a.ntracked; e++) {
                    const BinTrack t = s_trk[e];
                    if (t.base != 0xffff) {
                        if (g >= 0) ll[g] = off * 128;
                        g++;
                        off = t.base;
                    }
                    off += min((uint32_t)(t.half - ones(t.high)), (uint32_t)t.cap) * t.stride;
                }
                for (; g < a.list_words; off = 0, g++) ll[g] = off * 128;
            }
            __syncwarp();
            for (int k0 = 0; k0 < steps; k0 += 2) {
                uint32_t alive[2] = {0xffffffffu, k0 + 1 < steps ? 0xffffffffu : 0u};
                for (int v = 0; v < a.list_words; v += 4) {
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        const uint4 o = *reinterpret_cast<const uint4 *>(list + (k0 + t) * a.list_words + v);
                        const auto at = [&](uint32_t off) {
                            return *reinterpret_cast<const uint32_t *>(zl + off);
                        };
                        alive[t] &= at(o.x) & at(o.y) & at(o.z) & at(o.w);
                    }
                    if ((v & 4) && !__any_sync(0xffffffffu, (alive[0] | alive[1]) != 0)) break;
                }
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const uint64_t c = c0 + k0 + t;
                    if ((c << BIN_LOW) < a.state_lo || ((c + 1) << BIN_LOW) > a.state_hi) {
                        // a window that starts or ends inside this chunk
                        uint32_t in = 0;
                        for (int k = 0; k < 32; k++) {
                            uint32_t i = (uint32_t)(k | (lane << 5)) ^ (uint32_t)((c & 1) << (BIN_LOW - 1));
                            i ^= i >> 1;
                            i ^= i >> 2;
                            i ^= i >> 4;
                            i ^= i >> 8;
                            const uint64_t g = (c << BIN_LOW) | i;
                            in |= (uint32_t)(g >= a.state_lo && g < a.state_hi) << k;
                        }
                        alive[t] &= in;
                    }
                    if (__any_sync(0xffffffffu, alive[t] != 0)) append(alive[t], k0 + t);
                }
            }
            if (qn > 0) evaluate(qn);       // the next batch has other base bytes
            __syncwarp();
        }
        unit = __shfl_sync(0xffffffffu, nx, 0);
    }
    if (terms > 0) FoldCols<NR, NL>::apply(acc, col, colt);

    // block reduction and result words: as the exact kernel
    __shared__ long long red[binary_max_threads(NPAD) / 32][NL];
    __shared__ int any_abort;
    if (threadIdx.x == 0) any_abort = 0;
    __syncthreads();
    if (aborted) any_abort = 1;
#pragma unroll
    for (int l = 0; l < NL; l++) {
        long long v = (l == NL - 1) ? (long long)(int32_t)acc[l] : (long long)acc[l];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) red[warp][l] = v;
    }
    __syncthreads();
    exact_epilogue<NL>(red, any_abort, a.acc, a.part, a.status);
}

template <int NPAD, int G>
cudaError_t launch_binary_glynn(const BinaryArgs &args, int blocks, cudaStream_t stream) {
    const size_t smem = binary_smem(NPAD, args.entries, args.list_words, args.warps);
    cudaError_t e = cudaFuncSetAttribute(binary_glynn_kernel<NPAD, G>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    binary_glynn_kernel<NPAD, G><<<blocks, 32 * args.warps, smem, stream>>>(args);
    return cudaGetLastError();
}

// Compiled shapes (binary_inst_*.cu): NPAD in {32, 40, 48}, G in {5, 6, 7,
// 8, 10}.  Orders below BINARY_MIN_N, and matrices whose sampled share of
// states without a zero row exceeds BINARY_MAX_SURVIVORS, use the exact
// kernel.  EXACT_BINARY=0 sends every 0/1 matrix to the exact kernel (for
// comparisons).
constexpr int BINARY_MIN_N = 24;
constexpr double BINARY_MAX_SURVIVORS = 0.25;
#ifndef EXACT_BINARY
#define EXACT_BINARY 1
#endif
int binary_npad(int n);
bool binary_compiled(int NPAD, int G);
cudaError_t launch_binary_any(int NPAD, int G, const BinaryArgs &args, int blocks,
                              cudaStream_t stream);

// Packs even-degree rows with caps[e] + 1 table entries each into few enough
// table groups (a multiple of four where that takes no more lookups) for the
// tables to fit beside the NPAD kernel's other shared memory, with the most
// warps that allow it; group[e] = the row's group.  Returns the number of
// groups, 0 if there is no such packing.
int binary_pack_groups(int NPAD, const int *caps, int rows, int *group, int *warps);

}  // namespace pg
