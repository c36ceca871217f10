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
// signs: bit k of lane l's word is the state whose low signs are k | l << 5
// (an aligned Gray window, in another order).  The high columns are common to
// the warp, so an even-degree row is zero exactly where the low columns hold
// x = deg_r / 2 - (ones in high minus columns) more, words that depend only
// on the lane and on x in 0..dlow_r (any other x: never zero).  Rows are
// packed into groups whose table of AND-ed "no zero" words, one entry per
// combination of the rows' x, fits in shared memory ([entry][32 lanes]: no
// bank conflicts); a chunk costs one load and AND per group, with a vote
// after every eight groups.  The 32 lanes prepare the entries of the 32
// chunks of a batch, whose signs differ in five columns: row counts are
// bytes, the warp's count minus a 32-row table's, four rows per subtraction.
//
// Rows without ones in the low columns need no table.  Such a row is zero in
// all of a chunk or none of it, one without ones in the five chunk columns
// either in all of a batch or none.  Batch rows are tested first, for 32
// batches at once, one a lane; then the chunk rows, by bytes.  A whole walk
// orders its columns so that such rows exist (binary_order_columns).  4x4x5
// grid with a few bonds removed and columns shuffled: 34.9 ms without these
// tests, 25.7 with them (one batch at a time), 6.2 with ordered columns; 2.6-4.7
// by which bonds are removed with the batches of a unit tested together and taken from all over the
// walk (neighbours are zero together, and warps ran dry).
//
// Evaluation.  Surviving states are appended to a per-warp queue; whenever
// 32 are queued every lane evaluates one exactly.  The row sums come as
// bytes: base bytes of the chunk minus a table of the ten low
// columns, four rows per subtraction, and one byte permute per row; then the
// exact multi-word term of exact_glynn.cuh (row groups, signed running
// product, 64-bit column accumulators).  Counting the signs by popcount took
// 40 issues of the quarter-rate pipe per 32 states.
//
// Rows are padded to NPAD (pad rows: degree 1, no toggled column, s = 1) so
// that one instantiation serves a range of orders; the walk itself runs the
// true order's 2^(n-1) states.  Accumulation, the block reduction and the
// per-block result slots are those of the exact kernel.
//
// Issue bound (65-80 % of the issue slots).  Whole calls against a
// bit-sliced tracker that updated one state per lane and step and evaluated
// by popcount: 4x4x5 grid (40 x 40, 0.08 % survive) 441 -> 3.9 ms, 36 x 36
// Bernoulli(1/2) (6-13 % survive) 67-76 -> 18-29 ms by the matrix.
#pragma once

#include "exact_glynn.cuh"

namespace pg {

constexpr int BIN_LOW = 10;        // columns spread over word bits (5) and lanes (5)
constexpr int BIN_QCAP = 320;      // queue entries per warp (31 pending + 32 lanes x 8 bits)
constexpr size_t BIN_SMEM = 222 * 1024;   // dynamic shared memory of a block, at most

// One even-degree row, in table-group order.
struct BinTrack {
    uint64_t high;      // the row's ones in toggled columns BIN_LOW, ... (bit 0 the first)
    uint16_t low;       // the row's ones in the columns below
    uint8_t half;       // deg / 2
    uint8_t cap;        // ones in `low`, plus 1: the entry of "never zero"
    uint16_t stride;    // entries per unit of this row's x in its group's table
    uint16_t base;      // the group's first entry on its first row, else 0xffff
};

struct BinaryArgs {
    const uint64_t *rmask;     // [NPAD] toggled-column bits of each row (group order)
    const int32_t *deg;        // [NPAD] row degrees (pad rows 1)
    // Even-degree rows: batch rows (no ones below the columns common to a
    // batch of 32 chunks), then chunk rows (none in the low columns), then
    // table rows; the first two padded to a multiple of four
    const BinTrack *trk;       // [ntracked]
    int batch_rows, uniform_rows, ntracked;   // ends of the three, ntracked <= BIN_TRACK
    int entries;               // table entries (entry 0: no row is zero)
    int list_words;            // words of a chunk's list: the byte offset of each group's
                               // entry, padded with entry 0 to a multiple of four
    int warps;                 // warps of a block
    unsigned long long *acc;   // [NL] per-word sums (exact kernel layout)
    int *status;
    unsigned long long *part;  // [NL][gridDim] per-block slots (exact_epilogue), or nullptr
    unsigned long long *next;  // work units taken beyond each warp's first: zero at launch,
                               // re-zeroed by the finishing kernel
    volatile const int *abort_flag;
    uint64_t state_lo, state_hi;   // Gray states to walk
    int log_steps;             // chunks of a batch (<= 5)
    int log_batches;           // batches of the window, rounded up
    int log_unit;              // batches of a work unit (<= 5, <= log_batches)
};

// threads of a block, at most: as many warps as the registers allow
// (fewer when the tables leave no room for their lists)
__host__ __device__ constexpr int binary_max_threads(int NPAD) { return NPAD > 40 ? 512 : 768; }
// words of a state's row bytes, padded for 8-byte loads
__host__ __device__ constexpr int binary_row_words(int NPAD) { return (NPAD / 4 + 1) & ~1; }
constexpr int BIN_TRACK = 56;           // even-degree rows (at most 48) with their padding
constexpr int BIN_TRACK_WORDS = BIN_TRACK / 4;
__host__ __device__ constexpr size_t binary_warp_bytes(int NPAD, int list_words) {
    return (size_t)32 * binary_row_words(NPAD) * 4 + (size_t)32 * list_words * 4 + BIN_QCAP * 2 +
           BIN_TRACK_WORDS * 4 + 48;
}
__host__ __device__ constexpr size_t binary_smem(int NPAD, int entries, int list_words, int warps) {
    return (size_t)entries * 128 + (size_t)(1024 + 32) * binary_row_words(NPAD) * 4 +
           32 * BIN_TRACK_WORDS * 4 + warps * ((binary_warp_bytes(NPAD, list_words) + 15) & ~(size_t)15);
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
    constexpr int NW = NPAD / 4, LS = binary_row_words(NPAD), TW = BIN_TRACK_WORDS;
    constexpr int LOW = BIN_LOW, HI = LOW + 5;         // first column common to a batch of 32 chunks
    extern __shared__ uint4 bin_shared[];
    uint32_t *ztab = reinterpret_cast<uint32_t *>(bin_shared);      // [entries][32]
    uint32_t *ltab = ztab + (size_t)a.entries * 32;             // [1024][LS]
    uint32_t *ctab = ltab + 1024 * LS;                // [32][LS] bytes of the five chunk columns
    uint32_t *xtab = ctab + 32 * LS;                  // [32][TW] the same of the even rows
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    char *mine = reinterpret_cast<char *>(xtab + 32 * TW) +
                 warp * ((binary_warp_bytes(NPAD, a.list_words) + 15) & ~(size_t)15);
    uint32_t *list = reinterpret_cast<uint32_t *>(mine);            // [32][list_words]
    uint32_t *base = list + 32 * a.list_words;                      // [32][LS]
    uint32_t *ucnt = base + 32 * LS;                                    // row bytes, then even rows'
    uint32_t *xcnt = ucnt + 12;
    uint16_t *q = reinterpret_cast<uint16_t *>(xcnt + TW);
    __shared__ BinTrack s_trk[BIN_TRACK];
    __shared__ uint4 s_rec[BIN_TRACK];         // cap, stride bytes, group's first byte + 1 on its last row
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
    for (int e0 = a.uniform_rows; e0 < a.ntracked;) {            // table groups
        int e1 = e0 + 1, size = s_trk[e0].cap + 1;
        for (; e1 < a.ntracked && s_trk[e1].base == 0xffff; e1++) size *= s_trk[e1].cap + 1;
        if ((int)threadIdx.x >= e0 && (int)threadIdx.x < e1)
            s_rec[threadIdx.x] = make_uint4(s_trk[threadIdx.x].cap, s_trk[threadIdx.x].stride * 128u,
                                            (int)threadIdx.x == e1 - 1 ? s_trk[e0].base * 128u + 1 : 0, 0);
        for (int idx = warp; idx < size; idx += warps) {
            uint32_t w = 0xffffffffu;
            for (int e = e0, rem = idx; e < e1; e++) {
                const int cap = s_trk[e].cap, low = s_trk[e].low;
                const int x = rem % (cap + 1), y = x - __popc((low >> 5) & lane);
                rem /= cap + 1;
                if (x < cap && y >= 0 && y <= 5) w &= ~s_eq[low & 31][y];
            }
            ztab[(s_trk[e0].base + idx) * 32 + lane] = w;
        }
        e0 = e1;
    }
    // twice the ones of four rows among the minus columns of `bits`
    auto row_bytes = [&](int v, int shift, uint32_t bits) {
        uint32_t b = 0;
#pragma unroll
        for (int t = 0; t < 4; t++)
            b |= (uint32_t)(2 * __popc((uint32_t)(s_rm[4 * v + t] >> shift) & bits)) << (8 * t);
        return b;
    };
    for (int i = threadIdx.x; i < 1024 * NW; i += blockDim.x)
        ltab[(i & 1023) * LS + (i >> 10)] = row_bytes(i >> 10, 0, (uint32_t)(i & 1023));
    for (int i = threadIdx.x; i < 32 * NW; i += blockDim.x)
        ctab[(i & 31) * LS + (i >> 5)] = row_bytes(i >> 5, LOW, (uint32_t)(i & 31));
    for (int i = threadIdx.x; i < 32 * TW; i += blockDim.x) {
        uint32_t b = 0;
        for (int t = 0; t < 4; t++) {
            const int e = 4 * (i >> 5) + t;
            if (e < a.ntracked) b |= (uint32_t)__popc((uint32_t)s_trk[e].high & (uint32_t)(i & 31)) << (8 * t);
        }
        xtab[(i & 31) * TW + (i >> 5)] = b;
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
        // low signs, chunk of the batch (5 bits)
        const uint32_t e = live ? q[qn + lane] : 0, k = e >> LOW;
        uint32_t d[LS];
#pragma unroll
        for (int v = 0; v < LS / 2; v++) {
            const uint2 x = reinterpret_cast<const uint2 *>(base + k * LS)[v];
            const uint2 y = reinterpret_cast<const uint2 *>(ltab + (e & 1023u) * LS)[v];
            // bytes 128 + s_r, no borrow between them; then two's complement
            d[2 * v + 0] = (x.x - y.x) ^ 0x80808080u;
            d[2 * v + 1] = (x.y - y.y) ^ 0x80808080u;
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
        // batches start at even chunks or hold one
        exact_term_col<NPAD, G, 0>(s, col, colt, (__popc(e & ((1u << LOW) - 1)) ^ k ^ c_odd) & 1u,
                                   terms == 0);
        if (++terms == FOLD) {
            FoldCols<NR, NL>::apply(acc, col, colt);
            terms = 0;
        }
        __syncwarp();
    };
    // Appends the states of `alive` (tag: chunk), placed by a scan over the
    // lanes' counts: all at once while they fit the queue, else 256 at most.
    auto scan = [&](uint32_t part) {
        int inc = __popc(part);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        return inc;
    };
    auto push = [&](uint32_t part, uint32_t tag, int inc, int total) {
        int pos = qn + inc - __popc(part);
        while (part) {
            const uint32_t rest = part & (part - 1);
            q[pos++] = (uint16_t)(tag | (lane << 5) | __popc((part ^ rest) - 1));
            part = rest;
        }
        qn += total;
        while (qn >= 32) evaluate(32);
    };
    auto append = [&](uint32_t alive, uint32_t tag) {
        if (!__any_sync(0xffffffffu, alive != 0)) return;
        const int inc = scan(alive), total = __shfl_sync(0xffffffffu, inc, 31);
        if (qn + total <= BIN_QCAP) {
            push(alive, tag, inc, total);
        } else {
            for (int o = 0; o < 32; o += 8) {
                const uint32_t part = alive & (0xffu << o);
                const int pi = scan(part);
                push(part, tag, pi, __shfl_sync(0xffffffffu, pi, 31));
            }
        }
    };

    // Work units go to warps from a counter (the share of surviving states
    // varies strongly along the walk with the signs of the columns), one
    // ahead, so that the atomic's round trip overlaps the work.  A unit is
    // 2^log_unit batches of 2^log_steps chunks from all over the walk (an odd
    // multiple of their number modulo a power of two): neighbours share their
    // zero rows and would leave whole units empty and others full.
    const uint64_t c_lo = a.state_lo >> LOW;
    const uint64_t c_hi = (a.state_hi + (1u << LOW) - 1) >> LOW;
    const uint64_t units = 1ull << (a.log_batches - a.log_unit);
    const char *zl = reinterpret_cast<const char *>(ztab + lane);
    bool aborted = false;
    uint32_t polls = 0;
    for (uint64_t unit = (uint64_t)warp * gridDim.x + blockIdx.x; unit < units && !aborted;) {
        unsigned long long nx = 0;
        if (lane == 0) nx = (uint64_t)gridDim.x * warps + atomicAdd(a.next, 1ull);
        // the unit's batches, one a lane: not those beyond the window, nor
        // those with a batch row that is zero (in all of the batch)
        const uint64_t number = ((unit << a.log_unit | lane) * 0x9e3779b97f4a7c15ull) &
                                ((1ull << a.log_batches) - 1);
        const uint64_t mine_c0 = ((c_lo >> a.log_steps) + number) << a.log_steps;
        bool go;
        {
            const uint64_t b5 = mine_c0 >> 5;
            const uint32_t hw = (uint32_t)(b5 ^ (b5 >> 1));
            go = lane < (1 << a.log_unit) && mine_c0 < c_hi;
            for (int r = 0; r < a.batch_rows; r++)
                go &= (int)s_trk[r].half != __popc((uint32_t)(s_trk[r].high >> 5) & hw);
        }
        // the host-mapped abort word is read once per 128 batches that are
        // searched (4096 units without one), from the warp's second period on
        polls++;
        for (uint32_t todo = __ballot_sync(0xffffffffu, go); todo; todo &= todo - 1) {
            // chunks c0 + k0 .. c0 + k1 - 1 of the batch lie in the window
            const uint64_t c0 = __shfl_sync(0xffffffffu, mine_c0, __ffs(todo) - 1);
            const int k1 = c_hi - c0 < (1ull << a.log_steps) ? (int)(c_hi - c0) : 1 << a.log_steps;
            const int kfirst = c_lo > c0 ? (int)(c_lo - c0) : 0;
            polls += 32;
            // the batch's common high signs: gray(c0 >> 5) in columns HI and up
            const uint64_t b5 = c0 >> 5;
            const uint32_t hw = (uint32_t)(b5 ^ (b5 >> 1));
            auto ones = [&](uint64_t m) { return __popc((uint32_t)m & hw); };
            for (int r = a.batch_rows + lane; r < a.ntracked; r += 32)
                reinterpret_cast<uint8_t *>(xcnt)[r] = (uint8_t)(128 + s_trk[r].half - ones(s_trk[r].high >> 5));
            __syncwarp();
            // this lane's chunk: the signs of the five columns below those; a
            // chunk row with x = 0 (a zero byte) is zero in the whole chunk
            const uint32_t l5 = ((uint32_t)c0 + lane) & 31u;
            const uint32_t x5 = l5 ^ (l5 >> 1) ^ (((uint32_t)b5 & 1u) << 4);
            uint32_t zero = 0;
            for (int e = a.batch_rows >> 2; e < a.uniform_rows >> 2; e++) {
                const uint32_t x = (xcnt[e] - xtab[x5 * TW + e]) ^ 0x80808080u;
                zero |= (x - 0x01010101u) & ~x & 0x80808080u;
            }
            uint32_t chunks = __ballot_sync(0xffffffffu, zero == 0 && lane >= kfirst && lane < k1);
            __syncwarp();               // xcnt is read
            if (!chunks) continue;
            c_odd = (uint32_t)c0;
            const bool edge = ((c0 + kfirst) << LOW) < a.state_lo || ((c0 + k1) << LOW) > a.state_hi;
            for (int r = lane; r < NPAD; r += 32)
                reinterpret_cast<uint8_t *>(ucnt)[r] = (uint8_t)(128 + s_deg[r] - 2 * ones(s_rm[r] >> HI));
            __syncwarp();
            {
                const uint32_t *cb = ctab + x5 * LS;
                uint32_t *o = base + lane * LS;
#pragma unroll
                for (int v = 0; v < NW; v++) o[v] = ucnt[v] - cb[v];
            }
            {
                uint32_t *ll = list + lane * a.list_words;
                int g = 0;
                uint32_t off = 0;
                for (int e = a.uniform_rows; e < a.ntracked; e += 4) {
                    // bytes of x in two's complement: negative ones exceed every cap
                    const uint32_t x = (xcnt[e >> 2] - xtab[x5 * TW + (e >> 2)]) ^ 0x80808080u;
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        if (e + t >= a.ntracked) break;
                        const uint4 rec = s_rec[e + t];
                        off += min(__byte_perm(x, 0, 0x4440 + t), rec.x) * rec.y;
                        if (rec.z) {
                            ll[g++] = off + rec.z - 1;
                            off = 0;
                        }
                    }
                }
                for (; g < a.list_words; g++) ll[g] = 0;
            }
            __syncwarp();
            while (chunks) {            // two chunks at a time
                int kk[2];
                kk[0] = __ffs(chunks) - 1;
                chunks &= chunks - 1;
                const bool pair = chunks != 0;
                kk[1] = pair ? __ffs(chunks) - 1 : kk[0];
                chunks &= chunks - 1;
                uint32_t alive[2] = {0xffffffffu, pair ? 0xffffffffu : 0u};
                for (int v = 0; v < a.list_words; v += 4) {
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        const uint4 o = *reinterpret_cast<const uint4 *>(list + kk[t] * a.list_words + v);
                        const auto at = [&](uint32_t off) {
                            return *reinterpret_cast<const uint32_t *>(zl + off);
                        };
                        alive[t] &= at(o.x) & at(o.y) & at(o.z) & at(o.w);
                    }
                    if ((v & 4) && !__any_sync(0xffffffffu, (alive[0] | alive[1]) != 0)) break;
                }
                if (edge) {             // a window that starts or ends inside a chunk
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        const uint64_t c = c0 + kk[t];
                        uint32_t in = 0;
                        for (int k = 0; k < 32; k++) {
                            uint32_t i = (uint32_t)(k | (lane << 5)) ^ (uint32_t)((c & 1) << (LOW - 1));
                            i ^= i >> 1;
                            i ^= i >> 2;
                            i ^= i >> 4;
                            i ^= i >> 8;
                            const uint64_t g = (c << LOW) | i;
                            in |= (uint32_t)(g >= a.state_lo && g < a.state_hi) << k;
                        }
                        alive[t] &= in;
                    }
                }
#pragma unroll
                for (int t = 0; t < 2; t++) append(alive[t], (uint32_t)(kk[t] << LOW));
            }
            if (qn > 0) evaluate(qn);       // the next batch has other base bytes
            __syncwarp();
        }
        if (polls >= 4096) {
            polls = 0;
            aborted = __any_sync(0xffffffffu, *a.abort_flag != 0);
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

// Compiled shapes (binary_inst_*.cu): NPAD in {24, 28, ..., 48}, G in {5, 6,
// 7, 8, 10}.  Orders below BINARY_MIN_N, and matrices whose sampled share of
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
// tables to fit beside the NPAD kernel's other shared memory, and for a walk
// of `chunks` chunks a block not to spend its time on their entries, with the
// most warps that allow it; group[e] = the row's group.  Returns the number of
// groups, -1 if there is no such packing.
int binary_pack_groups(int NPAD, const int *caps, int rows, double chunks, int *group, int *warps);

}  // namespace pg
