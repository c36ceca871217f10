// Host side of the FP64 Glynn engine: forward (f64_forward.cuh, orders 2..32)
// and forward with gradient (f64_gradient.cuh) for batches of real matrices,
// complex forward, and the reductions of the warps' slots.  Orders above 32
// and Gray windows run f64_wide.cuh (pg_f64_wide.cu).
#include "pg_internal.h"
#include "f64_gradient.cuh"
#include "f64_wide.cuh"

#include <cmath>
#include <cstring>
#include <vector>

namespace pg {

// Adds the warps' slots of each matrix (one warp per matrix, a fixed order)
// and removes the row scaling and 2^(n-1).
__global__ void glynn_forward_reduce(const double *Are, const double *Aim, const double *slots,
                                     int n, int per_matrix, double *re, double *im,
                                     double *abs_sum) {
    const int b = blockIdx.x, lane = threadIdx.x;
    const double *base = slots + (size_t)b * per_matrix * FWD_SLOT;
    double sr = 0, cr = 0, si = 0, ci = 0, as = 0;
    for (int w = lane; w < per_matrix; w += 32) {
        kahan(sr, cr, base[w * FWD_SLOT]);
        kahan(si, ci, base[w * FWD_SLOT + 1]);
        as += base[w * FWD_SLOT + 2];
    }
    sr -= cr;
    si -= ci;
    int e = 0;
    if (lane < n) {
        const size_t row = (size_t)b * n * n + (size_t)lane * n;
        e = fwd_row_exponent(Are + row, Aim ? Aim + row : nullptr, n, fwd_bound_log(Aim != nullptr));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
        as += __shfl_xor_sync(0xffffffffu, as, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
    }
    if (lane != 0) return;
    re[b] = ldexp(sr, -e - (n - 1));
    if (im) im[b] = ldexp(si, -e - (n - 1));
    if (abs_sum) abs_sum[b] = ldexp(as, -e - (n - 1));
}

constexpr int F64_BLOCKS_SM = 32;    // resident blocks of an SM, at most

// Launch shape of the forward walk of `batch` matrices of order 2..32 (Aim
// null: real): fills a.batch, a.log_block, a.blocks_per; returns the slots'
// bytes, 0 where a warp takes a whole real matrix and writes its result.
static size_t forward_shape(const double *Are, const double *Aim, int batch, int n, int sms,
                            FwdArgs *out) {
    FwdArgs &a = *out;
    a.Are = Are;
    a.Aim = Aim;
    a.batch = batch;
    a.resident = F64_BLOCKS_SM * sms;
    a.log_block = std::min(FWD_LOG_BLOCK, n - 1);
    // shorter real blocks (down to 8 states a thread) while fewer than four
    // waves of warps are busy; complex ones keep the length that fixes the
    // order of their |term| sums
    while (!Aim && a.log_block > 8 &&
           ((uint64_t)batch << (n - 1 - a.log_block)) < (uint64_t)sms * 64)
        a.log_block--;
    // thread blocks: a power of two per matrix, so that every warp takes the
    // same number of blocks of states
    const uint64_t tasks = 1ull << (n - 1 - a.log_block);
    a.blocks_per = 1;
    if (!Aim && tasks == 1) return 0;
    while ((uint64_t)a.blocks_per * FWD_WARPS < tasks &&
           (uint64_t)batch * a.blocks_per * 2 <= (uint64_t)sms * 64)
        a.blocks_per *= 2;
    return (size_t)batch * a.blocks_per * FWD_WARPS * FWD_SLOT * sizeof(double);
}

// The walk and its reduction, asynchronous on s; a.slots null: no slots.
static int forward_launch(FwdArgs a, int n, double *re, double *im, double *abs_sum,
                          cudaStream_t s) {
    a.re = re;
    a.abs_sum = abs_sum;
    PG_CUDA(!a.Aim ? launch_forward_real(n, a, s)
            : n <= 22 ? launch_forward_cplx_lo(n, a, s) : launch_forward_cplx_hi(n, a, s));
    if (!a.slots) return PG_OK;
    glynn_forward_reduce<<<a.batch, 32, 0, s>>>(a.Are, a.Aim, a.slots, n, a.blocks_per * FWD_WARPS,
                                                re, im, abs_sum);
    PG_CUDA(cudaGetLastError());
    return PG_OK;
}

static int f64_finish(const int *status, cudaStream_t s) {
    int hstatus = 0;
    PG_CUDA(cudaMemcpyAsync(&hstatus, status, sizeof(int), cudaMemcpyDeviceToHost, s));
    PG_CUDA(cudaStreamSynchronize(s));
    if (hstatus) return fail(PG_EABORT, "FP64 launch aborted by pg_abort()");
    return PG_OK;
}

// per(A) of `batch` device matrices of order 2..32 (Aim null: real).
static int glynn_forward_run(const double *Are, const double *Aim, int batch, int n, double *re,
                             double *im, double *abs_sum, cudaStream_t stream) {
    DeviceInfo dev;
    int st = device_info(&dev);
    if (st != PG_OK) return st;
    FwdArgs a;
    volatile int *abort_dev;
    st = abort_flag_device(&abort_dev);
    if (st != PG_OK) return st;
    const size_t bytes = forward_shape(Are, Aim, batch, n, dev.sm_count, &a);
    Workspace *ws;
    st = workspace(&ws, bytes + 256, 64);
    if (st != PG_OK) return st;
    cudaStream_t s = stream ? stream : ws->stream;
    a.status = (int *)ws->dev;
    a.slots = bytes ? (double *)((char *)ws->dev + 256) : nullptr;
    a.abort_flag = abort_dev;
    PG_CUDA(cudaMemsetAsync(a.status, 0, sizeof(int), s));
    if ((st = forward_launch(a, n, re, im, abs_sum, s)) != PG_OK) return st;
    return f64_finish(a.status, s);
}

// One block per matrix and gradient row: warp v adds the slots v, v + 8, ...
// (lane = column), the first warp adds the eight sums; all in a fixed order.
__global__ void __launch_bounds__(256) glynn_gradient_reduce(
    const double *A, const double *slots, int n, int per_matrix, double *grad, double *grad_abs) {
    const int b = blockIdx.x, i = blockIdx.y, lane = threadIdx.x & 31, v = threadIdx.x >> 5;
    const int sd = grad_slot(n);
    const double *base = slots + (size_t)b * per_matrix * sd;
    __shared__ double part[8][32], rows[8];
    __shared__ int ex[32];
    double s = 0, c = 0, as = 0;
    for (int w = v; w < per_matrix; w += 8) {
        const double *sl = base + (size_t)w * sd;
        if (lane < n) {
            kahan(s, c, sl[i * n + lane]);
            kahan(s, c, -sl[n * n + i * n + lane]);
        }
        if (lane == 0) as += sl[2 * n * n + i];
    }
    part[v][lane] = s - c;
    if (lane == 0) rows[v] = as;
    if (threadIdx.x < 32)
        ex[lane] = lane < n ? fwd_row_exponent(A + ((size_t)b * n + lane) * n, nullptr, n,
                                               fwd_bound_log(false)) : 0;
    __syncthreads();
    if (v != 0) return;
    int total = 0;
    for (int r = 0; r < n; r++) total += ex[r];
    // E_i was formed from the scaled rows l != i
    const int shift = -(total - ex[i]) - (n - 1);
    double g = 0, gc = 0;
    for (int u = 0; u < 8; u++) kahan(g, gc, part[u][lane]);
    if (lane < n) grad[((size_t)b * n + i) * n + lane] = ldexp(g - gc, shift);
    if (lane != 0 || !grad_abs) return;
    double tg = 0;
    for (int u = 0; u < 8; u++) tg += rows[u];
    grad_abs[(size_t)b * n + i] = ldexp(tg, shift);
}

constexpr size_t GRAD_SLOT_BYTES = 256u << 20;   // of one launch's slots, at most

// The permanents come from the forward walk, so that they do not depend on
// whether the gradient is asked for (a tenth of the gradient's time).
static int glynn_gradient_run(const double *A, int batch, int n, double *per, double *grad,
                              double *abs_sum, double *grad_abs, cudaStream_t stream) {
    DeviceInfo dev;
    int st = device_info(&dev);
    if (st != PG_OK) return st;
    volatile int *abort_dev;
    st = abort_flag_device(&abort_dev);
    if (st != PG_OK) return st;
    GradArgs a;
    a.A = A;
    a.batch = batch;
    a.resident = F64_BLOCKS_SM * dev.sm_count;
    int lw, rmax;
    gradient_shape(n, &lw, &rmax);
    // shorter ranges (down to 2^5 states) while a warp per range leaves less
    // than two resident waves of blocks
    const uint64_t resident = 2 * (uint64_t)dev.sm_count;
    a.log_range = rmax;
    const auto tasks_of = [&](int R) { return n - 1 > R + lw ? 1ull << (n - 1 - R - lw) : 1ull; };
    while (a.log_range > 5 &&
           (uint64_t)batch * tasks_of(a.log_range) < 2 * GRAD_WARPS * resident)
        a.log_range--;
    const uint64_t tasks = tasks_of(a.log_range);
    FwdArgs f;
    const size_t fwd_bytes = forward_shape(A, nullptr, batch, n, dev.sm_count, &f);
    Workspace *ws;
    a.abort_flag = f.abort_flag = abort_dev;
    a.blocks_per = 1;
    if (tasks == 1) {                    // a warp a matrix, no slots
        if ((st = workspace(&ws, 256 + fwd_bytes, 64)) != PG_OK) return st;
        cudaStream_t s = stream ? stream : ws->stream;
        a.status = f.status = (int *)ws->dev;
        f.slots = fwd_bytes ? (double *)((char *)ws->dev + 256) : nullptr;
        a.slots = nullptr;
        a.grad = grad;
        a.grad_abs = grad_abs;
        PG_CUDA(cudaMemsetAsync(a.status, 0, sizeof(int), s));
        if ((st = forward_launch(f, n, per, nullptr, abs_sum, s)) != PG_OK) return st;
        PG_CUDA(launch_gradient_lo(n, a, s));
        return f64_finish(a.status, s);
    }
    // blocks per matrix: the fewest waves times ranges per warp; more blocks
    // also cost slots and their reduction, so ties go to fewer
    uint64_t best = ~0ull;
    for (uint64_t p = 1; p <= resident && (p == 1 || (p - 1) * GRAD_WARPS < tasks); p++) {
        if (p > 1 && (uint64_t)batch * p > 8 * resident) break;
        const uint64_t waves = ((uint64_t)batch * p + resident - 1) / resident;
        const uint64_t cost = waves * ((tasks + GRAD_WARPS * p - 1) / (GRAD_WARPS * p));
        if (cost < best) {
            best = cost;
            a.blocks_per = (int)p;
        }
    }
    const size_t warps = (size_t)a.blocks_per * GRAD_WARPS;
    // The matrices go in equal parts whose slots stay within GRAD_SLOT_BYTES
    // (thousands of matrices, many waves: 131072 of 16x16 175.4 ms in nine parts,
    // 174.8 with 2.2 GB of slots at once).
    const size_t each = warps * grad_slot(n) * sizeof(double);
    const int parts = (int)((batch * each + GRAD_SLOT_BYTES - 1) / GRAD_SLOT_BYTES);
    const int most = (batch + parts - 1) / parts;
    const size_t bytes = most * each + 256;
    if ((st = workspace(&ws, bytes + fwd_bytes, 64)) != PG_OK) return st;
    cudaStream_t s = stream ? stream : ws->stream;
    a.status = f.status = (int *)ws->dev;
    a.slots = (double *)((char *)ws->dev + 256);
    a.grad = a.grad_abs = nullptr;
    f.slots = fwd_bytes ? (double *)((char *)ws->dev + bytes) : nullptr;
    PG_CUDA(cudaMemsetAsync(a.status, 0, sizeof(int), s));
    if ((st = forward_launch(f, n, per, nullptr, abs_sum, s)) != PG_OK) return st;
    for (int b = 0; b < batch; b += most) {
        a.A = A + (size_t)b * n * n;
        a.batch = std::min(most, batch - b);
        PG_CUDA(cudaMemsetAsync(a.slots, 0, a.batch * each, s));
        PG_CUDA(n <= 16 ? launch_gradient_lo(n, a, s)
                : n <= 24 ? launch_gradient_mid(n, a, s) : launch_gradient_hi(n, a, s));
        glynn_gradient_reduce<<<dim3(a.batch, n), 256, 0, s>>>(
            a.A, a.slots, n, (int)warps, grad + (size_t)b * n * n,
            grad_abs ? grad_abs + (size_t)b * n : nullptr);
        PG_CUDA(cudaGetLastError());
    }
    return f64_finish(a.status, s);
}

}  // namespace pg

extern "C" int pg_glynn_f64_dev(const double *A, int batch, int n, double *per, double *grad,
                                double *abs_sum, double *grad_abs, void *stream) {
    using namespace pg;
    if (batch < 0 || n < 0 || n > 63) return fail(PG_ERANGE, "FP64 engine supports 0 <= n <= 63");
    if (batch == 0) return PG_OK;
    if (!A || !per) return fail(PG_EINVAL, "null argument");
    if (n <= 1) return fail(PG_ERANGE, "orders 0 and 1 are handled by the caller");
    if (n > 32) {
        // orders 33..63: forward only, two rows per lane (f64_wide.cuh)
        if (grad || grad_abs)
            return fail(PG_ERANGE, "the FP64 gradient supports n <= 32 (forward up to 63)");
        return glynn_wide_run(A, nullptr, batch, n, 0, 1ull << (n - 1), true, per, nullptr,
                              abs_sum, (cudaStream_t)stream);
    }
    return grad ? glynn_gradient_run(A, batch, n, per, grad, abs_sum, grad_abs, (cudaStream_t)stream)
                : glynn_forward_run(A, nullptr, batch, n, per, nullptr, abs_sum,
                                    (cudaStream_t)stream);
}

extern "C" int pg_glynn_c64_dev(const double *Are, const double *Aim, int batch, int n,
                                double *per_re, double *per_im, double *abs_sum, void *stream) {
    using namespace pg;
    if (batch < 0 || n < 2 || n > 63) return fail(PG_ERANGE, "complex FP64 engine supports 2 <= n <= 63");
    if (batch == 0) return PG_OK;
    if (!Are || !Aim || !per_re || !per_im) return fail(PG_EINVAL, "null argument");
    if (n > 32)   // two rows per lane (f64_wide.cuh)
        return glynn_wide_run(Are, Aim, batch, n, 0, 1ull << (n - 1), true, per_re, per_im,
                              abs_sum, (cudaStream_t)stream);
    return glynn_forward_run(Are, Aim, batch, n, per_re, per_im, abs_sum, (cudaStream_t)stream);
}

// Host-pointer form of pg_glynn_f64_dev for callers without device memory of
// their own (ctypes users, other languages' FFIs): device buffers for the
// call are allocated here (the library's workspace is the kernel's own
// scratch), the results are copied back and the buffers freed.
extern "C" int pg_glynn_f64_fwd_bwd(const double *A, int batch, int n, double *per,
                                    double *grad, double *abs_sum) {
    using namespace pg;
    if (batch < 0 || n < 0 || n > 63) return fail(PG_ERANGE, "FP64 engine supports 0 <= n <= 63");
    if (batch == 0) return PG_OK;
    if (!per || (n > 0 && !A)) return fail(PG_EINVAL, "null argument");
    if (n > 32 && grad)
        return fail(PG_ERANGE, "the FP64 gradient supports n <= 32 (forward up to 63)");
    if (n <= 1) {
        for (int b = 0; b < batch; b++) {
            per[b] = n == 0 ? 1.0 : A[b];
            if (grad && n == 1) grad[b] = 1.0;
            if (abs_sum) abs_sum[b] = n == 0 ? 1.0 : std::fabs(A[b]);
        }
        return PG_OK;
    }
    DeviceInfo dev;
    int st = device_info(&dev);
    if (st != PG_OK) return st;
    const size_t na = (size_t)batch * n * n;
    const size_t bytes = (na + (grad ? na : 0) + 2 * (size_t)batch) * sizeof(double);
    double *d = nullptr;
    PG_CUDA(cudaMalloc(&d, bytes));
    double *dA = d, *dgrad = grad ? d + na : nullptr;
    double *dper = d + na + (grad ? na : 0), *dabs = dper + batch;
    cudaError_t e = cudaMemcpy(dA, A, na * sizeof(double), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d);
        return cuda_fail(e, "cudaMemcpy(A)");
    }
    st = pg_glynn_f64_dev(dA, batch, n, dper, dgrad, dabs, nullptr, nullptr);
    if (st == PG_OK) {
        e = cudaMemcpy(per, dper, (size_t)batch * sizeof(double), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && grad)
            e = cudaMemcpy(grad, dgrad, na * sizeof(double), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && abs_sum)
            e = cudaMemcpy(abs_sum, dabs, (size_t)batch * sizeof(double), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) st = cuda_fail(e, "cudaMemcpy(results)");
    }
    cudaFree(d);
    return st;
}

// pg_glynn_c64_dev with host pointers: the real and imaginary planes
// [batch][n][n] in, per_re/per_im[batch] and abs_sum[batch] (nullable)
// out; 0 <= n <= 63 (n <= 1 on the host).  Device buffers for the call are
// allocated and freed inside.  Replaces permanent_parallel_complex
// (perm_parallel_cuda.cu:416-498), host planes in and host values out.
extern "C" int pg_glynn_c64(const double *Are, const double *Aim, int batch, int n,
                            double *per_re, double *per_im, double *abs_sum) {
    using namespace pg;
    if (batch < 0 || n < 0 || n > 63)
        return fail(PG_ERANGE, "complex FP64 engine supports 0 <= n <= 63");
    if (batch == 0) return PG_OK;
    if (!per_re || !per_im || (n > 0 && (!Are || !Aim))) return fail(PG_EINVAL, "null argument");
    if (n <= 1) {
        for (int b = 0; b < batch; b++) {
            per_re[b] = n == 0 ? 1.0 : Are[b];
            per_im[b] = n == 0 ? 0.0 : Aim[b];
            if (abs_sum) abs_sum[b] = n == 0 ? 1.0 : std::hypot(Are[b], Aim[b]);
        }
        return PG_OK;
    }
    DeviceInfo dev;
    int st = device_info(&dev);
    if (st != PG_OK) return st;
    const size_t na = (size_t)batch * n * n;
    const size_t bytes = (2 * na + 3 * (size_t)batch) * sizeof(double);
    double *d = nullptr;
    PG_CUDA(cudaMalloc(&d, bytes));
    double *dre = d, *dim = d + na, *dpre = d + 2 * na, *dpim = dpre + batch,
           *dabs = dpim + batch;
    cudaError_t e = cudaMemcpy(dre, Are, na * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dim, Aim, na * sizeof(double), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d);
        return cuda_fail(e, "cudaMemcpy(A)");
    }
    st = pg_glynn_c64_dev(dre, dim, batch, n, dpre, dpim, dabs, nullptr);
    if (st == PG_OK) {
        e = cudaMemcpy(per_re, dpre, (size_t)batch * sizeof(double), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess)
            e = cudaMemcpy(per_im, dpim, (size_t)batch * sizeof(double), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && abs_sum)
            e = cudaMemcpy(abs_sum, dabs, (size_t)batch * sizeof(double), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) st = cuda_fail(e, "cudaMemcpy(results)");
    }
    cudaFree(d);
    return st;
}
