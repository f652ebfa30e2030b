// validate.cu -- result checking on the GPU.
//
// 1. Constant check with validate_C_kernel's rule (1D-row-block/mulmat_kernel.cu:165-222): an
//    element is invalid when |v - expected| > abs_tol AND |v - expected| / |expected| > rel_tol;
//    max absolute and relative error are reported.  The reference resolves its maxima with a
//    compare-and-swap loop per element; here each block reduces in registers and shared memory
//    and issues one atomic per quantity.  Non-finite elements also count as invalid (the
//    reference's comparisons are false for NaN, so it would pass them).
// 2. Error of a computed C against a double-double product (Dot2: TwoProd by FMA, Knuth TwoSum),
//    reduced to normwise, max relative, max componentwise and max absolute error.
#include <cfloat>
#include <cstring>
#include <cmath>
#include <mutex>

#include "mgx_common.cuh"

namespace mgx {
namespace val {

constexpr int THREADS = 256;

__device__ __forceinline__ void atomic_max_nonneg(unsigned long long *addr, double v)
{
    // For non-negative doubles the IEEE bit pattern orders like the value.
    if (v > 0.0) atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

// What one block of the constant check found.
struct ConstPart {
    unsigned long long invalid;
    double max_abs;
};

// Bound by reading C from HBM: two 16-byte loads in flight per thread and no division.  The relative
// error |v - expected| / |expected| grows with the absolute one (a correctly rounded division by a
// constant), so its maximum is one division of the maximal absolute error at the end, and an
// element's own quotient is needed only where its absolute error is beyond abs_tol.  8192 x 8192:
// 357 us with a division per element and one 8-byte load in flight, 94 us now (5.7 TB/s).
__global__ void __launch_bounds__(THREADS) validate_const_kernel(const double *__restrict__ C, size_t count,
                                                                 double expected, double abs_tol, double rel_tol,
                                                                 ConstPart *parts)
{
    unsigned long long bad = 0;
    double mabs = 0.0;
    const double aexp = fabs(expected);
    // within `lim` an element is finite and inside abs_tol (an abs_tol of NaN is never exceeded)
    const double lim = abs_tol < DBL_MAX ? abs_tol : DBL_MAX;
    auto check = [&](double v) {
        const double ae = fabs(v - expected);
        if (ae > mabs) mabs = ae;  // NaN compares false: it never enters the maximum
        if (!(ae <= lim)) {
            const double re = (aexp > 0.0) ? ae / aexp : 0.0;
            if ((ae > abs_tol && re > rel_tol) || !isfinite(v)) ++bad;
        }
    };
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    // a first element off the 16-byte grid, then pairs, then a last odd element
    const size_t head = ((reinterpret_cast<uintptr_t>(C) & 15) != 0) ? 1 : 0;
    const double2 *P = reinterpret_cast<const double2 *>(C + head);
    const size_t pairs = (count - head) / 2;
    size_t i = tid;
    for (; i + stride < pairs; i += 2 * stride) {
        const double2 a = __ldg(P + i), b = __ldg(P + i + stride);
        check(a.x);
        check(a.y);
        check(b.x);
        check(b.y);
    }
    if (i < pairs) {
        const double2 a = __ldg(P + i);
        check(a.x);
        check(a.y);
    }
    if (tid == 0) {
        if (head) check(C[0]);
        if (head + 2 * pairs < count) check(C[count - 1]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        bad += __shfl_xor_sync(0xffffffffu, bad, o);
        mabs = fmax(mabs, __shfl_xor_sync(0xffffffffu, mabs, o));
    }
    __shared__ unsigned long long s_bad[THREADS / 32];
    __shared__ double s_abs[THREADS / 32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        s_bad[w] = bad;
        s_abs[w] = mabs;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < THREADS / 32; ++k) {
            bad += s_bad[k];
            mabs = fmax(mabs, s_abs[k]);
        }
        parts[blockIdx.x] = ConstPart{bad, mabs};
    }
}

// ---------------------------------------------------------------- double-double error check
constexpr int DD_TM = 64, DD_TN = 64, DD_TK = 16;

struct ErrAcc {
    double sum_d2;
    double sum_r2;
    unsigned long long max_rel_bits;
    unsigned long long max_comp_bits;
    unsigned long long max_abs_bits;
};

__global__ void __launch_bounds__(256) dd_error_kernel(const double *__restrict__ A, const double *__restrict__ B,
                                                       const double *__restrict__ C, int m, int n, int k, int lda,
                                                       int ldb, int ldc, int row0, int rows, double floor_abs,
                                                       ErrAcc *acc)
{
    __shared__ double As[DD_TM][DD_TK + 1];
    __shared__ double Bs[DD_TK][DD_TN];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int bm = row0 + blockIdx.y * DD_TM, bn = blockIdx.x * DD_TN;
    double s[4][4], c[4][4], ab[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = c[i][j] = ab[i][j] = 0.0;
    const int row_end = row0 + rows;
    for (int k0 = 0; k0 < k; k0 += DD_TK) {
        for (int idx = threadIdx.x; idx < DD_TM * DD_TK; idx += 256) {
            const int r = idx / DD_TK, kk = idx % DD_TK;
            const int gr = bm + r, gk = k0 + kk;
            As[r][kk] = (gr < row_end && gk < k) ? A[(size_t)gr * lda + gk] : 0.0;
        }
        for (int idx = threadIdx.x; idx < DD_TK * DD_TN; idx += 256) {
            const int kk = idx / DD_TN, cc = idx % DD_TN;
            const int gk = k0 + kk, gc = bn + cc;
            Bs[kk][cc] = (gk < k && gc < n) ? B[(size_t)gk * ldb + gc] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < DD_TK; ++kk) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[ty + 16 * i][kk];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const double p = a[i] * b[j];
                    const double q = fma(a[i], b[j], -p);
                    const double t = s[i][j] + p;
                    const double z = t - s[i][j];
                    const double e = (s[i][j] - (t - z)) + (p - z);
                    s[i][j] = t;
                    c[i][j] += e + q;
                    ab[i][j] = fma(fabs(a[i]), fabs(b[j]), ab[i][j]);
                }
        }
        __syncthreads();
    }
    double d2 = 0.0, r2 = 0.0, mrel = 0.0, mcomp = 0.0, mabs = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gr = bm + ty + 16 * i, gc = bn + tx + 16 * j;
            if (gr < row_end && gc < n) {
                const double hi = s[i][j] + c[i][j];
                const double lo = c[i][j] - (hi - s[i][j]);
                const double d = (C[(size_t)gr * ldc + gc] - hi) - lo;
                const double ad = fabs(d);
                d2 += d * d;
                r2 += hi * hi;
                mabs = fmax(mabs, ad);
                if (fabs(hi) >= floor_abs && hi != 0.0) mrel = fmax(mrel, ad / fabs(hi));
                if (ab[i][j] > 0.0) mcomp = fmax(mcomp, ad / ab[i][j]);
            }
        }
    for (int o = 16; o > 0; o >>= 1) {
        d2 += __shfl_xor_sync(0xffffffffu, d2, o);
        r2 += __shfl_xor_sync(0xffffffffu, r2, o);
        mrel = fmax(mrel, __shfl_xor_sync(0xffffffffu, mrel, o));
        mcomp = fmax(mcomp, __shfl_xor_sync(0xffffffffu, mcomp, o));
        mabs = fmax(mabs, __shfl_xor_sync(0xffffffffu, mabs, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&acc->sum_d2, d2);
        atomicAdd(&acc->sum_r2, r2);
        atomic_max_nonneg(&acc->max_rel_bits, mrel);
        atomic_max_nonneg(&acc->max_comp_bits, mcomp);
        atomic_max_nonneg(&acc->max_abs_bits, mabs);
    }
}

__global__ void max_abs_kernel(const double *__restrict__ C, int rows, int n, int ldc,
                               unsigned long long *out_bits)
{
    double mx = 0.0;
    const size_t total = (size_t)rows * n;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / n, cidx = i % n;
        mx = fmax(mx, fabs(C[r * ldc + cidx]));
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(out_bits, mx);
}

}  // namespace val
}  // namespace mgx

using namespace mgx;

static double bits_to_double(unsigned long long b)
{
    double d;
    memcpy(&d, &b, sizeof d);
    return d;
}

namespace {

// Page-locked buffers that the constant check's blocks write their findings to and the calling thread
// reads.  A call takes an idle one of its context and hands it back once it has read it, so as many are
// held as calls ever ran at once, at most kIdle of 32 KiB (mgx_scratch_trim frees them), and a thread's
// end frees nothing: cudaFreeHost waits for all of the device's work.  Never destroyed: threads may
// still check while the process exits.  A buffer whose context a cudaDeviceReset has ended is gone with
// it and is never found again, as the context after it has another id; without an id (driver without the
// call) nothing is kept.  With device accumulators instead, the call had an allocation, a memset, a
// copy back through pageable memory and a free around its kernel.
constexpr int kParts = 2048;
constexpr int kIdle = 64;

class PartsPool {
public:
    struct Buffer {
        val::ConstPart *ptr;
        unsigned long long ctx;
    };

    int take(Buffer *out)
    {
        unsigned long long ctx = mgx_context_id();
        if (ctx == 0) {  // a thread's first call: no context current yet
            int d = 0;
            MGX_HOST_CHECK(cudaGetDevice(&d));
            MGX_HOST_CHECK(cudaSetDevice(d));
            ctx = mgx_context_id();
        }
        if (ctx != 0) {
            std::lock_guard<std::mutex> lk(mu_);
            for (int i = count_ - 1; i >= 0; --i)
                if (idle_[i].ctx == ctx) {
                    *out = remove(i);
                    return MGX_SUCCESS;
                }
        }
        MGX_HOST_CHECK(cudaHostAlloc(reinterpret_cast<void **>(&out->ptr), kParts * sizeof(val::ConstPart),
                                     cudaHostAllocPortable | cudaHostAllocMapped));
        out->ctx = ctx;
        return MGX_SUCCESS;
    }

    void give_back(const Buffer &b)
    {
        if (b.ctx != 0) {
            std::lock_guard<std::mutex> lk(mu_);
            if (count_ == kIdle && idle_[0].ctx != b.ctx) remove(0);  // of a context that may be gone
            if (count_ < kIdle) {
                idle_[count_++] = b;
                return;
            }
        }
        cudaFreeHost(b.ptr);
    }

    // Frees the idle buffers of the current context.
    void trim()
    {
        const unsigned long long ctx = mgx_context_id();
        Buffer mine[kIdle];
        int n = 0;
        {
            std::lock_guard<std::mutex> lk(mu_);
            for (int i = count_ - 1; i >= 0; --i)
                if (idle_[i].ctx == ctx) mine[n++] = remove(i);
        }
        while (n > 0) cudaFreeHost(mine[--n].ptr);
    }

private:
    Buffer remove(int i)
    {
        const Buffer b = idle_[i];
        for (--count_; i < count_; ++i) idle_[i] = idle_[i + 1];
        return b;
    }

    std::mutex mu_;
    Buffer idle_[kIdle];
    int count_ = 0;
};

PartsPool &parts_pool()
{
    static PartsPool *pool = new PartsPool;
    return *pool;
}

}  // namespace

void mgx_validate_trim() { parts_pool().trim(); }

int mgx_validate_impl(const double *d_c, size_t count, double expected, double abs_tol, double rel_tol,
                      mgx_validation_t *out, cudaStream_t stream)
{
    out->elements = count;
    out->invalid = 0;
    out->max_abs_error = out->max_rel_error = 0.0;
    if (count > 0) {
        PartsPool::Buffer buffer{};
        const int brc = parts_pool().take(&buffer);
        if (brc != MGX_SUCCESS) return brc;
        val::ConstPart *parts = buffer.ptr;
        size_t blocks = (count + 4 * val::THREADS - 1) / (4 * val::THREADS);  // four elements per step
        const size_t cap = (size_t)mgx_sm_count() * 8;
        if (blocks > cap) blocks = cap;
        if (blocks > kParts) blocks = kParts;
        val::validate_const_kernel<<<(unsigned)blocks, val::THREADS, 0, stream>>>(d_c, count, expected, abs_tol, rel_tol,
                                                                                  parts);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) {
            mgx_set_last_cuda_error(e, "constant validation", __FILE__, __LINE__);
            return MGX_E_CUDA;  // (the buffer is not handed back: the kernel may still write to it)
        }
        for (size_t b = 0; b < blocks; ++b) {
            out->invalid += parts[b].invalid;
            if (parts[b].max_abs > out->max_abs_error) out->max_abs_error = parts[b].max_abs;
        }
        parts_pool().give_back(buffer);
    }
    // an infinite `expected` gives NaN quotients, which never count
    const double rel = fabs(expected) > 0.0 ? out->max_abs_error / fabs(expected) : 0.0;
    out->max_rel_error = rel > 0.0 ? rel : 0.0;
    return MGX_SUCCESS;
}

extern "C" MGX_API int mgx_error_vs_dd(const double *A, const double *B, const double *C, int m, int n, int k,
                                       int lda, int ldb, int ldc, int row_start, int row_count, double floor_rel,
                                       mgx_error_t *out)
{
    if (!out || m < 0 || n < 0 || k < 0 || !A || !B || !C || row_start < 0 || row_start > m) {
        mgx_set_last_message("mgx_error_vs_dd: invalid arguments");
        return MGX_E_INVALID;
    }
    int rows = (row_count <= 0) ? m - row_start : row_count;
    if (row_start + rows > m) rows = m - row_start;
    memset(out, 0, sizeof *out);
    if (rows <= 0 || n <= 0) return MGX_SUCCESS;
    struct Scratch {
        val::ErrAcc acc;
        unsigned long long cmax_bits;
    };
    Scratch *d = nullptr;
    cudaStream_t s = nullptr;
    {
        const int arc = mgx_scratch_alloc(reinterpret_cast<void **>(&d), sizeof(Scratch), s);
        if (arc != MGX_SUCCESS) return arc;
    }
    Scratch h;
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof(Scratch), s);
    if (e == cudaSuccess) {
        val::max_abs_kernel<<<mgx_sm_count() * 4, 256, 0, s>>>(C + (size_t)row_start * ldc, rows, n, ldc, &d->cmax_bits);
        e = cudaMemcpyAsync(&h, d, sizeof h, cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) {
        const double floor_abs = floor_rel * bits_to_double(h.cmax_bits);
        dim3 grid((n + val::DD_TN - 1) / val::DD_TN, (rows + val::DD_TM - 1) / val::DD_TM);
        val::dd_error_kernel<<<grid, 256, 0, s>>>(A, B, C, m, n, k, lda, ldb, ldc, row_start, rows, floor_abs, &d->acc);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof h, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    cudaFreeAsync(d, s);
    if (e != cudaSuccess) {
        mgx_set_last_cuda_error(e, "double-double error check", __FILE__, __LINE__);
        return MGX_E_CUDA;
    }
    out->normwise = (h.acc.sum_r2 > 0.0) ? sqrt(h.acc.sum_d2) / sqrt(h.acc.sum_r2) : sqrt(h.acc.sum_d2);
    out->max_rel = bits_to_double(h.acc.max_rel_bits);
    out->max_componentwise = bits_to_double(h.acc.max_comp_bits);
    out->max_abs = bits_to_double(h.acc.max_abs_bits);
    out->rows_checked = (uint64_t)rows;
    return MGX_SUCCESS;
}
