// Dense complex linear algebra for the plain FP64 form: GEMV and Frobenius
// norms (the LU is in lu64.cu).  All matrices column-major complex FP64
// (double2).
#include "common.cuh"
#include "complex.cuh"

namespace bem {

// ---------------------------------------------------------------------------
// y = alpha A x + beta y (m x n).  Column chunks are reduced by the last CTA of
// each row block in a fixed order (deterministic).
constexpr int GV_ROWS = 256;
constexpr int GV_COLS = 256;
__global__ void __launch_bounds__(GV_ROWS) gemv64_kernel(int64_t m, int64_t n, const double2* __restrict__ A,
                                                         int64_t lda, const double2* __restrict__ x,
                                                         double2* __restrict__ y, z2 alpha, z2 beta,
                                                         double2* __restrict__ part, int* __restrict__ tickets) {
    __shared__ double2 xs[GV_COLS];
    __shared__ int last;
    int64_t i = blockIdx.x * (int64_t)GV_ROWS + threadIdx.x;
    int64_t j0 = (int64_t)blockIdx.y * GV_COLS;
    int64_t jn = min((int64_t)GV_COLS, n - j0);
    for (int t = threadIdx.x; t < jn; t += GV_ROWS) xs[t] = x[j0 + t];
    __syncthreads();
    double2 acc = make_double2(0, 0);
    if (i < m) {
        const double2* a = A + j0 * lda + i;
        int64_t q = 0;
        for (; q + 4 <= jn; q += 4) {
            double2 a0 = a[q * lda], a1 = a[(q + 1) * lda], a2 = a[(q + 2) * lda], a3 = a[(q + 3) * lda];
            cfma(acc, a0, xs[q]);
            cfma(acc, a1, xs[q + 1]);
            cfma(acc, a2, xs[q + 2]);
            cfma(acc, a3, xs[q + 3]);
        }
        for (; q < jn; ++q) cfma(acc, a[q * lda], xs[q]);
        part[(int64_t)blockIdx.y * m + i] = acc;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(&tickets[blockIdx.x], 1) == (int)gridDim.y - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (i < m) {
        double2 s = make_double2(0, 0);
        for (int c = 0; c < (int)gridDim.y; ++c) s = cadd(s, part[(int64_t)c * m + i]);
        double2 v = cmul(alpha, s);
        if (beta.x != 0.0 || beta.y != 0.0) cfma(v, beta, y[i]);
        y[i] = v;
    }
    if (threadIdx.x == 0) tickets[blockIdx.x] = 0;  // reset for the next launch
}

void gemv_fp64(Context& ctx, int64_t m, int64_t n, const double2* A, int64_t lda, const double2* x, double2* y,
               cd alpha, cd beta) {
    unsigned rb = (unsigned)((m + GV_ROWS - 1) / GV_ROWS), cb = (unsigned)((n + GV_COLS - 1) / GV_COLS);
    ctx.w_small.ensure(sizeof(double2) * (size_t)cb * m + 4096 * sizeof(int));
    // tickets live after the partials; zeroed once and reset by the kernel
    static_assert(sizeof(int) == 4, "");
    double2* part = ctx.w_small.as<double2>();
    int* tickets = reinterpret_cast<int*>(part + (size_t)cb * m);
    require(rb <= 4096, "gemv: too many row blocks");
    BEM_CUDA(cudaMemsetAsync(tickets, 0, sizeof(int) * rb, ctx.stream));
    dim3 grid(rb, cb);
    gemv64_kernel<<<grid, GV_ROWS, 0, ctx.stream>>>(m, n, A, lda, x, y, make_double2(alpha.re, alpha.im),
                                                    make_double2(beta.re, beta.im), part, tickets);
    BEM_CHECK_LAUNCH(&ctx);
}

// ---------------------------------------------------------------------------
__global__ void frob64_kernel(int64_t m, int64_t n, const double2* __restrict__ A, int64_t lda,
                              double* __restrict__ part) {
    __shared__ double red[256];
    double s = 0;
    int64_t total = m * n;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t j = t / m, i = t - j * m;
        double2 v = A[j * lda + i];
        s += v.x * v.x + v.y * v.y;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

double frob_norm_fp64(Context& ctx, int64_t m, int64_t n, const double2* A, int64_t lda) {
    const int nb = 1024;
    DevBuf d;
    d.ensure(sizeof(double) * nb);
    frob64_kernel<<<nb, 256, 0, ctx.stream>>>(m, n, A, lda, d.as<double>());
    BEM_CHECK_LAUNCH(&ctx);
    std::vector<double> h(nb);
    BEM_CUDA(cudaMemcpyAsync(h.data(), d.p, sizeof(double) * nb, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    double s = 0;
    for (double v : h) s += v;
    return std::sqrt(s);
}

}  // namespace bem
