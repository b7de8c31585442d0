// FP64 GEMM for the SCF's small dense matrices (n x n with n of a few hundred).
//
// At n = 200 cuBLAS' DGEMM takes ~60 us: its tiles are large enough that the
// product runs on a few dozen SMs, and FP64 is only ~2 FMAs per cycle per SM on
// this GPU.  Here a block owns an 8 x 8 tile of C and stages its 8 rows of op(A)
// and 8 columns of op(B) whole in shared memory (stride k + 1, so the dot
// products read without bank conflicts), which spreads a 200 x 200 product over
// 625 blocks and every SM.  Each output's dot product is split into two k-halves
// (128 threads, one warp per sub-partition: a warp-wide FP64 FMA holds its
// sub-partition's FP64 pipe ~64 cycles, and 64-thread blocks left two of an SM's
// four pipes with the work).  Flags tell it which operand is triangular (the k beyond
// are not visited) and whether the result is symmetric (one triangle is computed, both
// are written): X^T F X and X Y X^T with a triangular X take 3/8 of their dense work
// each.  Used for m, n, k <= 512; larger products go to
// cuBLAS.
#include "internal.h"

namespace hfgpu {

namespace {

constexpr int GS_T = 8;
constexpr int GS_MAX = 512;

constexpr int GS_KS = 2;  // k-slices per output
constexpr int GS_THREADS = GS_T * GS_T * GS_KS;

template <bool TA, bool TB>
__global__ void __launch_bounds__(GS_THREADS) gemm_small_kernel(int m, int n, int k, double alpha,
                                                                const double* __restrict__ A, int lda,
                                                                const double* __restrict__ B, int ldb, double beta,
                                                                double* C, int ldc, int flags)
{
    extern __shared__ double gs_sh[];
    const int ld = k + 1;
    double* As = gs_sh;            // row r of op(A): As[r * ld + kk]
    double* Bs = gs_sh + GS_T * ld;  // column c of op(B): Bs[c * ld + kk]
    double* part = Bs + GS_T * ld;   // partial sums of the second k-half
    const int i0 = blockIdx.x * GS_T, j0 = blockIdx.y * GS_T;
    const int t = threadIdx.x;
    if ((flags & GEMM_SYMMETRIC) && j0 < i0) return;  // the mirrored tile writes this one
    // the k that meet non-zeros of a triangular operand
    const int lo = max((flags & GEMM_K_GE_I) ? i0 : 0, (flags & GEMM_K_GE_J) ? j0 : 0);
    const int hi = min(k, min((flags & GEMM_K_LE_I) ? i0 + GS_T : k, (flags & GEMM_K_LE_J) ? j0 + GS_T : k));
    const int kr = max(hi - lo, 0);
    for (int e = t; e < GS_T * kr; e += GS_THREADS) {
        // consecutive threads take consecutive addresses of A and of B
        int r, ka;
        if (TA) { r = e / kr; ka = lo + e - r * kr; } else { r = e % GS_T; ka = lo + e / GS_T; }
        const int i = i0 + r;
        As[r * ld + ka] = i < m ? (TA ? A[ka + (size_t)i * lda] : A[i + (size_t)ka * lda]) : 0.0;
        int c, kb;
        if (TB) { c = e % GS_T; kb = lo + e / GS_T; } else { c = e / kr; kb = lo + e - c * kr; }
        const int j = j0 + c;
        Bs[c * ld + kb] = j < n ? (TB ? B[j + (size_t)kb * ldb] : B[kb + (size_t)j * ldb]) : 0.0;
    }
    __syncthreads();
    const int o = t % (GS_T * GS_T), h = t / (GS_T * GS_T);  // output, k-half
    const int r = o % GS_T, c = o / GS_T;
    const int i = i0 + r, j = j0 + c;
    const double* a = As + r * ld;
    const double* b = Bs + c * ld;
    const int kh = (kr + 1) / 2, k0 = lo + h * kh, k1 = h == 0 ? lo + kh : lo + kr;
    double s0 = 0.0, s1 = 0.0;  // two chains: half the FMA latency on the critical path
    int kk = k0;
    for (; kk + 1 < k1; kk += 2) {
        s0 = fma(a[kk], b[kk], s0);
        s1 = fma(a[kk + 1], b[kk + 1], s1);
    }
    if (kk < k1) s0 = fma(a[kk], b[kk], s0);
    if (h == 1) part[o] = s0 + s1;
    __syncthreads();
    if (h == 1 || i >= m || j >= n) return;
    const double acc = (s0 + s1) + part[o];
    double* cp = C + i + (size_t)j * ldc;
    const double v = beta == 0.0 ? alpha * acc : fma(alpha, acc, beta * *cp);
    if ((flags & GEMM_SYMMETRIC) && j0 == i0) {  // a diagonal tile: its upper half decides
        if (j < i) return;
    }
    *cp = v;
    if ((flags & GEMM_SYMMETRIC) && i != j) C[j + (size_t)i * ldc] = v;
}

template <bool TA, bool TB>
void launch_small(Context& ctx, int m, int n, int k, double alpha, const double* A, int lda, const double* B, int ldb,
                  double beta, double* C, int ldc, int flags)
{
    const size_t smem = (2 * (size_t)GS_T * (k + 1) + GS_T * GS_T) * sizeof(double);
    static std::once_flag once;
    std::call_once(once, [] {
        cudaFuncSetAttribute(gemm_small_kernel<TA, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)((2 * (size_t)GS_T * (GS_MAX + 1) + GS_T * GS_T) * sizeof(double)));
    });
    const dim3 grid((unsigned)((m + GS_T - 1) / GS_T), (unsigned)((n + GS_T - 1) / GS_T));
    gemm_small_kernel<TA, TB><<<grid, GS_THREADS, smem, ctx.stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, flags);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

}  // namespace

void gemm(Context& ctx, bool ta, bool tb, int m, int n, int k, double alpha, const double* A, int lda,
          const double* B, int ldb, double beta, double* C, int ldc, int flags)
{
    if (m <= 0 || n <= 0) return;
    if (k <= 0 || m > GS_MAX || n > GS_MAX || k > GS_MAX) {
        HF_CUBLAS(cublasDgemm(ctx.blas, ta ? CUBLAS_OP_T : CUBLAS_OP_N, tb ? CUBLAS_OP_T : CUBLAS_OP_N, m, n, k,
                              &alpha, A, lda, B, ldb, &beta, C, ldc));
        return;
    }
    if (ta && tb) launch_small<true, true>(ctx, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, flags);
    else if (ta) launch_small<true, false>(ctx, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, flags);
    else if (tb) launch_small<false, true>(ctx, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, flags);
    else launch_small<false, false>(ctx, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, flags);
}

}  // namespace hfgpu
