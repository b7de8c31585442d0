// Fock two-electron part G = J - K/2 from the packed integrals.
//
// Replaces formG/formG2 (src/scf.f90:26-58), G(i,j) = sum_kl P(k,l) TT(k,l,i,j)
// with TT(k,l,i,j) = (ij|kl) - (il|kj)/2, without the dense n^4 TT the
// reference precomputes (src/scf.f90:79-105): each unique integral of the
// 8-fold packed array is read once from HBM and scattered.
//
// For a unique v = (ij|kl), i>=j, k>=l, ij>=kl, let w = v f with
// f = 1/2 per coincidence (i==j, k==l, ij==kl).  Summing the integral's 8
// index permutations gives the half-matrix updates
//   Jh[i][j] += w P_kl,  Jh[k][l] += w P_ij,
//   Kh[i][k] += w P_jl,  Kh[j][k] += w P_il,  Kh[i][l] += w P_jk,  Kh[j][l] += w P_ik,
// J = 2 (Jh + Jh^T), K = Kh + Kh^T and G = J - K / 2.
// A warp walks one row ij of the packed matrix (contiguous kl, so consecutive l), and
// everything indexed by l has it as the fast index: the reads of P (from its transpose)
// and the updates, which may go to either of (a, b) and (b, a).  The row's Jh[i][j] term
// is reduced in the warp before one atomic.
// Bound: the FP64 pipe and the L2's atomics, about 7 FP64 instructions and 5 atomics an
// integral.  5 waters (125 functions) 0.85 -> 0.64 ms against the form with l as the slow
// index, J and K's factors on every term and atomicAdd; formG at 150 and 200 functions, with
// its copies, 7.1 and 18.5 -> 5.2 and 15.2 ms.
#include "internal.h"
#include "jk_blocks.cuh"

namespace hfgpu {

__global__ void __launch_bounds__(256) jk_packed_kernel(int n, int64_t m, const double* __restrict__ ints,
                                                        const double* __restrict__ P, const double* __restrict__ Pt,
                                                        const int2* __restrict__ pairs, double* Jh, double* Kh)
{
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t ij = warp; ij < m; ij += nwarps) {
        const int2 pij = pairs[ij];
        const int i = pij.x, j = pij.y;
        const int64_t in = (int64_t)i * n, jn = (int64_t)j * n;
        const double fij = (i == j) ? 0.5 : 1.0;
        const double Pij = P[i + jn] * fij;
        const double* row = ints + ij * (ij + 1) / 2;
        double gij = 0.0;
        for (int kl = lane; kl <= (int)ij; kl += 32) {
            const double v = row[kl];
            // screened-out quartets contribute nothing (integer test: keeps the FP64 pipe free)
            if (!digest_nonzero(v)) continue;
            const int2 pkl = pairs[kl];
            const int k = pkl.x, l = pkl.y;
            const int64_t kn = (int64_t)k * n;
            double w = v;  // without fij, which J_kl has in Pij and the row sum gets at the end
            if (k == l) w *= 0.5;
            if (kl == (int)ij) w *= 0.5;
            gij = fma(w, Pt[l + kn], gij);
            red_add(&Jh[l + kn], w * Pij);
            if (i == j) w *= 0.5;
            red_add(&Kh[k + in], w * Pt[l + jn]);
            red_add(&Kh[k + jn], w * Pt[l + in]);
            red_add(&Kh[l + in], w * P[j + kn]);
            red_add(&Kh[l + jn], w * P[i + kn]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) gij += __shfl_xor_sync(0xffffffffu, gij, o);
        if (lane == 0) red_add(&Jh[i + jn], fij * gij);
    }
}

// Pt = P^T, and both half matrices zero
__global__ void jk_start_kernel(int n, const double* __restrict__ P, double* Pt, double* Jh, double* Kh)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n * n) return;
    const int i = idx % n, j = idx / n;
    Pt[idx] = P[j + (int64_t)i * n];
    Jh[idx] = Kh[idx] = 0.0;
}

// J and K (G null), or G = J - K / 2, from the half matrices
__global__ void jk_finish_kernel(int n, const double* __restrict__ Jh, const double* __restrict__ Kh, double* J,
                                 double* K, double* G)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n * n) return;
    const int i = idx % n, j = idx / n;
    const double jj = 2.0 * (Jh[idx] + Jh[j + (int64_t)i * n]), kk = Kh[idx] + Kh[j + (int64_t)i * n];
    if (G) {
        G[idx] = fma(-0.5, kk, jj);
    } else {
        J[idx] = jj;
        K[idx] = kk;
    }
}

struct PairTable {
    int n = -1;
    DBuf<int2> d;
};

static const int2* pair_table(Context& ctx, int n)
{
    static thread_local PairTable tab;
    if (tab.n != n || tab.d.st != ctx.stream) {
        std::vector<int2> h((size_t)n * (n + 1) / 2);
        for (int i = 0; i < n; i++)
            for (int j = 0; j <= i; j++) h[(size_t)i * (i + 1) / 2 + j] = make_int2(i, j);
        tab.d = to_device(h, ctx.stream);
        tab.n = n;
    }
    return tab.d.p;
}

static void jk_packed(Context& ctx, int n, const double* d_int2, const double* dP, double* dJ, double* dK, double* dG)
{
    const int2* pairs = pair_table(ctx, n);
    const int64_t m = (int64_t)n * (n + 1) / 2, nn = (int64_t)n * n;
    HF_CHECK(m < (1ll << 31) && nn < (1ll << 31), HFGPU_ERR_UNSUPPORTED, "basis too large for 32-bit pair indices");
    DBuf<double> work(3 * nn, ctx.stream);
    double *Jh = work.p, *Kh = Jh + nn, *Pt = Kh + nn;
    const unsigned cover = (unsigned)((nn + 255) / 256);
    jk_start_kernel<<<cover, 256, 0, ctx.stream>>>(n, dP, Pt, Jh, Kh);
    count_launch();
    const int blocks = (int)std::min<int64_t>((m + 7) / 8, (int64_t)ctx.num_sms * 16);
    jk_packed_kernel<<<blocks, 256, 0, ctx.stream>>>(n, m, d_int2, dP, Pt, pairs, Jh, Kh);
    count_launch();
    HF_CUDA(cudaGetLastError());
    jk_finish_kernel<<<cover, 256, 0, ctx.stream>>>(n, Jh, Kh, dJ, dK, dG);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

void jk_separate_from_packed(Context& ctx, int n, const double* d_int2, const double* dP, double* dJ, double* dK)
{
    jk_packed(ctx, n, d_int2, dP, dJ, dK, nullptr);
}

void jk_from_packed(Context& ctx, int n, const double* d_int2, const double* dP, double* dG)
{
    cudaEvent_t e0, e1;
    HF_CUDA(cudaEventCreate(&e0));
    HF_CUDA(cudaEventCreate(&e1));
    HF_CUDA(cudaEventRecord(e0, ctx.stream));
    jk_packed(ctx, n, d_int2, dP, nullptr, nullptr, dG);
    HF_CUDA(cudaEventRecord(e1, ctx.stream));
    HF_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    HF_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    ctx.stat_fock_ms += ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
}

}  // namespace hfgpu
