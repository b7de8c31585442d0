// AO -> MO half transform on the tensor cores, and MBPT2 from it.
//
// The (ia|jb) that transform_int2 (src/mbpt.f90:11-79) feeds to term1
// (src/mbpt2.f90:8-31), ordered as a half transform so that every contraction is one
// "tall A times coefficient block" GEMM in the exact bf16-sliced form of tcgemm.cu
// (FP64 inputs and outputs; six digits for the mixed-precision path, nine for the
// plain FP64 one):
//   1. Y[p][j][la]  = sum_si (mu nu|la si) C1[si, j]     p = pair(mu >= nu)
//   2. Z[p][j][b]   = sum_la Y[p][j][la] C2[la, b]
//   3. W[q][i][mu]  = sum_nu Z[pair(mu, nu)][q] C1[nu, i]    q = (j, b)
//   4. T[q][i][a]   = sum_mu W[q][i][mu] C2[mu, a]       T[j][b][i][a] = (ia|jb)
// The rows of A are gathered where they lie (the packed integrals, Z transposed, Y and
// W) and cut inside the GEMM.  Steps 1-2 run over blocks of pairs and steps 3-4 over
// blocks of q, so Y and W stay within a fixed device-memory budget.
#include <algorithm>
#include <vector>

#include "internal.h"
#include "scf.h"
#include "tcgemm.h"

namespace hfgpu {

static const int64_t BLOCK_ROWS = 1 << 20;  // GEMM rows of a block

// out[c][r] = in[r][c] for a rows x cols row-major matrix: 32 x 32 tiles through shared
// memory, both sides coalesced, a thread's loads in flight together.  Bound: DRAM (16
// waters, 80200 x 25600, 32.8 GB both ways: 5.2 -> 4.9 ms of 4.8 at copy speed; tiles
// of 64 6.4).
constexpr int TP_T = 32;
__global__ void __launch_bounds__(256) transpose_kernel(const double* __restrict__ in, int64_t rows, int64_t cols,
                                                        double* __restrict__ out)
{
    __shared__ double t[TP_T][TP_T + 1];
    const int64_t c0 = (int64_t)blockIdx.x * TP_T, r0 = (int64_t)blockIdx.y * TP_T;
    const int x = threadIdx.x % TP_T, y0 = threadIdx.x / TP_T;
    constexpr int DY = 256 / TP_T;
    double v[TP_T / DY];
#pragma unroll
    for (int k = 0; k < TP_T / DY; ++k) {
        const int64_t r = r0 + y0 + k * DY, c = c0 + x;
        v[k] = r < rows && c < cols ? __ldcs(in + r * cols + c) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < TP_T / DY; ++k) t[y0 + k * DY][x] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TP_T / DY; ++k) {
        const int y = y0 + k * DY;
        const int64_t c = c0 + y, r = r0 + x;
        if (r < rows && c < cols) out[c * rows + r] = t[x][y];
    }
}

void transpose_device(Context& ctx, const double* in, int64_t rows, int64_t cols, double* out)
{
    const dim3 grid((unsigned)((cols + TP_T - 1) / TP_T), (unsigned)((rows + TP_T - 1) / TP_T));
    transpose_kernel<<<grid, 256, 0, ctx.stream>>>(in, rows, cols, out);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

void ao2mo_sliced(Context& ctx, int n, const double* d_int2, const double* C1, int n1, const double* C2, int n2,
                  int digits, double* T)
{
    cudaStream_t st = ctx.stream;
    SlicedRun run(ctx);
    const int64_t npair = (int64_t)n * (n + 1) / 2, nq = (int64_t)n1 * n2;
    Sliced B1, B2;
    slice_dense(ctx, C1, n1, n, n, digits, B1);  // rows of B^T = columns of C1
    slice_dense(ctx, C2, n2, n, n, digits, B2);
    ctx.trace_mark("mp2 slice C");
    // row maxima of the gathered rows (the exponents of their digits), by coalesced
    // passes instead of a second gather inside the GEMM
    const int64_t pb = std::min(npair, std::max<int64_t>(8, BLOCK_ROWS / n / 8 * 8));
    const int64_t qb = std::min(nq, std::max<int64_t>(1, BLOCK_ROWS / std::max(n, n1)));
    DBuf<unsigned> rmax((size_t)std::max(npair, qb) * n, st), dmax((size_t)std::max(pb, qb) * n1, st);
    packed_row_max(ctx, d_int2, n, rmax.p);
    ctx.trace_mark("mp2 row max");
    DBuf<double> Z((size_t)npair * nq, st);
    {
        DBuf<double> Y((size_t)pb * n1 * n, st);
        for (int64_t p0 = 0; p0 < npair; p0 += pb) {
            const int64_t np = std::min(pb, npair - p0);
            sliced_gemm_packed(ctx, d_int2, p0, np, n, rmax.p, B1, Y.p, OutMap{n, n1});
            ctx.trace_mark("mp2 step 1");
            dense_row_max(ctx, Y.p, np * n1, n, n, dmax.p);
            sliced_gemm_dense(ctx, Y.p, np * n1, n, n, dmax.p, B2, Z.p + p0 * nq, OutMap{0, n2});
            ctx.trace_mark("mp2 step 2");
        }
    }
    // Z^T: one contiguous row of pairs per q, so that the (q, mu) rows of step 3
    // gather from one L2-resident row instead of one cache line per element
    DBuf<double> Zt((size_t)npair * nq, st);
    transpose_device(ctx, Z.p, npair, nq, Zt.p);
    Z.release();
    ctx.trace_mark("mp2 transpose");
    DBuf<double> W((size_t)qb * n1 * n, st);
    for (int64_t q0 = 0; q0 < nq; q0 += qb) {
        const int64_t nqb = std::min(qb, nq - q0);
        // rows (q, mu) over nu of Zt[q0 + q][pair(mu, nu)] -> W[q][i][mu]
        sympair_row_max(ctx, Zt.p + q0 * npair, npair, nqb, n, rmax.p);
        sliced_gemm_sympair(ctx, Zt.p + q0 * npair, npair, nqb, n, rmax.p, B1, W.p, OutMap{n, n1});
        ctx.trace_mark("mp2 step 3");
        // rows (q, i) -> T[q][i][a]
        dense_row_max(ctx, W.p, nqb * n1, n, n, dmax.p);
        sliced_gemm_dense(ctx, W.p, nqb * n1, n, n, dmax.p, B2, T + q0 * n1 * n2, OutMap{0, n2});
        ctx.trace_mark("mp2 step 4");
    }
    run.settle();
}

// one block per pair i >= j: sum_ab (ia|jb) [2 (ia|jb) - (ib|ja)] / (e_i + e_j - e_a - e_b)
// from T[j][b][i][a] (relative error of each term ~1e-14 from the refined reciprocal).
// For fixed (i, j) the v x v block X[b][a] = (ia|jb) has rows of consecutive a, and
// (ib|ja) = X[a][b] is its transpose: 32 x 32 tiles of X and of the mirrored tile are
// staged in shared memory with coalesced row reads.  (a, b) and (b, a) have one
// denominator, so tiles below the diagonal stand for both:
//   x (2x - y) + y (2y - x) = 2 ((x - y)^2 + x y).
// Bound: the FP64 pipe (9 instructions per two terms; 10 per term with each (a, b) on
// its own): 8 and 16 waters 0.52 and 6.5 -> 0.33 and 3.4 ms.
__global__ void __launch_bounds__(256) mp2_pair_energy_kernel(int o, int v, const double* __restrict__ T,
                                                             const double* __restrict__ eps, double* partial)
{
    __shared__ double A[32][33], B[32][33], eb[32];
    // block p = the pair i >= j (p = i (i + 1) / 2 + j): the (j, i) block holds the
    // same terms with a and b exchanged ((jb|ia) = (ia|jb)), so it counts twice
    const int p = blockIdx.x;
    int i = (int)((sqrtf(8.0f * (float)p + 1.0f) - 1.0f) * 0.5f);
    while (i * (i + 1) / 2 > p) --i;
    while ((i + 1) * (i + 2) / 2 <= p) ++i;
    const int j = p - i * (i + 1) / 2;
    const double eij = eps[i] + eps[j];
    const int64_t rs = (int64_t)o * v;  // stride between consecutive b (rows of X)
    const double* X = T + ((int64_t)j * v * o + i) * v;  // X[b][a] = X[b * rs + a]
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    double s_diag = 0.0, s_off = 0.0;
    for (int b0 = 0; b0 < v; b0 += 32)
        for (int a0 = 0; a0 <= b0; a0 += 32) {
            const bool off = a0 != b0;
            double va[4], vb[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = ty + 8 * k, b = b0 + r, a = a0 + tx, bb = a0 + r, aa = b0 + tx;
                va[k] = (b < v && a < v) ? X[b * rs + a] : 0.0;            // X[b0 + r][a0 + tx]
                vb[k] = off && bb < v && aa < v ? X[bb * rs + aa] : va[k];  // X[a0 + r][b0 + tx]
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                A[ty + 8 * k][tx] = va[k];
                B[ty + 8 * k][tx] = vb[k];
            }
            if (ty == 0) eb[tx] = b0 + tx < v ? eps[o + b0 + tx] : 0.0;
            const double da = a0 + tx < v ? eij - eps[o + a0 + tx] : 0.0;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = ty + 8 * k;
                if (b0 + r < v && a0 + tx < v) {
                    const double x = A[r][tx], y = B[tx][r];  // (ia|jb), (ib|ja)
                    const double d = da - eb[r];
                    // 1/d: FP32 reciprocal (24 bits) and one Newton step in FP64
                    // (~48 bits), instead of an FP64 division on the narrow FP64 pipe
                    const double r0 = (double)__frcp_rn((float)d);
                    const double rd = r0 * fma(-d, r0, 2.0);
                    const double u = x - y;
                    if (off)
                        s_off = fma(fma(u, u, x * y), rd, s_off);
                    else
                        s_diag = fma(x * (x + u), rd, s_diag);
                }
            }
            __syncthreads();
        }
    const double s = fma(2.0, s_off, s_diag);
    __shared__ double sh[256];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if ((int)threadIdx.x < k) sh[threadIdx.x] += sh[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = (i == j ? 1.0 : 2.0) * sh[0];
}

double mp2_energy_mixed(Context& ctx, int n, const double* d_int2, const double* dC, int o, const double* d_eps)
{
    const int v = n - o;
    if (o <= 0 || v <= 0) return 0.0;
    DBuf<double> T((size_t)o * v * o * v, ctx.stream);
    HF_CHECK(n <= slice_kmax(SLICE_MIXED), HFGPU_ERR_UNSUPPORTED,
             "mixed-precision transform supports up to 512 functions");
    ao2mo_sliced(ctx, n, d_int2, dC, o, dC + (size_t)n * o, v, SLICE_MIXED, T.p);
    const int npairs = o * (o + 1) / 2;
    DBuf<double> part((size_t)npairs, ctx.stream);
    mp2_pair_energy_kernel<<<npairs, 256, 0, ctx.stream>>>(o, v, T.p, d_eps, part.p);
    count_launch();
    HF_CUDA(cudaGetLastError());
    std::vector<double> h((size_t)npairs);
    part.download(h.data(), h.size());
    HF_CUDA(cudaStreamSynchronize(ctx.stream));
    double E = 0;
    for (double x : h) E += x;
    return E;
}

}  // namespace hfgpu
