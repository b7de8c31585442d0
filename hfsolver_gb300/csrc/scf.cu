// Closed-shell RHF SCF loop on the GPU.
//
// Follows doscf (src/scf.f90:72-136): P = 0 start, F = H + G(P),
// E0 = sum P (H + F) / 2, generalised eigenproblem F C = S C lam solved with
// the same LAPACK routine the reference calls (dsygvd, lower triangle,
// src/linalg.f90:241-280; here cuSOLVER's device implementation),
// P = 2 C_occ C_occ^T (formP, :12-24), dP = sqrt(sum (P - Pold)^2 / 4),
// convergence from the 4th iteration when dP < tolP and the last four energies
// span less than tolE, otherwise linear mixing P = (1-alpha) Pold + alpha P.
// Optionally Pulay's DIIS (commutator error F P S - S P F) extrapolates F
// instead of mixing P.  Everything stays on the device; each iteration reads
// back two scalars (E0, dP) for the convergence test.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "internal.h"
#include "eigh.h"
#include "gridsync.cuh"
#include "scf.h"

namespace hfgpu {

// ---- the elementwise passes of an iteration, with their sums ----------------
// Every sum over n^2 elements: each block's part goes to partial[], and the block that
// finishes last adds them in block order (deterministic), writes the result and resets
// the counter for the next launch.  One block alone took 30 us for 400 functions.
constexpr int RED_BLOCK = 256, RED_MAX_BLOCKS = 128, RED_MAX = 20;  // RED_MAX sums at once
struct RedWork {
    double* partial;  // RED_MAX_BLOCKS x RED_MAX
    unsigned* count;
};

static unsigned red_blocks(int64_t nn)
{
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(RED_MAX_BLOCKS, (nn + 2 * RED_BLOCK - 1) / (2 * RED_BLOCK)));
}

// The block's sums of v[0 .. m) (m <= M) to partial; true in the last block to finish, with
// the totals over all blocks in tot[0 .. m) (shared memory).
template <int M>
__device__ bool grid_sums(const double (&v)[M], int m, const RedWork w, double* tot)
{
    __shared__ double sh[M][RED_BLOCK / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < M; ++k) {
        if (k >= m) break;
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) sh[k][warp] = x;
    }
    __syncthreads();
    if ((int)threadIdx.x < m) {
        double x = 0;
        for (int i = 0; i < RED_BLOCK / 32; ++i) x += sh[threadIdx.x][i];
        w.partial[blockIdx.x * RED_MAX + threadIdx.x] = x;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(w.count, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    for (int k = warp; k < m; k += RED_BLOCK / 32) {
        double x = 0;
        for (int i = lane; i < (int)gridDim.x; i += 32) x += __ldcg(w.partial + i * RED_MAX + k);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) tot[k] = x;
    }
    if (threadIdx.x == 0) *w.count = 0;
    __syncthreads();
    return true;
}

// what an iteration reports to the host, in one copy
struct Sp2Sync {
    unsigned count;
    int err, steps;
    double trace;  // tr X of the result
};
// the course of an FP64 purification from F: X_0 = shift I - scale F; dif = ||F - Fprev||_F
// where there is an Fprev; per step w = tr(X - X^2)
// and tr X before it, and its stretch alpha (negative: a 2X - X^2 step)
constexpr int SP2_LOG = 64;
struct Sp2Log {
    double scale, shift, dif, alpha[SP2_LOG];
    long long w[SP2_LOG], tr[SP2_LOG];  // in units of 2^-50
};
struct ScfReport {
    double E0, dP;
    Sp2Sync sp2[2];  // density purification: [0] FP32, [1] FP64
    Sp2Log log;
};

// F = H + G (with acc: G is added to the running acc first, F = H + acc), F's copy in the
// DIIS history, Pold = P, E0 = sum P (H + F) / 2; clears the purification's barriers
__global__ void __launch_bounds__(RED_BLOCK) fock_kernel(int64_t nn, const double* __restrict__ H,
                                                         const double* __restrict__ G, double* acc,
                                                         const double* __restrict__ P, double* __restrict__ F,
                                                         double* __restrict__ Fhist, double* __restrict__ Pold, RedWork w,
                                                         ScfReport* rep)
{
    __shared__ double tot[1];
    double s[1] = {0.0};
    for (int64_t i = (int64_t)blockIdx.x * RED_BLOCK + threadIdx.x; i < nn; i += (int64_t)gridDim.x * RED_BLOCK) {
        double g = G[i];
        if (acc) {
            g += acc[i];
            acc[i] = g;
        }
        const double h = H[i], f = h + g, p = P[i];
        F[i] = f;
        if (Fhist) Fhist[i] = f;
        Pold[i] = p;
        s[0] += p * (h + f);
    }
    if (grid_sums(s, 1, w, tot) && threadIdx.x == 0) {
        rep->E0 = 0.5 * tot[0];
        rep->sp2[0] = rep->sp2[1] = Sp2Sync{0u, 0, 0, 0.0};
    }
}

// D = P - Pold (the next incremental build's density), dP = sqrt(sum D^2 / 4)
__global__ void __launch_bounds__(RED_BLOCK) density_change_kernel(int64_t nn, const double* __restrict__ P,
                                                                   const double* __restrict__ Pold, double* D, RedWork w,
                                                                   ScfReport* rep)
{
    __shared__ double tot[1];
    double s[1] = {0.0};
    for (int64_t i = (int64_t)blockIdx.x * RED_BLOCK + threadIdx.x; i < nn; i += (int64_t)gridDim.x * RED_BLOCK) {
        const double d = P[i] - Pold[i];
        if (D) D[i] = d;
        s[0] += d * d;
    }
    if (grid_sums(s, 1, w, tot) && threadIdx.x == 0) rep->dP = sqrt(tot[0] / 4);
}

__global__ void __launch_bounds__(RED_BLOCK) dot_kernel(int64_t nn, const double* __restrict__ A,
                                                        const double* __restrict__ B, RedWork w, double* out)
{
    __shared__ double tot[1];
    double s[1] = {0.0};
    for (int64_t i = (int64_t)blockIdx.x * RED_BLOCK + threadIdx.x; i < nn; i += (int64_t)gridDim.x * RED_BLOCK)
        s[0] += A[i] * B[i];
    if (grid_sums(s, 1, w, tot) && threadIdx.x == 0) *out = tot[0];
}

// P = (1 - alpha) Pold + alpha P and D = P - Pold
__global__ void mix_kernel(int64_t nn, double alpha, const double* __restrict__ Pold, double* P, double* D)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const double p = (1 - alpha) * Pold[i] + alpha * P[i];
    P[i] = p;
    if (D) D[i] = p - Pold[i];
}

static unsigned nblk(int64_t n) { return (unsigned)((n + 255) / 256); }

// ---- density by purification (SP2, Niklasson, Phys. Rev. B 66, 155115 (2002)) ----
// Gershgorin bounds of a symmetric matrix: b[0] <= lowest, b[1] >= highest eigenvalue.
// One warp per column (the matrix is symmetric, so column sums are row sums):
// coalesced reads, shuffle sums.
__global__ void gersh_kernel(int n, const double* __restrict__ A, double* b)
{
    __shared__ double lo[32], hi[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double l = 1e300, h = -1e300;
    for (int i = warp; i < n; i += nw) {
        const double* col = A + (int64_t)i * n;
        double r = 0;
        for (int j = lane; j < n; j += 32)
            if (j != i) r += fabs(col[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        const double d = col[i];
        l = fmin(l, d - r);
        h = fmax(h, d + r);
    }
    if (lane == 0) {
        lo[warp] = l;
        hi[warp] = h;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < nw; ++w) {
            l = fmin(l, lo[w]);
            h = fmax(h, hi[w]);
        }
        b[0] = l;
        b[1] = h;
    }
}

// X2 = X X for symmetric X (n <= 1024), upper-triangle 16x16 tiles mirrored;
// the diagonal of X2 is added to trX2 (one SP2 step's tr X^2).
constexpr int SQ_T = 16;
__global__ void __launch_bounds__(SQ_T* SQ_T) sym_square_kernel(int n, const double* __restrict__ X, double* X2,
                                                                double* trX2)
{
    __shared__ double As[SQ_T][SQ_T + 1], Bs[SQ_T][SQ_T + 1];
    // blockIdx.x -> tile pair (ti <= tj), row-major over the upper triangle
    const int nt = (n + SQ_T - 1) / SQ_T;
    int b = blockIdx.x, ti = 0;
    while (b >= nt - ti) {
        b -= nt - ti;
        ++ti;
    }
    const int tj = ti + b;
    const int ty = threadIdx.x / SQ_T, tx = threadIdx.x % SQ_T;
    const int i = ti * SQ_T + ty, j = tj * SQ_T + tx;
    double acc = 0.0;
    for (int k0 = 0; k0 < n; k0 += SQ_T) {
        const int ka = k0 + tx, kb = k0 + ty;
        As[ty][tx] = (i < n && ka < n) ? X[i + (int64_t)ka * n] : 0.0;  // X[i][k]
        Bs[ty][tx] = (kb < n && j < n) ? X[kb + (int64_t)j * n] : 0.0;  // X[k][j]
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SQ_T; ++k) acc = fma(As[ty][k], Bs[k][tx], acc);
        __syncthreads();
    }
    if (i < n && j < n) {
        X2[i + (int64_t)j * n] = acc;
        if (ti != tj) X2[j + (int64_t)i * n] = acc;
        if (i == j) atomicAdd(trX2, acc);
    }
}

// The whole density purification of one Fock matrix as one cooperative launch: the
// spectral bounds, the initial iterate and the SP2 recursion, one block per tt x tt
// upper-triangle tile of the iterate, one grid barrier per step.
// what a block leaves for the others at a barrier: its share of tr X and ||X||_F^2 in
// units of 2^-50, or of the traces of F and its spectral bounds
struct __align__(16) Sp2Slot {
    long long a, c;
};
struct __align__(16) Sp2Bounds {
    double tr, nrm, lo, hi, dif, pad;
};
// The shares are summed as integers: a warp-wide FP64 add holds its sub-partition's pipe
// 64 cycles and a shuffle sum of two doubles takes a thousand, a third of a step.  (|X| <= 1
// and ||X||^2 <= n: sums below 2^60, each element within 2^-51.)
constexpr double SP2_UNIT = 1125899906842624.0;  // 2^50

enum { SP2_FROM_F = 0, SP2_FROM_F32 = 1 };

// Start: SP2_FROM_F: X_0 = (hi I - F) / (hi - lo), the spectrum of F mapped into [0, 1] by
// its Gershgorin bounds with the occupied states near 1 (the blocks share the rows of F
// and meet at one barrier; X_0 itself is never stored: step 0 maps F as it stages it);
// SP2_FROM_F32: X_0 is the FP32 result of an earlier coarse launch.
// A step: every block sums the others' shares of tr X_k and ||X_k||_F^2 = tr X_k^2 (X_k
// symmetric) in a fixed order, so all blocks take the same choice between X^2 and 2X - X^2
// and the same convergence decision; squares its tile from its tt rows and tt columns of
// X_k, staged whole in shared memory (stride n + 1: no bank conflicts); writes it with its
// shares and arrives at the barrier.  The iterate alternates between X0 and X1 and ends in
// X0.  T = float for the coarse steps of early SCF iterations.  The tile edge tt (8 .. 32)
// and the number of k-slices ks each output's dot product is split into (their partial
// sums meet in shared memory) are chosen so that the FP64 work spreads evenly over the SMs
// and over each SM's four sub-partitions (sp2_shape).
// Stretched steps: of an earlier F (Fprev) the last occupied energy is known to be at most
// homo and the first virtual one at least lumo (sp2_gap); F's are within ||F - Fprev||_F
// of them.  With the virtual states' X in [0, l] and the occupied ones' in [1 - m, 1], the
// square of a X + (1 - a) I, a = 2 / (2 - l), maps 0 and l to the same (l / (2 - l))^2
// where X^2 leaves l^2, and keeps the order and [0, 1]; I - (I - a X)^2, a = 2 / (2 - m),
// does the same for the holes.  The larger of l and m is taken until both are below
// SP2_STRETCH; the plain recursion ends the work.  l, m and a are one thread's work while
// the block waits at the barrier.  (Rubensson, J. Chem. Theory Comput. 7, 1233 (2011).)
// Steps of a density: 28 plain and 19 stretched (1 water, from the eleventh of 48
// iterations on), 30 and 19 (6 waters), 31 and 18 (16 waters); all FP64 purifications of an
// SCF of 1, 6, 9 and 16 waters 5.8, 9.9, 20.0 and 23.4 ms plain, 4.9, 8.8, 17.3 and 17.1 so.
// Once tr(X - X^2) < tol_idem the recursion takes `polish` (0 or 2) more steps, one
// square and one 2X - X^2: an occupation 1 - d goes to 1 - 2d and 1 - 4d^2 (or 1 - d^2
// and 1 - 2d^2), one at d to the mirror image, so a sum of 1e-7 left by the test ends
// at 4e-14, the rounding of the sum, on both sides.
// Bound: the FP64 pipe at a few hundred functions, the latency of a step below: one
// barrier and one round of L2 loads (shares and tiles together); every warp-wide FP64
// instruction outside the dot products (sums, tests) lengthens it by 64 cycles.  Per
// purification of 28 steps, with the bounds and X_0 in a chain of small kernels before:
// 25 functions 0.154 -> 0.11 ms, 50: 0.20 -> 0.14, 150: 0.54 -> 0.38; the 17 densities of
// an 8-water SCF (8 of them FP32 first) 7.4 -> 5.3 ms, the 18 of 16 waters 31.3 -> 26.7 (all
// steps plain).
// x^2 in units of 2^-50: the scale goes to x's exponent (|x| < 2^-900 counts as zero)
__device__ __forceinline__ long long square_fixed(double x)
{
    const int hi = __double2hiint(x);
    const double y = (hi & 0x7FF00000) < (123 << 20) ? 0.0 : __hiloint2double(hi + (25 << 20), __double2loint(x));
    return __double2ll_rn(y * y);
}

constexpr double SP2_STRETCH = 0.02;  // (0.1: a step more at times; below, a is 1.01 and less)

template <typename T, int FROM>
__global__ void __launch_bounds__(1024) sp2_kernel(int n, int nocc, int tt, int ks, const void* src, T* X0, T* X1,
                                                   Sp2Slot* slots, int maxs, double tol_idem, double tol_n, int polish,
                                                   Sp2Sync* sync, const double* Fprev, double homo, double lumo,
                                                   Sp2Log* log)
{
    extern __shared__ __align__(16) unsigned char sp2_smem[];
    __shared__ long long red[2][32];
    __shared__ double rb[5][32], tot[4];
    __shared__ long long s_trace, s_w;
    __shared__ int s_go, s_conv, s_square;
    __shared__ int s_stretch;      // this step: 0 plain, 1 stretched square, 2 stretched 2X - X^2
    __shared__ double s_alpha[4];  // its a, and the factors of X^2, X and I
    const int ld = n + 1, nblk = gridDim.x;
    T* Ar = (T*)sp2_smem;    // rows i0 .. i0+tt-1 of X_k, all k
    T* Bc = Ar + tt * ld;    // columns j0 .. j0+tt-1 (rows by symmetry)
    T* part = Bc + tt * ld;  // partial dot products of k-slices 1 .. ks-1
    const int nt = (n + tt - 1) / tt;
    int b = blockIdx.x, ti = 0;
    while (b >= nt - ti) {
        b -= nt - ti;
        ++ti;
    }
    const int tj = ti + b;
    const int i0 = ti * tt, j0 = tj * tt;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // ks x tt x tt workers: output (ty, tx) of k-slice `slice`; the block is rounded up to
    // whole warps
    const int outs = tt * tt;
    const bool worker = (int)threadIdx.x < ks * outs;
    const int slice = (int)threadIdx.x / outs, o = (int)threadIdx.x - slice * outs;
    const int ty = o / tt, tx = o % tt;
    const int i = i0 + ty, j = j0 + tx;
    const int kc = (n + ks - 1) / ks, k0 = slice * kc, k1 = min(n, k0 + kc);
    const bool own = worker && slice == 0 && i < n && j < n;

    // this thread's place in the staging of a panel, and its stride
    const int st_r = (int)threadIdx.x % tt, st_k = (int)threadIdx.x / tt;
    const int st_dr = (int)blockDim.x % tt, st_dk = (int)blockDim.x / tt;
    auto fixed = [](double x) { return __double2ll_rn(x * SP2_UNIT); };
    Sp2Bounds* bounds = reinterpret_cast<Sp2Bounds*>(slots + 2 * nblk);
    // arrive at barrier number `epoch` (thread 0, after the block's writes); false after a timeout
    auto barrier = [&](unsigned epoch) {
        if (threadIdx.x == 0) s_go = grid_arrive_wait(&sync->count, &sync->err, (unsigned)nblk, epoch);
        __syncthreads();
        return s_go != 0;
    };
    // the next step's stretch from l and m, which go on to the step's results (one thread).
    // a in single precision, l and m for the a taken; non-negative doubles compare as integers
    double l = 0.0, m = 0.0;
    auto stretch = [&] {
        int k = 0;
        const long long li = __double_as_longlong(l), mi = __double_as_longlong(m);
        if (max(li, mi) > __double_as_longlong(SP2_STRETCH)) {
            k = li >= mi ? 1 : 2;
            const double x = k == 1 ? l : m, y = k == 1 ? m : l;
            const double a = (double)__fdividef(2.0f, 2.0f - (float)x);
            const double q = 1.0 - a, p = fma(a, x, q), r = fma(-a, y, 1.0);
            s_alpha[0] = a;
            s_alpha[1] = k == 1 ? a * a : -a * a;
            s_alpha[2] = (k == 1 ? q : 1.0) * (a + a);
            const double qq = q * q, pp = p * p, small = fma(-r, r, 1.0);
            s_alpha[3] = k == 1 ? qq : 0.0;
            const double big = __double_as_longlong(qq) > __double_as_longlong(pp) ? qq : pp;
            l = k == 1 ? big : small;
            m = k == 1 ? small : big;
        }
        s_stretch = k;
    };
    const bool planner = threadIdx.x == blockDim.x - 1;  // (not of warp 0: the block has two at least)
    // the block's share of the traces into its slot of set `set`, then the barrier
    auto share = [&](long long a, long long c, int set, unsigned epoch) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, d);
            c += __shfl_xor_sync(0xffffffffu, c, d);
        }
        if (lane == 0) {
            red[0][warp] = a;
            red[1][warp] = c;
        }
        __syncthreads();  // (and every thread's part of X is written)
        if (threadIdx.x == 0) {
            for (int w = 1; w < nw; ++w) {
                a += red[0][w];
                c += red[1][w];
            }
            slots[set * nblk + blockIdx.x] = Sp2Slot{a, c};
        }
        if (planner) stretch();
        return barrier(epoch);
    };
    // What step `it` does, from tr X and ||X||^2 in units of 2^-50 (one thread, in integers:
    // every FP64 compare would cost all warps 64 cycles each)
    const long long N = (long long)nocc << 50, tol_i = fixed(tol_idem), tol_t = fixed(tol_n);
    auto decide = [&](long long a, long long c) {
        s_trace = a;
        s_w = a - c;
        s_conv = llabs(a - c) < tol_i && llabs(a - N) < tol_t;
        s_square = llabs(c - N) <= llabs(2 * a - c - N);
    };
    // the sums over all slots of set `set` and the decision, by warp 0; ready after the next
    // __syncthreads
    auto gather = [&](int set) {
        if (warp == 0) {
            long long a = 0, c = 0;
            for (int s = lane; s < nblk; s += 32) {
                const longlong2 u = __ldcg(reinterpret_cast<const longlong2*>(slots + set * nblk + s));
                a += u.x;
                c += u.y;
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                a += __shfl_xor_sync(0xffffffffu, a, d);
                c += __shfl_xor_sync(0xffffffffu, c, d);
            }
            if (lane == 0) decide(a, c);
        }
    };

    unsigned epoch = 0;
    double scale = 0.0, shift = 0.0;  // X_0 = shift I - scale F
    if (FROM == SP2_FROM_F) {
        const double* F = (const double*)src;
        double tr = 0, nrm = 0, lo = 1e300, hi = -1e300, dif = 0;
        for (int r = (int)blockIdx.x * nw + warp; r < n; r += nblk * nw) {  // one warp per row (column: F is symmetric)
            double s = 0, q = 0;
            for (int k = lane; k < n; k += 32) {
                const double f = F[k + (int64_t)r * n];
                s += fabs(f);
                q = fma(f, f, q);
                if (Fprev) {
                    const double d = f - Fprev[k + (int64_t)r * n];
                    dif = fma(d, d, dif);
                }
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                s += __shfl_xor_sync(0xffffffffu, s, d);
                q += __shfl_xor_sync(0xffffffffu, q, d);
            }
            const double f = F[r + (int64_t)r * n], rad = s - fabs(f);
            lo = fmin(lo, f - rad);
            hi = fmax(hi, f + rad);
            if (lane == 0) {
                tr += f;
                nrm += q;
            }
        }
        if (Fprev)
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) dif += __shfl_xor_sync(0xffffffffu, dif, d);
        if (lane == 0) {
            rb[4][warp] = dif;
            rb[0][warp] = tr;
            rb[1][warp] = nrm;
            rb[2][warp] = lo;
            rb[3][warp] = hi;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < nw; ++w) {
                tr += rb[0][w];
                nrm += rb[1][w];
                lo = fmin(lo, rb[2][w]);
                hi = fmax(hi, rb[3][w]);
                dif += rb[4][w];
            }
            bounds[blockIdx.x] = Sp2Bounds{tr, nrm, lo, hi, dif, 0.0};
        }
        if (!barrier(++epoch)) return;
        if (warp == 0) {
            tr = nrm = dif = 0;
            lo = 1e300, hi = -1e300;
            for (int s = lane; s < nblk; s += 32) {
                const double2* p = reinterpret_cast<const double2*>(bounds + s);
                const double2 u = __ldcg(p), v = __ldcg(p + 1);
                if (Fprev) dif += __ldcg(p + 2).x;
                tr += u.x;
                nrm += u.y;
                lo = fmin(lo, v.x);
                hi = fmax(hi, v.y);
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                tr += __shfl_xor_sync(0xffffffffu, tr, d);
                nrm += __shfl_xor_sync(0xffffffffu, nrm, d);
                lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, d));
                hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, d));
                if (Fprev) dif += __shfl_xor_sync(0xffffffffu, dif, d);
            }
            if (lane == 0) {  // X_0 = shift I - scale F, its trace and squared norm
                const double sc = 1.0 / (hi - lo), sf = hi * sc;
                decide(fixed(n * sf - sc * tr), fixed(n * sf * sf - 2.0 * sf * sc * tr + sc * sc * nrm));
                tot[0] = sc;
                tot[1] = sf;
                tot[2] = tot[3] = 0.0;
                if (Fprev) {
                    const double e = sqrt(dif);
                    const double l0 = fmax(sf - sc * (lumo - e), 0.0), m0 = fmax(1.0 - sf + sc * (homo + e), 0.0);
                    if (l0 + m0 < 1.0) {  // (also false for NaN)
                        tot[2] = l0;
                        tot[3] = m0;
                    }
                }
                if (log && blockIdx.x == 0) {
                    log->scale = sc;
                    log->shift = sf;
                    log->dif = sqrt(dif);
                }
            }
        }
        __syncthreads();
        scale = tot[0];
        shift = tot[1];
        if (planner) {
            l = tot[2];
            m = tot[3];
            stretch();  // (read after the first panels' __syncthreads)
        }
    } else {
        long long tr = 0, nrm = 0;
        const float* S = (const float*)src;
        if (own) {
            const double x = (double)S[i + (int64_t)j * n];
            if (i == j) tr = fixed(x);
            nrm = square_fixed(x) << (ti != tj ? 1 : 0);
        }
        if (!share(tr, nrm, 0, ++epoch)) return;
        gather(0);
    }

    int left = -1;  // polishing steps still to do (-1: not converged yet)
    bool last_square = false;
    for (int it = 0; it < maxs; ++it) {
        T* Xc = (it & 1) ? X1 : X0;
        T* Xn = (it & 1) ? X0 : X1;
        if (it > 0) gather(it & 1);
        // U elements of each panel in flight per thread: one at a time, a step at 150
        // functions (four warps a block) spent 8 us here; r fastest: tt consecutive elements
        // of a column
        constexpr int U = 6;
        for (int r = st_r, k = st_k; k < n;) {
            T x[U], y[U];
            int rr[U], kk[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                rr[u] = r;
                kk[u] = k;
                x[u] = y[u] = T(0);
                if (k < n) {
                    const int a = i0 + r, c = j0 + r;
                    if (it == 0 && FROM == SP2_FROM_F) {
                        const double* F = (const double*)src;
                        if (a < n) x[u] = (T)((a == k ? shift : 0.0) - scale * F[a + k * n]);
                        if (c < n) y[u] = (T)((c == k ? shift : 0.0) - scale * F[c + k * n]);
                    } else if (it == 0) {
                        const float* S = (const float*)src;
                        if (a < n) x[u] = (T)S[a + k * n];
                        if (c < n) y[u] = (T)S[c + k * n];
                    } else {
                        if (a < n) x[u] = __ldcg(Xc + a + k * n);
                        if (c < n) y[u] = __ldcg(Xc + c + k * n);
                    }
                }
                r += st_dr;
                k += st_dk;
                if (r >= tt) {
                    r -= tt;
                    ++k;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (kk[u] < n) {
                    Ar[rr[u] * ld + kk[u]] = x[u];
                    Bc[rr[u] * ld + kk[u]] = y[u];
                }
        }
        __syncthreads();
        const bool conv = s_conv != 0, sq = s_square != 0;
        if (left < 0 && conv) left = polish;
        if (left == 0) {
            if (own && ((it & 1) || it == 0)) {  // X_k is in X1, or was never stored: this block's tile to X0
                X0[i + (int64_t)j * n] = Ar[ty * ld + j];
                if (ti != tj) X0[j + (int64_t)i * n] = Ar[ty * ld + j];
            }
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                sync->steps = it;
                sync->trace = (double)s_trace * (1.0 / SP2_UNIT);
            }
            return;
        }
        const int st = left < 0 ? s_stretch : 0;
        // the last of the polishing steps is the opposite of the one before it
        const bool square = st ? st == 1 : left == 1 ? !last_square : sq;
        if (log && blockIdx.x == 0 && threadIdx.x == 0 && it < SP2_LOG) {
            const double a = st ? s_alpha[0] : 1.0;
            log->w[it] = s_w;
            log->tr[it] = s_trace;
            log->alpha[it] = square ? a : -a;
        }
        last_square = square;
        if (left > 0) --left;
        T acc = 0;
        if (worker) {
            const T* ar = Ar + ty * ld;
            const T* bc = Bc + tx * ld;
            for (int k = k0; k < k1; ++k) acc = fma(ar[k], bc[k], acc);
            if (slice > 0) part[(slice - 1) * outs + o] = acc;
        }
        if (ks > 1) {
            __syncthreads();
            if (worker && slice == 0)
                for (int q = 1; q < ks; ++q) acc += part[(q - 1) * outs + o];
        }
        long long pt = 0, pn = 0;
        if (own) {
            const T y = Ar[ty * ld + j];
            const T x = st ? (T)fma(s_alpha[1], (double)acc, fma(s_alpha[2], (double)y, i == j ? s_alpha[3] : 0.0))
                           : square ? acc : T(2) * y - acc;
            Xn[i + (int64_t)j * n] = x;
            if (ti != tj) Xn[j + (int64_t)i * n] = x;
            if (i == j) pt = fixed((double)x);
            pn = square_fixed((double)x) << (ti != tj ? 1 : 0);
        }
        // (its __syncthreads also guard Ar, Bc, part and tot)
        if (!share(pt, pn, (it + 1) & 1, ++epoch)) return;
    }
    if (blockIdx.x == 0) {  // maxs is even: X is in X0
        gather(maxs & 1);
        if (threadIdx.x == 0) {
            sync->steps = maxs;
            sync->trace = (double)s_trace * (1.0 / SP2_UNIT);
        }
    }
}

// Sum of v over the block into *dst (one atomic per block).
__device__ __forceinline__ void block_add(double v, double* dst)
{
    __shared__ double part[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) part[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += part[w];
        if (s != 0.0) atomicAdd(dst, s);
    }
    __syncthreads();
}

// The launch-per-step form (bases whose recursion does not fit one launch):
// X = (emax I - F) / (emax - emin): spectrum mapped into [0, 1], occupied states
// near 1; trX[0] = tr X and trX[1] = ||X||_F^2 of this initial iterate
__global__ void sp2_init2_kernel(int n, const double* __restrict__ F, const double* __restrict__ b, double* X,
                                 double* trX)
{
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double t = 0.0, q = 0.0;
    if (idx < (int64_t)n * n) {
        const int i = idx % n, j = idx / n;
        const double x = ((i == j ? b[1] : 0.0) - F[idx]) / (b[1] - b[0]);
        X[idx] = x;
        if (i == j) t = x;
        q = x * x;
    }
    block_add(t, trX);
    block_add(q, trX + 1);
}

// one SP2 step from the traces of this step (t[0] = tr X, t[1] = tr X^2);
// accumulates tr of the new iterate into tnext[0]
__global__ void sp2_step_kernel(int n, int nocc, const double* __restrict__ t, const double* __restrict__ X2,
                                double* X, double* tnext)
{
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)n * n) return;
    const bool square = fabs(t[1] - nocc) <= fabs(2 * t[0] - t[1] - nocc);
    const double x = square ? X2[idx] : 2 * X[idx] - X2[idx];
    X[idx] = x;
    const int i = idx % n, j = idx / n;
    if (i == j) atomicAdd(tnext, x);
}

static int sp2_threads(int tt, int ks) { return (ks * tt * tt + 31) / 32 * 32; }
static size_t sp2_smem_bytes(int n, int tt, int ks, size_t elem)
{
    return (2 * (size_t)tt * (n + 1) + (size_t)(ks - 1) * tt * tt) * elem;
}
static unsigned sp2_tiles(int n, int tt)
{
    const int nt = (n + tt - 1) / tt;
    return (unsigned)(nt * (nt + 1) / 2);
}

// can all blocks of the persistent SP2 kernel with tile edge tt be resident at once?
static bool coop_ok(Context& ctx, int n, int tt, int ks)
{
    int coop = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx.device) != cudaSuccess || !coop) return false;
    // the attribute is per process: set it once, to the most a block may have,
    // so that concurrent molecules of other sizes never lower it
    // (the block's opt-in maximum less the kernels' static shared memory)
    static std::once_flag once;
    static bool attr_ok = false;
    static size_t most = 0;
    const int dev = ctx.device;
    std::call_once(once, [dev] {
        int optin = 0;
        const void* fns[] = {(const void*)sp2_kernel<double, SP2_FROM_F>, (const void*)sp2_kernel<double, SP2_FROM_F32>,
                             (const void*)sp2_kernel<float, SP2_FROM_F>};
        size_t fixed = 0;
        bool ok = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess;
        for (const void* f : fns) {
            cudaFuncAttributes fa{};
            ok = ok && cudaFuncGetAttributes(&fa, f) == cudaSuccess;
            fixed = std::max(fixed, fa.sharedSizeBytes);
        }
        most = (size_t)optin - fixed;
        for (const void* f : fns)
            ok = ok && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) == cudaSuccess;
        attr_ok = ok;
        if (!attr_ok) (void)cudaGetLastError();  // no pending error for the next launch check
    });
    if (!attr_ok || n > 512 || sp2_smem_bytes(n, tt, ks, sizeof(double)) > most) return false;
    int per_sm32 = 0;
    const size_t smem = sp2_smem_bytes(n, tt, ks, sizeof(double));
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sp2_kernel<double, SP2_FROM_F>, sp2_threads(tt, ks),
                                                      smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm32, sp2_kernel<double, SP2_FROM_F32>, sp2_threads(tt, ks),
                                                      smem) != cudaSuccess)
        return false;
    return (int64_t)std::min(per_sm, per_sm32) * ctx.num_sms >= (int64_t)sp2_tiles(n, tt);
}

// tile edge tt and k-slices ks of the persistent SP2 kernel.  Per step, a warp's
// FP64 FMA keeps its sub-partition's FP64 pipe ~64 cycles busy on this GPU, so the
// busiest sub-partition of the busiest SM takes ceil(resident warps / 4) x n/ks
// such instructions; every block adds ~40 cycles of the barrier's atomic and of the
// shares that all others read.  Take the (tt in 8 .. 32, ks in 1 .. 4, at most 1024 threads) with
// the least of both among those whose grid can be co-resident (n = 400: edge 17
// or 25, where 8 .. 16 would need more blocks per SM than shared memory allows).
// tt = 0: none fits.
struct Sp2Shape {
    int tt = 0, ks = 1;
};

static Sp2Shape sp2_shape(Context& ctx, int n)
{
    // ~100 occupancy queries a size: kept per (device, size)
    static std::mutex mu;
    static std::map<std::pair<int, int>, Sp2Shape> cache;
    std::lock_guard<std::mutex> lk(mu);
    const auto known = cache.find({ctx.device, n});
    if (known != cache.end()) return known->second;
    Sp2Shape best;
    int64_t best_cost = 0;
    for (int tt = 32; tt >= 8; --tt)
        for (int ks = 1; ks <= 4; ++ks) {
            if (ks * tt * tt > 1024 || !coop_ok(ctx, n, tt, ks)) continue;
            const int64_t tiles = sp2_tiles(n, tt);
            const int64_t per_sm = (tiles + ctx.num_sms - 1) / ctx.num_sms;
            const int64_t warps = sp2_threads(tt, ks) / 32;
            const int64_t cost = (per_sm * warps + 3) / 4 * ((n + ks - 1) / ks) * 64 + 40 * tiles;
            if (best.tt == 0 || cost < best_cost) {
                best.tt = tt;
                best.ks = ks;
                best_cost = cost;
            }
        }
    return cache[{ctx.device, n}] = best;
}

// Bounds on the last occupied and the first virtual energy of F from the course of its
// purification in `steps` steps to a projector of the right trace: before step i every
// eigenvalue x of X_i has x (1 - x) <= w_i = tr(X_i - X_i^2), so where nocc of them are
// near 1 the virtual ones are below (1 - sqrt(1 - 4 w_i)) / 2 and the occupied ones as
// close to 1; the inverse steps take both to X_0 and F.  Late steps have few eigenvalues left in w_i and are the
// tightest; 1e-5 and up is far above w_i's rounding.  false: none, or no gap left.
static bool sp2_gap(const Sp2Log& log, int steps, int nocc, double& homo, double& lumo)
{
    double l0 = 1.0, h0 = 0.0;
    if (steps > SP2_LOG) return false;
    for (int i = 0; i < steps; ++i) {
        const double w = (double)log.w[i] / SP2_UNIT * (1.0 + 1e-6);
        if (!(w > 1e-5 && w < 0.2)) continue;
        // (all but w / 0.72 of the trace is the number of eigenvalues near 1)
        if (std::fabs((double)log.tr[i] / SP2_UNIT - nocc) > 0.2) continue;
        double x = 0.5 * (1.0 - std::sqrt(1.0 - 4.0 * w)), y = 1.0 - x;
        for (int j = i - 1; j >= 0; --j) {
            const double a = std::fabs(log.alpha[j]);
            if (log.alpha[j] > 0) {
                x = (std::sqrt(x) - 1.0 + a) / a;
                y = (std::sqrt(y) - 1.0 + a) / a;
            } else {
                x = (1.0 - std::sqrt(1.0 - x)) / a;
                y = (1.0 - std::sqrt(1.0 - y)) / a;
            }
        }
        l0 = std::min(l0, x);
        h0 = std::max(h0, y);
    }
    l0 += 1e-8;  // far above the rounding of the steps
    h0 -= 1e-8;
    homo = (log.shift - h0) / log.scale;
    lumo = (log.shift - l0) / log.scale;
    return l0 < h0;
}

struct Purifier {
    int n = 0, nocc = 0;
    int tile = 0;  // persistent-kernel tile edge (sp2_shape); -1: per-step fallback
    int kslices = 1;
    DBuf<double> X, T1, T2, T3, B, tr;  // orthogonaliser L^-T and work
    DBuf<float> Xf;                     // FP32 iterate of the coarse steps
    DBuf<Sp2Slot> slots;
    // X^T F X of this density, and of the one whose bounds (sp2_gap) are known
    DBuf<double> Fx, Fprev;
    bool gap = false, from_f = false;
    double homo = 0, lumo = 0;
    ScfReport* rep = nullptr;         // device: barriers and outcome, cleared before each density()
    const ScfReport* hrep = nullptr;  // its host copy, read by converged()
    void setup(Context& ctx, int n_, int nocc_, const double* dS, ScfReport* rep_, const ScfReport* hrep_)
    {
        n = n_;
        nocc = nocc_;
        rep = rep_;
        hrep = hrep_;
        const int64_t nn = (int64_t)n * n;
        cudaStream_t st = ctx.stream;
        X.alloc(nn, st);
        T1.alloc(nn, st);
        T2.alloc(nn, st);
        // orthogonaliser X = L^-T from the Cholesky factor S = L L^T (X^T S X = I):
        // a factorisation and a triangular solve instead of an eigensolve
        cholesky_orthogonalizer(ctx, n, dS, X.p);
    }
    // One cooperative launch of the whole recursion, barrier state slot `which`.
    template <typename T, int FROM>
    void run(Context& ctx, const void* src, T* X0, T* X1, double tol_idem, double tol_n, int polish, int which,
             const double* prev = nullptr, Sp2Log* log = nullptr)
    {
        int n_ = n, nocc_ = nocc, tt_ = tile, ks_ = kslices, maxs = limit;
        Sp2Slot* sl = slots.p;
        Sp2Sync* sp = rep->sp2 + which;
        void* args[] = {&n_, &nocc_, &tt_, &ks_, &src, &X0, &X1, &sl, &maxs, &tol_idem, &tol_n, &polish, &sp,
                        &prev, &homo, &lumo, &log};
        HF_CUDA(cudaLaunchCooperativeKernel((const void*)sp2_kernel<T, FROM>, dim3(sp2_tiles(n, tile)),
                                            dim3(sp2_threads(tile, kslices)), args,
                                            sp2_smem_bytes(n, tile, kslices, sizeof(T)), ctx.stream));
        count_launch();
    }
    // The outcome of the last cooperative purification (barrier timeouts, final trace)
    // travels to the host with the iteration's report.
    bool pending = false;
    static constexpr int MAXS = 160;
    // Steps that the recursion may take (even), and its estimate for a spectrum of this
    // width and gap: each step shrinks their ratio 1.24 times.  Where an eigensolve can take
    // over, more than slow() steps are slower than it: 4 us a step at 25 functions, 6 us at
    // 75 and 13 us at 150 against 0.2, 0.7 and 2 ms.  One such density costs little (of one
    // water's Fock matrices after the core Hamiltonian the first has a gap of 0.0045 and takes 52
    // steps, the others 24 to 38), so it is given up at twice as many.
    int limit = MAXS;
    int slow() const { return std::min(MAXS, std::max(40, 20 + 5 * n / 4)); }
    int steps() const { return hrep->sp2[1].steps; }
    static double steps_for(double width, double gap) { return gap > 0 ? 9.0 + 10.9 * std::log10(1.5 * width / gap) : 1e9; }
    // Did the last density() end with tr X = nocc?  strict: and by the idempotency
    // test, not at the step limit.  (True when nothing is pending.)
    bool converged(bool strict)
    {
        if (!pending) return true;
        pending = false;
        HF_CHECK(hrep->sp2[0].err == 0 && hrep->sp2[1].err == 0, HFGPU_ERR_CUDA,
                 "density purification: grid barrier timed out");
        const bool idem = hrep->sp2[1].steps < limit, trace = fabs(hrep->sp2[1].trace - nocc) < 1e-6;
        if (from_f) {  // the bounds of this F for the next
            double h = 0, l = 0;
            const bool found = idem && trace && sp2_gap(hrep->log, hrep->sp2[1].steps, nocc, h, l);
            // a stretched course reaches back with the bounds it was given at best: the
            // last ones moved by the change of F are tighter once that is small
            homo = gap && found ? std::min(h, homo + hrep->log.dif) : h;
            lumo = gap && found ? std::max(l, lumo - hrep->log.dif) : l;
            gap = found;
            std::swap(Fx, Fprev);
        }
        return trace && !(strict && !idem);
    }
    // is the whole recursion one cooperative launch at this size?
    bool one_launch(Context& ctx)
    {
        if (tile == 0) {
            const Sp2Shape sh = sp2_shape(ctx, n);
            tile = sh.tt == 0 ? -1 : sh.tt;
            kslices = sh.ks;
        }
        return tile > 0;
    }
    // P = 2 X proj(X^T F X) X^T: the closed-shell density of F without diagonalising it.
    // coarse: run the recursion in FP32 until tr(X - X^2) < 1e-3, then finish in
    // FP64 (a few steps); the result is idempotent to FP64 precision but its
    // occupied subspace carries FP32 rounding (~1e-7), which is fine while the
    // SCF is far from convergence.
    void density(Context& ctx, const double* dF, double* dP, bool coarse = false)
    {
        const int64_t nn = (int64_t)n * n;
        cudaStream_t st = ctx.stream;
        // X is upper triangular: X^T F sums k <= i, (X^T F) X k <= j and is symmetric
        gemm(ctx, true, false, n, n, n, 1.0, X.p, n, dF, n, 0.0, T1.p, n, GEMM_K_LE_I);
        const bool one = one_launch(ctx);
        if (one && !slots.p) {
            slots.alloc(5 * (size_t)sp2_tiles(n, tile), st);  // two sets, and the bounds
            T3.alloc(nn, st);
            Fx.alloc(nn, st);
            Fprev.alloc(nn, st);
        }
        double* f = one ? Fx.p : T2.p;
        gemm(ctx, false, false, n, n, n, 1.0, T1.p, n, X.p, n, 0.0, f, n, GEMM_K_LE_J | GEMM_SYMMETRIC);
        ctx.trace_mark("sp2 X^T F X");
        if (one) {
            if (coarse) {
                if (Xf.n < (size_t)(2 * nn)) Xf.alloc(2 * nn, st);
                run<float, SP2_FROM_F>(ctx, f, Xf.p, Xf.p + nn, 1e-3, 1e-3, 0, 0);
                ctx.trace_mark("sp2 fp32");
                run<double, SP2_FROM_F32>(ctx, Xf.p, T1.p, T3.p, 1e-7, 1e-6, 2, 1);
            } else {
                run<double, SP2_FROM_F>(ctx, f, T1.p, T3.p, 1e-7, 1e-6, 2, 1, gap ? Fprev.p : nullptr, &rep->log);
            }
            from_f = !coarse;
            ctx.trace_mark("sp2 fp64");
            pending = true;
        } else {
            per_step(ctx);
        }
        // X Y sums k >= i, (X Y) X^T k >= j and is symmetric
        gemm(ctx, false, false, n, n, n, 1.0, X.p, n, T1.p, n, 0.0, T2.p, n, GEMM_K_GE_I);
        gemm(ctx, false, true, n, n, n, 2.0, T2.p, n, X.p, n, 0.0, dP, n, GEMM_K_GE_J | GEMM_SYMMETRIC);
    }
    // launch-per-step form: T2 = X^T F X to the projector in T1
    void per_step(Context& ctx)
    {
        const int64_t nn = (int64_t)n * n;
        cudaStream_t st = ctx.stream;
        const int CHECK = 8;
        B.alloc(4, st);
        gersh_kernel<<<1, 1024, 0, st>>>(n, T2.p, B.p);
        count_launch();
        // per-step trace slots [step][tr X, tr X^2], zeroed once; tr[2k+1] is accumulated
        // by the square kernel
        tr.alloc(2 * (MAXS + 1), st);
        HF_CUDA(cudaMemsetAsync(tr.p, 0, sizeof(double) * 2 * (MAXS + 1), st));
        sp2_init2_kernel<<<nblk(nn), 256, 0, st>>>(n, T2.p, B.p, T1.p, tr.p);  // T1 = iterate
        count_launch();
        HF_CUDA(cudaMemsetAsync(tr.p + 1, 0, sizeof(double), st));
        const int nt = (n + SQ_T - 1) / SQ_T;
        const unsigned tiles = (unsigned)(nt * (nt + 1) / 2);
        double h[2] = {0, 1};
        bool done = false;
        for (int it = 0; it < MAXS && !done; ++it) {
            sym_square_kernel<<<tiles, SQ_T * SQ_T, 0, st>>>(n, T1.p, T2.p, tr.p + 2 * it + 1);
            count_launch();
            sp2_step_kernel<<<nblk(nn), 256, 0, st>>>(n, nocc, tr.p + 2 * it, T2.p, T1.p, tr.p + 2 * (it + 1));
            count_launch();
            if (it % CHECK == CHECK - 1) {
                // traces of step it (tr X, tr X^2) are complete once its kernels ran
                HF_CUDA(cudaMemcpyAsync(h, tr.p + 2 * it, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
                HF_CUDA(cudaStreamSynchronize(st));
                done = fabs(h[0] - h[1]) < 1e-13 * n && fabs(h[0] - nocc) < 1e-6;
            }
        }
        HF_CHECK(fabs(h[0] - nocc) < 1e-6, HFGPU_ERR_LINALG, "density purification did not converge (no gap?)");
    }
};

// P = 2 C_occ C_occ^T
static void form_density(Context& ctx, int n, int nocc, const double* C, double* P)
{
    const double two = 2.0, zero = 0.0;
    if (nocc == 0) {
        HF_CUDA(cudaMemsetAsync(P, 0, sizeof(double) * n * n, ctx.stream));
        return;
    }
    gemm(ctx, false, true, n, n, nocc, 2.0, C, n, C, n, 0.0, P, n);
}

// The DIIS step: e = Y - Y^T (the commutator F P S - S P F) into the history slot `head`,
// its products with the nhist errors kept, and in the last block the DIIS system
// [[B / scale, -1], [-1, 0]] c = [0 .. 0, -1], solved by Gaussian elimination with partial
// pivoting by one warp (B, nd x nd, keeps <e_k, e_l> from one call to the next); c gets the
// nhist coefficients, or selects the newest Fock matrix alone when the system is singular.
constexpr int DIIS_MAX = RED_MAX;  // the history length run_scf allows
__global__ void __launch_bounds__(RED_BLOCK) diis_error_kernel(int n, const double* __restrict__ Y, double* Eh, int nd,
                                                               int nhist, int head, double* __restrict__ Bd,
                                                               double* __restrict__ cvec, RedWork w)
{
    __shared__ double tot[DIIS_MAX];
    __shared__ double A[DIIS_MAX + 1][DIIS_MAX + 2], x[DIIS_MAX + 1];
    const int64_t nn = (int64_t)n * n;
    double s[DIIS_MAX];
#pragma unroll
    for (int k = 0; k < DIIS_MAX; ++k) s[k] = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * RED_BLOCK + threadIdx.x; i < nn; i += (int64_t)gridDim.x * RED_BLOCK) {
        const int r = (int)(i % n), c = (int)(i / n);
        const double e = Y[i] - Y[c + (int64_t)r * n];
        Eh[head * nn + i] = e;
#pragma unroll
        for (int k = 0; k < DIIS_MAX; ++k)
            if (k < nhist) s[k] = fma(k == head ? e : Eh[k * nn + i], e, s[k]);
    }
    if (!grid_sums(s, nhist, w, tot)) return;
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x, m = nhist + 1;
    if (lane < nhist) {
        Bd[head * nd + lane] = tot[lane];
        Bd[lane * nd + head] = tot[lane];
    }
    __syncwarp();
    double scale = 0;
    for (int k = 0; k < nhist; ++k) scale = fmax(scale, fabs(Bd[k * nd + k]));
    if (scale <= 0) scale = 1;
    // lane = column; column m is the right-hand side
    for (int r = 0; r < m; ++r)
        if (lane <= m)
            A[r][lane] = lane < nhist ? (r < nhist ? Bd[r * nd + lane] / scale : -1.0)
                         : lane == nhist ? (r < nhist ? -1.0 : 0.0) : (r == nhist ? -1.0 : 0.0);
    __syncwarp();
    bool ok = true;
    for (int c = 0; c < m && ok; ++c) {
        int piv = c;
        for (int r = c + 1; r < m; ++r)
            if (fabs(A[r][c]) > fabs(A[piv][c])) piv = r;
        if (fabs(A[piv][c]) < 1e-300) ok = false;
        __syncwarp();
        if (ok && lane <= m && piv != c) {
            const double t = A[c][lane];
            A[c][lane] = A[piv][lane];
            A[piv][lane] = t;
        }
        __syncwarp();
        if (ok)
            for (int r = c + 1; r < m; ++r) {
                const double f = A[r][c] / A[c][c];
                __syncwarp();
                if (lane >= c && lane <= m) A[r][lane] = fma(-f, A[c][lane], A[r][lane]);
                __syncwarp();
            }
    }
    if (ok && lane == 0)
        for (int c = m - 1; c >= 0; --c) {
            double v = A[c][m];
            for (int k = c + 1; k < m; ++k) v = fma(-A[c][k], x[k], v);
            x[c] = v / A[c][c];
        }
    __syncwarp();
    if (lane < nd) cvec[lane] = ok ? (lane < nhist ? x[lane] : 0.0) : (lane == head ? 1.0 : 0.0);
}

// out = sum_k c_k Fh_k over the nhist kept Fock matrices
__global__ void diis_mix_kernel(int64_t nn, const double* __restrict__ Fh, const double* __restrict__ c, int nhist,
                                double* __restrict__ out)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    double s = 0.0;
    for (int k = 0; k < nhist; ++k) s = fma(__ldg(c + k), Fh[k * nn + i], s);
    out[i] = s;
}

constexpr int SP2_MIN = 8;  // smallest basis whose iteration densities come from purification by default

ScfOut run_scf(Context& ctx, const ScfIn& in, double* dC, double* dP, double* dLam)
{
    cudaStream_t st = ctx.stream;
    const int n = in.n;
    const int64_t nn = (int64_t)n * n;
    HF_CHECK(in.nocc >= 0 && in.nocc <= n, HFGPU_ERR_INVALID, "nocc out of range");
    SideStreams beside(in.begin ? &ctx : nullptr);  // until `end`
    if (in.begin) in.begin(in.hook_user);
    DBuf<double> G(nn, st), F(nn, st), Fw(nn, st), Sw(nn, st), Pold(nn, st), partial(RED_MAX_BLOCKS * RED_MAX, st);
    DBuf<unsigned> redcount(1, st);
    redcount.zero();
    const RedWork red{partial.p, redcount.p};
    const unsigned rb = red_blocks(nn);
    DBuf<ScfReport> rep(1, st);
    ScfReport* h = (ScfReport*)ctx.pinned(Context::PIN_SCF, sizeof(ScfReport));
    DBuf<int> info(1, st);
    info.zero();  // written by dsygvd; the own eigensolver reports errors by exception
    if (in.dP0)
        HF_CUDA(cudaMemcpyAsync(dP, in.dP0, sizeof(double) * nn, cudaMemcpyDeviceToDevice, st));
    else
        HF_CUDA(cudaMemsetAsync(dP, 0, sizeof(double) * nn, st));
    int lwork = 0;
    HF_CUSOLVER(cusolverDnDsygvd_bufferSize(ctx.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                            CUBLAS_FILL_MODE_LOWER, n, Fw.p, n, Sw.p, n, dLam, &lwork));
    DBuf<double> work(std::max(lwork, 1), st);

    const bool diis = in.accel == HFGPU_SCF_DIIS;
    const int nd = std::max(2, std::min(in.diis_size, 20));
    DBuf<double> Fh, Eh, Y, cvec, Bd;
    if (diis) {
        Fh.alloc((size_t)nd * nn, st);
        Eh.alloc((size_t)nd * nn, st);
        Y.alloc(nn, st);
        cvec.alloc(nd, st);
        Bd.alloc((size_t)nd * nd, st);
        Bd.zero();
    }
    int nhist = 0, head = 0;

    // eigensolver: our own (eigh.cu) where it fits, with the purifier's X; cuSOLVER's
    // dsygvd otherwise
    Purifier pur;
    Eigh eig;
    const bool own_eigh = in.eigensolver == 0 && Eigh::supported(ctx, n);
    if (in.purify || own_eigh) pur.setup(ctx, n, in.nocc, in.dS, rep.p, h);
    if (own_eigh) eig.setup(ctx, n);
    const double* Xorth = pur.X.p;
    // Densities of the iterations: with the own eigensolver they too come from FP64
    // purification, whose projector is the occupied eigenvectors' to rounding (its
    // last two steps square the idempotency error away), and an eigensolve follows
    // only where that does not converge (no gap) and for the final orbitals.  The
    // eigensolve walks n columns with a grid barrier each and waits for the host's
    // tridiagonal solve; purification takes about 30 steps and no host.  At n = 225:
    // 3.0 ms an iteration by eigensolve.  Below SP2_MIN functions, for a tolP near
    // rounding, and where the recursion does not fit one launch, the eigensolve
    // stays.
    const bool sp2_density = in.purify || (own_eigh && in.nocc > 0 && in.nocc < n && n >= SP2_MIN &&
                                           in.tolP >= 1e-11 && pur.one_launch(ctx));
    // After a purification that found no gap, or two slow ones in a row, none is tried until
    // the energies of the eigensolves instead of it show a gap for a fast one (and after the
    // third such not at all): 20 iterations of 25 functions without a gap, or with one of 1e-6,
    // took 19 and 10 ms, 6.3 with eigensolves alone.
    bool rest = false;
    int misses = 0, slow = 0;
    if (sp2_density && !in.purify) pur.limit = std::min(Purifier::MAXS, 2 * pur.slow());
    // orbitals C (may alias F) and energies of F C = S C diag(lam); with the own
    // eigensolver only the lowest ncol orbitals are formed (ncol <= 0: all)
    auto eigh = [&](const double* Fm, double* Cm, int ncol) {
        if (own_eigh) {
            eig.solve(ctx, Xorth, Fm, Cm, dLam, ncol);
            return;
        }
        if (Cm != Fm) HF_CUDA(cudaMemcpyAsync(Cm, Fm, sizeof(double) * nn, cudaMemcpyDeviceToDevice, st));
        HF_CUDA(cudaMemcpyAsync(Sw.p, in.dS, sizeof(double) * nn, cudaMemcpyDeviceToDevice, st));
        HF_CUSOLVER(cusolverDnDsygvd(ctx.solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER,
                                     n, Cm, n, Sw.p, n, dLam, work.p, lwork, info.p));
    };

    std::vector<double> Escf;
    ScfOut out;
    // incremental Fock builds: Gacc = G(Pold); each iteration adds G(P - Pold)
    const bool inc = in.direct_jk && in.inc_screen > 0;
    DBuf<double> Gacc, D;
    if (inc) {
        Gacc.alloc(nn, st);
        D.alloc(nn, st);
    }
    // near convergence (dP < 100 tolP) every build is a full one, so the last
    // iterations converge exactly like the full-build SCF
    int since_full = 0;
    bool last_full = true, endgame = false;
    double last_dP = 1.0;
    const double* last_F = nullptr;  // the Fock matrix of the last eigensolve
    ctx.trace_mark("scf setup");
    if (in.end) in.end(in.hook_user);
    beside.joined();
    for (int it = 1; it <= in.nscf; ++it) {
        const double* Gcur = G.p;
        double* acc = nullptr;
        if (inc) {
            last_full = it == 1 || endgame || since_full >= in.inc_rebuild;
            if (last_full) {
                in.direct_jk(ctx, in.direct_ctx, dP, Gacc.p, 0.0);
                Gcur = Gacc.p;
                since_full = 0;
            } else {
                in.direct_jk(ctx, in.direct_ctx, D.p, G.p, in.inc_screen);
                acc = Gacc.p;
                ++since_full;
            }
        } else if (in.direct_jk) {
            in.direct_jk(ctx, in.direct_ctx, dP, G.p, 0.0);
        } else {
            jk_from_packed(ctx, n, in.d_int2, dP, G.p);
        }
        ctx.trace_mark("fock");
        // the first iteration of a P = 0 start has a commutator that vanishes
        // trivially: keep it out of the DIIS history
        const bool extrapolate = diis && (it >= 2 || in.dP0);
        fock_kernel<<<rb, RED_BLOCK, 0, st>>>(nn, in.dH, Gcur, acc, dP, F.p, extrapolate ? Fh.p + head * nn : nullptr,
                                              Pold.p, red, rep.p);
        count_launch();
        HF_CUDA(cudaGetLastError());
        const double* Fsolve = F.p;
        if (extrapolate) {
            // error = F P S - S P F = Y - Y^T with Y = F P S
            gemm(ctx, false, false, n, n, n, 1.0, F.p, n, dP, n, 0.0, G.p, n);
            gemm(ctx, false, false, n, n, n, 1.0, G.p, n, in.dS, n, 0.0, Y.p, n);
            nhist = std::min(nhist + 1, nd);
            diis_error_kernel<<<rb, RED_BLOCK, 0, st>>>(n, Y.p, Eh.p, nd, nhist, head, Bd.p, cvec.p, red);
            count_launch();
            HF_CUDA(cudaGetLastError());
            ctx.trace_mark("diis error");
            if (nhist >= 2) {
                diis_mix_kernel<<<nblk(nn), 256, 0, st>>>(nn, Fh.p, cvec.p, nhist, Y.p);
                count_launch();
                HF_CUDA(cudaGetLastError());
                Fsolve = Y.p;
            }
            head = (head + 1) % nd;
            ctx.trace_mark("diis extrap");
        }
        const bool sp2_now = sp2_density && !rest;
        if (sp2_now) {
            // with the purify option, FP32 steps while the density is still far from converged
            pur.density(ctx, Fsolve, dP, in.purify && it > 1 && !endgame && last_dP > 1e-4);
        } else {
            // the density needs the occupied orbitals only; all are formed once converged
            eigh(Fsolve, Fw.p, in.nocc);
            form_density(ctx, n, in.nocc, Fw.p, dP);
        }
        last_F = Fsolve;
        ctx.trace_mark("density");
        auto report = [&] {  // dP, and everything the host reads of this iteration
            density_change_kernel<<<rb, RED_BLOCK, 0, st>>>(nn, dP, Pold.p, inc ? D.p : nullptr, red, rep.p);
            count_launch();
            HF_CUDA(cudaGetLastError());
            HF_CUDA(cudaMemcpyAsync(h, rep.p, sizeof(ScfReport), cudaMemcpyDeviceToHost, st));
        };
        report();
        int hinfo = 0;
        if (!own_eigh) info.download(&hinfo, 1);  // dsygvd's; the own eigensolver throws
        HF_CUDA(cudaStreamSynchronize(st));
        if (rest) {
            const double* w = eig.energies();
            rest = misses >= 3 || Purifier::steps_for(w[n - 1] - w[0], w[in.nocc] - w[in.nocc - 1]) > pur.slow() - 6;
        }
        const bool fell_back = sp2_now && !pur.converged(!in.purify);
        slow = sp2_now && !in.purify && pur.steps() > pur.slow() ? slow + 1 : 0;
        if (fell_back || slow >= 2) {
            rest = true;
            ++misses;
        }
        if (fell_back) {
            HF_CHECK(!in.purify, HFGPU_ERR_LINALG, "density purification did not converge (no gap?)");
            eigh(Fsolve, Fw.p, in.nocc);
            form_density(ctx, n, in.nocc, Fw.p, dP);
            report();
            HF_CUDA(cudaStreamSynchronize(st));
        }
        ctx.trace_mark("convergence");
        HF_CHECK(hinfo == 0, HFGPU_ERR_LINALG,
                 "eigh: dsygvd returned info = " + std::to_string(hinfo) +
                     (hinfo > n ? " (S is not positive definite)" : ""));
        const double E0 = h->E0, dPv = h->dP;
        last_dP = dPv;
        if (dPv < 100 * in.tolP) endgame = true;
        Escf.push_back(E0);
        out.E0 = E0;
        out.dP = dPv;
        out.niter = it;
        if (it > 3) {
            double emax = *std::max_element(Escf.end() - 4, Escf.end());
            double emin = *std::min_element(Escf.end() - 4, Escf.end());
            if (dPv < in.tolP && emax - emin < in.tolE && !last_full) {
                endgame = true;  // accept convergence only on a fully built Fock matrix
            } else if (dPv < in.tolP && emax - emin < in.tolE) {
                if (sp2_density) {
                    // orbitals and orbital energies of the last Fock matrix, as the reference returns them
                    eigh(last_F, Fw.p, 0);
                    form_density(ctx, n, in.nocc, Fw.p, dP);
                    info.download(&hinfo, 1);
                    HF_CUDA(cudaStreamSynchronize(st));
                    HF_CHECK(hinfo == 0, HFGPU_ERR_LINALG, "eigh: dsygvd returned info = " + std::to_string(hinfo));
                } else if (own_eigh && in.nocc < n) {
                    eigh(last_F, Fw.p, 0);  // the virtual orbitals too (same occupied ones)
                }
                HF_CUDA(cudaMemcpyAsync(dC, Fw.p, sizeof(double) * nn, cudaMemcpyDeviceToDevice, st));
                HF_CUDA(cudaStreamSynchronize(st));
                ctx.trace_mark("orbitals");
                out.converged = true;
                return out;
            }
        }
        if (!diis && in.alpha != 1.0) {
            mix_kernel<<<nblk(nn), 256, 0, st>>>(nn, in.alpha, Pold.p, dP, inc ? D.p : nullptr);
            count_launch();
        }
    }
    // not converged: orbitals of the last Fock matrix, and P as the last iteration left it (mixed)
    if ((sp2_density || own_eigh) && last_F) eigh(last_F, Fw.p, 0);
    HF_CUDA(cudaMemcpyAsync(dC, Fw.p, sizeof(double) * nn, cudaMemcpyDeviceToDevice, st));
    HF_CUDA(cudaStreamSynchronize(st));
    out.converged = false;
    return out;
}

double device_dot(Context& ctx, int64_t nn, const double* A, const double* B)
{
    DBuf<double> s(1, ctx.stream), partial(RED_MAX_BLOCKS * RED_MAX, ctx.stream);
    DBuf<unsigned> count(1, ctx.stream);
    count.zero();
    dot_kernel<<<red_blocks(nn), RED_BLOCK, 0, ctx.stream>>>(nn, A, B, RedWork{partial.p, count.p}, s.p);
    count_launch();
    HF_CUDA(cudaGetLastError());
    double h = 0;
    s.download(&h, 1);
    HF_CUDA(cudaStreamSynchronize(ctx.stream));
    return h;
}

}  // namespace hfgpu
