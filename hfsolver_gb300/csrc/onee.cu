// One-electron integrals S, T, V over contracted Cartesian GTOs on the GPU.
//
// Same matrices as hfsolver's getS/getT/getV (src/qc.c:6-93 over
// src/cints.c:186-307), evaluated with McMurchie-Davidson expansions:
//   S_ab = sum c_a c_b K_ab (pi/p)^{3/2} Ex^{ab}_0 Ey^{ab}_0 Ez^{ab}_0
//   T_ab from overlaps with the ket power raised/lowered by 2 (the same
//        kinetic formula as cints.c:186-210)
//   V_ab = -sum_C Z_C sum c_a c_b K_ab (2 pi/p) sum_tuv E^{ab}_{tuv} R_tuv(p, P-C)
// A group of lanes per shell pair and chunk of nuclei (every component pair of the
// shells at once); n x n column-major like the reference.
#include <algorithm>
#include <vector>

#include "boys.cuh"
#include "internal.h"
#include "md.cuh"

namespace hfgpu {

struct ShellOne {
    const int* L;
    const int* nprim;
    const int* prim0;
    const int* coef0;
    const int* cfn0;
    const double* xyz;  // 3 per shell
    const double* alpha;
    const double* coef;
    const int* comp_fn;
};

// 1-D Hermite coefficients E[i][j][t] (Helgaker et al. eqs. 9.5.6-9.5.7) for
// i <= IA, j <= JB, with compile-time bounds so the table stays in registers
template <int IA, int JB>
__device__ __forceinline__ void e1d_ct(double (&E)[IA + 1][JB + 1][IA + JB + 1], double xpa, double xpb, double i2p)
{
#pragma unroll
    for (int i = 0; i <= IA; ++i)
#pragma unroll
        for (int j = 0; j <= JB; ++j)
#pragma unroll
            for (int t = 0; t <= IA + JB; ++t) E[i][j][t] = 0.0;
    E[0][0][0] = 1.0;
#pragma unroll
    for (int i = 0; i < IA; ++i)
#pragma unroll
        for (int t = 0; t <= i + 1; ++t) {
            double v = xpa * E[i][0][t];
            if (t > 0) v = fma(i2p, E[i][0][t - 1], v);
            if (t + 1 <= i) v = fma((double)(t + 1), E[i][0][t + 1], v);
            E[i + 1][0][t] = v;
        }
#pragma unroll
    for (int i = 0; i <= IA; ++i)
#pragma unroll
        for (int j = 0; j < JB; ++j)
#pragma unroll
            for (int t = 0; t <= i + j + 1; ++t) {
                double v = xpb * E[i][j][t];
                if (t > 0) v = fma(i2p, E[i][j][t - 1], v);
                if (t + 1 <= i + j) v = fma((double)(t + 1), E[i][j][t + 1], v);
                E[i][j + 1][t] = v;
            }
}

// The shell pairs of one type, sorted by primitive count: `split` lanes of a warp
// share the primitive pairs of each shell pair of a segment.
struct OneeSeg {
    int warp0, pair0, npairs, split;
};
constexpr int ONEE_SEGS = 6;  // split = 1 .. 32
struct OneeSegs {
    OneeSeg s[ONEE_SEGS];
    int nseg, nwarps;
};

// acc summed over aligned groups of split lanes
template <int N>
__device__ __forceinline__ void lane_sums(double (&acc)[N], int split)
{
    for (int o = split >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
}

// One group of split lanes per shell pair (A, B) of one pair type (l_A >= l_B) and
// blockIdx.y: 0 forms S and T, y > 0 adds the attraction of nuclei
// [(y - 1) atoms, y atoms) to V (zeroed by the caller) atomically, or with vrow > 0 writes
// it to a matrix of its own at V + (y - 1) vrow.  The 1-D tables
// of a primitive pair serve every component pair, and the Boys values and R_tuv of
// a nucleus serve every component pair as well.  A == B: only component pairs with
// a >= b are formed (both triangle entries are written from them).
//
// Bound by latency below ~9 waters: one FP64 instruction of a warp takes 64 clocks
// whatever its lanes do, and a thread that walks a pair's 36 primitive pairs over
// four nuclei runs ~4000 of them in a row.  With one thread per pair and the types one
// after the other the six launches took 1.24 ms for 2 waters (and held up the Schwarz
// bounds on their stream); so, the whole set-up of 1, 2, 3 and 8 waters is 0.46, 0.52,
// 0.62 and 1.8 ms (1.20, 1.52, 1.6 and 2.6 with those launches).
template <int LA, int LB>
__global__ void __launch_bounds__(64) onee_shell_kernel(ShellOne sh, const int2* __restrict__ pairs, OneeSegs segs,
                                                        int n, int nat, int atoms, const int* __restrict__ Z,
                                                        const double* __restrict__ C, const double* __restrict__ boys,
                                                        double* S, double* T, double* V, int64_t vrow)
{
    constexpr double PI = 3.14159265358979323846;
    constexpr int NA = ncart(LA), NB = ncart(LB), L = LA + LB;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= segs.nwarps) return;
    OneeSeg sg = segs.s[0];
#pragma unroll
    for (int i = 1; i < ONEE_SEGS; ++i)
        if (i < segs.nseg && w >= segs.s[i].warp0) sg = segs.s[i];
    const int lane = threadIdx.x & 31, sub = lane & (sg.split - 1);
    const int q = (w - sg.warp0) * (32 / sg.split) + lane / sg.split;
    const bool active = q < sg.npairs;
    const int2 pr = pairs[sg.pair0 + (active ? q : sg.npairs - 1)];
    const int A = pr.x, B = pr.y;
    const double ax = sh.xyz[3 * A], ay = sh.xyz[3 * A + 1], az = sh.xyz[3 * A + 2];
    const double bx = sh.xyz[3 * B], by = sh.xyz[3 * B + 1], bz = sh.xyz[3 * B + 2];
    const double rab2 = (ax - bx) * (ax - bx) + (ay - by) * (ay - by) + (az - bz) * (az - bz);
    const int npa = sh.nprim[A], npb = sh.nprim[B], npp = npa * npb;
    const double* alA = sh.alpha + sh.prim0[A];
    const double* alB = sh.alpha + sh.prim0[B];
    const double* coA = sh.coef + sh.coef0[A];
    const double* coB = sh.coef + sh.coef0[B];
    const int* fa = sh.comp_fn + sh.cfn0[A];
    const int* fb = sh.comp_fn + sh.cfn0[B];
    if (blockIdx.y == 0) {
        if (!S && !T) return;
        double sacc[NA * NB], tacc[NA * NB];
#pragma unroll
        for (int k = 0; k < NA * NB; ++k) sacc[k] = tacc[k] = 0.0;
        for (int pp = sub; pp < npp; pp += sg.split) {
            const int pa = pp / npb, pb = pp - pa * npb;
            const double a = alA[pa], b = alB[pb];
            const double p = a + b, ip = 1.0 / p;
            const double px = (a * ax + b * bx) * ip, py = (a * ay + b * by) * ip, pz = (a * az + b * bz) * ip;
            const double K = exp(-a * b * ip * rab2);
            // overlap and kinetic (cints.c:186-232 in terms of 1-D overlaps):
            // E_0 tables with the ket power raised by up to 2
            double Ex[LA + 1][LB + 3][LA + LB + 3], Ey[LA + 1][LB + 3][LA + LB + 3], Ez[LA + 1][LB + 3][LA + LB + 3];
            e1d_ct<LA, LB + 2>(Ex, px - ax, px - bx, 0.5 * ip);
            e1d_ct<LA, LB + 2>(Ey, py - ay, py - by, 0.5 * ip);
            e1d_ct<LA, LB + 2>(Ez, pz - az, pz - bz, 0.5 * ip);
            const double pre = K * PI * ip * sqrt(PI * ip);
#pragma unroll
            for (int i = 0; i < NA; ++i)
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    const Cart c1_ = cart(LA, i), c2 = cart(LB, j);
                    const double sx = Ex[c1_.l][c2.l][0], sy = Ey[c1_.m][c2.m][0], sz = Ez[c1_.n][c2.n][0];
                    const double s0 = sx * sy * sz;
                    const double t0 = b * (2 * (c2.l + c2.m + c2.n) + 3) * s0;
                    const double t1 = -2 * b * b *
                                      (Ex[c1_.l][c2.l + 2][0] * sy * sz + sx * Ey[c1_.m][c2.m + 2][0] * sz +
                                       sx * sy * Ez[c1_.n][c2.n + 2][0]);
                    double t2 = 0.0;
                    if (c2.l >= 2) t2 += c2.l * (c2.l - 1) * Ex[c1_.l][c2.l - 2][0] * sy * sz;
                    if (c2.m >= 2) t2 += c2.m * (c2.m - 1) * sx * Ey[c1_.m][c2.m - 2][0] * sz;
                    if (c2.n >= 2) t2 += c2.n * (c2.n - 1) * sx * sy * Ez[c1_.n][c2.n - 2][0];
                    // component coefficients c_a(pa), c_b(pb)
                    const double wc = pre * coA[i * npa + pa] * coB[j * npb + pb];
                    sacc[i * NB + j] = fma(wc, s0, sacc[i * NB + j]);
                    tacc[i * NB + j] = fma(wc, t0 + t1 - 0.5 * t2, tacc[i * NB + j]);
                }
        }
        lane_sums(sacc, sg.split);
        lane_sums(tacc, sg.split);
        if (!active || sub != 0) return;
#pragma unroll
        for (int i = 0; i < NA; ++i)
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                const int x = fa[i], y = fb[j];
                if (x < 0 || y < 0 || (A == B && i < j)) continue;
                const int64_t o1 = x + (int64_t)y * n, o2 = y + (int64_t)x * n;
                if (S) S[o1] = S[o2] = sacc[i * NB + j];
                if (T) T[o1] = T[o2] = tacc[i * NB + j];
            }
        return;
    }
    const int c0 = (blockIdx.y - 1) * atoms, c1 = min(nat, c0 + atoms);
    double vacc[NA * NB];
#pragma unroll
    for (int k = 0; k < NA * NB; ++k) vacc[k] = 0.0;
    for (int pp = sub; pp < npp; pp += sg.split) {
        const int pa = pp / npb, pb = pp - pa * npb;
        const double a = alA[pa], b = alB[pb];
        const double p = a + b, ip = 1.0 / p;
        const double px = (a * ax + b * bx) * ip, py = (a * ay + b * by) * ip, pz = (a * az + b * bz) * ip;
        const double K = exp(-a * b * ip * rab2);
        double Ex[LA + 1][LB + 1][L + 1], Ey[LA + 1][LB + 1][L + 1], Ez[LA + 1][LB + 1][L + 1];
        e1d_ct<LA, LB>(Ex, px - ax, px - bx, 0.5 * ip);
        e1d_ct<LA, LB>(Ey, py - ay, py - by, 0.5 * ip);
        e1d_ct<LA, LB>(Ez, pz - az, pz - bz, 0.5 * ip);
        const double vpre = K * 2 * PI * ip;
        for (int c = c0; c < c1; ++c) {
            const double X = px - C[3 * c], Y = py - C[3 * c + 1], Zc = pz - C[3 * c + 2];
            double F[L + 1];
            boys_scaled<L>(p * (X * X + Y * Y + Zc * Zc), 1.0, -2.0 * p, boys, F);
            double R[nherm(L)];
            r_ct<L>(R, F, X, Y, Zc);
            const double zc = -(double)Z[c] * vpre;
#pragma unroll
            for (int i = 0; i < NA; ++i)
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    const Cart c1_ = cart(LA, i), c2 = cart(LB, j);
                    double acc = 0.0;
#pragma unroll
                    for (int t = 0; t <= c1_.l + c2.l; ++t) {
                        double su = 0.0;
#pragma unroll
                        for (int u = 0; u <= c1_.m + c2.m; ++u) {
                            double sv = 0.0;
#pragma unroll
                            for (int v = 0; v <= c1_.n + c2.n; ++v)
                                sv = fma(Ez[c1_.n][c2.n][v], R[hidx(t, u, v)], sv);
                            su = fma(Ey[c1_.m][c2.m][u], sv, su);
                        }
                        acc = fma(Ex[c1_.l][c2.l][t], su, acc);
                    }
                    vacc[i * NB + j] = fma(zc * coA[i * npa + pa] * coB[j * npb + pb], acc, vacc[i * NB + j]);
                }
        }
    }
    lane_sums(vacc, sg.split);
    if (!active || sub != 0) return;
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int x = fa[i], y = fb[j];
            if (x < 0 || y < 0 || (A == B && i < j)) continue;
            const int64_t o1 = x + (int64_t)y * n, o2 = y + (int64_t)x * n;
            if (vrow > 0) {
                double* Vr = V + (blockIdx.y - 1) * vrow;
                Vr[o1] = Vr[o2] = vacc[i * NB + j];
                continue;
            }
            atomicAdd(V + o1, vacc[i * NB + j]);
            if (o2 != o1) atomicAdd(V + o2, vacc[i * NB + j]);
        }
}

// V = the sum of the block rows' matrices, in their order
__global__ void onee_sum_kernel(int64_t nn, int rows, const double* __restrict__ part, double* __restrict__ V)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    double s = 0.0;
    for (int r = 0; r < rows; ++r) s += part[r * nn + i];
    V[i] = s;
}

// nuclei per block row: ONEE_ATOMS share a primitive pair's 1-D tables, unless that
// leaves fewer warps (of whole shell pairs) than the GPU has FP64 pipes
constexpr int ONEE_ATOMS = 4;

// lanes that share a shell pair of npp primitive pairs: with few pairs, at most two
// primitive pairs a lane; with many, each lane keeps up to 16 (fewer sums over
// lanes, no idle ones)
static int onee_lanes(int npp, bool wide)
{
    int s = 1;
    while (s < 32 && (wide ? 2 * s <= npp : 16 * s < npp)) s <<= 1;
    return s;
}

void onee_compute(Context& ctx, const Basis& b, int nat, const int* atno, const double* x, const double* y,
                  const double* z, double* dS, double* dT, double* dV, cudaStream_t on, bool fixed_lanes)
{
    cudaStream_t st = on ? on : ctx.stream;
    const int n = b.nbf;
    const int ns = (int)b.shells.size();
    std::vector<int> L(ns), np(ns), p0(ns), c0(ns), f0(ns);
    std::vector<double> xyz(3 * ns);
    for (int s = 0; s < ns; ++s) {
        const Shell& sh = b.shells[s];
        HF_CHECK(sh.L <= 2, HFGPU_ERR_UNSUPPORTED, "one-electron integrals support s, p and d shells");
        L[s] = sh.L; np[s] = sh.nprim; p0[s] = sh.prim0; c0[s] = sh.coef0; f0[s] = sh.cfn0;
        xyz[3 * s] = sh.x; xyz[3 * s + 1] = sh.y; xyz[3 * s + 2] = sh.z;
    }
    // shell pairs by pair type, the larger angular momentum first, most primitives first
    const bool wide = !fixed_lanes &&
                      (int64_t)ns * (ns + 1) / 2 * ((nat + ONEE_ATOMS - 1) / ONEE_ATOMS) / 32 < (int64_t)ctx.num_sms * 4;
    // (block rows past 65535 are not launchable: point charges by the ten thousand share them)
    const int atoms = std::max(wide ? 1 : ONEE_ATOMS, (nat + 65533) / 65534);
    std::vector<int2> pairs;
    int off[NPTYPE] = {};
    OneeSegs segs[NPTYPE] = {};
    {
        std::vector<int2> by[NPTYPE];
        for (int s1 = 0; s1 < ns; ++s1)
            for (int s2 = 0; s2 <= s1; ++s2) {
                const int A = L[s1] >= L[s2] ? s1 : s2, B = A == s1 ? s2 : s1;
                by[ptype_of(L[A], L[B])].push_back(make_int2(A, B));
            }
        auto lanes = [&](const int2& p) { return fixed_lanes ? 1 : onee_lanes(np[p.x] * np[p.y], wide); };
        for (int t = 0; t < NPTYPE; ++t) {
            std::stable_sort(by[t].begin(), by[t].end(), [&](int2 x, int2 y) { return lanes(x) > lanes(y); });
            OneeSegs& sg = segs[t];
            for (size_t i = 0; i < by[t].size(); ++i) {
                const int s = lanes(by[t][i]);
                if (i == 0 || s != sg.s[sg.nseg - 1].split) sg.s[sg.nseg++] = OneeSeg{0, (int)i, 0, s};
                ++sg.s[sg.nseg - 1].npairs;
            }
            for (int k = 0; k < sg.nseg; ++k) {
                const int ppw = 32 / sg.s[k].split;
                sg.s[k].warp0 = sg.nwarps;
                sg.nwarps += (sg.s[k].npairs + ppw - 1) / ppw;
            }
            off[t] = (int)pairs.size();
            pairs.insert(pairs.end(), by[t].begin(), by[t].end());
        }
    }
    std::vector<int> Z(nat > 0 ? nat : 1);
    std::vector<double> C(3 * (nat > 0 ? nat : 1));
    for (int i = 0; i < nat; i++) {
        Z[i] = atno[i];
        C[3 * i] = x[i]; C[3 * i + 1] = y[i]; C[3 * i + 2] = z[i];
    }
    auto dL = to_device(L, st);
    auto dn = to_device(np, st);
    auto dp0 = to_device(p0, st);
    auto dc0 = to_device(c0, st);
    auto df0 = to_device(f0, st);
    auto dxyz = to_device(xyz, st);
    auto dal = to_device(b.alpha, st);
    auto dco = to_device(b.coef, st);
    auto dcf = to_device(b.comp_fn, st);
    auto dpairs = to_device(pairs, st);
    auto dZ = to_device(Z, st);
    auto dC = to_device(C, st);
    ShellOne sh{dL.p, dn.p, dp0.p, dc0.p, df0.p, dxyz.p, dal.p, dco.p, dcf.p};
    // a nucleus per block row: the rows' matrices are summed in order, so that V does not
    // change from call to call (as one block row's does not; with more nuclei a row, 9
    // waters and up, the rows meet in atomics)
    const int64_t nn = (int64_t)n * n;
    DBuf<double> parts;
    const int vrows = (nat + atoms - 1) / atoms;
    if (dV && wide && nat > 0)
        parts.alloc((size_t)(nn * vrows), st);
    else if (dV)
        HF_CUDA(cudaMemsetAsync(dV, 0, sizeof(double) * nn, st));
    double* v = parts.p ? parts.p : dV;
    const int64_t vrow = parts.p ? nn : 0;
    // one small launch per pair type: side by side, the longest first
    const unsigned rows = 1 + (dV ? (unsigned)vrows : 0u);
    static_assert(NPTYPE <= Context::NAUX, "one side stream per pair type");
    HF_CUDA(cudaEventRecord(ctx.fork_ev, st));
    for (int t = NPTYPE - 1; t >= 0; --t) {
        if (segs[t].nwarps == 0) continue;
        const dim3 grid((unsigned)((segs[t].nwarps + 1) / 2), rows);
        const int2* pp = dpairs.p + off[t];
        cudaStream_t on_t = ctx.aux[t];
        if (on_t != st) HF_CUDA(cudaStreamWaitEvent(on_t, ctx.fork_ev, 0));
        auto launch = [&](auto kernel) {
            kernel<<<grid, 64, 0, on_t>>>(sh, pp, segs[t], n, nat, atoms, dZ.p, dC.p, ctx.boys, dS, dT, v, vrow);
        };
        switch (t) {
            case 0: launch(onee_shell_kernel<0, 0>); break;
            case 1: launch(onee_shell_kernel<1, 0>); break;
            case 2: launch(onee_shell_kernel<2, 0>); break;
            case 3: launch(onee_shell_kernel<1, 1>); break;
            case 4: launch(onee_shell_kernel<2, 1>); break;
            default: launch(onee_shell_kernel<2, 2>); break;
        }
        count_launch();
        HF_CUDA(cudaGetLastError());
        if (on_t != st) HF_CUDA(cudaEventRecord(ctx.join_ev[t], on_t));
    }
    // st frees the tables: after every launch
    for (int t = 0; t < NPTYPE; ++t)
        if (segs[t].nwarps && ctx.aux[t] != st) HF_CUDA(cudaStreamWaitEvent(st, ctx.join_ev[t], 0));
    if (parts.p) {
        onee_sum_kernel<<<(unsigned)((nn + 127) / 128), 128, 0, st>>>(nn, vrows, parts.p, dV);
        count_launch();
        HF_CUDA(cudaGetLastError());
    }
}

}  // namespace hfgpu
