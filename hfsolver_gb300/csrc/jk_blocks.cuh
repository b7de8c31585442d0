// Fock two-electron term G = J - K/2 from the class-wise quartet blocks that
// the ERI kernels leave in HBM (EriArgs::blocks).
//
// Same G as formG (src/scf.f90:26-58) and as jk_packed_kernel, but only the
// quartets that survived Schwarz screening are read (no zeros), reads are
// coalesced (block element e of quartet q is at e * nq + q), and each thread
// folds its whole quartet block into J/K partial sums before the atomics.
//
// Degeneracy: a block holds every component quartet of the shell quartet,
// including both orders when A == B, C == D or bra pair == ket pair; weighting
// every element by 1/2 per coincidence of shells makes the sum over the block
// equal to the sum over unique integrals with the usual 8-fold weights.  The
// ERI pass stores the blocks with that (exact) weight w applied, and the J and
// K terms go to two half matrices without their factors,
//   Jh[a][b] += w v P_cd, Jh[c][d] += w v P_ab,
//   Kh[a][c] += w v P_bd, Kh[b][c] += w v P_ad, Kh[a][d] += w v P_bc, Kh[b][d] += w v P_ac,
// so that G = 2 (Jh + Jh^T) - (Kh + Kh^T) / 2 takes them once per matrix element.
//
// Bound: the FP64 pipe.  A warp-wide FP64 instruction holds its sub-partition's
// pipe ~64 cycles here, whatever it computes, so the six FMAs per element should
// be all there is: no weights, no partial-sum adds (each chain continues from
// the stored sum, partial J and K sums meet in the atomics, which the L2
// performs), no FP64 in the screening (single precision, rounded up), no idle
// lanes.  Measured, a full build at 8 waters (36 M elements, 0.35 ms of FP64
// pipe): 1.16 ms with weights per output, 64-bit compares, value-returning atomics
// and 21 launches; 0.64 ms now; at 16 waters (2.0 ms of pipe) 5.3 and 3.3 ms.  The
// rest is the atomics (0.1 ms of the 0.64) and load latency.
#pragma once
#include "eri_kernel.cuh"

namespace hfgpu {

// one quartet class of a build
struct DigestClass {
    int id;       // 6 tb + tk
    int block0;   // first thread block of the class within its launch
    int nq;       // quartets (below 2^31, checked when the plan is made)
    int split;    // warps that share the bra component rows of the same 32 x rounds quartets
    int rounds;   // a warp screens rounds x 32 quartets and digests the survivors (1 to 8)
    const double* blocks;
    const int2* qlist;  // the (bra, ket) pair ids of every quartet, written by the ERI pass
};

struct DigestArgs {
    ShellDev sh;
    PairDev pr;
    const double* P;
    int n;
    double* Gh;  // Jh (n x n), then Kh
    // density-difference screening (screen > 0): pair Schwarz bounds Q and the
    // largest |P| element of each shell pair, Dm[S1 * ns + S2] (both rounded up)
    float screen;
    const float* Q;
    const float* Dm;
    int ns;
    // batched plans (mol_n != null): per molecule its basis size, density,
    // half-matrix outputs, screen (< 0: not part of this build), shell-pair
    // maximum table, shell count and first shell, and the molecule of every pair;
    // the scalars above are unused
    const int* mol_n;
    const double* const* mol_P;
    double* const* mol_Gh;
    const float* mol_screen;
    const float* const* mol_Dm;
    const int* mol_ns;
    const int* mol_sh0;
    const int* pair_mol;
};

// The classes of a build go out in three launches by ket type, so that one
// launch's classes need about the same registers: kets ss and ps (<= 80), ds and
// pp (<= 150), dp and dd (255).  21 launches over eight streams cost 0.08 ms a
// build before any work (3 waters: 0.105 ms a build for 0.017 ms of FP64 time).
constexpr int DIGEST_TIERS = 3, DIGEST_TIER_MAX = 11;
__host__ __device__ constexpr int digest_tier(int tk) { return tk / 2; }
struct DigestLaunch {
    DigestArgs a;
    int ncls, nblocks;
    DigestClass cls[DIGEST_TIER_MAX];
};

// the per-molecule view of a batched build (the arguments themselves for one molecule)
struct DigestMol {
    int n, ns, sh0;
    const double* P;
    double* Gh;
    float screen;
    const float* Dm;
};

__device__ __forceinline__ bool digest_mol(const DigestArgs& a, int mol, DigestMol& m)
{
    if (!a.mol_n) {
        m = DigestMol{a.n, a.ns, 0, a.P, a.Gh, a.screen, a.Dm};
        return true;
    }
    m.screen = a.mol_screen[mol];
    if (m.screen < 0.0f) return false;
    m.n = a.mol_n[mol];
    m.ns = a.mol_ns[mol];
    m.sh0 = a.mol_sh0[mol];
    m.P = a.mol_P[mol];
    m.Gh = a.mol_Gh[mol];
    m.Dm = a.mol_Dm ? a.mol_Dm[mol] : nullptr;
    return true;
}

// quartet qg of the class: its bra and ket pair ids and its molecule
__device__ __forceinline__ void digest_quartet(const DigestArgs& a, const DigestClass& c, int qg, int& bra, int& ket, int& mol)
{
    const int2 e = __ldg(c.qlist + qg);
    bra = e.x;
    ket = e.y;
    mol = a.pair_mol ? __ldg(a.pair_mol + bra) : 0;
}

// true if the quartet's whole contribution is below the screening threshold:
// |(ab|cd)| <= Q_bra Q_ket, and the largest density factor it meets is
// 2|P_ab|, 2|P_cd| (Coulomb) or |P_ac|/2 ... (exchange).  In single precision,
// rounded up: never true where the FP64 test would be false.
__device__ __forceinline__ bool digest_skip(const DigestArgs& a, const DigestMol& m, int bra, int ket, int A, int B,
                                            int C, int D)
{
    if (m.screen <= 0.0f) return false;
    const float* Dm = m.Dm;
    const int ns = m.ns;
    A -= m.sh0; B -= m.sh0; C -= m.sh0; D -= m.sh0;
    const float dj = fmaxf(Dm[A * ns + B], Dm[C * ns + D]);
    const float dk = fmaxf(fmaxf(Dm[A * ns + C], Dm[B * ns + D]), fmaxf(Dm[A * ns + D], Dm[B * ns + C]));
    return __fmul_ru(__fmul_ru(a.Q[bra], a.Q[ket]), fmaxf(2.0f * dj, 0.5f * dk)) < m.screen;
}

// v != 0 on the two 32-bit halves (-0 counts as zero): FP64 and 64-bit integer
// compares both run on the FP64 pipe
__device__ __forceinline__ bool digest_nonzero(double v) { return (__double2loint(v) | (__double2hiint(v) << 1)) != 0; }

// *p += v with no result: a red on a global address.  atomicAdd on a generic
// pointer compiles to an atom that returns a value, and the warp waits for it.
__device__ __forceinline__ void red_add(double* p, double v)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "d"(v) : "memory");
}

constexpr int DIGEST_MAX_Q = 256;  // quartets screened per warp: 32 x 8 rounds
// threads per block of the digest kernels (two warps: a class with few quartets
// still reaches most SMs)
constexpr int DIGEST_BLOCK = 64, DIGEST_WARPS = DIGEST_BLOCK / 32;

// Screen the warp's quartets q0 .. q0 + cnt - 1 (density-difference screen,
// molecules not in this build) and leave the offsets of the survivors in the
// warp's list; returns their number.  The survivors are then digested in full
// warps, instead of each warp idling on the lanes whose quartets were skipped.
__device__ __forceinline__ int digest_compact(const DigestArgs& a, const DigestClass& c, int q0, int cnt, int* list, int lane)
{
    int ns = 0;
    for (int r = 0; r < cnt; r += 32) {
        const int k = r + lane;
        const int qg = q0 + k;
        bool keep = false;
        if (k < cnt && (unsigned)qg < (unsigned)c.nq) {
            int bra, ket, mol;
            digest_quartet(a, c, qg, bra, ket, mol);
            DigestMol mm;
            if (digest_mol(a, mol, mm))
                keep = !digest_skip(a, mm, bra, ket, a.pr.A[bra], a.pr.B[bra], a.pr.A[ket], a.pr.B[ket]);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) list[ns + __popc(m & ((1u << lane) - 1u))] = k;
        ns += __popc(m);
    }
    __syncwarp();
    return ns;
}

// One thread digests the bra component rows r0 .. r1 - 1 (row ia NB + ib) of one
// quartet: J_cd and P_cd, and K_ac and K_ad of the current ia, in registers, K_bc
// and K_bd in registers (NB = 1) or local memory.
template <int TB, int TK>
__device__ __forceinline__ void digest_rows(const DigestArgs& a, const DigestClass& c, int qg, int r0, int r1)
{
    using CI = ClassInfo<TB, TK>;
    constexpr int NB = ncart(CI::LB), NC = ncart(CI::LC), ND = ncart(CI::LD);
    int bra, ket, mol;
    digest_quartet(a, c, qg, bra, ket, mol);
    DigestMol mm;
    digest_mol(a, mol, mm);
    const int A = a.pr.A[bra], B = a.pr.B[bra], C = a.pr.A[ket], D = a.pr.B[ket];
    int fc[NC], fd[ND];
#pragma unroll
    for (int i = 0; i < NC; ++i) fc[i] = a.sh.comp_fn[a.sh.cfn0[C] + i];
#pragma unroll
    for (int i = 0; i < ND; ++i) fd[i] = a.sh.comp_fn[a.sh.cfn0[D] + i];
    const int* fa = a.sh.comp_fn + a.sh.cfn0[A];
    const int* fb = a.sh.comp_fn + a.sh.cfn0[B];
    const int n = mm.n;
    const double* Pm = mm.P;
    auto Pv = [&](int x, int y) { return (x < 0 || y < 0) ? 0.0 : __ldg(Pm + x + y * n); };
    double* Jh = mm.Gh;
    double* Kh = Jh + n * n;
    auto add = [&](double* H, int x, int y, double v) {
        if (x >= 0 && y >= 0 && digest_nonzero(v)) red_add(H + x + y * n, v);
    };
    double jcd[NC * ND], Pcd[NC * ND], kbc[NB * NC], kbd[NB * ND];
#pragma unroll
    for (int i = 0; i < NB * NC; ++i) kbc[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NB * ND; ++i) kbd[i] = 0.0;
#pragma unroll
    for (int ic = 0; ic < NC; ++ic)
#pragma unroll
        for (int id = 0; id < ND; ++id) {
            jcd[ic * ND + id] = 0.0;
            Pcd[ic * ND + id] = Pv(fc[ic], fd[id]);
        }
    const int64_t nq = c.nq;
    const double* blk = c.blocks + (r0 * CI::NCDT) * nq + qg;
#pragma unroll 1
    for (int r = r0; r < r1;) {
        const int ia = r / NB;
        const int rend = min(r1, (ia + 1) * NB);
        const int xa = __ldg(fa + ia);
        double Pac[NC], Pad[ND], s_ac[NC], s_ad[ND];
#pragma unroll
        for (int ic = 0; ic < NC; ++ic) {
            Pac[ic] = Pv(xa, fc[ic]);
            s_ac[ic] = 0.0;
        }
#pragma unroll
        for (int id = 0; id < ND; ++id) {
            Pad[id] = Pv(xa, fd[id]);
            s_ad[id] = 0.0;
        }
#pragma unroll 1
        for (; r < rend; ++r) {
            const int ib = NB == 1 ? 0 : r - ia * NB;
            const int xb = __ldg(fb + ib);
            const double Pab = Pv(xa, xb);
            double Pbd[ND], s_ab = 0.0, s_bd[ND];
#pragma unroll
            for (int id = 0; id < ND; ++id) {
                Pbd[id] = Pv(xb, fd[id]);
                s_bd[id] = kbd[ib * ND + id];
            }
#pragma unroll
            for (int ic = 0; ic < NC; ++ic) {
                const double Pbc = Pv(xb, fc[ic]);
                double s_bc = kbc[ib * NC + ic];
#pragma unroll
                for (int id = 0; id < ND; ++id) {
                    const double v = __ldg(blk);
                    blk += nq;
                    s_ab = fma(v, Pcd[ic * ND + id], s_ab);
                    jcd[ic * ND + id] = fma(v, Pab, jcd[ic * ND + id]);
                    s_ac[ic] = fma(v, Pbd[id], s_ac[ic]);
                    s_bc = fma(v, Pad[id], s_bc);
                    s_ad[id] = fma(v, Pbc, s_ad[id]);
                    s_bd[id] = fma(v, Pac[ic], s_bd[id]);
                }
                kbc[ib * NC + ic] = s_bc;
            }
#pragma unroll
            for (int id = 0; id < ND; ++id) kbd[ib * ND + id] = s_bd[id];
            add(Jh, xa, xb, s_ab);
        }
#pragma unroll
        for (int ic = 0; ic < NC; ++ic) add(Kh, xa, fc[ic], s_ac[ic]);
#pragma unroll
        for (int id = 0; id < ND; ++id) add(Kh, xa, fd[id], s_ad[id]);
    }
#pragma unroll
    for (int ic = 0; ic < NC; ++ic)
#pragma unroll
        for (int id = 0; id < ND; ++id) add(Jh, fc[ic], fd[id], jcd[ic * ND + id]);
    // the ib that rows r0 .. r1 - 1 met
    const int nb = min(NB, r1 - r0);
#pragma unroll 1
    for (int k = 0; k < nb; ++k) {
        const int ib = NB == 1 ? 0 : (r0 + k) % NB;
        const int xb = __ldg(fb + ib);
#pragma unroll
        for (int ic = 0; ic < NC; ++ic) add(Kh, xb, fc[ic], kbc[ib * NC + ic]);
#pragma unroll
        for (int id = 0; id < ND; ++id) add(Kh, xb, fd[id], kbd[ib * ND + id]);
    }
}

// One warp = 32 x rounds quartets (32 at a time, one per lane) and 1 / split of
// their bra component rows: all lanes do the same rows, so none idles, the block
// reads are 32 consecutive quartets of one element plane, and classes of few
// large blocks ((dd|dd): a few hundred quartets of 1296 elements at 200
// functions) still make many warps.
template <int TB, int TK>
__device__ __forceinline__ void digest_block(const DigestArgs& a, const DigestClass& c, int* list)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qpw = 32 * c.rounds;
    const int w = ((int)blockIdx.x - c.block0) * DIGEST_WARPS + warp;
    const int chunk = w / c.split, sub = w - chunk * c.split;
    const int q0 = chunk * qpw;
    if ((unsigned)q0 >= (unsigned)c.nq) return;  // the whole warp
    constexpr int ROWS = ClassInfo<TB, TK>::NAB;
    const int per = ROWS / c.split;  // split divides the rows
    const int r0 = sub * per, r1 = r0 + per;
    if (a.screen <= 0.0f && !a.mol_n) {  // nothing is screened: no list
        for (int k = lane; k < qpw; k += 32)
            if ((unsigned)(q0 + k) < (unsigned)c.nq) digest_rows<TB, TK>(a, c, q0 + k, r0, r1);
        return;
    }
    list += warp * DIGEST_MAX_Q;
    const int ns = digest_compact(a, c, q0, qpw, list, lane);
    for (int base = 0; base < ns; base += 32)
        if (base + lane < ns) digest_rows<TB, TK>(a, c, q0 + list[base + lane], r0, r1);
}

template <int TIER>
__global__ void __launch_bounds__(DIGEST_BLOCK) digest_kernel(const __grid_constant__ DigestLaunch l)
{
    __shared__ int list[DIGEST_WARPS * DIGEST_MAX_Q];
    int k = 0;
    while (k + 1 < l.ncls && (int)blockIdx.x >= l.cls[k + 1].block0) ++k;
    const DigestClass& c = l.cls[k];
#define HF_D(B, K) \
    case 6 * B + K: digest_block<B, K>(l.a, c, list); break;
    if constexpr (TIER == 0) {
        switch (c.id) { HF_D(0, 0) HF_D(0, 1) HF_D(1, 1) }
    } else if constexpr (TIER == 1) {
        switch (c.id) { HF_D(0, 2) HF_D(1, 2) HF_D(2, 2) HF_D(0, 3) HF_D(1, 3) HF_D(2, 3) HF_D(3, 3) }
    } else {
        switch (c.id) {
            HF_D(0, 4) HF_D(1, 4) HF_D(2, 4) HF_D(3, 4) HF_D(4, 4)
            HF_D(0, 5) HF_D(1, 5) HF_D(2, 5) HF_D(3, 5) HF_D(4, 5) HF_D(5, 5)
        }
    }
#undef HF_D
}

// launches the classes of l (all of one tier) on stream s (jk_blocks.cu, one
// translation unit per tier)
void launch_digest_tier(int tier, const DigestLaunch& l, cudaStream_t s);

}  // namespace hfgpu
