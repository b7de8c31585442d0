// FP64-accurate GEMM on the tcgen05 tensor cores (sm_103a) by exact bf16 slicing.
//
// C[r, c] = sum_k A[r, k] B[k, c] for FP64 A and B, as used by the AO->MO
// transforms.  Each row of A (and each column of B) is scaled by a power of two 2^e
// so that |x| < 2^e, rounded to a fixed-point integer and cut into NSL balanced
// 7-bit digits d_0 .. d_{NSL-1} (slice_bits.cuh), stored as bf16.  This is the
// error-free splitting of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59, 95
// (2012)) with bf16 tensor-core products: digit pairs (i, j) with i + j = t share a
// weight and are accumulated together in group t (t < NSL); every group's FP32 sum
// is exact; the epilogue recombines the groups in int64 and applies the row and
// column scales.  Six digits (21 products) keep each entry to 2^-42 of its row's or
// column's scale; nine digits (45 products) keep 2^-62, and entries that are small against
// those scales are formed again in FP64 (fp64_entries_kernel).
//
// Kernel: persistent CTAs, one per SM, walk the 128 x T output tiles; a K step of 32
// is one pipeline stage.
//   * A: 16 producer warps gather their rows' FP64 elements (Src, gather_rows.cuh),
//     cut them and store the digits straight into the stage's shared-memory tiles in
//     the 64-byte-swizzled K-major layout the MMA reads (16-byte chunk c of row r at
//     c ^ ((r >> 1) & 3)).  Thread t: row t % 128, K quarter t / 128 (8 elements, one
//     chunk per plane); the elements of the next two steps are in flight.
//   * B: its planes are stacked as PLANES T rows of one K-major tile (one bulk copy
//     a stage, laid out by slice_kernel), so that digit plane i of A multiplies
//     consecutive planes of B in one product: column block j lands on group i + j by
//     starting at TMEM column (i + j) T.  The groups are taken in slots of three, so
//     that consecutive products write the same columns: 9 tcgen05.mma of up to 240
//     columns per 16 k instead of 21 of T.  (One product over all the planes that i
//     meets, whose column ranges overlap in part from one i to the next, ran 30%
//     slower: 44 against 34 ms for 16 waters' step 1 with the cutting left out.)
//   * The 17th warp issues the B loads (ahead, into every free stage) and the products.
//   * Producers read the accumulators of a finished tile back (tcgen05.ld) after they
//     have filled the first stage of the next one, so that the products have a stage to
//     go on with; with PLANES T <= 256 columns two sets of accumulators fit TMEM and the
//     products go on meanwhile too.
// Bound: the producers' instructions (gather, cut, read back), then shared-memory
// bandwidth (a 32 k step of 80 columns reads 180 KB for its products beside the 78 KB
// written).  Transform step 1 against separate products per digit pair, accumulators
// read back at a tile barrier and B as tensor-map tiles: 8 waters (N = 40) 6.9 ->
// 3.5 ms, 16 waters (N = 80) 77 -> 55 ms; all four steps 12.4 -> 7.0 and 187 -> 130.
// Every wait on an mbarrier is bounded and reports a timeout through an error flag
// instead of spinning forever.
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <type_traits>

#include "internal.h"
#include "gather_rows.cuh"
#include "slice_bits.cuh"
#include "tcgemm.h"

namespace hfgpu {

constexpr int BM = 128, BK = 32;
constexpr int A_TILE = BM * BK * 2;  // 8 KiB: one digit plane of a stage
constexpr uint32_t TMEM_COLS = 512;
constexpr int WAIT_SPINS = 1 << 20;  // of up to 2 us each
constexpr int COPY_SPINS = 1 << 10;  // for a copy in flight, which needs microseconds
constexpr int GATHER_PRODUCERS = 512, PRODUCER_WARPS = GATHER_PRODUCERS / 32;
constexpr int GATHER_THREADS = GATHER_PRODUCERS + 32;
constexpr int MAX_STAGES = 4, MAX_OPS = 19;
// planes of a stage: the digits, and with nine the magnitudes (scaled_abs) whose product
// tells which entries the digits are good enough for
template <int NSL>
constexpr int PLANES = NSL + (NSL == SLICE_FP64 ? 1 : 0);

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}

// the same, suspended for up to about `ns` while the phase is open: polling would take
// issue slots from the warps that cut digits
__device__ __forceinline__ bool mbar_try_wait_ns(uint64_t* bar, uint32_t phase, uint32_t ns)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(bar)), "r"(phase), "r"(ns)
        : "memory");
    return ok != 0;
}

// bounded wait on an mbarrier phase; false after `spins` polls
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, int spins = WAIT_SPINS)
{
    for (int i = 0; i < spins; ++i)
        if (mbar_try_wait_ns(bar, phase, 2000)) return true;
    return false;
}

// contiguous copy into shared memory (16-byte aligned, bytes a multiple of 16)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, int bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(su32(dst)),
                 "l"(src), "r"(bytes), "r"(su32(bar))
                 : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand tile with 64-byte swizzle (rows of BK = 32
// bf16): 8-row groups 512 B apart
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;              // leading byte offset (not used by swizzled K-major)
    d |= (uint64_t)(512 >> 4) << 32;     // stride byte offset
    d |= (uint64_t)1 << 46;              // descriptor version
    d |= (uint64_t)4 << 61;              // 64-byte swizzle
    return d;
}

// kind::f16 instruction descriptor: BF16 x BF16 -> FP32, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t idesc(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t dt, uint64_t ad, uint64_t bd, uint32_t id, uint32_t acc)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dt),
        "l"(ad), "l"(bd), "r"(id), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(bar)) : "memory");
}

// four consecutive columns of the calling warp's 32 lanes (no wait)
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
// wait for the loads queued so far; the registers pass through so that nothing reads
// them earlier
template <int N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[N][4])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int t = 0; t < N; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) asm volatile("" : "+r"(r[t][i]));
}

// 2^e for any integer e (0 below the normal range, where the scaled values of
// the transform are far below anything that matters)
__device__ __forceinline__ double pow2(int e)
{
    if (e < -1022) return 0.0;
    if (e > 1023) e = 1023;
    return __longlong_as_double((int64_t)(e + 1023) << 52);
}

// v 2^E, by the exponent field where v is zero or |E| leaves the result normal (v is an
// integer below 2^120 in magnitude)
__device__ __forceinline__ double scale_pow2(double v, int E)
{
    const int hi = __double2hiint(v);
    if ((unsigned)(E + 900) <= 1800u) return __hiloint2double((hi << 1) == 0 ? hi : hi + (E << 20), __double2loint(v));
    return v * pow2(E);
}

__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}

// group sums (integers, |a_t| <= 2^24) -> sum_t a_t 2^(7 (NSL - 1 - t)), rounded once to
// FP64 and times 2^E: 32 x 32 + 64-bit multiply-adds, and one or two conversions on
// the FP64 pipe (they overlap the integer work of other warps).
template <int NSL>
__device__ __forceinline__ double recombine(const uint32_t (&a)[NSL], int E)
{
    int v[NSL];
#pragma unroll
    for (int t = 0; t < NSL; ++t) v[t] = __float2int_rn(__uint_as_float(a[t]));
    // groups 0 .. 3, below 2^47
    const long long hi = mad_wide(v[0], 1 << 21, mad_wide(v[1], 1 << 14, mad_wide(v[2], 1 << 7, v[3])));
    if constexpr (NSL == 6) {
        return scale_pow2((double)(mad_wide(v[4], 1 << 7, v[5]) + (hi << 14)), E);
    } else {  // both parts are exact in FP64 (below 2^53)
        const long long lo = mad_wide(v[4], 1 << 28, mad_wide(v[5], 1 << 21, mad_wide(v[6], 1 << 14, mad_wide(v[7], 1 << 7, v[8]))));
        return scale_pow2(fma((double)hi, 34359738368.0, (double)lo), E);
    }
}

// digit plane t of two elements as packed bf16 (element a in the low half)
template <int NSL, int T>
__device__ __forceinline__ uint32_t digit_word(uint64_t Ua, uint64_t Ub)
{
    uint32_t w;
    if constexpr (NSL == 6 && T == 0) {  // u - 128 with u <= 256, by FP32
        const float fa = __uint_as_float(0x4B000000u | digit_field<6>(Ua, 0)) - 8388736.0f;
        const float fb = __uint_as_float(0x4B000000u | digit_field<6>(Ub, 0)) - 8388736.0f;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(fb), "f"(fa));
    } else {
        const uint32_t u = 0x43004300u | digit_field<NSL>(Ua, T) | (digit_field<NSL>(Ub, T) << 16);
        asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(w) : "r"(u), "r"(0x43404340u));
    }
    return w;
}

template <int NSL, int T = 0>
__device__ __forceinline__ void digit_words(uint64_t Ua, uint64_t Ub, uint32_t (&w)[NSL])
{
    if constexpr (T < NSL) {
        w[T] = digit_word<NSL, T>(Ua, Ub);
        digit_words<NSL, T + 1>(Ua, Ub, w);
    }
}

constexpr unsigned HI_INF = 0x7FF00000u, HI_NORMAL = 1u << 20;  // upper words
constexpr int FAR_EXPONENT = 1 << 20;

// row exponent from the upper word of the largest |x| of the row: |x| < 2^e for every
// x in the row (0 for a row without normal numbers, whose digits are all zero)
__device__ __forceinline__ int row_exponent(unsigned amax_hi)
{
    return amax_hi < (1u << 20) ? 0 : (int)(amax_hi >> 20) - 1022;
}

// |x| 2^-e < 1 as bf16, rounded down (0 below 2^-126)
__device__ __forceinline__ uint32_t scaled_abs(double x, int e)
{
    const int u = ((__double2hiint(x) & 0x7FFFFFFF) >> 13) - ((896 + e) << 7);
    return u < 128 ? 0u : (uint32_t)u;
}

// the digits (and magnitudes) of two elements as packed bf16
template <int NSL>
__device__ __forceinline__ void cut2(double x0, double x1, int e, uint32_t (&w)[PLANES<NSL>])
{
    uint32_t d[NSL];
    digit_words<NSL>(biased_digits<NSL>((uint64_t)__double_as_longlong(x0), e),
                     biased_digits<NSL>((uint64_t)__double_as_longlong(x1), e), d);
#pragma unroll
    for (int t = 0; t < NSL; ++t) w[t] = d[t];
    if constexpr (NSL == SLICE_FP64) w[NSL] = scaled_abs(x0, e) | scaled_abs(x1, e) << 16;
}

// the digits of 8 consecutive elements of a row whose largest |x| has upper word amax_hi
template <int NSL>
__device__ __forceinline__ void cut8(const double (&x)[8], unsigned amax_hi, uint32_t (&w)[4][PLANES<NSL>])
{
    const int e = row_exponent(amax_hi);
#pragma unroll
    for (int j = 0; j < 8; j += 2) cut2<NSL>(x[j], x[j + 1], e, w[j / 2]);
}

// ------------------------------------------------------------------ slicing of B
// One warp per row (a column of B): its exponent, then every element's digits, laid out
// as the GEMM's stages take them: per column tile and K step, PLANES T rows (plane major)
// of 32 bf16, already swizzled, so that a stage's B is one contiguous bulk copy.  (As
// NSL tensor-map tiles of T 64-byte rows a step's B took longer to arrive than its A
// to be cut: 16 waters, step 1 70 ms; see the kernel.)
template <int NSL>
__global__ void slice_kernel(const double* __restrict__ A, int64_t ld, int64_t rows, int K, int T, int ksteps,
                             uint16_t* planes, int* rexp, double* b)
{
    constexpr int NP = PLANES<NSL>;
    const int lane = threadIdx.x & 31;
    const int64_t nwarp = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nwarp) {
        const double* row = A + r * ld;
        unsigned m = 0u;
        for (int k = lane; k < K; k += 32) m = max(m, (unsigned)__double2hiint(row[k]) & 0x7FFFFFFFu);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int e = row_exponent(m);
        // with nine digits, columns that digits cannot hold are told apart by their exponent
        if (lane == 0) rexp[r] = NSL == SLICE_FP64 && (m >= HI_INF || m < HI_NORMAL) ? FAR_EXPONENT : e;
        const int nt = (int)(r / T), c = (int)(r - (int64_t)nt * T);
        for (int k = lane; k < K; k += 32) {
            if (NSL == SLICE_FP64) b[k * rows + r] = row[k];
            uint32_t w[NP];
            cut2<NSL>(row[k], row[k], e, w);
#pragma unroll
            for (int t = 0; t < NP; ++t) {
                const int row = t * T + c;
                const int chunk = ((k & 31) >> 3) ^ ((row >> 1) & 3);  // 64-byte swizzle
                planes[(((int64_t)nt * ksteps + (k >> 5)) * (NP * T) + row) * BK + chunk * 8 + (k & 7)] = (uint16_t)w[t];
            }
        }
    }
}

// ------------------------------------------------------------------ GEMM kernel
// Nine digits stand in for plain FP64, so every entry has to be as good as an FP64 sum,
// which is within K 2^-53 S of it, S = sum_k |A_rk B_kc|.  Digits keep an element to 2^-63
// of its row's 2^e and leave out the products i + j >= 9, less than 1.01 2^-60 of 2^(ea + eb)
// each k: 1.26 K 2^(ea + eb - 60) in all, a third of K 2^-53 S where S = 2^(ea + eb - 5).  (On
// the average, sqrt(K) 2^(ea + eb - 63), the two meet there: rounding leaves about
// 2^-54.5 S in an FP64 sum of terms of random sign.)  Entries with a smaller S, their row
// and column large in different places as with orbitals on distant molecules, are left
// to fp64_entries_kernel: the magnitudes' product is S to 2 parts in 2^7, from below.  So
// are those whose scales leave FP64's range, and every entry of a row or column with
// an Inf or a NaN, which digits cannot hold, or with subnormals alone.
constexpr float FP64_S = 1.0f / 32;
constexpr long long TO_REDO = 0x7FF8DEADBEEF5EEDll;

struct GatherArgs {
    const unsigned char* b;  // B's stages (slice_kernel)
    int K, ksteps;
    int T, nst, stage, nbuf, slot;  // tile columns, pipeline stages, bytes of one, accumulator sets, groups of a slot
    int N, ntn, M, ntiles;
    const int* eb;
    double* out;
    OutMap om;
    int* err;
    int spins;  // of a wait (WAIT_SPINS; fewer to test what follows when one runs out)
};

template <class Src, int NSL>
__global__ void __launch_bounds__(GATHER_THREADS, 1)
    gather_gemm_kernel(const Src src, const GatherArgs g)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES];  // stage filled / its products done
    __shared__ uint64_t acc_full[2], acc_empty[2];            // accumulators complete / read back
    // the products of 16 k: TMEM column (bit 31: plane 0 of A, which writes its groups
    // first), descriptor offsets of A and B (16-byte units), instruction descriptor
    __shared__ uint4 ops[MAX_OPS];
    __shared__ uint32_t tslot;
    __shared__ int s_ok;
    constexpr int NP = PLANES<NSL>;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int T = g.T, nst = g.nst, nbuf = g.nbuf, ksteps = g.ksteps;
    if (tid == 0) {
        for (int s = 0; s < nst; ++s) {
            mbar_init(&full[s], PRODUCER_WARPS + 1);  // every producer warp + the B expect_tx
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], PRODUCER_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ok = 1;
        // slots of g.slot groups; plane i of A writes groups max(i, g0) .. g1 - 1 of each
        int k = 0;
        for (int g0 = (NSL - 1) / g.slot * g.slot; g0 >= 0; g0 -= g.slot) {
            const int g1 = min(g0 + g.slot, NSL);
            for (int i = 0; i < g1; ++i) {
                const int first = max(i, g0);
                ops[k++] = make_uint4((uint32_t)(first * T) | (i == 0 ? 0x80000000u : 0u), (uint32_t)(i * (A_TILE >> 4)),
                                      (uint32_t)((first - i) * T * (BK * 2) >> 4), idesc(((g1 - first) * T + 15) & ~15));
            }
        }
        if (NP > NSL)  // magnitudes: a group of their own
            ops[k] = make_uint4((uint32_t)(NSL * T) | 0x80000000u, (uint32_t)(NSL * (A_TILE >> 4)),
                                (uint32_t)(NSL * T * (BK * 2) >> 4), idesc(T));
    }
    const int nops = (g.slot == NSL ? NSL : NSL == 6 ? 9 : 18) + NP - NSL;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tslot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tslot;
    auto stage_a = [&](int s) { return smem + s * g.stage; };
    auto stage_b = [&](int s) { return smem + s * g.stage + NP * A_TILE; };

    bool ok = true;
    if (warp == PRODUCER_WARPS) {
        if (lane == 0) {
            // B loads run ahead into every stage already free; step q of the CTA's whole
            // sequence uses stage q % nst for the (q / nst)-th time
            int sl = 0, sl_use = 0;        // next stage to load, how often it was used
            int ks_l = 0;                  // its K step
            int tile_l = blockIdx.x;       // its tile
            int ahead = 0;                 // loads issued beyond the step being multiplied
            int last_commit = -1, last_commit_use = 0;
            int s = 0, use = 0, lt = 0;
            const int b_bytes = NP * T * BK * 2;
            for (int tile = blockIdx.x; tile < g.ntiles && ok; tile += gridDim.x, ++lt) {
                const int buf = nbuf == 2 ? lt & 1 : 0;
                const uint32_t acc = tmem + (uint32_t)(buf * 256);
                for (int ks = 0; ks < ksteps && ok; ++ks) {
                    while (tile_l < g.ntiles && ahead < nst) {
                        if (sl_use > 0) {
                            const uint32_t ph = (uint32_t)(sl_use - 1) & 1u;
                            if (ahead == 0) {
                                if (!mbar_wait(&empty[sl], ph, g.spins)) {
                                    ok = false;
                                    break;
                                }
                            } else if (!mbar_try_wait(&empty[sl], ph)) {
                                break;
                            }
                        }
                        mbar_expect_tx(&full[sl], b_bytes);
                        bulk_load(stage_b(sl), g.b + (int64_t)((tile_l % g.ntn) * ksteps + ks_l) * b_bytes, b_bytes,
                                  &full[sl]);
                        ++ahead;
                        if (++sl == nst) {
                            sl = 0;
                            ++sl_use;
                        }
                        if (++ks_l == ksteps) {
                            ks_l = 0;
                            tile_l += gridDim.x;
                        }
                    }
                    if (!ok) break;
                    if (ks == 0 && lt >= nbuf) {  // the tile that used these accumulators has been read back
                        if (!mbar_wait(&acc_empty[buf], (uint32_t)(lt / nbuf - 1) & 1u, g.spins)) {
                            ok = false;
                            break;
                        }
                    }
                    if (!mbar_wait(&full[s], (uint32_t)use & 1u, g.spins)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint64_t a0 = sdesc(su32(stage_a(s))), b0 = sdesc(su32(stage_b(s)));
                    const bool second = g.K - ks * BK > 16;  // the step's second 16 k hold elements
#pragma unroll 3
                    for (int k = 0; k < nops; ++k) {  // kk innermost: the same columns twice in a row
                        const uint4 op = ops[k];
                        const uint32_t dt = acc + (op.x & 0xFFFFu);
                        umma(dt, a0 + op.y, b0 + op.z, op.w, ks == 0 ? (op.x >> 31) ^ 1u : 1u);
                        if (second) umma(dt, a0 + op.y + 2, b0 + op.z + 2, op.w, 1u);
                    }
                    umma_commit(&empty[s]);
                    if (ks == ksteps - 1) umma_commit(&acc_full[buf]);
                    last_commit = s;
                    last_commit_use = use;
                    --ahead;
                    if (++s == nst) {
                        s = 0;
                        ++use;
                    }
                }
            }
            // every B copy and all products in flight land before shared memory and TMEM go
            // (a stage whose producers gave up never fills: its copy is waited out)
            if (!ok) {
                atomicExch(&s_ok, 0);
                for (; ahead > 0; --ahead) {
                    mbar_wait(&full[s], (uint32_t)use & 1u, COPY_SPINS);
                    if (++s == nst) {
                        s = 0;
                        ++use;
                    }
                }
            }
            if (last_commit >= 0) mbar_wait(&empty[last_commit], (uint32_t)last_commit_use & 1u);
        }
    } else {
        const int prow = tid & (BM - 1), part = tid / BM;  // row of the tile, K quarter of a stage
        const int chunk = part ^ ((prow >> 1) & 3);
        // the tile and step that are fetched next, up to two steps ahead of the cutting
        // (32-bit tile arithmetic: 64-bit divisions would cost as much as the digits)
        int tile_f = blockIdx.x, ks_f = 0;
        bool live_f = false;
        typename Src::Row row_f{};
        unsigned amax_f = 0;
        auto open_row = [&] {
            amax_f = 0;
            live_f = tile_f < g.ntiles && src.open((int)((unsigned)tile_f / (unsigned)g.ntn) * BM + prow, g.M, row_f, amax_f);
        };
        auto fetch = [&](double(&x)[8], unsigned& amax) {
            const int k0 = ks_f * BK + part * 8;
            amax = amax_f;
            if (live_f && k0 + 8 <= g.K) {
                src.load8(row_f, k0, x);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = (live_f && k0 + j < g.K) ? src.at(row_f, k0 + j) : 0.0;
            }
            if (++ks_f == ksteps) {
                ks_f = 0;
                tile_f += gridDim.x;
                open_row();
            }
        };
        // read the accumulators of the CTA's tile number lt back: TMEM lanes 32 (warp % 4),
        // every fourth group of four columns
        const int cstep = g.om.R > 0 ? (int)g.om.R : 1;
        auto epilogue = [&](int tile, int lt) {
            const int buf = nbuf == 2 ? lt & 1 : 0;
            const int mt = (int)((unsigned)tile / (unsigned)g.ntn), n0 = (tile - mt * g.ntn) * T;
            int64_t off = 0;
            unsigned amax = 0;
            const bool lv = src.place(mt * BM + (warp & 3) * 32 + lane, g.M, (int)g.om.R, g.om.ld, off, amax);
            const int er = NSL == SLICE_FP64 && amax >= HI_INF ? FAR_EXPONENT : row_exponent(amax);
            double* orow = g.out + off;
            // (lanes that disagreed on a wait would part before the warp's next barrier)
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(&acc_full[buf], (uint32_t)(nbuf == 2 ? lt >> 1 : lt) & 1u, g.spins)))
                return false;
            fence_after();
            const uint32_t ta = tmem + (uint32_t)(buf * 256) + ((uint32_t)((warp & 3) * 32) << 16);
            for (int c0 = (warp >> 2) * 4; c0 < T && n0 + c0 < g.N; c0 += PRODUCER_WARPS) {
                uint32_t f[NP][4];
#pragma unroll
                for (int t = 0; t < NP; ++t) tmem_ld4(ta + (uint32_t)(t * T + c0), f[t]);
                tmem_wait_ld(f);
                const int c = n0 + c0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t a[NSL];
#pragma unroll
                    for (int t = 0; t < NSL; ++t) a[t] = f[t][i];
                    if (lv && c + i < g.N) {
                        const int E = er + __ldg(g.eb + c + i);
                        double v = recombine<NSL>(a, E - SliceFmt<NSL>::SHIFT);
                        if constexpr (NSL == SLICE_FP64)
                            if ((unsigned)(E + 800) > 1600u || (amax != 0u && __uint_as_float(f[NSL][i]) < FP64_S))
                                v = __longlong_as_double(TO_REDO);
                        orow[(int64_t)(c + i) * cstep] = v;
                    }
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
            return true;
        };

        open_row();
        double x0[8], x1[8];
        unsigned m0, m1;
        fetch(x0, m0);
        fetch(x1, m1);
        int s = 0, use = 0, lt = 0, prev = -1, tile = blockIdx.x, ks = 0;
        // one K step from x; false at the end of the tiles or after a timeout.  (One copy of
        // this code, with the two buffers swapped after it: two copies, or a second way to
        // cut digits on the FP32 pipe, ran slower from instruction fetches.)
        auto step = [&](double(&x)[8], unsigned& amax) {
            uint32_t w[4][NP];
            const bool has = ks * BK + part * 8 < g.K;
            if (has) cut8<NSL>(x, amax, w);
            fetch(x, amax);  // in flight while this step is stored and the next one is cut
            if (use > 0 && !__all_sync(0xFFFFFFFFu, mbar_wait(&empty[s], (uint32_t)(use - 1) & 1u, g.spins)))
                return ok = false;
            unsigned char* dst = stage_a(s) + prow * 64 + chunk * 16;
#pragma unroll
            for (int t = 0; t < NP; ++t)
                *reinterpret_cast<uint4*>(dst + t * A_TILE) =
                    has ? make_uint4(w[0][t], w[1][t], w[2][t], w[3][t]) : make_uint4(0u, 0u, 0u, 0u);
            // the tensor core reads shared memory through the async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            if (++s == nst) {
                s = 0;
                ++use;
            }
            // the previous tile is read back once the first step of this one is filled
            if (ks == 0 && prev >= 0 && !epilogue(prev, lt - 1)) return ok = false;
            if (++ks == ksteps) {
                ks = 0;
                prev = tile;
                tile += gridDim.x;
                ++lt;
            }
            return tile < g.ntiles;
        };
        while (step(x0, m0)) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const double t = x0[j];
                x0[j] = x1[j];
                x1[j] = t;
            }
            const unsigned t = m0;
            m0 = m1;
            m1 = t;
        }
        if (ok && prev >= 0) ok = epilogue(prev, lt - 1);
        if (!ok) atomicExch(&s_ok, 0);
    }
    fence_before();
    __syncthreads();
    if (tid == 0 && !s_ok) atomicExch(g.err, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// ------------------------------------------------------------------ nine digits: entries in FP64
// Forms the entries that the GEMM left as TO_REDO as FP64 sums in the order of k, as the
// FP64 GEMM (dgemm_rows.cu) forms them.  A block walks 128-row tiles of the output, lists
// them and does them 256 at a time, one per thread, so that its warps are full however the
// entries lie.  Bound: the FP64 pipe, 83 to 94% busy at 6 waters (35 M entries of 150 terms
// in 12.2 ms).
struct Fp64Args {
    const double* b;  // K x N: the lanes of a warp mostly have one row and different columns, or the reverse
    int K, N, M;
    double* out;
    OutMap om;
};

constexpr int FP64_THREADS = 256, FP64_CHUNK = 4 * FP64_THREADS;

template <class Src>
__global__ void __launch_bounds__(FP64_THREADS) fp64_entries_kernel(const Src src, const Fp64Args g)
{
    __shared__ int2 list[FP64_THREADS + FP64_CHUNK];
    __shared__ int count, tiny[BM];
    __shared__ int64_t off[BM];
    const int t = threadIdx.x, R = (int)g.om.R;
    const int64_t cstep = R > 0 ? R : 1;
    auto redo = [&](int2 e) {
        typename Src::Row w{};
        unsigned m;
        src.open(e.x, g.M, w, m);
        const double* b = g.b + e.y;
        double s = 0.0;
        int k = 0;
        for (; k + 8 <= g.K; k += 8) {
            double x[8];
            src.load8(w, k, x);
#pragma unroll
            for (int j = 0; j < 8; ++j) s = fma(x[j], __ldg(b + (k + j) * g.N), s);
        }
        for (; k < g.K; ++k) s = fma(src.at(w, k), __ldg(b + k * g.N), s);
        int64_t o;
        src.place(e.x, g.M, R, g.om.ld, o, m);
        g.out[o + e.y * cstep] = s;
    };
    if (t == 0) count = 0;
    const int ntm = (g.M + BM - 1) / BM;
    for (int tile = blockIdx.x; tile < ntm; tile += gridDim.x) {
        __syncthreads();  // the last tile's off and tiny
        if (t < BM) {
            unsigned m = 0u;
            const bool live = src.place(tile * BM + t, g.M, R, g.om.ld, off[t], m);
            if (!live) off[t] = -1;
            tiny[t] = live && m == 0u ? -1 : 0;
        }
        __syncthreads();
        // the maxima are upper words: of a row with 0 there, is anything left below?
        if (tiny[t % BM]) {
            typename Src::Row w{};
            unsigned m, any = 0u;
            src.open(tile * BM + t % BM, g.M, w, m);
#pragma unroll 8
            for (int k = t / BM; k < g.K; k += FP64_THREADS / BM) any |= (unsigned)__double2loint(src.at(w, k));
            if (any) tiny[t % BM] = 1;
        }
        __syncthreads();
        for (int e0 = 0; e0 < BM * g.N; e0 += FP64_CHUNK) {
            for (int e = e0 + t; e < min(e0 + FP64_CHUNK, BM * g.N); e += FP64_THREADS) {
                // the outputs' order: rows fastest in blocks of R rows, else columns
                const int r = R > 0 ? e & (BM - 1) : e / g.N, c = R > 0 ? e / BM : e - r * g.N;
                if (off[r] < 0) continue;
                if (tiny[r] > 0 || __double_as_longlong(g.out[off[r] + c * cstep]) == TO_REDO)
                    list[atomicAdd(&count, 1)] = make_int2(tile * BM + r, c);
            }
            __syncthreads();
            int have = count;
            __syncthreads();
            if (have >= FP64_THREADS) {
                for (; have >= FP64_THREADS; have -= FP64_THREADS) redo(list[have - FP64_THREADS + t]);
                if (t == 0) count = have;
                __syncthreads();
            }
        }
    }
    __syncthreads();
    if (t < count) redo(list[t]);
}

template <class Src>
static void fp64_entries(Context& ctx, const Src& src, int M, int K, const Sliced& B, double* out, OutMap om)
{
    HF_CHECK(B.rows < (1 << 20), HFGPU_ERR_UNSUPPORTED, "sliced GEMM: column count");
    const Fp64Args g{B.b.p, K, (int)B.rows, M, out, om};
    const unsigned grid = (unsigned)std::min((M + BM - 1) / BM, ctx.num_sms * 8);
    fp64_entries_kernel<Src><<<grid, FP64_THREADS, 0, ctx.stream>>>(src, g);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------ host side
int slice_kmax(int digits) { return digits == SLICE_MIXED ? SliceFmt<6>::KMAX : SliceFmt<9>::KMAX; }

static int slice_planes(int digits) { return digits == SLICE_MIXED ? PLANES<SLICE_MIXED> : PLANES<SLICE_FP64>; }

// Columns of a tile for N columns of B: the fewest tiles (every tile gathers and cuts
// the A rows again) that fit the TMEM columns, evenly filled, a multiple of 16 (the
// granularity of a product's columns); or 40, for 33 to 40 columns of six digits: 240
// accumulator columns leave room for a second set, 48 x 6 would not (8 waters, step 1:
// 4.1 against 5.1 ms).
static int tile_columns(int64_t N, int digits)
{
    if (digits == SLICE_MIXED && N > 32 && N <= 40) return 40;
    const int most = (int)TMEM_COLS / slice_planes(digits) / 16 * 16;  // 80 with six digits, 48 with nine
    const int64_t ntn = (N + most - 1) / most;
    return (int)(((N + ntn - 1) / ntn + 15) / 16 * 16);
}

void slice_dense(Context& ctx, const double* A, int64_t rows, int K, int64_t ld, int digits, Sliced& s)
{
    HF_CHECK(K >= 1 && K <= slice_kmax(digits), HFGPU_ERR_UNSUPPORTED,
             "sliced GEMM supports 1 <= K <= " + std::to_string(slice_kmax(digits)));
    s.rows = rows;
    s.K = K;
    s.digits = digits;
    s.spins = WAIT_SPINS;
    s.tile = tile_columns(rows, digits);
    s.rows_pad = (rows + s.tile - 1) / s.tile * s.tile;
    s.ksteps = (K + BK - 1) / BK;
    const size_t need = (size_t)slice_planes(digits) * s.rows_pad * s.ksteps * BK;
    s.planes.alloc(need, ctx.stream);
    s.rexp.alloc(s.rows_pad, ctx.stream);
    if (digits == SLICE_FP64) s.b.alloc((size_t)rows * K, ctx.stream);
    HF_CUDA(cudaMemsetAsync(s.planes.p, 0, need * sizeof(__nv_bfloat16), ctx.stream));
    const int64_t warps = std::min<int64_t>(rows, (int64_t)ctx.num_sms * 64);
    const unsigned blocks = (unsigned)std::max<int64_t>(1, (warps * 32 + 255) / 256);
    uint16_t* pl = reinterpret_cast<uint16_t*>(s.planes.p);
    if (digits == SLICE_MIXED)
        slice_kernel<6><<<blocks, 256, 0, ctx.stream>>>(A, ld, rows, K, s.tile, s.ksteps, pl, s.rexp.p, s.b.p);
    else
        slice_kernel<9><<<blocks, 256, 0, ctx.stream>>>(A, ld, rows, K, s.tile, s.ksteps, pl, s.rexp.p, s.b.p);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

// (M: rows of the launch, dead ones included; M_rows: the live rows, for the flop count)
template <class Src, int NSL>
static void gather_gemm_n(Context& ctx, const Src& src, int64_t M, int64_t M_rows, int K, const Sliced& B, double* out,
                          OutMap om)
{
    HF_CHECK(K == B.K, HFGPU_ERR_INVALID, "gather GEMM: K mismatch");
    GatherArgs g;
    g.b = reinterpret_cast<const unsigned char*>(B.planes.p);
    g.K = K;
    g.ksteps = B.ksteps;
    g.T = B.tile;
    g.N = (int)B.rows;
    g.ntn = (int)(B.rows_pad / B.tile);
    const int64_t ntiles = (M + BM - 1) / BM * g.ntn;
    HF_CHECK(ntiles > 0 && M < (1ll << 30) && ntiles < (1ll << 30), HFGPU_ERR_INVALID, "gather GEMM: row count");
    HF_CHECK((std::is_same_v<Src, DenseRowsG> || om.R == K), HFGPU_ERR_INVALID, "gather GEMM: output placement");
    g.M = (int)M;
    g.ntiles = (int)ntiles;
    g.nbuf = PLANES<NSL> * g.T <= 256 ? 2 : 1;
    // slots of three groups where every product's columns are a multiple of 16; else all
    // groups in one: a padded product then writes only past the last group, into the 8
    // spare columns of a set (and reads B rows of the next plane)
    g.slot = g.T % 16 == 0 ? 3 : NSL;
    HF_CHECK(g.slot == 3 || NSL * g.T + 8 <= 256, HFGPU_ERR_INVALID, "gather GEMM: tile columns");
    g.stage = (PLANES<NSL> * (A_TILE + g.T * BK * 2) + 1023) / 1024 * 1024;  // the planes of A and of B
    g.eb = B.rexp.p;
    g.out = out;
    g.om = om;
    static std::once_flag once;
    static size_t most = 0;
    std::call_once(once, [] {
        int dev = 0, optin = 0;
        cudaFuncAttributes fa{};
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            cudaFuncGetAttributes(&fa, gather_gemm_kernel<Src, NSL>) != cudaSuccess)
            return;
        const size_t m = (size_t)optin - fa.sharedSizeBytes;
        if (cudaFuncSetAttribute(gather_gemm_kernel<Src, NSL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)m) ==
            cudaSuccess)
            most = m;
    });
    g.nst = (int)std::min<size_t>(MAX_STAGES, most > 1024 ? (most - 1024) / g.stage : 0);
    HF_CHECK(g.nst >= 2, HFGPU_ERR_CUDA, "gather GEMM: shared memory attribute");
    if (!ctx.tc_err) {
        HF_CUDA(cudaMalloc((void**)&ctx.tc_err, sizeof(int)));
        HF_CUDA(cudaMemsetAsync(ctx.tc_err, 0, sizeof(int), ctx.stream));
    }
    g.err = ctx.tc_err;
    g.spins = B.spins;
    Context::TcTimer t;
    HF_CUDA(cudaEventCreate(&t.a));
    HF_CUDA(cudaEventCreate(&t.b));
    t.step1 = std::is_same_v<Src, PackedRowsBlocked>;
    t.flops = 2.0 * (NSL * (NSL + 1) / 2) * (double)M_rows * (double)B.rows * (double)K;
    HF_CUDA(cudaEventRecord(t.a, ctx.stream));
    const unsigned grid = (unsigned)std::min<int64_t>(g.ntiles, ctx.num_sms);
    gather_gemm_kernel<Src, NSL><<<grid, GATHER_THREADS, g.nst * g.stage + 1024, ctx.stream>>>(src, g);
    count_launch();
    HF_CUDA(cudaGetLastError());
    HF_CUDA(cudaEventRecord(t.b, ctx.stream));
    ctx.tc_events.push_back(t);
    if constexpr (NSL == SLICE_FP64) fp64_entries(ctx, src, g.M, K, B, out, om);
}

template <class Src>
static void gather_gemm(Context& ctx, const Src& src, int64_t M, int64_t M_rows, int K, const Sliced& B, double* out,
                        OutMap om)
{
    if (B.digits == SLICE_MIXED)
        gather_gemm_n<Src, 6>(ctx, src, M, M_rows, K, B, out, om);
    else
        gather_gemm_n<Src, 9>(ctx, src, M, M_rows, K, B, out, om);
}

SlicedRun::~SlicedRun()
{
    if (ctx.tc_events.empty()) return;  // settled
    for (auto& t : ctx.tc_events) {
        cudaEventDestroy(t.a);
        cudaEventDestroy(t.b);
    }
    ctx.tc_events.clear();
    if (ctx.tc_err) cudaMemsetAsync(ctx.tc_err, 0, sizeof(int), ctx.stream);  // after the GEMMs
}

void SlicedRun::settle()
{
    int h = 0;
    if (ctx.tc_err) {
        HF_CUDA(cudaMemcpyAsync(&h, ctx.tc_err, sizeof(int), cudaMemcpyDeviceToHost, ctx.stream));
        HF_CUDA(cudaMemsetAsync(ctx.tc_err, 0, sizeof(int), ctx.stream));
    }
    HF_CUDA(cudaStreamSynchronize(ctx.stream));
    for (auto& t : ctx.tc_events) {
        float ms = 0;
        HF_CUDA(cudaEventElapsedTime(&ms, t.a, t.b));
        cudaEventDestroy(t.a);
        cudaEventDestroy(t.b);
        ctx.stat_tc_ms += ms;
        ctx.stat_tc_flops += t.flops;
        if (t.step1) {
            ctx.stat_tc_step1_ms += ms;
            ctx.stat_tc_step1_n += 1;
        }
    }
    ctx.tc_events.clear();
    HF_CHECK(h == 0, HFGPU_ERR_CUDA, "sliced GEMM: an mbarrier wait timed out");
}

// ---- row maxima for the gather-fed GEMM
// A row of the gather GEMM is (pair a, la) over si of M[a][pair(la, si)], or
// (q, mu) over nu of Zt[q][pair(mu, nu)]: the maximum |x| over si is the
// maximum over the elements of the symmetric pair-row a whose pair contains la.
// Only its exponent is used (row_exponent), so the maxima are kept as the upper
// 32 bits of |x| (sign cleared), which order like |x| down to the exponent and
// stay on 32-bit integer instructions (64-bit compares and conversions run on
// this GPU's narrow FP64 pipe).
// Folding a stored row (elements kl = (la, si), la >= si, kl < len) onto basis
// indices: a warp takes one run kl = tri(la) .. tri(la) + la (consecutive si,
// coalesced loads); the run's maximum counts for la, and a
// lane keeps those of its own si = lane + 32 j over all runs of its warp in registers
// (a shared-memory atomicMax per element otherwise).
__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }
// the same straight from memory: the upper 32-bit word of the element, loaded as an integer
__device__ __forceinline__ unsigned abs_hi_at(const double* p)
{
    return __ldg(reinterpret_cast<const unsigned*>(p) + 1) & 0x7FFFFFFFu;
}

__device__ __forceinline__ unsigned warp_max_u32(unsigned v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// one CTA per stored row a: PACKED rows are the lower triangle of the packed
// integrals (row a = M[a][0 .. a], at a (a + 1) / 2); otherwise rows of length
// len_full at src + a * ld.  out[a * n + idx] = folded maximum.
// NJ: runs of up to 32 NJ elements.
template <bool PACKED, int NJ>
__global__ void __launch_bounds__(256) row_max_tri_kernel(const double* __restrict__ src, int64_t ld, int len_full,
                                                          int n, unsigned* out)
{
    extern __shared__ unsigned smax32[];
    const int a = blockIdx.x;
    const double* row = PACKED ? src + (int64_t)a * (a + 1) / 2 : src + (int64_t)a * ld;
    const int len = PACKED ? a + 1 : len_full;
    for (int i = threadIdx.x; i < n; i += blockDim.x) smax32[i] = 0u;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    constexpr int NG = NJ < 4 ? NJ : 4;  // loads of a run in flight
    unsigned own[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) own[j] = 0u;
    for (int la = warp; la < n; la += nw) {
        const int t0 = la * (la + 1) / 2;
        if (t0 >= len) break;  // later runs start further out
        const int smx = min(len - 1 - t0, la);
        unsigned m = 0u;
#pragma unroll
        for (int j0 = 0; j0 < NJ; j0 += NG)
            if (32 * j0 <= smx) {
                unsigned v[NG];
#pragma unroll
                for (int j = 0; j < NG; ++j) {
                    const int si = lane + 32 * (j0 + j);
                    v[j] = si <= smx ? abs_hi_at(row + t0 + si) : 0u;
                }
#pragma unroll
                for (int j = 0; j < NG; ++j) {
                    own[j0 + j] = max(own[j0 + j], v[j]);
                    m = max(m, v[j]);
                }
            }
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) atomicMax(&smax32[la], m);
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j)
        if (lane + 32 * j < n) atomicMax(&smax32[lane + 32 * j], own[j]);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[(int64_t)a * n + i] = smax32[i];
}

template <bool PACKED>
static void row_max_tri(Context& ctx, const double* src, int64_t ld, int len_full, int n, int64_t rows, unsigned* out)
{
    HF_CHECK(n <= 512, HFGPU_ERR_UNSUPPORTED, "row maxima: basis too large");
    auto kernel = n <= 64    ? row_max_tri_kernel<PACKED, 2>
                  : n <= 128 ? row_max_tri_kernel<PACKED, 4>
                  : n <= 256 ? row_max_tri_kernel<PACKED, 8>
                  : n <= 384 ? row_max_tri_kernel<PACKED, 12>
                             : row_max_tri_kernel<PACKED, 16>;
    kernel<<<(unsigned)rows, 256, n * sizeof(unsigned), ctx.stream>>>(src, ld, len_full, n, out);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

// the column part of the packed rows: M[a][b] = M[b][a] for b > a lives in
// stored row b.  A CTA takes 32 consecutive a (one per lane, so a warp's loads of
// row b are one 256-byte segment); a warp takes pairs b = (la, si) of COLS_LA
// consecutive la and COLS_SI consecutive si: their la maxima stay in registers and
// the si ones are merged before they go to shared memory, laid out [idx][lane]
// (padded), so an element costs 1 / COLS_LA of an atomicMax there instead of two.
// The block's maxima are merged into out by atomicMax.
constexpr int COLS_LA = 4, COLS_SI = 64, COLS_THREADS = 256, COLS_SPLIT = 4;
__global__ void __launch_bounds__(COLS_THREADS) row_max_cols_kernel(const double* __restrict__ ints, int npair, int n,
                                                            unsigned* out)
{
    extern __shared__ unsigned smax32[];  // n x 33
    const int a0 = blockIdx.x * 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int i = threadIdx.x; i < n * 33; i += blockDim.x) smax32[i] = 0u;
    __syncthreads();
    const int a = a0 + lane;
    int first = (int)((sqrtf(8.0f * (float)a0 + 1.0f) - 1.0f) * 0.5f);  // the la of pair a0
    while (first * (first + 1) / 2 > a0) --first;
    while ((first + 1) * (first + 2) / 2 <= a0) ++first;
    const int nseg = (n + COLS_SI - 1) / COLS_SI, g0 = first / COLS_LA, ng = (n + COLS_LA - 1) / COLS_LA;
    for (int t = blockIdx.y * nw + warp; t < (ng - g0) * nseg; t += nw * gridDim.y) {
        const int la0 = (ng - 1 - t / nseg) * COLS_LA, s0 = t % nseg * COLS_SI;  // the longest runs first
        const int s1 = min(s0 + COLS_SI, min(la0 + COLS_LA, n));
        unsigned m[COLS_LA];
        int b[COLS_LA];
        const double* p[COLS_LA];  // element (b, a): advances by b + 1 with b
#pragma unroll
        for (int u = 0; u < COLS_LA; ++u) {
            m[u] = 0u;
            b[u] = (la0 + u) * (la0 + u + 1) / 2 + s0;
            p[u] = ints + (((int64_t)b[u] * (b[u] + 1)) >> 1) + a;
        }
#pragma unroll 2
        for (int s = s0; s < s1; ++s) {
            unsigned v[COLS_LA];
#pragma unroll
            for (int u = 0; u < COLS_LA; ++u) {
                v[u] = (la0 + u < n && s <= la0 + u && b[u] > a) ? abs_hi_at(p[u]) : 0u;
                p[u] += ++b[u];
            }
            unsigned x = 0u;
#pragma unroll
            for (int u = 0; u < COLS_LA; ++u) {
                m[u] = max(m[u], v[u]);
                x = max(x, v[u]);
            }
            atomicMax(&smax32[s * 33 + lane], x);
        }
#pragma unroll
        for (int u = 0; u < COLS_LA; ++u)
            if (la0 + u < n) atomicMax(&smax32[(la0 + u) * 33 + lane], m[u]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * 32; i += blockDim.x) {
        const int idx = i >> 5, l = i & 31;
        const unsigned v = smax32[idx * 33 + l];
        if (a0 + l < npair && v) atomicMax(out + (int64_t)(a0 + l) * n + idx, v);
    }
}

void packed_row_max(Context& ctx, const double* ints, int n, unsigned* out)
{
    const int npair = n * (n + 1) / 2;
    row_max_tri<true>(ctx, ints, 0, 0, n, npair, out);
    const size_t smem = (size_t)n * 33 * sizeof(unsigned);
    static std::once_flag once;
    std::call_once(once, [] {
        cudaFuncSetAttribute(row_max_cols_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    });
    HF_CHECK(smem <= 200 * 1024, HFGPU_ERR_UNSUPPORTED, "row maxima: basis too large");
    // the first pairs have a whole triangle of rows: COLS_SPLIT CTAs share each 32 of them.
    // Both passes of 16 waters read 51 GB, 7.6 ms at copy speed: 11.7 -> 10.1 ms (8 waters
    // 0.83 -> 0.74); one CTA of 1024 threads per 32 pairs 11.7, 1.13
    const dim3 grid((unsigned)((npair + 31) / 32), COLS_SPLIT);
    row_max_cols_kernel<<<grid, COLS_THREADS, smem, ctx.stream>>>(ints, npair, n, out);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

void sympair_row_max(Context& ctx, const double* Zt, int64_t ldz, int64_t nq, int n, unsigned* out)
{
    const int npair = n * (n + 1) / 2;
    row_max_tri<false>(ctx, Zt, ldz, npair, n, nq, out);
}

// one warp per row: the upper word of max |x| over the row's K elements
__global__ void dense_row_max_kernel(const double* __restrict__ A, int64_t rows, int K, int64_t ld, unsigned* out)
{
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= rows) return;
    const double* row = A + r * ld;
    unsigned m = 0u;
    for (int k = lane; k < K; k += 32) m = max(m, abs_hi_at(row + k));
    m = warp_max_u32(m);
    if (lane == 0) out[r] = m;
}

void dense_row_max(Context& ctx, const double* A, int64_t rows, int K, int64_t ld, unsigned* out)
{
    dense_row_max_kernel<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, ctx.stream>>>(A, rows, K, ld, out);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

void sliced_gemm_dense(Context& ctx, const double* A, int64_t rows, int K, int64_t ld, const unsigned* rmax,
                       const Sliced& B, double* out, OutMap om)
{
    gather_gemm(ctx, DenseRowsG(A, ld, rmax), rows, rows, K, B, out, om);
}

void sliced_gemm_packed(Context& ctx, const double* ints, int64_t p0, int64_t npairs, int n, const unsigned* rmax,
                        const Sliced& B, double* out, OutMap om)
{
    const int nlg = (n + 15) / 16;
    const PackedRowsBlocked src{ints, p0, npairs, n, nlg, rmax};
    gather_gemm(ctx, src, (npairs + 7) / 8 * nlg * 128, npairs * n, n, B, out, om);
}

void sliced_gemm_sympair(Context& ctx, const double* Zt, int64_t ldz, int64_t nq, int n, const unsigned* rmax,
                         const Sliced& B, double* out, OutMap om)
{
    const SymPairRows src{Zt, ldz, n, rmax};
    gather_gemm(ctx, src, nq * n, nq * n, n, B, out, om);
}

}  // namespace hfgpu
