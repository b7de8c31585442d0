// Row sources of the gather-fed GEMMs (tcgemm.cu on the tensor cores,
// dgemm_rows.cu in FP64): each maps a row index r of the A operand to the
// elements of that row, gathered straight from where the transform keeps them
// (the packed AO integrals, Z transposed, or a dense row-major matrix), so that
// no unpacked copy of A goes through HBM.
//   row(r)       per-row state, computed once per row
//   at(w, k)     element k of the row
//   load8(w, k0, x)  elements k0 .. k0 + 7 (all within the row; k0 a multiple of 8)
//   live(r)      false for padding rows of blocked layouts (not loaded or stored)
//   out_row(r)   the row's place in the output's row order
//   open(r, M, w, amax)  false for a dead row (or r >= M); else its state and the upper
//                word of its largest |element|
//   place(r, M, R, ld, off, amax)  the same test; the output offset of column 0 and the
//                distance between columns is R (1 for R = 0), as OutMap places rows
// r is the row of a 128-row tile (r = 128 tile + row), below 2^31.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace hfgpu {

// dense row-major rows with stride ld (row maxima from dense_row_max)
struct DenseRowsG {
    const double* p;
    int64_t ld;
    const unsigned* rmax;
    bool pairs;  // every row starts on a 16-byte boundary (p and ld): 16-byte loads
    using Row = const double*;
    DenseRowsG(const double* p_, int64_t ld_, const unsigned* rmax_)
        : p(p_), ld(ld_), rmax(rmax_), pairs(((uintptr_t)p_ & 15) == 0 && (ld_ & 1) == 0)
    {
    }
    __device__ Row row(int64_t r) const { return p + r * ld; }
    __device__ double at(Row w, int k) const { return __ldg(w + k); }
    __device__ void load8(Row w, int k0, double (&x)[8]) const
    {
        if (pairs) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const double2 v = __ldg(reinterpret_cast<const double2*>(w + k0 + j));
                x[j] = v.x;
                x[j + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = __ldg(w + k0 + j);
        }
    }
    __device__ bool open(int r, int M, Row& w, unsigned& amax) const
    {
        if (r >= M) return false;
        w = p + r * ld;
        amax = __ldg(rmax + r);
        return true;
    }
    __device__ bool place(int r, int M, int R, int64_t ldo, int64_t& off, unsigned& amax) const
    {
        if (r >= M) return false;
        amax = __ldg(rmax + r);
        if (R > 0) {
            const int b = r / R;
            off = (int64_t)b * R * ldo + (r - b * R);
        } else {
            off = r * ldo;
        }
        return true;
    }
    __device__ bool live(int64_t) const { return true; }
    __device__ int64_t out_row(int64_t r) const { return r; }
};

// Rows (pair p, la), k = si of the packed (mu nu|la si), pairs mu >= nu from p0 (pair
// p is the packed pair index itself), in 2-D blocks: a warp's 32 rows are 8
// consecutive pairs x 4 consecutive indices la, a 128-row tile 8 pairs x 16
// indices.  For a fixed si, the elements with pair(la, si) > pair p sit in one
// stored row at consecutive p (one 64-byte run per la), and those with
// pair(la, si) <= p in runs over consecutive la or si: about 40% fewer memory
// transactions per load than rows running over la alone.  Rows past the last
// pair or index are dead (not loaded, not stored).
struct PackedRowsBlocked {
    const double* ints;
    int64_t p0, np;  // pairs p0 .. p0 + np
    int n, nlg;      // nlg = ceil(n / 16) index groups
    const unsigned* rmax;  // row maxima (upper word of |x|) of every pair row, [p][la]
    struct Row {
        const double* own;  // stored row p: own[kl] for kl <= p
        const double* col;  // column p: col[kl (kl + 1) / 2] for kl >= p
        int ij, la, tla;    // p, la, la (la + 1) / 2 (p < 2^31)
    };
    __device__ void decode(int64_t r, int& p, int& la) const
    {
        const int t = (int)(r >> 7);
        const int q = (int)(r & 127), w = q >> 5, l = q & 31;
        p = (t / nlg) * 8 + (l & 7);
        la = (t % nlg) * 16 + w * 4 + (l >> 3);
    }
    __device__ bool live(int64_t r) const
    {
        int p, la;
        decode(r, p, la);
        return p < (int)np && la < n;
    }
    __device__ int64_t out_row(int64_t r) const  // the row's place in p-major order (p n + la)
    {
        int p, la;
        decode(r, p, la);
        return (int64_t)p * n + la;
    }
    __device__ Row row(int64_t r) const
    {
        int p, la;
        decode(r, p, la);
        const int ij = (int)p0 + p;
        return Row{ints + (((int64_t)ij * (ij + 1)) >> 1), ints + ij, ij, la, la * (la + 1) / 2};
    }
    __device__ bool open(int r, int, Row& w, unsigned& amax) const
    {
        int p, la;
        decode(r, p, la);
        if (p >= (int)np || la >= n) return false;
        const int ij = (int)p0 + p;
        w = Row{ints + (((int64_t)ij * (ij + 1)) >> 1), ints + ij, ij, la, la * (la + 1) / 2};
        amax = __ldg(rmax + (int64_t)ij * n + la);
        return true;
    }
    __device__ bool place(int r, int, int R, int64_t ldo, int64_t& off, unsigned& amax) const
    {
        int p, la;
        decode(r, p, la);
        if (p >= (int)np || la >= n) return false;
        amax = __ldg(rmax + (p0 + p) * n + la);
        off = R == n ? (int64_t)p * n * ldo + la : 0;  // OutMap{n, .}: whole pairs (checked by the host)
        return true;
    }
    // 32-bit index arithmetic up to the address (64-bit compares would run on the
    // FP64 pipe); kl (kl + 1) / 2 elements are kl 4 (kl + 1) bytes, one wide multiply
    __device__ double elem(const Row& w, unsigned kl) const
    {
        const char* a = reinterpret_cast<const char*>(w.own) + (uint64_t)kl * 8u;
        const char* b = reinterpret_cast<const char*>(w.col) + (uint64_t)kl * ((kl + 1u) * 4u);
        return __ldg(reinterpret_cast<const double*>((int)kl <= w.ij ? a : b));
    }
    __device__ double at(const Row& w, int si) const
    {
        return elem(w, si <= w.la ? w.tla + si : si * (si + 1) / 2 + w.la);
    }
    __device__ void load8(const Row& w, int k0, double (&x)[8]) const
    {
        int t = k0 * (k0 + 1) / 2;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int si = k0 + j;
            x[j] = elem(w, si <= w.la ? w.tla + si : t + w.la);
            t += si + 1;
        }
    }
};

struct SymPairRows {  // rows (q, mu), k = nu of Zt[q * ldz + pair(mu, nu)] (Z transposed: one row per q)
    const double* Zt;
    int64_t ldz;
    int n;
    const unsigned* rmax = nullptr;  // row maxima (upper word of |x|), [q][mu] (gather GEMM)
    __device__ bool live(int64_t) const { return true; }
    __device__ int64_t out_row(int64_t r) const { return r; }
    struct Row {
        const double* z;
        int mu, tmu;
    };
    __device__ Row row(int64_t r) const
    {
        const int64_t q = r / n;
        const int mu = (int)(r - q * n);
        return Row{Zt + q * ldz, mu, mu * (mu + 1) / 2};
    }
    __device__ bool open(int r, int M, Row& w, unsigned& amax) const
    {
        if (r >= M) return false;
        const int q = r / n, mu = r - q * n;
        w = Row{Zt + q * ldz, mu, mu * (mu + 1) / 2};
        amax = __ldg(rmax + r);
        return true;
    }
    __device__ bool place(int r, int M, int R, int64_t ldo, int64_t& off, unsigned& amax) const
    {
        if (r >= M) return false;
        const int q = r / n, mu = r - q * n;
        amax = __ldg(rmax + r);
        off = R == n ? (int64_t)q * n * ldo + mu : 0;  // OutMap{n, .} (checked by the host)
        return true;
    }
    __device__ double at(const Row& w, int nu) const
    {
        return __ldg(w.z + (nu <= w.mu ? w.tmu + nu : nu * (nu + 1) / 2 + w.mu));
    }
    __device__ void load8(const Row& w, int k0, double (&x)[8]) const
    {
        int t = k0 * (k0 + 1) / 2;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int nu = k0 + j;
            x[j] = __ldg(w.z + (nu <= w.mu ? w.tmu + nu : t + w.mu));
            t += nu + 1;
        }
    }
};

}  // namespace hfgpu
