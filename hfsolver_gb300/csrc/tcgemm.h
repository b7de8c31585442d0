// Exactly sliced FP64 GEMMs on tcgen05 tensor cores (tcgemm.cu).
#pragma once
#include <cuda_bf16.h>

#include "internal.h"

namespace hfgpu {

// Output placement: element (r, c) goes to r*ld + c (R == 0), or, with R > 0,
// to (r/R)*(R*ld) + c*R + r%R (the rows transposed within blocks of R).
struct OutMap {
    int64_t R;
    int64_t ld;
};

// Digits a double is cut into: 6 (2^-42 of its row's scale) or 9 (2^-62).
enum SliceDigits { SLICE_MIXED = 6, SLICE_FP64 = 9 };
// the longest K whose FP32 accumulation is exact with that many digits
int slice_kmax(int digits);

// The B operand of a sliced GEMM: the rows of B^T cut into bf16 digit planes, laid out
// as the GEMM's pipeline stages (whole tiles of `tile` columns, K steps of 32), plus
// one power-of-two exponent per row; with nine digits also a plane of magnitudes, and B
// itself in FP64.
struct Sliced {
    DBuf<__nv_bfloat16> planes;
    DBuf<int> rexp;
    DBuf<double> b;  // [k][row]
    int64_t rows = 0, rows_pad = 0;
    int K = 0, ksteps = 0, digits = 0, tile = 0;
    int spins = 0;  // polls of the GEMM's waits before it gives up
};
// rows of a row-major FP64 matrix (stride ld)
void slice_dense(Context& ctx, const double* A, int64_t rows, int K, int64_t ld, int digits, Sliced& s);

// out = A B^T with A's rows gathered and sliced inside the GEMM (no A planes in
// HBM), B's digits deciding the precision:
// rows (pair p, la) over si of the packed (mu nu|la si), pairs p0 .. p0 + npairs (rmax:
// the rows' maxima from packed_row_max, for all pairs) ...
void sliced_gemm_packed(Context& ctx, const double* ints, int64_t p0, int64_t npairs, int n, const unsigned* rmax,
                        const Sliced& B, double* out, OutMap om);
// ... or rows (q, mu), q < nq, over nu of Zt[q * ldz + pair(mu, nu)] (rmax from
// sympair_row_max for these nq rows) ...
void sliced_gemm_sympair(Context& ctx, const double* Zt, int64_t ldz, int64_t nq, int n, const unsigned* rmax,
                         const Sliced& B, double* out, OutMap om);
// ... or dense row-major rows (rows x K, stride ld; rmax from dense_row_max)
void sliced_gemm_dense(Context& ctx, const double* A, int64_t rows, int K, int64_t ld, const unsigned* rmax,
                       const Sliced& B, double* out, OutMap om);
// max |x| of every gather row, as the upper 32 bits of |x| (enough for its
// exponent): packed integrals, rows (pair p, la) of all n (n + 1) / 2 pairs ->
// out[p * n + la]; Zt rows (q, mu) -> out[q * n + mu]
void packed_row_max(Context& ctx, const double* ints, int n, unsigned* out);
void dense_row_max(Context& ctx, const double* A, int64_t rows, int K, int64_t ld, unsigned* out);
void sympair_row_max(Context& ctx, const double* Zt, int64_t ldz, int64_t nq, int n, unsigned* out);
// Held around the sliced GEMMs of a call.  settle() waits for them, adds their times to
// the context's counters and throws if one of them timed out; where an exception ends
// the call between two of them, what they left in the context goes with this object.
class SlicedRun {
    Context& ctx;

public:
    explicit SlicedRun(Context& c) : ctx(c) {}
    SlicedRun(const SlicedRun&) = delete;
    ~SlicedRun();
    void settle();
};
// (ia|jb) by the half transform on sliced GEMMs of `digits` digits, T[j][b][i][a]
// (mp2_mixed.cu); n <= slice_kmax(digits)
void ao2mo_sliced(Context& ctx, int n, const double* d_int2, const double* C1, int n1, const double* C2, int n2,
                  int digits, double* T);
// out[c][r] = in[r][c] for a rows x cols row-major FP64 matrix (mp2_mixed.cu)
void transpose_device(Context& ctx, const double* in, int64_t rows, int64_t cols, double* out);

}  // namespace hfgpu
