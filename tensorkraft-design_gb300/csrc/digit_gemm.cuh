// digit_gemm.cuh -- FP64 products on the fp16 tensor cores (digit_gemm.cu).
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "tk_internal.hpp"

namespace tk {

// An operand row x is held as seven fp16 integer digits on a grid of its own,
//   x = 2^(e - 57) * sum_j d_j 2^(8 (6 - j)),  |d_0| <= 2^9, |d_j| <= 2^7,
// e the exponent of the row's largest element (all |x| < 2^e): every element
// to 2^(e - 58), five bits below the last place of the largest one.
constexpr int kDigits = 7;
constexpr int kDigitValue = 1, kDigitWait = 2;  // *redo: an operand's values / a wait that ran out
constexpr int kDigitRing = 2;  // shared-memory stages of 32 K of a product

// Programmatic dependent launch: a kernel's prologue overlaps the tail of the
// one before it; it touches nothing another kernel writes before dep_wait(),
// which returns once the previous kernel is complete and its memory visible.
#ifdef __CUDACC__
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_dependent(void (*k)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k, P(args)...);
}
#endif

// A digit operand in the operand-stack layout (K-major 64-wide chunks, see
// TcTables): `rows` rows of seven digits of 64 elements each, one after the
// other, and the biased exponent of every row of chunk 0 (kTcBM entries more, for
// tiles without K: they have no rows, a_row = b_row = 0, and their sums are zeros
// whatever the exponents).
struct DigitStack {
    __half* q = nullptr;
    int32_t* ex = nullptr;
    int64_t rows = 0;
};
inline size_t digit_stack_bytes(int64_t rows) { return (size_t)rows * kTcBK * kDigits * sizeof(__half); }

// Rows [row, row + n) of a stack whose chunks are `cs` rows apart; `kx` >= 0:
// the index of the power-of-two scales of its k (launch_digit_columns); `ex0`
// >= 0: row 0's exponent in the table that launch_digit_columns gets.
struct DigitRows {
    int32_t row, n, cs, kch, kx, ex0;
};
// The same of a complex stack: its digits go to rows to .. of a stack whose
// chunks are cs_out rows apart (the imaginary part's chunks behind the real
// part's), the second form of a B operand n_dual rows further.
struct DigitRowsC {
    int32_t row, n, cs, kch, kx, to, cs_out, n_dual;
};
// Columns [0, cols) (at most 32) at src of a psi sub-block (rows x pitch), as
// rows to .. of a B operand; complex vectors' second form n_dual rows further.
// `kx`: the index of the scales of its k.
struct DigitPsi {
    int64_t src;
    int32_t rows, cols, pitch, to, cs, n_dual, kx, pad;
};
constexpr int kDigitRowsPerCta = 8;

// Tensor maps of one product's operands: A in boxes of 32, 64, 96 or 128 rows
// x 32 k x all digits, B in boxes of 32 rows.
struct DigitMaps {
    CUtensorMap a[4], b;
};
bool digit_maps(DigitMaps& m, const DigitStack& a, const DigitStack& b, std::string& err);

// Where a product goes: rows through a row table (TcTile mode 1), columns
// through column tables (mode 2), or C = alpha A B + beta C with strides
// (mode 0: a
// single product whose tiles need no table).
struct DigitOut {
    double* out;
    double* out_im;  // mode 1, complex products: where a tile's columns from `split` on go
    const int64_t* rowtab;
    const int64_t* colbase;
    const int32_t* colstride;
    int64_t c_rs, c_cs;
    double alpha, beta;
    int tiles;    // mode 0: tiles of the C grid
    int m, n, k;  // mode 0: the product's size (its operands' stacks have m and n rows a chunk)
};

// Once per process and device before the first launch.
cudaError_t digit_setup();
// Deals the tiles of a product out to `ctas` CTAs: CTA c runs out[begin[c] ..
// begin[c + 1]), heaviest first, the sums of the estimated times as equal as
// longest-first dealing makes them; in 32-wide halves where that ends sooner
// (fewer tiles than SMs).
void digit_schedule(const std::vector<TcTile>& in, int ctas, std::vector<TcTile>& out, std::vector<int32_t>& begin);

// Runs the tiles' products (mode 0: the C grid's, dealt in turn).  Nothing is
// written once *redo is non-zero (an operand row held an infinity or a NaN); a
// bounded wait that ran out sets it too.  Whoever launches this computes the
// product in another way when it ends up non-zero.
cudaError_t launch_digit_gemm(int mode, const TcTile* tiles, const int32_t* begin, int ctas, const DigitMaps& maps,
                              const int32_t* exa, const int32_t* exb, const DigitOut& out, int* redo, cudaStream_t s);

// Exponents of a stack's columns: kx[j.kx + k] = floor(log2 max |x|) over the
// rows [row, row + n) of job j at k, of x 2^(1023 - ex[j.ex0 + r]) with a table ex
// (leaving out rows of kNoGain); kDeadColumn for a column of zeros, far below the others:
// what the other operand holds at that k is multiplied by zeros, so it must neither set
// its row's exponent nor take up its digits.
constexpr int kNoGain = INT32_MIN, kDeadColumn = -8192;
cudaError_t launch_digit_columns(const DigitRows* jobs, int n_jobs, int max_kch, const double* q64, const double* q64_im,
                                 const int32_t* ex, int32_t* kx, cudaStream_t s);
// Digits of FP64 operand stacks (rows of 64 doubles per chunk), of
// x 2^(sign * kx) where the job has scales.
cudaError_t launch_digit_rows(const DigitRows* jobs, int n_jobs, const double* q64, const int32_t* kx, int sign,
                              const DigitStack& out, int* redo, cudaStream_t s);
cudaError_t launch_digit_rows_complex(const DigitRowsC* jobs, int n_jobs, const double* re, const double* im,
                                      const int32_t* kx, int sign, bool dual, const DigitStack& out, int* redo,
                                      cudaStream_t s);
// Digits of both operands of a dense product (*redo is set where an output might be
// less exact than by an FP64 chain): row r, k of K at x[r * rs + k * ks], into stacks
// whose chunks are `rows` rows apart.  `top`, *inexact and *wide start at zero.
struct DigitMatrix {
    const double* x;
    int64_t rs, ks;
    int rows;
    DigitStack out;
    uint32_t* top;  // scratch: a value a row,
    int* inexact;   // one value,
    float* sample;  // kDigitSamples values a row
};
constexpr int kDigitSamples = 64;
cudaError_t launch_digit_matrices(const DigitMatrix& a, const DigitMatrix& b, int K, int* wide, int* redo, cudaStream_t s);
// Digits of psi sub-blocks (jobs of at most `cols` columns, 32 or 8, and max_k
// rows) times 2^kx, of both parts with x_im.
cudaError_t launch_digit_psi(const DigitPsi* jobs, int n_jobs, int cols, int max_k, const double* x, const double* x_im,
                             const int32_t* kx, const DigitStack& out, int* redo, cudaStream_t s);

}  // namespace tk
