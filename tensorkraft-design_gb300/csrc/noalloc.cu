// noalloc.cu -- tk_gemm_f64_noalloc: the FP64 GEMM of tk_gemm_f64 without any
// memory allocation.
//
// Who needs it: callers that must not allocate device memory at call time.
// A sweep that works out of a pre-sized arena (tensorkraft's SweepArena
// design forbids allocation inside the Krylov loop), a host runtime that
// hands the library only the memory it manages itself, and latency-bound
// loops, which tk_gemm_f64 would make wait for each product.
//
// How: the task is a kernel argument and every CTA works its tile out from its
// index (dense_gemm_f64_kernel), so nothing is allocated, freed or copied.
//
// Limits and rules:
//   * outputs of at most kNoallocMaxTiles 64x64 squares (about 16k x 16k): a limit
//     of the interface, from the table that the call once kept in a fixed device
//     array; larger calls are rejected with TK_ERR_INVALID_ARG;
//   * the call is stream-ordered and does not synchronise: C is complete when
//     the stream reaches the end of the call's work.
#include <cuda_runtime.h>

#include <climits>
#include <cstdlib>
#include <string>

#include "kernels.cuh"
#include "tk_internal.hpp"

namespace {

constexpr int64_t kNoallocMaxTiles = 65520;
constexpr int kMaxDevices = 64;

tk_status fail(const std::string& msg, tk_status code) {
    tk::set_error(msg);
    return code;
}

}  // namespace

extern "C" tk_status tk_gemm_f64_noalloc(tk_ctx* ctx, double alpha, const tk_mat* a, const tk_mat* b, double beta,
                                         tk_mat_mut* c, void* stream) {
    if (!a || !b || !c || !a->data || !b->data || !c->data)
        return fail("tk_gemm_f64_noalloc: null argument", TK_ERR_INVALID_ARG);
    if (a->cols != b->rows || c->rows != a->rows || c->cols != b->cols)
        return fail("tk_gemm_f64_noalloc: shape mismatch", TK_ERR_INVALID_ARG);
    if (c->rows == 0 || c->cols == 0) return TK_OK;
    const int64_t lim = INT32_MAX;
    if (a->rows > lim || a->cols > lim || b->cols > lim || std::llabs(a->row_stride) > lim ||
        std::llabs(a->col_stride) > lim || std::llabs(b->row_stride) > lim || std::llabs(b->col_stride) > lim ||
        std::llabs(c->row_stride) > lim || std::llabs(c->col_stride) > lim)
        return fail("tk_gemm_f64_noalloc: dimensions or strides exceed 32 bits", TK_ERR_UNSUPPORTED);
    const int64_t ntm = (c->rows + 63) / 64, ntn = (c->cols + 63) / 64;
    if (ntm * ntn > kNoallocMaxTiles)
        return fail("tk_gemm_f64_noalloc: output of " + std::to_string(ntm * ntn) + " 64x64 squares, more than the " +
                        std::to_string(kNoallocMaxTiles) + " this call takes (its former no-allocation scratch); use tk_gemm_f64",
                    TK_ERR_INVALID_ARG);
    const int dev = ctx ? ctx->device : 0;
    if (dev < 0 || dev >= kMaxDevices) return fail("tk_gemm_f64_noalloc: device index out of range", TK_ERR_INVALID_ARG);
    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    cudaError_t e = cudaSetDevice(dev);
    if (e != cudaSuccess) return fail(std::string("tk_gemm_f64_noalloc: cudaSetDevice: ") + cudaGetErrorString(e), TK_ERR_CUDA);
    struct Restore {
        int d;
        ~Restore() {
            if (d >= 0) cudaSetDevice(d);
        }
    } restore{prev};
    tk::GemmTask task{};
    task.M = (int32_t)a->rows;
    task.N = (int32_t)b->cols;
    task.c_rs = (int32_t)c->row_stride;
    task.c_cs = (int32_t)c->col_stride;
    task.alpha = alpha;
    task.beta = beta;
    tk::GemmSeg seg{};
    seg.a_rs = (int32_t)a->row_stride;
    seg.a_cs = (int32_t)a->col_stride;
    seg.b_rs = (int32_t)b->row_stride;
    seg.b_cs = (int32_t)b->col_stride;
    seg.K = (int32_t)a->cols;
    e = tk::launch_dense_gemm_f64(task, seg, a->data, b->data, c->data, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(std::string("tk_gemm_f64_noalloc: GEMM launch: ") + cudaGetErrorString(e), TK_ERR_CUDA);
    return TK_OK;
}
