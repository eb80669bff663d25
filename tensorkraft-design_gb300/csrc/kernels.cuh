// kernels.cuh -- launch wrappers of the device kernels.
#pragma once
#include <cuda_runtime.h>

#include "tk_internal.hpp"

namespace tk {

// FP64 grouped segmented GEMM over a list of kF64Tile-square tiles, one CTA each.
// C = amul * alpha * A B (+ beta C, or + C when `accumulate`), per task.
cudaError_t launch_gemm_f64(const GemmTile* tiles, int n_tiles, const GemmTask* tasks, const GemmSeg* segs,
                            const double* A, const double* B, double* C, cudaStream_t s, double amul = 1.0,
                            bool accumulate = false);
// One dense product of M x K by K x N, without tables: the estimated time in
// seconds, with the CTAs that share a tile's K in *split; and the launch.
double dense_gemm_f64_plan(int64_t M, int64_t N, int64_t K, int* split = nullptr);
cudaError_t launch_dense_gemm_f64(const GemmTask& task, const GemmSeg& seg, const double* A, const double* B,
                                  double* C, cudaStream_t s);
// The tables of launch_gemm_f64 on planar complex operands (four launches): C = A B, or
// conj(A) B with conj_a; the tasks must overwrite their output (beta = 0).
cudaError_t launch_gemm_c64(const GemmTile* tiles, int n_tiles, const GemmTask* tasks, const GemmSeg* segs,
                            const double* Ar, const double* Ai, const double* Br, const double* Bi, double* Cr,
                            double* Ci, bool conj_a, cudaStream_t s);

// Channel combine: one CTA per job.
cudaError_t launch_combine_f64(const CombJob* jobs, int n_jobs, const CombTerm* terms, const double* in,
                               double* out, cudaStream_t s);

// Vector kernels used by the device Lanczos.
cudaError_t launch_fill_start_vector(double* v, int64_t n, cudaStream_t s);

}  // namespace tk
