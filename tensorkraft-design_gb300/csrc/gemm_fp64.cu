// gemm_fp64.cu -- FP64 sector-GEMM path of the two-site H_eff.
//
// grouped_gemm_f64: one CTA per 16 x 16 output tile.  A tile's task is one
// output block; its K dimension is a list of segments (one per contributing
// sector pair), accumulated in registers, so every output element is written
// exactly once and no atomics are needed.  Operand tiles are staged through
// shared memory with the load mapping chosen per segment so that the
// unit-stride direction of each operand is the one walked by consecutive
// threads (coalesced for K-major and N-major operands alike).
//
// What bounds it is the FP64 pipe (1.2 TFLOP/s over the chip, so a 64 x 64 x 240
// tile keeps one SM busy for a quarter of a millisecond), not the loads (1 byte a
// multiply-add even at 16 x 16).  Hence the small edge: the pipe does hardly any
// work for padding and the longest tile is short beside the whole.  With edges of
// 64, 32 or 16 by task, the growth of an environment of 2 x 78 MFLOP (hubbard,
// D = 2048) took 139 + 281 us, its pipe 2 x 105; with 16 everywhere
// 82 + 85 us, its pipe 2 x 69.
//
// combine_f64: applies the fused two-site MPO W_ij between the two GEMM
// stages, out = sum_t coef_t * in_t over equally shaped slabs.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"

namespace tk {

namespace {

constexpr int NT = 256;
constexpr int BK = 16;
constexpr int E = kF64Tile;
constexpr int kSegs = 32;  // segments of a task kept in shared memory at a time

__device__ __forceinline__ void store_out(const GemmTask& task, double* __restrict__ C, int gm, int gn, double acc,
                                          double amul, int accumulate) {
    double* c = C + task.c_off + (int64_t)gm * task.c_rs + (int64_t)gn * task.c_cs;
    double v = amul * task.alpha * acc;
    if (accumulate)
        v += *c;
    else if (task.beta != 0.0)
        v += task.beta * *c;
    *c = v;
}

// The threads are laid over the valid mv x nv outputs (thread t owns
// (t / nv, t % nv)), so that a sector block of 13 x 13 keeps six warps busy and
// leaves two idle rather than spreading its outputs over all eight.  Every
// output sums its segments in order and k ascending inside each.  A step of k
// past a segment's K is not issued: a predicated-off FMA holds the pipe as long
// as a real one.  The next 16 k are on their way from memory while the present
// ones are multiplied.
__global__ void __launch_bounds__(NT, 6) grouped_gemm_f64_kernel(const GemmTile* __restrict__ tiles, int n_tiles,
                                                                 const GemmTask* __restrict__ tasks,
                                                                 const GemmSeg* __restrict__ segs,
                                                                 const double* __restrict__ A,
                                                                 const double* __restrict__ B,
                                                                 double* __restrict__ C, double amul, int accumulate) {
    __shared__ double As[2][BK][E + 1];
    __shared__ double Bs[2][BK][E + 1];
    __shared__ GemmSeg sseg[kSegs];
    if ((int)blockIdx.x >= n_tiles) return;
    const GemmTile tile = tiles[blockIdx.x];
    const GemmTask& task = tasks[tile.task];
    const int tid = threadIdx.x, lo = tid & 15, hi = tid >> 4;
    const int mv = min(E, task.M - tile.m0), nv = min(E, task.N - tile.n0);
    const int seg_begin = task.seg_begin, seg_end = task.seg_end;
    const bool mine = tid < mv * nv;
    const int ty = mine ? tid / nv : 0, tx = mine ? tid - ty * nv : 0;
    const bool warp_busy = (tid & ~31) < mv * nv;
    double acc = 0.0;
    int p = 0;
    for (int s0 = seg_begin; s0 < seg_end; s0 += kSegs) {
        const int ns = min(kSegs, seg_end - s0);
        // the last reads of the batch before lie ahead of that batch's last barrier
        for (int i = tid; i < ns; i += NT) sseg[i] = segs[s0 + i];
        __syncthreads();
        double va, vb;
        auto fetch = [&](const GemmSeg& sg, int k0) {
            const bool ak = sg.a_cs == 1, bn = sg.b_cs == 1;
            const int am = ak ? hi : lo, ka = k0 + (ak ? lo : hi);
            const int bc = bn ? lo : hi, kb = k0 + (bn ? hi : lo);
            va = am < mv && ka < sg.K ? A[sg.a_off + (int64_t)(tile.m0 + am) * sg.a_rs + (int64_t)ka * sg.a_cs] : 0.0;
            vb = bc < nv && kb < sg.K ? B[sg.b_off + (int64_t)kb * sg.b_rs + (int64_t)(tile.n0 + bc) * sg.b_cs] : 0.0;
        };
        int s = 0, k0 = 0;
        fetch(sseg[0], 0);
        while (s < ns) {
            const bool ak = sseg[s].a_cs == 1, bn = sseg[s].b_cs == 1;
            const int K = sseg[s].K, kl = min(BK, K - k0);
            As[p][ak ? lo : hi][ak ? hi : lo] = va;
            Bs[p][bn ? hi : lo][bn ? lo : hi] = vb;
            __syncthreads();
            k0 += BK;
            if (k0 >= K) {
                ++s;
                k0 = 0;
            }
            if (s < ns) fetch(sseg[s], k0);
            if (warp_busy) {
                if (kl == BK) {
#pragma unroll
                    for (int k = 0; k < BK; ++k) acc = fma(As[p][k][ty], Bs[p][k][tx], acc);
                } else {
#pragma unroll 1
                    for (int k = 0; k < kl; ++k) acc = fma(As[p][k][ty], Bs[p][k][tx], acc);
                }
            }
            p ^= 1;
        }
    }
    if (mine) store_out(task, C, tile.m0 + ty, tile.n0 + tx, acc, amul, accumulate);
}

// 64 x 64 tiles of one dense product, where 16 x 16 ones would not fit the
// caller's table: thread (tx, ty) owns the outputs (ty + 16 i, tx + 16 j).
__global__ void __launch_bounds__(NT) wide_gemm_f64_kernel(const GemmTile* __restrict__ tiles, int n_tiles,
                                                           const GemmTask* __restrict__ tasks,
                                                           const GemmSeg* __restrict__ segs,
                                                           const double* __restrict__ A, const double* __restrict__ B,
                                                           double* __restrict__ C) {
    constexpr int W = kF64WideTile, R = W / 16;
    __shared__ double As[BK][W + 1];
    __shared__ double Bs[BK][W + 1];
    if ((int)blockIdx.x >= n_tiles) return;
    const GemmTile tile = tiles[blockIdx.x];
    const GemmTask task = tasks[tile.task];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    double acc[R][R];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i][j] = 0.0;
    for (int s = task.seg_begin; s < task.seg_end; ++s) {
        const GemmSeg sg = segs[s];
        for (int k0 = 0; k0 < sg.K; k0 += BK) {
#pragma unroll
            for (int r = 0; r < (W * BK) / NT; ++r) {
                const int e = tid + r * NT;
                const bool ak = sg.a_cs == 1, bn = sg.b_cs == 1;
                const int m = ak ? e / BK : e % W, ka = ak ? e % BK : e / W;
                const int n = bn ? e % W : e / BK, kb = bn ? e / W : e % BK;
                const int gm = tile.m0 + m, gn = tile.n0 + n;
                As[ka][m] = gm < task.M && k0 + ka < sg.K
                                ? A[sg.a_off + (int64_t)gm * sg.a_rs + (int64_t)(k0 + ka) * sg.a_cs] : 0.0;
                Bs[kb][n] = gn < task.N && k0 + kb < sg.K
                                ? B[sg.b_off + (int64_t)(k0 + kb) * sg.b_rs + (int64_t)gn * sg.b_cs] : 0.0;
            }
            __syncthreads();
            const int kl = min(BK, sg.K - k0);
#pragma unroll 4
            for (int k = 0; k < kl; ++k) {
                double a[R], b[R];
#pragma unroll
                for (int i = 0; i < R; ++i) a[i] = As[k][ty + 16 * i];
#pragma unroll
                for (int j = 0; j < R; ++j) b[j] = Bs[k][tx + 16 * j];
#pragma unroll
                for (int i = 0; i < R; ++i)
#pragma unroll
                    for (int j = 0; j < R; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int gm = tile.m0 + ty + 16 * i, gn = tile.n0 + tx + 16 * j;
            if (gm < task.M && gn < task.N) store_out(task, C, gm, gn, acc[i][j], 1.0, 0);
        }
}

__global__ void __launch_bounds__(256) combine_f64_kernel(const CombJob* __restrict__ jobs,
                                                          const CombTerm* __restrict__ terms,
                                                          const double* __restrict__ in,
                                                          double* __restrict__ out) {
    const CombJob j = jobs[blockIdx.x];
    const int nterm = j.term_end - j.term_begin;
    __shared__ CombTerm st[64];
    const int n = j.rows * j.cols;
    for (int t0 = 0; t0 < max(nterm, 1); t0 += 64) {
        const int tn = min(64, nterm - t0);
        __syncthreads();
        if (threadIdx.x < tn) st[threadIdx.x] = terms[j.term_begin + t0 + threadIdx.x];
        __syncthreads();
        for (int e = threadIdx.x; e < n; e += blockDim.x) {
            const int r = e / j.cols, c = e - r * j.cols;
            double acc = 0.0;
            for (int t = 0; t < tn; ++t) acc = fma(st[t].coef, in[st[t].in_off + (int64_t)r * st[t].in_rs + c], acc);
            double* o = out + j.out_off + (int64_t)r * j.out_rs + c;
            *o = (t0 == 0) ? acc : (*o + acc);
        }
    }
}

__global__ void start_vector_kernel(double* v, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[i] = (double)((i * 7 + 13) % 97) / 97.0 - 0.5;
}

}  // namespace

cudaError_t launch_gemm_f64(const GemmTile* tiles, int n_tiles, const GemmTask* tasks, const GemmSeg* segs,
                            const double* A, const double* B, double* C, cudaStream_t s, double amul,
                            bool accumulate) {
    if (n_tiles <= 0) return cudaSuccess;
    grouped_gemm_f64_kernel<<<n_tiles, NT, 0, s>>>(tiles, n_tiles, tasks, segs, A, B, C, amul, accumulate ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_wide_gemm_f64(const GemmTile* tiles, int n_tiles, const GemmTask* tasks, const GemmSeg* segs,
                                 const double* A, const double* B, double* C, cudaStream_t s) {
    if (n_tiles <= 0) return cudaSuccess;
    wide_gemm_f64_kernel<<<n_tiles, NT, 0, s>>>(tiles, n_tiles, tasks, segs, A, B, C);
    return cudaGetLastError();
}

cudaError_t launch_gemm_c64(const GemmTile* tiles, int n_tiles, const GemmTask* tasks, const GemmSeg* segs,
                            const double* Ar, const double* Ai, const double* Br, const double* Bi, double* Cr,
                            double* Ci, bool conj_a, cudaStream_t s) {
    // (Ar + i Ai)^(*) (Br + i Bi): re = Ar Br -+ Ai Bi, im = Ar Bi +- Ai Br
    const double si = conj_a ? 1.0 : -1.0;
    cudaError_t e;
    if ((e = launch_gemm_f64(tiles, n_tiles, tasks, segs, Ar, Br, Cr, s, 1.0, false)) != cudaSuccess) return e;
    if ((e = launch_gemm_f64(tiles, n_tiles, tasks, segs, Ai, Bi, Cr, s, si, true)) != cudaSuccess) return e;
    if ((e = launch_gemm_f64(tiles, n_tiles, tasks, segs, Ar, Bi, Ci, s, 1.0, false)) != cudaSuccess) return e;
    return launch_gemm_f64(tiles, n_tiles, tasks, segs, Ai, Br, Ci, s, -si, true);
}

cudaError_t launch_combine_f64(const CombJob* jobs, int n_jobs, const CombTerm* terms, const double* in,
                               double* out, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    combine_f64_kernel<<<n_jobs, 256, 0, s>>>(jobs, terms, in, out);
    return cudaGetLastError();
}

cudaError_t launch_fill_start_vector(double* v, int64_t n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    int blocks = (int)std::min<int64_t>((n + 255) / 256, 152 * 8);
    start_vector_kernel<<<blocks, 256, 0, s>>>(v, n);
    return cudaGetLastError();
}

}  // namespace tk
