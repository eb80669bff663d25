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
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "kernels.cuh"

namespace cg = cooperative_groups;

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

// One dense product C = alpha A B + beta C, its task and segment passed by
// value (no tables, no upload).  `split` CTAs of a cluster share a tile's K and
// the first sums their parts in order through distributed shared memory: a
// 16 x 16 x 2048 tile alone takes one SM 160 us, and with 49 such tiles
// (100 x 100 x 2000) two thirds of the SMs have nothing to do.
__global__ void __launch_bounds__(NT, 6) dense_gemm_f64_kernel(const GemmTask task, const GemmSeg sg, int ntn,
                                                               int split, const double* __restrict__ A,
                                                               const double* __restrict__ B,
                                                               double* __restrict__ C) {
    __shared__ double As[2][BK][E + 1];
    __shared__ double Bs[2][BK][E + 1];
    __shared__ double part[NT];
    const int tile = blockIdx.x / split, rank = blockIdx.x % split;
    const int m0 = tile / ntn * E, n0 = tile % ntn * E;
    const int tid = threadIdx.x, lo = tid & 15, hi = tid >> 4;
    const int mv = min(E, task.M - m0), nv = min(E, task.N - n0);
    const bool mine = tid < mv * nv;
    const int ty = mine ? tid / nv : 0, tx = mine ? tid - ty * nv : 0;
    const bool warp_busy = (tid & ~31) < mv * nv;
    const bool ak = sg.a_cs == 1, bn = sg.b_cs == 1;
    const int am = ak ? hi : lo, ka = ak ? lo : hi, bc = bn ? lo : hi, kb = bn ? hi : lo;
    const double* pa = A + (int64_t)(m0 + am) * sg.a_rs;
    const double* pb = B + (int64_t)(n0 + bc) * sg.b_cs;
    const int64_t per = ((int64_t)sg.K + BK * split - 1) / (BK * split) * BK;  // k of each CTA
    const int64_t k_end = min((int64_t)sg.K, per * (rank + 1));
    double acc = 0.0, va, vb;
    auto fetch = [&](int64_t k0) {
        va = am < mv && k0 + ka < k_end ? pa[(k0 + ka) * sg.a_cs] : 0.0;
        vb = bc < nv && k0 + kb < k_end ? pb[(k0 + kb) * sg.b_rs] : 0.0;
    };
    int p = 0;
    int64_t k0 = per * rank;
    fetch(k0);
    for (; k0 < k_end; k0 += BK, p ^= 1) {
        As[p][ka][am] = va;
        Bs[p][kb][bc] = vb;
        __syncthreads();
        fetch(k0 + BK);
        if (warp_busy) {
            if (k_end - k0 >= BK) {
#pragma unroll
                for (int k = 0; k < BK; ++k) acc = fma(As[p][k][ty], Bs[p][k][tx], acc);
            } else {
                const int kl = (int)(k_end - k0);
#pragma unroll 1
                for (int k = 0; k < kl; ++k) acc = fma(As[p][k][ty], Bs[p][k][tx], acc);
            }
        }
    }
    if (split > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        part[tid] = acc;
        cluster.sync();
        if (rank == 0)
            for (int r = 1; r < split; ++r) acc += cluster.map_shared_rank(part, r)[tid];
        cluster.sync();  // the parts are there until they are read
    }
    if (mine && rank == 0) store_out(task, C, m0 + ty, n0 + tx, acc, 1.0, 0);
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

double dense_gemm_f64_plan(int64_t M, int64_t N, int64_t K, int* split) {
    // 85 ns a k for a tile on its SM's pipe; the SM with the most tiles counts.
    // A share has at least 64 k.  Eight shares against one: 16 x 16 x 2048 28 us
    // against 175, 100 x 100 x 2000 61 against 171, 200 x 200 x 1000 93 against 139;
    // with the chip full (2048 x 32 x 2048) 241 against 274.
    const double tiles = (double)((M + E - 1) / E) * ((N + E - 1) / E);
    double best = 0.0;
    for (int s = 1; s <= 8; s *= 2) {
        if (s > 1 && K < 64 * s) break;
        const double per = (double)((K + (int64_t)BK * s - 1) / ((int64_t)BK * s) * BK);
        const double t = std::ceil(tiles * s / 152.0) * per * 85e-9 + (s > 1 ? 2e-6 : 0.0);
        if (s == 1 || t < 0.9 * best) {
            best = t;
            if (split) *split = s;
        }
    }
    return best + 8e-6;
}

cudaError_t launch_dense_gemm_f64(const GemmTask& task, const GemmSeg& seg, const double* A, const double* B,
                                  double* C, cudaStream_t s) {
    int split = 1;
    dense_gemm_f64_plan(task.M, task.N, seg.K, &split);
    const int64_t ntn = (task.N + (int64_t)E - 1) / E, ntm = (task.M + (int64_t)E - 1) / E;
    if (ntm * ntn * split > INT32_MAX) return cudaErrorInvalidConfiguration;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)split;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ntm * ntn * split));
    cfg.blockDim = dim3(NT);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = split > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, dense_gemm_f64_kernel, task, seg, (int)ntn, split, A, B, C);
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
