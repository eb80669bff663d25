// stack_f64.cu -- the FP64 matvec on operand stacks (TK_SCHED_STACKED).
//
// The grouped FP64 schedule runs one GEMM task per output sector block; with
// sector dimensions around 13 and one or two MPO channels per slab, most of
// its tasks are a few rows tall and a square tile covers them sparsely (about
// 60 % of the FP64 FMAs it issues are useful on Hubbard D=2048).  This
// schedule regroups the same work the way the split-precision path does
// (TcTables, built with every psi column read through its table and no
// fused stage 3):
//   stage 1, one stack per ket sector A of L: T1 = L_stack(A) * psi_A, the
//     stack's rows every L slab (A', w, A), its columns every psi sub-block
//     (p, A, B), K = D_A;
//   combine: T2 = sum coef * T1 over the W_i W_j terms, written in the
//     stage-3 operand layout (K-major 64-wide chunks, zero padding);
//   stage 3, one stack per bra sector B' of R: y = T2_stack * R_stack^T
//     through the y row table.
// The operands are the split path's stacks in FP64; the GEMMs run on the
// FP64 pipe (this GPU's FP64 tensor rate is no higher than its CUDA-core
// FP64 rate).  On this GPU an FP64 FMA occupies its pipe some thirty times
// longer than any other instruction a thread runs, so the kernels are laid
// out to issue as few FP64 FMAs as possible, index arithmetic being free
// next to them:
//   - a piece (the work of one CTA) is at most 32 x 64 outputs, laid densely
//     over the 256 threads (DenseMap);
//   - k steps over the piece's K segments only: stage 1 the stack's true K,
//     stage 3 the column ranges of T2 that its rows hold (the combine leaves
//     the rest of a T2 stack zero: the W_i W_j channels that do not reach
//     those rows), with no predicated-off FMA past a segment's end;
//   - pieces are cut so that each holds at most a share of the stage's
//     FMAs, and go out longest first.
// The launches are chained by programmatic dependent launch: for small plans they
// are most of the time (Heisenberg D = 64: 17.4 -> 10.9 us).
// Every output sums its k in ascending order.
//
// Large plans run the same stacks on the fp16 tensor cores instead
// (digit_gemm.cu): digits of psi, T1 by digit products, the same combine,
// digits of T2, y by digit products.  Hubbard D = 2048: 701 -> 143 us; cylinder
// D = 2048: 40.9 -> 1.60 ms, relative error 2.6e-15 -> 1.5e-15; a complex plan
// takes both parts as one K twice as long.  The columns of L and R, and with them
// psi's and T2's elements at that k, are scaled by powers of two: R's to even
// magnitudes, L's by what they come to in the result (row_gains).  So the largest
// element of every digit row reaches the result at full size, and the error by norm
// stays within an FP64 chain's bound whatever the environments' scales (1 % of the
// matvec; without L's scales, ket scales of 2^-20 .. 2^20 left a relative error of
// 2e-6).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <set>
#include <string>

#include "digit_gemm.cuh"
#include "tk_plan.cuh"

namespace tk {
namespace {

constexpr int SBN = kTcBN;  // 64 columns per piece (the stacks' column tiles)
constexpr int SBK = 16;     // k step through shared memory
constexpr int ST = 256;
constexpr int SBM = 32;     // rows per piece at most
constexpr int RPT = SBM * SBN / ST;  // outputs per thread of a full piece

// One CTA's work: rows [a_row, a_row + m_valid) (operand rows of chunk 0) of
// a stack against n_valid columns, over the K segments segs[seg0, seg0 + nseg).
struct F64Piece {
    int32_t a_row, a_cs, b_row, b_cs;
    int32_t m_valid, n_valid;
    int32_t ldc, n0;   // stage 1: T1 row of the first row; stage 3: y column offset
    int64_t out_off;   // stage 1: column-table index of column 0; stage 3: y row-table index of row 0
    int32_t seg0, nseg;
};
struct KSeg {
    int32_t kb, ke;  // k in [kb, ke)
};

// The outputs of a piece lie densely over the threads: output e (row e / nv,
// column e % nv of the m_valid x nv block) belongs to thread e % ST, its
// round e / ST.  A warp runs only the rounds that hold one of its outputs,
// so the FMAs it issues are the piece's outputs times K, rounded up to whole
// warps.
struct DenseMap {
    int nv, total, rounds;  // columns, outputs, rounds of this warp
    __device__ DenseMap(int m_valid, int n_valid, int warp) : nv(n_valid), total(m_valid * n_valid) {
        rounds = total > 32 * warp ? (total - 32 * warp + ST - 1) / ST : 0;
    }
};

// acc[r] += sum over k < kl of A[k][m_r] * B[k][n_r], k ascending; complex
// (CPLX): (ar + i ai)(br + i bi) accumulated as re += ar br - ai bi and
// im += ar bi + ai br.  A full step is unrolled; a short one loops exactly kl
// times, so that no FMA past the segment's end is issued (predicated off, it
// would still hold the pipe).
template <bool CPLX>
__device__ __forceinline__ void dense_kstep(const double (*Ar)[SBM + 1], const double (*Ai)[SBM + 1],
                                            const double (*Br)[SBN + 1], const double (*Bi)[SBN + 1], int kl,
                                            const DenseMap& d, int tid, double* accr, double* acci) {
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        if (r < d.rounds) {
            const int e = min(tid + ST * r, d.total - 1);  // lanes past the end read a valid element
            const int m = e / d.nv, n = e - m * d.nv;
            double sr = accr[r], si = CPLX ? acci[r] : 0.0;
            auto step = [&](int k) {
                sr = fma(Ar[k][m], Br[k][n], sr);
                if constexpr (CPLX) {
                    sr = fma(-Ai[k][m], Bi[k][n], sr);
                    si = fma(Ar[k][m], Bi[k][n], si);
                    si = fma(Ai[k][m], Br[k][n], si);
                }
            };
            if (kl == SBK) {
#pragma unroll
                for (int k = 0; k < SBK; ++k) step(k);
            } else {
#pragma unroll 1
                for (int k = 0; k < kl; ++k) step(k);
            }
            accr[r] = sr;
            if constexpr (CPLX) acci[r] = si;
        }
    }
}

// k in [k0, k0 + kl) of a stack operand (rows m < rows_valid of chunk-0 row
// `row`, `cs` rows between chunks) into S[k][m].
__device__ __forceinline__ void load_op_a(double (*S)[SBM + 1], const double* __restrict__ q, int32_t row, int32_t cs,
                                          int rows_valid, int k0, int kl, int tid) {
#pragma unroll
    for (int r = 0; r < SBM * SBK / ST; ++r) {
        const int e = tid + ST * r, k = e & 15, m = e >> 4, kk = k0 + k;
        double v = 0.0;
        if (m < rows_valid && k < kl) v = q[(((int64_t)row + (int64_t)(kk >> 6) * cs + m) << 6) + (kk & 63)];
        S[k][m] = v;
    }
}

__device__ __forceinline__ void load_op_b(double (*S)[SBN + 1], const double* __restrict__ q, int32_t row, int32_t cs,
                                          int rows_valid, int k0, int kl, int tid) {
#pragma unroll
    for (int r = 0; r < SBN * SBK / ST; ++r) {
        const int e = tid + ST * r, k = e & 15, n = e >> 4, kk = k0 + k;
        double v = 0.0;
        if (n < rows_valid && k < kl) v = q[(((int64_t)row + (int64_t)(kk >> 6) * cs + n) << 6) + (kk & 63)];
        S[k][n] = v;
    }
}

// Shared memory of one piece.
template <bool CPLX>
struct PieceTiles {
    double Ar[SBK][SBM + 1], Br[SBK][SBN + 1];
    double Ai[CPLX ? SBK : 1][SBM + 1], Bi[CPLX ? SBK : 1][SBN + 1];
};

// Stage 1: T1 = L stacks * psi (CPLX: both complex, planar).
template <bool CPLX>
__device__ __forceinline__ void stack_piece1(const F64Piece t, PieceTiles<CPLX>& sm, const KSeg* __restrict__ segs,
                                             const double* __restrict__ lq, const double* __restrict__ lq_im,
                                             const double* __restrict__ x, const double* __restrict__ x_im,
                                             const int64_t* __restrict__ xsrc, const int32_t* __restrict__ xstride,
                                             const int64_t* __restrict__ colbase,
                                             const int32_t* __restrict__ colstride, double* __restrict__ t1,
                                             double* __restrict__ t1_im) {
    auto& Ar = sm.Ar;
    auto& Br = sm.Br;
    auto& Ai = sm.Ai;
    auto& Bi = sm.Bi;
    const int tid = threadIdx.x;
    const int ln = tid & 63;  // the B column this thread loads
    const bool lv = ln < t.n_valid;
    const int64_t src = lv ? xsrc[t.out_off + ln] : 0;
    const int32_t str = lv ? xstride[t.out_off + ln] : 0;
    const DenseMap d(t.m_valid, t.n_valid, tid >> 5);
    double accr[RPT], acci[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) accr[r] = acci[r] = 0.0;
    for (int sg = t.seg0; sg < t.seg0 + t.nseg; ++sg) {
        const KSeg g = segs[sg];
        for (int k0 = g.kb; k0 < g.ke; k0 += SBK) {
            const int kl = min(SBK, g.ke - k0);
            load_op_a(Ar, lq, t.a_row, t.a_cs, t.m_valid, k0, kl, tid);
            if constexpr (CPLX) load_op_a(Ai, lq_im, t.a_row, t.a_cs, t.m_valid, k0, kl, tid);
#pragma unroll
            for (int r = 0; r < SBN * SBK / ST; ++r) {
                const int k = (tid >> 6) + 4 * r, kk = k0 + k;
                const bool ok = lv && k < kl;
                Br[k][ln] = ok ? x[src + (int64_t)kk * str] : 0.0;
                if constexpr (CPLX) Bi[k][ln] = ok ? x_im[src + (int64_t)kk * str] : 0.0;
            }
            __syncthreads();
            dense_kstep<CPLX>(Ar, Ai, Br, Bi, kl, d, tid, accr, acci);
            __syncthreads();
        }
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int e = tid + ST * r;
        if (r < d.rounds && e < d.total) {
            const int m = e / d.nv, n = e - m * d.nv;
            const int64_t o = colbase[t.out_off + n] + (int64_t)(t.ldc + m) * colstride[t.out_off + n];
            t1[o] = accr[r];
            if constexpr (CPLX) t1_im[o] = acci[r];
        }
    }
}

template <bool CPLX>
__global__ void __launch_bounds__(ST, 4) stack_gemm1_f64_kernel(const F64Piece* __restrict__ pieces,
                                                                const KSeg* __restrict__ segs,
                                                                const double* __restrict__ lq,
                                                                const double* __restrict__ lq_im,
                                                                const double* __restrict__ x,
                                                                const double* __restrict__ x_im,
                                                                const int64_t* __restrict__ xsrc,
                                                                const int32_t* __restrict__ xstride,
                                                                const int64_t* __restrict__ colbase,
                                                                const int32_t* __restrict__ colstride,
                                                                double* __restrict__ t1, double* __restrict__ t1_im) {
    __shared__ PieceTiles<CPLX> sm;
    const F64Piece t = pieces[blockIdx.x];  // a plan constant
    dep_launch();
    dep_wait();
    stack_piece1<CPLX>(t, sm, segs, lq, lq_im, x, x_im, xsrc, xstride, colbase, colstride, t1, t1_im);
}

// Stage 3: y = T2 stacks * R stacks^T (CPLX: both complex, planar).
template <bool CPLX>
__device__ __forceinline__ void stack_piece3(const F64Piece t, PieceTiles<CPLX>& sm, const KSeg* __restrict__ segs,
                                             const double* __restrict__ t2, const double* __restrict__ t2_im,
                                             const double* __restrict__ rq, const double* __restrict__ rq_im,
                                             const int64_t* __restrict__ yrow, double* __restrict__ y,
                                             double* __restrict__ y_im) {
    auto& Ar = sm.Ar;
    auto& Br = sm.Br;
    auto& Ai = sm.Ai;
    auto& Bi = sm.Bi;
    const int tid = threadIdx.x;
    const DenseMap d(t.m_valid, t.n_valid, tid >> 5);
    double accr[RPT], acci[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) accr[r] = acci[r] = 0.0;
    for (int sg = t.seg0; sg < t.seg0 + t.nseg; ++sg) {
        const KSeg g = segs[sg];
        for (int k0 = g.kb; k0 < g.ke; k0 += SBK) {
            const int kl = min(SBK, g.ke - k0);
            load_op_a(Ar, t2, t.a_row, t.a_cs, t.m_valid, k0, kl, tid);
            load_op_b(Br, rq, t.b_row, t.b_cs, t.n_valid, k0, kl, tid);
            if constexpr (CPLX) {
                load_op_a(Ai, t2_im, t.a_row, t.a_cs, t.m_valid, k0, kl, tid);
                load_op_b(Bi, rq_im, t.b_row, t.b_cs, t.n_valid, k0, kl, tid);
            }
            __syncthreads();
            dense_kstep<CPLX>(Ar, Ai, Br, Bi, kl, d, tid, accr, acci);
            __syncthreads();
        }
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int e = tid + ST * r;
        if (r < d.rounds && e < d.total) {
            const int m = e / d.nv, n = e - m * d.nv;
            const int64_t o = yrow[t.out_off + m] + t.n0 + n;
            y[o] = accr[r];
            if constexpr (CPLX) y_im[o] = acci[r];
        }
    }
}

template <bool CPLX>
__global__ void __launch_bounds__(ST, 4) stack_gemm3_f64_kernel(const F64Piece* __restrict__ pieces,
                                                                const KSeg* __restrict__ segs,
                                                                const double* __restrict__ t2,
                                                                const double* __restrict__ t2_im,
                                                                const double* __restrict__ rq,
                                                                const double* __restrict__ rq_im,
                                                                const int64_t* __restrict__ yrow,
                                                                double* __restrict__ y, double* __restrict__ y_im) {
    __shared__ PieceTiles<CPLX> sm;
    const F64Piece t = pieces[blockIdx.x];  // a plan constant
    dep_launch();
    dep_wait();
    stack_piece3<CPLX>(t, sm, segs, t2, t2_im, rq, rq_im, yrow, y, y_im);
}

// T2 = sum coef * T1 for one combine job (rows r0 .. r0 + rows of a slab),
// written into the chunked stage-3 operand layout.
__device__ __forceinline__ void stack_combine_job(const TcCombJob& j, const TcCombTerm* __restrict__ terms,
                                                  const double* __restrict__ coef, const double* __restrict__ t1,
                                                  double* __restrict__ t2) {
    const int n = j.rows * j.cols;
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int rl = e / j.cols, c = e - rl * j.cols, r = j.r0 + rl;
        double acc = 0.0;
        for (int q = j.term_begin; q < j.term_end; ++q)
            acc = fma(coef[q], t1[terms[q].in_off + (int64_t)r * terms[q].in_rs + c], acc);
        const int k = j.k0 + c;
        t2[(((int64_t)j.t2row + (int64_t)(k >> 6) * j.cstride + r) << 6) + (k & 63)] = acc;
    }
}

template <bool CPLX>
__global__ void __launch_bounds__(256) stack_combine_f64_kernel(const TcCombJob* __restrict__ jobs,
                                                                const TcCombTerm* __restrict__ terms,
                                                                const double* __restrict__ coef,
                                                                const double* __restrict__ t1,
                                                                double* __restrict__ t2,
                                                                const double* __restrict__ t1_im,
                                                                double* __restrict__ t2_im) {
    const TcCombJob j = jobs[blockIdx.x];  // a plan constant
    dep_launch();
    dep_wait();
    // the W_i W_j coefficients are real: they act on each part (blockIdx.y)
    if (!CPLX)
        stack_combine_job(j, terms, coef, t1, t2);
    else
        stack_combine_job(j, terms, coef, blockIdx.y ? t1_im : t1, blockIdx.y ? t2_im : t2);
}

// The whole FP64 matvec in one launch, after a digit matvec that could not
// stand: *redo set by an operand with infinities or NaNs, or by a bounded wait
// that ran out.  Otherwise it ends at once (launched behind every digit matvec).
// Its CTAs, as many as the GPU holds, take each stage's work from a queue; a stage
// starts when the one before it is done.  A CTA waits only with nothing in hand,
// for work that running CTAs have taken, so not all CTAs need be on the GPU at
// once.  (As one cluster of eight CTAs, with the cluster's barrier between the
// stages, cylinder D = 1000 took 225 ms, as the FP64 launches 8.1.)
struct RedoQueue {
    unsigned next[3], done[2], left, late;
};
struct RedoArgs {
    const F64Piece *pieces1, *pieces3;
    const KSeg* segs;
    const TcCombJob* jobs;
    const TcCombTerm* terms;
    const double *coef, *lq, *rq, *lq_im, *rq_im;
    const int64_t *xsrc, *colbase, *yrow;
    const int32_t *xstride, *colstride;
    double *t1, *t2, *t1_im, *t2_im;
    RedoQueue* queue;
    int n1, n3, njobs;
};
constexpr int kRedoCtasPerSm = 2;         // 9.2 ms, with 4: 8.3, but each digit matvec 0.7 us more
constexpr int kRedoJobs = 8;              // combine jobs taken at a time
constexpr unsigned kRedoPolls = 1u << 24;  // without progress of the others, some ten seconds
template <bool CPLX>
__global__ void __launch_bounds__(ST, kRedoCtasPerSm)
    stack_redo_f64_kernel(const RedoArgs a, const double* __restrict__ x, const double* __restrict__ x_im,
                          double* __restrict__ y, double* __restrict__ y_im, int* redo) {
    __shared__ PieceTiles<CPLX> sm;
    __shared__ int item;
    dep_launch();
    dep_wait();
    if (*(volatile int*)redo == 0) return;
    RedoQueue& q = *a.queue;
    const int tid = threadIdx.x;
    // the next of n items of stage s, -1 when all are taken
    auto take = [&](int s, int n) {
        __syncthreads();
        if (tid == 0) item = (int)atomicAdd(&q.next[s], 1u);
        __syncthreads();
        return item < n ? item : -1;
    };
    auto finish = [&](int s) {
        __threadfence();
        __syncthreads();
        if (tid == 0) atomicAdd(&q.done[s], 1u);
    };
    // until all n items of stage s are done; false when the others stand still
    auto wait = [&](int s, int n) {
        __syncthreads();
        if (tid == 0) {
            unsigned seen = 0, last = 0, polls = 0;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&q.done[s]) : "memory");
                if (seen >= (unsigned)n || ++polls > kRedoPolls) break;
                if (seen != last) polls = 0;
                last = seen;
                __nanosleep(200);
            }
            item = seen >= (unsigned)n;
            if (!item) atomicExch(&q.late, 1u);
        }
        __syncthreads();
        return item != 0;
    };
    const int batches = (a.njobs + kRedoJobs - 1) / kRedoJobs;
    for (int i; (i = take(0, a.n1)) >= 0; finish(0))
        stack_piece1<CPLX>(a.pieces1[i], sm, a.segs, a.lq, a.lq_im, x, x_im, a.xsrc, a.xstride, a.colbase, a.colstride,
                           a.t1, a.t1_im);
    if (wait(0, a.n1)) {
        for (int i; (i = take(1, batches)) >= 0; finish(1))
            for (int j = i * kRedoJobs; j < min(a.njobs, (i + 1) * kRedoJobs); ++j) {
                stack_combine_job(a.jobs[j], a.terms, a.coef, a.t1, a.t2);
                if constexpr (CPLX) stack_combine_job(a.jobs[j], a.terms, a.coef, a.t1_im, a.t2_im);
            }
        if (wait(1, batches))
            for (int i; (i = take(2, a.n3)) >= 0;)
                stack_piece3<CPLX>(a.pieces3[i], sm, a.segs, a.t2, a.t2_im, a.rq, a.rq_im, a.yrow, y, y_im);
    }
    // the last CTA leaves the queue as it found it; if a wait ran out, nothing of y stands
    __threadfence();
    __syncthreads();
    if (tid == 0) item = atomicAdd(&q.left, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!item) return;
    __threadfence();
    if (*(volatile unsigned*)&q.late)
        for (int i = 0; i < a.n3; ++i) {
            const F64Piece t = a.pieces3[i];
            for (int e = tid; e < t.m_valid * t.n_valid; e += ST) {
                const int64_t o = a.yrow[t.out_off + e / t.n_valid] + t.n0 + e % t.n_valid;
                y[o] = NAN;
                if constexpr (CPLX) y_im[o] = NAN;
            }
        }
    __syncthreads();
    if (tid == 0) {
        q = RedoQueue{};
        *redo = 0;
    }
}

double seg_len(const std::vector<KSeg>& segs, int32_t s0, int32_t n) {
    double k = 0.0;
    for (int32_t s = s0; s < s0 + n; ++s) k += segs[(size_t)s].ke - segs[(size_t)s].kb;
    return k;
}

// One run of rows [r_begin, r_end) of a 128-row stack tile that share the K
// segments segs[seg0, seg0 + nseg): cut into pieces of at most SBM rows, and
// more where a piece would exceed `target` FMAs (down to one row).  A piece
// is the tile with its first row moved: stage 1 (mode 2) shifts the operand
// row and the T1 row (ldc), stage 3 (mode 1) the operand row and the y
// row-table index.
void cut_run(const TcTile& t, int r_begin, int r_end, int32_t seg0, int32_t nseg, double klen, double target,
             std::vector<F64Piece>& out) {
    const int R = r_end - r_begin;
    const double cost = (double)R * t.n_valid * klen;
    const int64_t want = std::max<int64_t>((R + SBM - 1) / SBM, (int64_t)std::ceil(cost / target));
    const int pieces = (int)std::min<int64_t>(want, R);
    const int rows = (R + pieces - 1) / pieces;
    for (int r0 = r_begin; r0 < r_end; r0 += rows) {
        F64Piece p;
        p.a_row = t.a_row + r0;
        p.a_cs = t.a_cs;
        p.b_row = t.b_row;
        p.b_cs = t.b_cs;
        p.m_valid = std::min(rows, r_end - r0);
        p.n_valid = t.n_valid;
        p.ldc = t.mode == 2 ? t.ldc + r0 : t.ldc;
        p.n0 = t.n0;
        p.out_off = t.mode == 2 ? t.out_off : t.out_off + r0;
        p.seg0 = seg0;
        p.nseg = nseg;
        out.push_back(p);
    }
}

void sort_longest_first(std::vector<F64Piece>& v, const std::vector<KSeg>& segs) {
    std::vector<std::pair<double, size_t>> c(v.size());
    for (size_t i = 0; i < v.size(); ++i)
        c[i] = {-(double)v[i].m_valid * v[i].n_valid * seg_len(segs, v[i].seg0, v[i].nseg), i};
    std::stable_sort(c.begin(), c.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
    std::vector<F64Piece> o(v.size());
    for (size_t i = 0; i < v.size(); ++i) o[i] = v[c[i].second];
    v.swap(o);
}

// Stage 1: every row of a stack needs all of its K = D_A.
void stage1_pieces(const std::vector<TcTile>& tiles, std::vector<F64Piece>& out, std::vector<KSeg>& segs) {
    double total = 0.0;
    for (const TcTile& t : tiles) total += (double)t.m_valid * t.n_valid * t.k_valid;
    const double target = std::max(1.0, total / (152.0 * 16.0));
    for (const TcTile& t : tiles) {
        const int32_t s0 = (int32_t)segs.size();
        segs.push_back({0, t.k_valid});
        cut_run(t, 0, t.m_valid, s0, 1, t.k_valid, target, out);
    }
    sort_longest_first(out, segs);
}

// Stage 3: row r of a T2 stack holds the columns the combine jobs write to
// it (each job one rectangle of rows and K columns); a run of consecutive
// rows with the same merged column ranges becomes pieces over those ranges.
bool stage3_pieces(const TcTables& C, std::vector<F64Piece>& out, std::vector<KSeg>& segs, std::string& err) {
    // column ranges per operand row of chunk 0 (the rows tiles and jobs index)
    std::vector<std::vector<KSeg>> rowk((size_t)std::max<int64_t>(C.t2q_rows, 0));
    for (const TcCombJob& j : C.jobs)
        for (int r = j.r0; r < j.r0 + j.rows; ++r) rowk[(size_t)j.t2row + r].push_back({j.k0, j.k0 + j.cols});
    for (std::vector<KSeg>& v : rowk) {
        if (v.empty()) continue;
        std::sort(v.begin(), v.end(), [](const KSeg& a, const KSeg& b) { return a.kb < b.kb; });
        std::vector<KSeg> m;
        for (const KSeg& g : v) {
            if (!m.empty() && g.kb <= m.back().ke)
                m.back().ke = std::max(m.back().ke, g.ke);
            else
                m.push_back(g);
        }
        v.swap(m);
    }
    auto klen = [](const std::vector<KSeg>& v) {
        double k = 0.0;
        for (const KSeg& g : v) k += g.ke - g.kb;
        return k;
    };
    auto same = [](const std::vector<KSeg>& a, const std::vector<KSeg>& b) {
        if (a.size() != b.size()) return false;
        for (size_t i = 0; i < a.size(); ++i)
            if (a[i].kb != b[i].kb || a[i].ke != b[i].ke) return false;
        return true;
    };
    // a bra sector without blocks of R has tiles without K: no rows of T2 are theirs
    const std::vector<KSeg> none;
    auto row_of = [&](const TcTile& t, int m) -> const std::vector<KSeg>& {
        return t.kch > 0 ? rowk[(size_t)t.a_row + m] : none;
    };
    double total = 0.0;
    for (const TcTile& t : C.tiles3)
        for (int m = 0; m < t.m_valid; ++m) total += (double)t.n_valid * klen(row_of(t, m));
    const double target = std::max(1.0, total / (152.0 * 16.0));
    for (const TcTile& t : C.tiles3) {
        int m = 0;
        while (m < t.m_valid) {
            const std::vector<KSeg>& ks = row_of(t, m);
            if (!ks.empty() && (ks.front().kb < 0 || ks.back().ke > t.k_valid)) {
                err = "stacked FP64 stage-3 row reaches past its stack's K";
                return false;
            }
            int e = m + 1;
            while (e < t.m_valid && same(row_of(t, e), ks)) ++e;
            // rows no combine job writes get a piece without segments: it stores zeros
            const int32_t s0 = (int32_t)segs.size();
            segs.insert(segs.end(), ks.begin(), ks.end());
            cut_run(t, m, e, s0, (int32_t)ks.size(), klen(ks), target, out);
            m = e;
        }
    }
    sort_longest_first(out, segs);
    return true;
}

}  // namespace

// The digit form of a stacked plan (digit_gemm.cu): the operand stacks as
// digits, their tiles, and the rows to turn into digits on every matvec.
struct F64Digits {
    DevBuf<unsigned char> mem;       // one allocation for all of it
    DigitStack l, r, t2, x;
    const int32_t* kx = nullptr;     // scales of the R and L stacks' columns
    const TcTile *tiles1 = nullptr, *tiles3 = nullptr;   // dealt out to `sms` CTAs:
    const int32_t *begin1 = nullptr, *begin3 = nullptr;
    const DigitPsi* psi = nullptr;
    const DigitRows* rows = nullptr;  // of T2
    // complex plans: the same for planar operands, T1's column tables for both parts
    const DigitRowsC* rows_c = nullptr;
    const int64_t* colbase = nullptr;
    const int32_t* colstride = nullptr;
    int* redo = nullptr;
    RedoQueue* queue = nullptr;
    DigitMaps m1, m3;
    int npsi = 0, max_k = 0, psi_cols = 32, nrows = 0, sms = 0;
};

struct F64Stack {
    std::unique_ptr<F64Digits> dg;  // null: the FP64 kernels run
    DevBuf<double> lq, rq, t1, t2, coef;
    DevBuf<double> lq_im, rq_im, t1_im, t2_im;  // complex environments only
    bool cplx = false;
    DevBuf<F64Piece> pieces1, pieces3;
    DevBuf<KSeg> segs;
    DevBuf<TcCombJob> jobs;
    DevBuf<TcCombTerm> terms;
    DevBuf<int64_t> yrow, colbase, xsrc;
    DevBuf<int32_t> colstride, xstride;
    int n1 = 0, n3 = 0, njobs = 0, comb_threads = 0;
    double bytes[3] = {0.0, 0.0, 0.0};  // per stage, without the psi / y vectors
};

void F64StackDeleter::operator()(F64Stack* p) const { delete p; }

// The rows of a stack, kDigitRowsPerCta a job.
static void digit_rows_of(std::vector<DigitRows>& out, int32_t row, int n, int32_t cs, int32_t kch, int32_t kx) {
    for (int r = 0; r < n; r += kDigitRowsPerCta)
        out.push_back({row + r, std::min(kDigitRowsPerCta, n - r), cs, kch, kx, -1});
}

// Whether a plan's FP64 matvec runs on digits: from 1.2 million multiply-adds in
// stage 1.  Below, the FP64 kernels finish before the digit kernels' latencies
// add up (Heisenberg D = 128, 0.4 million: 17 us against 29; Hubbard D = 256,
// 0.4 million: 31 against 28); above, their pipe is the limit (Hubbard D = 362,
// 1.3 million: 38 against 31 us; D = 512: 50 against 33; D = 2048, 230 million:
// 701 against 143; Heisenberg D = 512, 25 million: 151 against 48; cylinder D =
// 2048, 13 billion: 40.9 ms against 1.60).  A plan of less than a dozen stage-3
// tiles keeps its three launches up to 8 million: small plans of a few sectors
// are relied on to be three launches (digits would take 58 us against 85 at 6.2
// million on ten tiles).
bool f64stack_on_digits(const TcTables& C, bool cplx) {
    double f = 0.0;
    for (const std::vector<TcTile>* v : {&C.tiles1, &C.tiles1x})
        for (const TcTile& t : *v) f += (cplx ? 4.0 : 1.0) * t.m_valid * t.n_valid * t.k_valid;
    return f >= (C.tiles3.size() + C.tiles3f.size() < 12 ? 8e6 : 1.2e6);
}

// Where a K of several chunks leaves less than two 32-column jobs an SM, they are
// cut to eight columns: a job reads its K twice, one load after the other
// (Heisenberg D = 1024, 162 jobs: 10.1 -> 7.5 us).
static void psi_jobs(std::vector<DigitPsi>& psi, F64Digits& d) {
    for (const DigitPsi& j : psi) d.max_k = std::max(d.max_k, j.rows);
    if (d.max_k <= kTcBK || psi.size() >= 304) return;
    std::vector<DigitPsi> cut;
    for (const DigitPsi& j : psi)
        for (int c = 0; c < j.cols; c += 8) {
            DigitPsi q = j;
            q.src += c;
            q.to += c;
            q.cols = std::min(8, j.cols - c);
            cut.push_back(q);
        }
    psi.swap(cut);
    d.psi_cols = 8;
}

// Room behind the tables for the digits and the column scales; the tables go up
// in one copy, everything in one allocation.
static cudaError_t digits_alloc(F64Digits& d, const Blob& blob, const int64_t (&rows)[4], int32_t nk, int32_t** kx) {
    std::vector<unsigned char> host(blob.size());
    blob.copy_to(host.data());
    size_t total = blob.size(), q[4], x[4];
    auto take = [&](size_t n) {
        const size_t at = (total + 1023) & ~(size_t)1023;
        total = at + n;
        return at;
    };
    DigitStack* st[4] = {&d.l, &d.r, &d.t2, &d.x};
    for (int i = 0; i < 4; ++i) {
        st[i]->rows = std::max<int64_t>(rows[i], 1);
        q[i] = take(digit_stack_bytes(st[i]->rows));
        x[i] = take(sizeof(int32_t) * (size_t)(st[i]->rows + kTcBM));
    }
    const size_t k = take(sizeof(int32_t) * (size_t)std::max(nk, 1));
    cudaError_t e;
    // at most half of what is free: the solvers' vectors and other plans come later
    size_t free_bytes = 0, all = 0;
    if ((e = cudaMemGetInfo(&free_bytes, &all)) != cudaSuccess) return e;
    if (total > free_bytes / 2) return cudaErrorMemoryAllocation;
    if ((e = d.mem.alloc(total)) != cudaSuccess ||
        (e = cudaMemcpy(d.mem.p, host.data(), host.size(), cudaMemcpyHostToDevice)) != cudaSuccess)
        return e;
    for (int i = 0; i < 4; ++i) {
        st[i]->q = reinterpret_cast<__half*>(d.mem.p + q[i]);
        st[i]->ex = reinterpret_cast<int32_t*>(d.mem.p + x[i]);
    }
    *kx = reinterpret_cast<int32_t*>(d.mem.p + k);
    d.kx = *kx;
    // digit_psi_kernel writes a column's k up to a multiple of 16; a product's boxes of
    // 32 rows take in more of neighbouring columns (outputs that nothing uses)
    return cudaMemset(d.x.q, 0, digit_stack_bytes(d.x.rows));
}

// What a row of an L stack can come to in the result: the largest coefficient times
// column of R that the combine's terms give a row of T1 (binary exponents, kNoGain
// where no term reads it), as launch_digit_columns takes it for that row's unit.
// The scales of L's columns go by it: with psi's element at k on 2^kx, where some
// row's L 2^gain reaches 2^kx, the largest scaled element of a psi column does reach
// the result at full size, and no row's error can come to more than 2^-58 of it.
// (By the rows' own sizes instead, a channel that is large but hardly counts at the k
// where psi is large left relative errors up to 2e-7.)  kx3: exponents of R's columns;
// stack3: a stack-3 tile's first row of T2 -> its scales.
static std::vector<int32_t> row_gains(const TcTables& C, const std::map<int32_t, int32_t>& stack3,
                                      const std::vector<int32_t>& kx3) {
    const std::vector<std::pair<int32_t, int32_t>> stacks(stack3.begin(), stack3.end());
    std::vector<int32_t> gain((size_t)C.lq_rows, kNoGain);
    int32_t slab = -1, r = 0;  // the jobs of a slab have its terms in common
    for (const TcCombJob& j : C.jobs) {
        if (j.term_begin != slab) {
            slab = j.term_begin;
            const auto st = std::upper_bound(stacks.begin(), stacks.end(), j.t2row,
                                             [](int32_t v, const auto& x) { return v < x.first; });
            const int32_t* k = kx3.data() + std::prev(st)->second + j.k0;
            r = *std::max_element(k, k + j.cols);
        }
        if (r <= kDeadColumn) continue;
        for (int t = j.term_begin; t < j.term_end; ++t) {
            const double c = C.term_coef64[(size_t)t];
            if (c == 0.0) continue;
            uint64_t bits;
            std::memcpy(&bits, &c, sizeof(bits));
            const int32_t g = (int32_t)((bits >> 52) & 0x7FF) - 1023 + r, step = C.terms[(size_t)t].in_rs / j.cols;
            int32_t* x = gain.data() + C.term_row[(size_t)t] + (int64_t)j.r0 * step;
            // (a slab's rows are all raised together)
            if (*x >= g) continue;
            for (int i = 0; i < j.rows; ++i) x[(int64_t)i * step] = g;
        }
    }
    for (int32_t& g : gain)
        if (g != kNoGain) g = 1023 - g;  // the unit of a row's exponents
    return gain;
}

// The digit form of a complex plan: the same products on operands of two parts.
// Row (A, T2): (re | im); column (psi, R): re (re | -im), im (im | re), the im
// columns behind the re ones, so that one tile may hold both.
static cudaError_t digits_create_complex(const TcTables& C, F64Stack& p, std::unique_ptr<F64Digits> d, std::string& err) {
    struct Stack {
        int32_t M = 0, N = 0, K = 0, kch = 0, a = INT32_MAX, b = INT32_MAX;  // rows, columns, K; first rows of A and B
        int64_t out = INT64_MAX;  // first entry of the column table (stage 1) or row table (stage 3)
        int32_t kx = 0;           // stage 1: scales of its k
    };
    if (std::max({C.lq_rows, C.rq_rows, C.t2q_rows, C.xq_rows}) > INT32_MAX / 4) return cudaSuccess;  // 32-bit rows
    std::map<int32_t, Stack> s1, s3;  // by the first row of the operand that names the stack
    std::vector<TcTile> w3;
    for (const std::vector<TcTile>* v : {&C.tiles1x, &C.tiles3})
        for (const TcTile& t : *v) {
            if (t.kch == 0) {  // zeros, in either part: no operands; the second tile's columns all lie behind the split
                TcTile z = t;
                z.a_row = z.b_row = 0;
                w3.push_back(z);
                z.n0 += 1;
                z.split = 1;
                w3.push_back(z);
                continue;
            }
            Stack& s = t.mode == 2 ? s1[t.a_row - t.ldc] : s3[t.b_row - t.n0];
            s.M = t.a_cs, s.N = t.b_cs, s.K = t.k_valid, s.kch = t.kch;
            s.a = std::min(s.a, t.a_row), s.b = std::min(s.b, t.b_row), s.out = std::min(s.out, t.out_off);
        }
    std::vector<TcTile> w1, t1, t3;
    std::vector<int32_t> b1, b3;
    std::vector<DigitRowsC> lrows, rrows, trows;
    std::vector<DigitRows> rcols, lcols;
    std::vector<DigitPsi> psi;
    std::vector<int64_t> colbase(2 * C.t1col_base.size());
    std::vector<int32_t> colstride(2 * C.t1col_stride.size());
    const int64_t im = p.t1_im.p - p.t1.p;  // from T1's real part to its imaginary part
    int32_t nk = 0;
    auto rows = [](std::vector<DigitRowsC>& out, int32_t row, int n, int32_t cs, int32_t kch, int32_t kx, int32_t to,
                   int32_t cs_out, int32_t n_dual) {
        for (int r = 0; r < n; r += kDigitRowsPerCta)
            out.push_back({row + r, std::min(kDigitRowsPerCta, n - r), cs, kch, kx, to + r, cs_out, n_dual});
    };
    auto tiles = [](std::vector<TcTile>& out, const Stack& s, int mode) {
        for (int32_t m = 0; m < s.M; m += kTcBM)
            for (int32_t n = 0; n < 2 * s.N; n += kTcBN) {
                TcTile t{};
                t.a_row = 2 * s.a + m, t.a_cs = s.M;
                t.b_row = 4 * s.b + n, t.b_cs = 2 * s.N;
                t.kch = s.kch, t.k_valid = s.K, t.parts = 2;
                t.m_valid = std::min(kTcBM, s.M - m), t.n_valid = std::min(kTcBN, 2 * s.N - n);
                t.mode = mode;
                t.ldc = m, t.n0 = n;
                t.out_off = mode == 2 ? 2 * s.out + n : s.out + m;
                t.split = mode == 1 ? s.N : 0;
                out.push_back(t);
            }
    };
    std::map<int32_t, const Stack*> by_psi;  // stage-1 stacks by their first psi row
    int kch1 = 0;
    std::map<int32_t, int32_t> stack3;  // first row of T2 -> scales
    for (auto& [key, s] : s1) {
        by_psi[s.b] = &s;
        tiles(w1, s, 2);
        s.kx = nk;
        nk += s.kch * kTcBK;
        kch1 = std::max(kch1, s.kch);
        lcols.push_back({s.a, s.M, s.M, s.kch, s.kx, s.a});
        rows(lrows, s.a, s.M, s.M, s.kch, s.kx, 2 * s.a, s.M, 0);
        for (int32_t c = 0; c < s.N; ++c)
            for (int h = 0; h < 2; ++h) {
                colbase[(size_t)(2 * s.out + h * s.N + c)] = C.t1col_base[(size_t)(s.out + c)] + h * im;
                colstride[(size_t)(2 * s.out + h * s.N + c)] = C.t1col_stride[(size_t)(s.out + c)];
            }
    }
    for (const TcSplitJob& j : C.split) {
        if (j.a0 != 0) continue;
        auto it = by_psi.upper_bound(j.xrow);
        if (it == by_psi.begin()) {
            err = "digit operands: psi sub-block outside every stack";
            return cudaErrorInvalidValue;
        }
        const Stack& s = *std::prev(it)->second;
        psi.push_back({j.src + j.b0, j.rows, std::min(32, j.cols - j.b0), j.cols, 4 * s.b + (j.xrow - s.b) + j.b0, 2 * s.N,
                       s.N, s.kx, 0});
    }
    psi_jobs(psi, *d);
    for (const auto& [key, s] : s3) {
        tiles(w3, s, 1);
        rcols.push_back({s.b, s.N, s.N, s.kch, nk, -1});
        stack3[s.a] = nk;
        rows(rrows, s.b, s.N, s.N, s.kch, nk, 4 * s.b, 2 * s.N, s.N);
        rows(trows, s.a, s.M, s.M, s.kch, nk, 2 * s.a, s.M, 0);
        nk += s.kch * kTcBK;
    }
    cudaError_t e;
    int redo = 0, dev = 0;
    int32_t* kx = nullptr;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = digit_setup()) != cudaSuccess)
        return e;
    digit_schedule(w1, d->sms, t1, b1);
    digit_schedule(w3, d->sms, t3, b3);
    Blob blob;
    auto table = [&](const auto& v) { return blob.add(v.data(), sizeof(v[0]) * v.size()); };
    const RedoQueue queue{};
    const size_t o_redo = blob.add(&redo, sizeof(redo)), o_q = blob.add(&queue, sizeof(queue)), o_t1 = table(t1), o_t3 = table(t3), o_b1 = table(b1),
                 o_b3 = table(b3), o_psi = table(psi), o_rows = table(trows), o_l = table(lrows), o_r = table(rrows),
                 o_c = table(rcols), o_lc = table(lcols), o_cb = table(colbase), o_cs = table(colstride);
    if ((e = digits_alloc(*d, blob, {2 * C.lq_rows, 4 * C.rq_rows, 2 * C.t2q_rows, 4 * C.xq_rows}, nk, &kx)) != cudaSuccess)
        return e;
    unsigned char* m = d->mem.p;
    d->tiles1 = reinterpret_cast<const TcTile*>(m + o_t1);
    d->tiles3 = reinterpret_cast<const TcTile*>(m + o_t3);
    d->begin1 = reinterpret_cast<const int32_t*>(m + o_b1);
    d->begin3 = reinterpret_cast<const int32_t*>(m + o_b3);
    d->psi = reinterpret_cast<const DigitPsi*>(m + o_psi);
    d->rows_c = reinterpret_cast<const DigitRowsC*>(m + o_rows);
    d->colbase = reinterpret_cast<const int64_t*>(m + o_cb);
    d->colstride = reinterpret_cast<const int32_t*>(m + o_cs);
    d->redo = reinterpret_cast<int*>(m + o_redo);
    d->queue = reinterpret_cast<RedoQueue*>(m + o_q);
    if (!digit_maps(d->m1, d->l, d->x, err) || !digit_maps(d->m3, d->t2, d->r, err)) {
        err.clear();
        return cudaSuccess;
    }
    std::vector<int32_t> kx3((size_t)std::max(nk, 1)), gain;
    if ((e = cudaMemset(kx, 0, sizeof(int32_t) * (size_t)nk)) != cudaSuccess ||
        (e = launch_digit_columns(reinterpret_cast<const DigitRows*>(m + o_c), (int)rcols.size(), C.max_kch3, p.rq.p,
                                  p.rq_im.p, nullptr, kx, 0)) != cudaSuccess ||
        (e = cudaMemcpy(kx3.data(), kx, sizeof(int32_t) * (size_t)nk, cudaMemcpyDeviceToHost)) != cudaSuccess)
        return e;
    gain = row_gains(C, stack3, kx3);
    if ((e = cudaMemcpy(d->l.ex, gain.data(), sizeof(int32_t) * gain.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = launch_digit_columns(reinterpret_cast<const DigitRows*>(m + o_lc), (int)lcols.size(), kch1, p.lq.p, p.lq_im.p,
                                  d->l.ex, kx, 0)) != cudaSuccess ||
        (e = launch_digit_rows_complex(reinterpret_cast<const DigitRowsC*>(m + o_l), (int)lrows.size(), p.lq.p, p.lq_im.p,
                                       kx, -1, false, d->l, d->redo, 0)) != cudaSuccess ||
        (e = launch_digit_rows_complex(reinterpret_cast<const DigitRowsC*>(m + o_r), (int)rrows.size(), p.rq.p, p.rq_im.p,
                                       kx, -1, true, d->r, d->redo, 0)) != cudaSuccess ||
        (e = cudaMemcpy(&redo, d->redo, sizeof(int), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return e;
    d->npsi = (int)psi.size();
    d->nrows = (int)trows.size();
    if (redo == 0) p.dg = std::move(d);
    return cudaSuccess;
}

// Builds the digit form of p; left out (dg null) where the constant operands
// hold infinities or NaNs, without tensor maps, and (cudaErrorMemoryAllocation) where there is no
// memory for it.
static cudaError_t digits_create(const TcTables& C, F64Stack& p, std::string& err) {
    std::unique_ptr<F64Digits> d(new F64Digits);
    if (p.cplx) return digits_create_complex(C, p, std::move(d), err);
    std::vector<DigitRows> lrows, rrows, trows, rcols, lcols;
    std::vector<DigitPsi> psi;
    std::set<int32_t> seen;
    int32_t nk = 0;
    int kch1 = 0;
    // stage 1: the columns of L on scales of their own (row_gains), which psi takes up
    std::map<int32_t, int32_t> kx1;  // stack (its first psi row) -> scales
    for (const TcTile& t : C.tiles1x) {
        if (kx1.insert({t.b_row - t.n0, nk}).second) {
            const int32_t a = t.a_row - t.ldc;
            lcols.push_back({a, t.a_cs, t.a_cs, t.kch, nk, a});
            nk += t.kch * kTcBK;
            kch1 = std::max(kch1, t.kch);
        }
        if (seen.insert(t.a_row).second)
            digit_rows_of(lrows, t.a_row, t.m_valid, t.a_cs, t.kch, kx1[t.b_row - t.n0]);
    }
    for (const TcSplitJob& j : C.split) {
        if (j.a0 != 0) continue;
        auto it = kx1.upper_bound(j.xrow);
        if (it == kx1.begin()) {
            err = "digit operands: psi sub-block outside every stack";
            return cudaErrorInvalidValue;
        }
        psi.push_back({j.src + j.b0, j.rows, std::min(32, j.cols - j.b0), j.cols, j.xrow + j.b0, j.cstride, 0,
                       std::prev(it)->second, 0});
    }
    psi_jobs(psi, *d);
    // stage 3: the columns of R on scales of their own, which T2 takes up, so
    // that no channel's magnitude (an energy against an identity) costs the
    // others digits
    std::map<int32_t, int32_t> kx, stack3;  // stack (its first row of R, a tile's first row of T2) -> scales
    std::vector<TcTile> w3(C.tiles3);
    for (TcTile& t : w3) {
        if (t.kch == 0) {  // zeros, without operands
            t.a_row = t.b_row = 0;
            continue;
        }
        const int32_t base = t.b_row - t.n0;
        if (kx.insert({base, nk}).second) {
            rcols.push_back({base, t.b_cs, t.b_cs, t.kch, nk, -1});
            nk += t.kch * kTcBK;
        }
        if (seen.insert(-1 - t.b_row).second) digit_rows_of(rrows, t.b_row, t.n_valid, t.b_cs, t.kch, kx[base]);
        if (t.n0 == 0) digit_rows_of(trows, t.a_row, t.m_valid, t.a_cs, t.kch, kx[base]);
        stack3[t.a_row] = kx[base];
    }
    std::vector<TcTile> t1, t3;
    std::vector<int32_t> b1, b3;
    cudaError_t e;
    int redo = 0, dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = digit_setup()) != cudaSuccess)
        return e;
    digit_schedule(C.tiles1x, d->sms, t1, b1);
    digit_schedule(w3, d->sms, t3, b3);
    // the tables first (one copy), then what the device writes
    Blob blob;
    auto table = [&](const auto& v) { return blob.add(v.data(), sizeof(v[0]) * v.size()); };
    const RedoQueue queue{};
    const size_t o_redo = blob.add(&redo, sizeof(redo)), o_q = blob.add(&queue, sizeof(queue)), o_t1 = table(t1), o_t3 = table(t3), o_b1 = table(b1),
                 o_b3 = table(b3), o_psi = table(psi), o_rows = table(trows), o_l = table(lrows), o_r = table(rrows),
                 o_c = table(rcols), o_lc = table(lcols);
    int32_t* kxd = nullptr;
    if ((e = digits_alloc(*d, blob, {C.lq_rows, C.rq_rows, C.t2q_rows, C.xq_rows}, nk, &kxd)) != cudaSuccess) return e;
    unsigned char* m = d->mem.p;
    d->tiles1 = reinterpret_cast<const TcTile*>(m + o_t1);
    d->tiles3 = reinterpret_cast<const TcTile*>(m + o_t3);
    d->begin1 = reinterpret_cast<const int32_t*>(m + o_b1);
    d->begin3 = reinterpret_cast<const int32_t*>(m + o_b3);
    d->psi = reinterpret_cast<const DigitPsi*>(m + o_psi);
    d->rows = reinterpret_cast<const DigitRows*>(m + o_rows);
    d->redo = reinterpret_cast<int*>(m + o_redo);
    d->queue = reinterpret_cast<RedoQueue*>(m + o_q);
    if (!digit_maps(d->m1, d->l, d->x, err) || !digit_maps(d->m3, d->t2, d->r, err)) {
        err.clear();
        return cudaSuccess;
    }
    std::vector<int32_t> kx3((size_t)std::max(nk, 1)), gain;
    if ((e = cudaMemset(kxd, 0, sizeof(int32_t) * (size_t)nk)) != cudaSuccess ||
        (e = launch_digit_columns(reinterpret_cast<const DigitRows*>(m + o_c), (int)rcols.size(), C.max_kch3, p.rq.p, nullptr,
                                  nullptr, kxd, 0)) != cudaSuccess ||
        (e = cudaMemcpy(kx3.data(), kxd, sizeof(int32_t) * (size_t)nk, cudaMemcpyDeviceToHost)) != cudaSuccess)
        return e;
    gain = row_gains(C, stack3, kx3);
    if ((e = cudaMemcpy(d->l.ex, gain.data(), sizeof(int32_t) * gain.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = launch_digit_columns(reinterpret_cast<const DigitRows*>(m + o_lc), (int)lcols.size(), kch1, p.lq.p, nullptr,
                                  d->l.ex, kxd, 0)) != cudaSuccess ||
        (e = launch_digit_rows(reinterpret_cast<const DigitRows*>(m + o_l), (int)lrows.size(), p.lq.p, kxd, -1, d->l,
                               d->redo, 0)) != cudaSuccess ||
        (e = launch_digit_rows(reinterpret_cast<const DigitRows*>(m + o_r), (int)rrows.size(), p.rq.p, kxd, -1, d->r,
                               d->redo, 0)) != cudaSuccess ||
        (e = cudaMemcpy(&redo, d->redo, sizeof(int), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return e;
    d->npsi = (int)psi.size();
    d->nrows = (int)trows.size();
    if (redo == 0) p.dg = std::move(d);
    return cudaSuccess;
}

tk_status f64stack_create(const TcTables& C, std::unique_ptr<F64Stack, F64StackDeleter>& out, std::string& err) {
    if (!C.tiles1.empty() || !C.tiles3f.empty()) {
        err = "stacked FP64 tables without a psi copy's layout, or with fused tiles";
        return TK_ERR_INVALID_ARG;
    }
    for (const std::vector<TcTile>* v : {&C.tiles1x, &C.tiles3})
        for (const TcTile& t : *v)
            if (t.m_valid <= 0 || t.m_valid > kTcBM || t.n_valid <= 0 || t.n_valid > SBN) {
                err = "stacked FP64 tile shape";
                return TK_ERR_INVALID_ARG;
            }
    std::vector<KSeg> segs;
    std::vector<F64Piece> p1, p3;
    stage1_pieces(C.tiles1x, p1, segs);
    if (!stage3_pieces(C, p3, segs, err)) return TK_ERR_INVALID_ARG;
    std::unique_ptr<F64Stack, F64StackDeleter> p(new F64Stack);
    cudaError_t e = cudaSuccess;
    if ((e = p->lq.upload(C.lq64)) != cudaSuccess || (e = p->rq.upload(C.rq64)) != cudaSuccess ||
        (e = p->pieces1.upload(p1)) != cudaSuccess || (e = p->pieces3.upload(p3)) != cudaSuccess ||
        (e = p->segs.upload(segs)) != cudaSuccess ||
        (e = p->jobs.upload(C.jobs)) != cudaSuccess || (e = p->terms.upload(C.terms)) != cudaSuccess ||
        (e = p->coef.upload(C.term_coef64)) != cudaSuccess || (e = p->yrow.upload(C.yrow)) != cudaSuccess ||
        (e = p->colbase.upload(C.t1col_base)) != cudaSuccess || (e = p->colstride.upload(C.t1col_stride)) != cudaSuccess ||
        (e = p->xsrc.upload(C.xsrc)) != cudaSuccess || (e = p->xstride.upload(C.xstride)) != cudaSuccess ||
        (e = p->t1.alloc((size_t)std::max<int64_t>(C.t1_total, 1))) != cudaSuccess ||
        (e = p->t2.alloc((size_t)std::max<int64_t>(C.t2q_rows * kTcBK, 1))) != cudaSuccess ||
        (e = cudaMemset(p->t2.p, 0, sizeof(double) * p->t2.n)) != cudaSuccess) {
        err = std::string("stacked FP64 operands: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? TK_ERR_OOM : TK_ERR_CUDA;
    }
    p->cplx = !C.lq64_im.empty() || !C.rq64_im.empty();
    if (p->cplx &&
        ((e = p->lq_im.upload(C.lq64_im)) != cudaSuccess || (e = p->rq_im.upload(C.rq64_im)) != cudaSuccess ||
         (e = p->t1_im.alloc(p->t1.n)) != cudaSuccess || (e = p->t2_im.alloc(p->t2.n)) != cudaSuccess ||
         (e = cudaMemset(p->t2_im.p, 0, sizeof(double) * p->t2_im.n)) != cudaSuccess)) {
        err = std::string("stacked FP64 imaginary operands: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? TK_ERR_OOM : TK_ERR_CUDA;
    }
    if (p->cplx && (C.lq64_im.size() != C.lq64.size() || C.rq64_im.size() != C.rq64.size())) {
        err = "stacked FP64 imaginary stacks of another size";
        return TK_ERR_INVALID_ARG;
    }
    // Bytes each stage must move at least: every stack element a piece reads
    // once (rows read by several column tiles count once), T1 written / read
    // once, T2 written / read once.
    auto stack_elems = [&](const std::vector<F64Piece>& v, bool a_side) {
        std::set<std::pair<int32_t, int32_t>> seen;
        double n = 0.0;
        for (const F64Piece& q : v)
            if (seen.insert({a_side ? q.a_row : q.b_row, a_side ? q.m_valid : q.n_valid}).second)
                n += (double)(a_side ? q.m_valid : q.n_valid) * seg_len(segs, q.seg0, q.nseg);
        return n;
    };
    double comb_reads = 0.0;
    for (const TcCombJob& j : C.jobs) comb_reads += (double)j.rows * j.cols * (j.term_end - j.term_begin);
    const double t2_elems = stack_elems(p3, true);
    p->bytes[0] = 8.0 * (stack_elems(p1, true) + (double)C.t1_total);
    p->bytes[1] = 8.0 * (std::min<double>((double)C.t1_total, comb_reads) + t2_elems);
    p->bytes[2] = 8.0 * (t2_elems + stack_elems(p3, false));
    p->n1 = (int)p1.size();
    p->n3 = (int)p3.size();
    p->njobs = (int)C.jobs.size();
    // Threads a combine job, whole matvecs in us at 256 / 128: Heisenberg D = 256
    // 32.8 / 35.8, D = 1024 89.1 / 91.1, cylinder D = 128 42.5 / 46.3, D = 512
    // 126 / 131; the other way round (combine_narrow) Hubbard D = 2048 145 / 142,
    // cylinder D = 64 17.4 / 17.0, and from 16 thousand jobs on: cylinder D = 1150
    // 508 / 497, D = 2048 1,599 / 1,580 (D = 1024, 17 thousand: 331 / 332).
    p->comb_threads = combine_narrow(C.jobs) || C.jobs.size() >= 16384 ? 128 : 256;
    if (f64stack_on_digits(C, p->cplx) && (e = digits_create(C, *p, err)) != cudaSuccess) {
        // without memory for the digits (7/4 of the stacks' bytes) the FP64 kernels run
        if (e != cudaErrorMemoryAllocation) {
            if (err.empty()) err = std::string("digit operands: ") + cudaGetErrorString(e);
            return TK_ERR_CUDA;
        }
        cudaGetLastError();
    }
    if (p->dg) {  // operands of two bytes a digit; those of psi and T2 written and read on top
        double psi = 0.0;
        for (const TcSplitJob& j : C.split)
            if (j.a0 == 0 && j.b0 == 0) psi += (double)j.rows * j.cols;
        constexpr double d = 2.0 * kDigits;
        p->bytes[0] = d * (stack_elems(p1, true) + 2.0 * psi) + 8.0 * (double)C.t1_total;
        p->bytes[1] += (8.0 + d) * t2_elems;
        p->bytes[2] = d * (t2_elems + stack_elems(p3, false));
    }
    out = std::move(p);
    return TK_OK;
}

// T2 from T1, both parts of a complex plan in one launch.
static cudaError_t combine_stage(const F64Stack& p, cudaStream_t s) {
    if (p.njobs == 0) return cudaSuccess;
    return launch_dependent(p.cplx ? stack_combine_f64_kernel<true> : stack_combine_f64_kernel<false>,
                            dim3((unsigned)p.njobs, p.cplx ? 2u : 1u), (unsigned)p.comb_threads, 0, s, p.jobs.p,
                            p.terms.p, p.coef.p, p.t1.p, p.t2.p, p.t1_im.p, p.t2_im.p);
}

static RedoArgs redo_args(const F64Stack& p) {
    return RedoArgs{p.pieces1.p, p.pieces3.p, p.segs.p,  p.jobs.p,    p.terms.p,     p.coef.p, p.lq.p, p.rq.p, p.lq_im.p,
                    p.rq_im.p,   p.xsrc.p,    p.colbase.p, p.yrow.p,  p.xstride.p, p.colstride.p, p.t1.p,   p.t2.p, p.t1_im.p,
                    p.t2_im.p,   p.dg->queue, p.n1,      p.n3,       p.njobs};
}

// The stand-by: at most kRedoCtasPerSm CTAs an SM, fewer where a stage has not so much work.
template <bool CPLX>
static cudaError_t launch_redo(const F64Stack& p, const double* x, const double* x_im, double* y, double* y_im,
                               cudaStream_t s) {
    const int ctas = std::min(kRedoCtasPerSm * p.dg->sms, std::max({p.n1, p.n3, 1}));
    return launch_dependent(stack_redo_f64_kernel<CPLX>, ctas, ST, 0, s, redo_args(p), x, x_im, y, y_im, p.dg->redo);
}

// One stage of the digit matvec.
static cudaError_t digits_stage(F64Stack& p, const double* x, double* y, cudaStream_t s, int stage) {
    F64Digits& d = *p.dg;
    cudaError_t e;
    DigitOut o{};
    if (stage == 0) {
        if ((e = launch_digit_psi(d.psi, d.npsi, d.psi_cols, d.max_k, x, nullptr, d.kx, d.x, d.redo, s)) != cudaSuccess) return e;
        o.out = p.t1.p;
        o.colbase = p.colbase.p;
        o.colstride = p.colstride.p;
        return launch_digit_gemm(2, d.tiles1, d.begin1, d.sms, d.m1, d.l.ex, d.x.ex, o, d.redo, s);
    }
    if (stage == 1) {
        if ((e = combine_stage(p, s)) != cudaSuccess) return e;
        return launch_digit_rows(d.rows, d.nrows, p.t2.p, d.kx, 1, d.t2, d.redo, s);
    }
    o.out = y;
    o.rowtab = p.yrow.p;
    if ((e = launch_digit_gemm(1, d.tiles3, d.begin3, d.sms, d.m3, d.t2.ex, d.r.ex, o, d.redo, s)) != cudaSuccess) return e;
    return launch_redo<false>(p, x, nullptr, y, nullptr, s);
}

// The digit matvec on planar vectors.
static cudaError_t digits_apply_complex(F64Stack& p, const double* xr, const double* xi, double* yr, double* yi,
                                        cudaStream_t s) {
    F64Digits& d = *p.dg;
    cudaError_t e = launch_digit_psi(d.psi, d.npsi, d.psi_cols, d.max_k, xr, xi, d.kx, d.x, d.redo, s);
    DigitOut o{};
    o.out = p.t1.p;
    o.colbase = d.colbase;
    o.colstride = d.colstride;
    if (e == cudaSuccess) e = launch_digit_gemm(2, d.tiles1, d.begin1, d.sms, d.m1, d.l.ex, d.x.ex, o, d.redo, s);
    if (e == cudaSuccess) e = combine_stage(p, s);
    if (e == cudaSuccess)
        e = launch_digit_rows_complex(d.rows_c, d.nrows, p.t2.p, p.t2_im.p, d.kx, 1, false, d.t2, d.redo, s);
    o = DigitOut{};
    o.out = yr;
    o.out_im = yi;
    o.rowtab = p.yrow.p;
    if (e == cudaSuccess) e = launch_digit_gemm(1, d.tiles3, d.begin3, d.sms, d.m3, d.t2.ex, d.r.ex, o, d.redo, s);
    if (e != cudaSuccess) return e;
    return launch_redo<true>(p, xr, xi, yr, yi, s);
}

cudaError_t f64stack_stage(F64Stack& p, const double* x, double* y, cudaStream_t s, int stage) {
    if (p.dg) return digits_stage(p, x, y, s, stage);
    if (stage == 0 && p.n1 > 0)
        return launch_dependent(stack_gemm1_f64_kernel<false>, p.n1, ST, 0, s, p.pieces1.p, p.segs.p, p.lq.p, nullptr, x,
                                nullptr, p.xsrc.p, p.xstride.p, p.colbase.p, p.colstride.p, p.t1.p, nullptr);
    if (stage == 1) return combine_stage(p, s);
    if (stage == 2 && p.n3 > 0)
        return launch_dependent(stack_gemm3_f64_kernel<false>, p.n3, ST, 0, s, p.pieces3.p, p.segs.p, p.t2.p, nullptr,
                                p.rq.p, nullptr, p.yrow.p, y, nullptr);
    return cudaSuccess;
}

cudaError_t f64stack_apply(F64Stack& p, const double* x, double* y, cudaStream_t s) {
    for (int stage = 0; stage < 3; ++stage) {
        cudaError_t e = f64stack_stage(p, x, y, s, stage);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t f64stack_apply_complex(F64Stack& p, const double* xr, const double* xi, double* yr, double* yi,
                                   cudaStream_t s) {
    if (!p.cplx) return cudaErrorInvalidValue;
    if (p.dg) return digits_apply_complex(p, xr, xi, yr, yi, s);
    cudaError_t e = cudaSuccess;
    if (p.n1 > 0)
        e = launch_dependent(stack_gemm1_f64_kernel<true>, p.n1, ST, 0, s, p.pieces1.p, p.segs.p, p.lq.p, p.lq_im.p, xr, xi,
                             p.xsrc.p, p.xstride.p, p.colbase.p, p.colstride.p, p.t1.p, p.t1_im.p);
    if (e == cudaSuccess) e = combine_stage(p, s);
    if (e == cudaSuccess && p.n3 > 0)
        e = launch_dependent(stack_gemm3_f64_kernel<true>, p.n3, ST, 0, s, p.pieces3.p, p.segs.p, p.t2.p, p.t2_im.p,
                             p.rq.p, p.rq_im.p, p.yrow.p, yr, yi);
    return e;
}

int f64stack_launches(const F64Stack& p) {
    const int n = (p.n1 > 0) + (p.njobs > 0) + (p.n3 > 0);
    return p.dg ? n + (p.dg->npsi > 0) + (p.dg->nrows > 0) + 1 : n;
}

void f64stack_bytes(const F64Stack& p, double out[3]) {
    for (int i = 0; i < 3; ++i) out[i] = p.bytes[i];
}

}  // namespace tk
