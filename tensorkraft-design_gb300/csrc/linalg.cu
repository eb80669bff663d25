// linalg.cu -- LinAlgBackend::gemm, SparseLinAlgBackend::{block_gemm, spmv}
// on the device, through the same grouped segmented FP64 GEMM kernel as the
// H_eff path.
//
// block_gemm follows tk-linalg/src/device/faer.rs:390-575 and
// tk-linalg/src/tasks.rs:36-81,180-188: a task for every (key_a, key_b) pair
// whose contracted quantum numbers are equal and whose output sector
// satisfies row (+) dual(col) == flux_a (+) flux_b; contributions to the same
// output key are summed (here in registers, one output block per task); the
// output keys are ascending; output legs [a.legs[0], b.legs[1]] with
// directions [a.dirs[0], b.dirs[1]].
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "digit_gemm.cuh"
#include "kernels.cuh"
#include "tk_bsgemm.hpp"
#include "tk_internal.hpp"
#include "tk_plan.cuh"

using namespace tk;

namespace {

struct Guard {
    int prev = -1;
    explicit Guard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        cudaSetDevice(dev);
    }
    ~Guard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

tk_status fail(const char* op, cudaError_t e) {
    set_error(std::string(op) + ": " + cudaGetErrorName(e) + ": " + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? TK_ERR_OOM : TK_ERR_CUDA;
}

struct Scratch {
    std::vector<void*> ptrs;
    ~Scratch() {
        for (void* p : ptrs) cudaFree(p);
    }
    template <class T>
    cudaError_t put(const std::vector<T>& v, T** out) {
        *out = nullptr;
        if (v.empty()) return cudaSuccess;
        cudaError_t e = cudaMalloc((void**)out, sizeof(T) * v.size());
        if (e != cudaSuccess) return e;
        ptrs.push_back(*out);
        return cudaMemcpy(*out, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
    }
    template <class T>
    cudaError_t make(size_t n, T** out) {
        *out = nullptr;
        if (n == 0) return cudaSuccess;
        cudaError_t e = cudaMalloc((void**)out, sizeof(T) * n);
        if (e == cudaSuccess) ptrs.push_back(*out);
        return e;
    }
};

#define CK(op)                                        \
    do {                                              \
        cudaError_t e_ = (op);                        \
        if (e_ != cudaSuccess) return fail(#op, e_);  \
    } while (0)


// A device buffer for one tk_gemm_f64 call; null where there is no memory (the
// caller takes another path).  The call waits for its stream before it gives the
// buffer back, so any thread's next call on the context may take it; at most
// kGemmKeep bytes stay with the context (the digits of 4096^3), until memory runs
// out (release_scratch).
constexpr size_t kGemmKeep = (size_t)512 << 20;
struct GemmBuffer {
    tk_ctx* ctx;
    void* p = nullptr;
    size_t n = 0;
    GemmBuffer(tk_ctx* c, size_t bytes) : ctx(c) {
        if (ctx) {
            std::lock_guard<std::mutex> lock(ctx->gemm_mutex);
            auto best = ctx->gemm_free.end();
            for (auto it = ctx->gemm_free.begin(); it != ctx->gemm_free.end(); ++it)
                if (it->second >= bytes && (best == ctx->gemm_free.end() || it->second < best->second)) best = it;
            if (best != ctx->gemm_free.end()) {
                p = best->first;
                n = best->second;
                ctx->gemm_free.erase(best);
                return;
            }
        }
        if (dev_malloc(&p, bytes) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        n = bytes;
    }
    ~GemmBuffer() {
        if (!p) return;
        if (ctx) {
            std::lock_guard<std::mutex> lock(ctx->gemm_mutex);
            size_t kept = n;
            for (auto& b : ctx->gemm_free) kept += b.second;
            try {
                // the smaller ones make room: the largest serves every call
                std::sort(ctx->gemm_free.begin(), ctx->gemm_free.end(),
                          [](const auto& a, const auto& b) { return a.second < b.second; });
                while (kept > kGemmKeep && !ctx->gemm_free.empty() && ctx->gemm_free.front().second < n) {
                    kept -= ctx->gemm_free.front().second;
                    cudaFree(ctx->gemm_free.front().first);
                    ctx->gemm_free.erase(ctx->gemm_free.begin());
                }
                if (kept <= kGemmKeep) {
                    ctx->gemm_free.push_back({p, n});
                    return;
                }
            } catch (const std::bad_alloc&) {
            }
        }
        cudaFree(p);
    }
    GemmBuffer(const GemmBuffer&) = delete;
    GemmBuffer& operator=(const GemmBuffer&) = delete;
};

// The dense product on the fp16 tensor cores (digit_gemm.cu).  *done is left
// false where the FP64 kernel is to run instead: an output that might be less
// exact on digits, no memory for them, no tensor maps.
tk_status gemm_digits(tk_ctx* ctx, double alpha, const tk_mat* a, const tk_mat* b, double beta, tk_mat_mut* c,
                      cudaStream_t s, bool* done) {
    *done = false;
    const int64_t M = a->rows, N = b->cols, K = a->cols, kch = (K + kTcBK - 1) / kTcBK;
    DigitMatrix A{a->data, a->row_stride, a->col_stride, (int)M, {}, nullptr, nullptr, nullptr};
    DigitMatrix B{b->data, b->col_stride, b->row_stride, (int)N, {}, nullptr, nullptr, nullptr};
    A.out.rows = M * kch;
    B.out.rows = N * kch;
    size_t total = 256;  // the flags
    auto take = [&](size_t n) {
        const size_t at = total;
        total += (n + 255) & ~(size_t)255;
        return at;
    };
    const size_t ta = take(sizeof(uint32_t) * M), tb = take(sizeof(uint32_t) * N), zeroed = total;
    const size_t ea = take(sizeof(int32_t) * M), eb = take(sizeof(int32_t) * N);
    const size_t sa = take(sizeof(float) * kDigitSamples * M), sb = take(sizeof(float) * kDigitSamples * N);
    const size_t qa = take(digit_stack_bytes(A.out.rows)), qb = take(digit_stack_bytes(B.out.rows));
    GemmBuffer buf(ctx, total);
    if (!buf.p) return TK_OK;
    unsigned char* p = static_cast<unsigned char*>(buf.p);
    int* redo = reinterpret_cast<int*>(p);
    A.out.q = reinterpret_cast<__half*>(p + qa);
    B.out.q = reinterpret_cast<__half*>(p + qb);
    A.out.ex = reinterpret_cast<int32_t*>(p + ea);
    B.out.ex = reinterpret_cast<int32_t*>(p + eb);
    A.top = reinterpret_cast<uint32_t*>(p + ta);
    B.top = reinterpret_cast<uint32_t*>(p + tb);
    A.inexact = redo + 2;
    B.inexact = redo + 3;
    A.sample = reinterpret_cast<float*>(p + sa);
    B.sample = reinterpret_cast<float*>(p + sb);
    DigitMaps maps;
    std::string err;
    if (!digit_maps(maps, A.out, B.out, err)) return TK_OK;
    DigitOut o{};
    o.out = c->data;
    o.c_rs = c->row_stride;
    o.c_cs = c->col_stride;
    o.alpha = alpha;
    o.beta = beta;
    o.m = (int)M;
    o.n = (int)N;
    o.k = (int)K;
    o.tiles = (int)(((M + kTcBM - 1) / kTcBM) * ((N + kTcBN - 1) / kTcBN));
    int state = 0;
    cudaError_t e = digit_setup();
    if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, zeroed, s);
    if (e == cudaSuccess) e = launch_digit_matrices(A, B, (int)K, redo + 1, redo, s);
    if (e == cudaSuccess) e = launch_digit_gemm(0, nullptr, nullptr, std::min(o.tiles, 152), maps, A.out.ex, B.out.ex, o, redo, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&state, redo, sizeof(int), cudaMemcpyDeviceToHost, s);
    // the buffer goes back when the stream is done with it, whatever failed
    const cudaError_t w = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = w;
    if (e != cudaSuccess) return fail("tk_gemm_f64", e);
    if (state == kDigitWait && beta != 0.0) {  // part of C is written: it cannot be computed again
        set_error("tk_gemm_f64: a bounded wait of the tensor-core kernel ran out");
        return TK_ERR_TIMEOUT;
    }
    *done = state == 0;
    return TK_OK;
}

// The faster of the two kernels for a product.  The digits cost 45 us however
// small it is, then 4 us for 64 k of as many 128 x 64 tiles as there are SMs and
// 6 us for the tiles' ends (estimates, 10 to 15 % above what large products take);
// the FP64 kernel's estimate is its own.  Whole calls, digits against FP64 kernel:
// 200 x 200 x 1000 97 us against 98, 300^3 67 against 71, 512 x 512 x 128 56
// against 71, 2048 x 64 x 300 69 against 90, 400^3 69 against 142, 2048 x 32 x
// 2048 143 against 245, 2048^3 0.51 ms against 13.9; on the other side 256^3 and
// 512 x 512 x 64 stay with the FP64 kernel (53 and 48 us).  Operands that the gate
// refuses have cost 50 us and the digits' passes when the FP64 kernel starts.
// Digits of more than 2 GB are not laid out.
bool gemm_on_digits(int64_t M, int64_t N, int64_t K) {
    if (K <= 0 || (double)(M + N) * (K + kTcBK) * kDigits * 2.0 > 2147483648.0) return false;
    const double tiles = (double)((M + kTcBM - 1) / kTcBM) * ((N + kTcBN - 1) / kTcBN);
    const double waves = std::ceil(tiles / 152.0), kch = (double)((K + kTcBK - 1) / kTcBK);
    return 45e-6 + waves * (6e-6 + 4e-6 * kch) < dense_gemm_f64_plan(M, N, K);
}

}  // namespace

extern "C" {

tk_status tk_gemm_f64(tk_ctx* ctx, double alpha, const tk_mat* a, const tk_mat* b, double beta, tk_mat_mut* c,
                      void* stream) {
    (void)ctx;
    if (!a || !b || !c || !a->data || !b->data || !c->data) {
        set_error("tk_gemm_f64: null argument");
        return TK_ERR_INVALID_ARG;
    }
    if (a->cols != b->rows || c->rows != a->rows || c->cols != b->cols) {
        set_error("tk_gemm_f64: shape mismatch");
        return TK_ERR_INVALID_ARG;
    }
    if (c->rows == 0 || c->cols == 0) return TK_OK;
    const int64_t lim = INT32_MAX;
    if (a->rows > lim || a->cols > lim || b->cols > lim || std::llabs(a->row_stride) > lim ||
        std::llabs(a->col_stride) > lim || std::llabs(b->row_stride) > lim || std::llabs(b->col_stride) > lim ||
        std::llabs(c->row_stride) > lim || std::llabs(c->col_stride) > lim) {
        set_error("tk_gemm_f64: dimensions or strides exceed 32 bits");
        return TK_ERR_UNSUPPORTED;
    }
    int dev = 0;
    if (ctx) dev = ctx->device;
    Guard gd(dev);
    cudaStream_t s = (cudaStream_t)stream;
    if (gemm_on_digits(a->rows, b->cols, a->cols)) {
        bool done = false;
        const tk_status st = gemm_digits(ctx, alpha, a, b, beta, c, s, &done);
        if (st != TK_OK || done) return st;
    }
    GemmTask t{};
    t.M = (int32_t)a->rows;
    t.N = (int32_t)b->cols;
    t.c_off = 0;
    t.c_rs = (int32_t)c->row_stride;
    t.c_cs = (int32_t)c->col_stride;
    t.alpha = alpha;
    t.beta = beta;
    GemmSeg sg{};
    sg.a_rs = (int32_t)a->row_stride; sg.a_cs = (int32_t)a->col_stride;
    sg.b_rs = (int32_t)b->row_stride; sg.b_cs = (int32_t)b->col_stride;
    sg.K = (int32_t)a->cols;
    CK(launch_dense_gemm_f64(t, sg, a->data, b->data, c->data, s));
    CK(cudaStreamSynchronize(s));
    return TK_OK;
}

// Output header of a block GEMM (legs of A's rows and B's columns, their
// directions, the output flux) and its key / offset arrays; data unallocated.
static tk_status fill_out_header(const tk_bst* a_abi, const tk_bst* b_abi, const Rank2& A, const Rank2& B,
                                 const BlockGemmPlan& P, tk_bst_out* out, bool with_data) {
    out->qn_kind = A.kind;
    out->rank = 2;
    out->legs[0] = a_abi->legs[0];
    out->legs[1] = b_abi->legs[1];
    out->leg_dirs[0] = A.dirs[0];
    out->leg_dirs[1] = B.dirs[1];
    out->flux[0] = P.target.c[0];
    out->flux[1] = P.target.c[1];
    out->n_blocks = (int64_t)P.okeys.size();
    out->total = P.total;
    out->keys = (uint64_t*)std::malloc(sizeof(uint64_t) * std::max<size_t>(P.okeys.size(), 1));
    out->block_offsets = (int64_t*)std::malloc(sizeof(int64_t) * std::max<size_t>(P.ooffs.size(), 1));
    out->data = with_data ? (double*)std::malloc(sizeof(double) * (size_t)std::max<int64_t>(P.total, 1)) : nullptr;
    if (!out->keys || !out->block_offsets || (with_data && !out->data)) {
        tk_bst_free(out);
        set_error("block gemm: host allocation failed");
        return TK_ERR_OOM;
    }
    std::copy(P.okeys.begin(), P.okeys.end(), out->keys);
    std::copy(P.ooffs.begin(), P.ooffs.end(), out->block_offsets);
    return TK_OK;
}

// Grouped-GEMM tables of a block GEMM, packed for one copy.
struct TableBlob {
    size_t tasks = 0, segs = 0, tiles = 0;
};
static TableBlob add_tables(Blob& b, const GemmTable& g) {
    TableBlob t;
    t.tasks = b.add(g.tasks.data(), sizeof(GemmTask) * g.tasks.size());
    t.segs = b.add(g.segs.data(), sizeof(GemmSeg) * g.segs.size());
    t.tiles = b.add(g.tiles.data(), sizeof(GemmTile) * g.tiles.size());
    return t;
}

// Copies `blob` through the context's page-locked staging into its device
// scratch on `s`; *dev receives the scratch base (at least blob.device_size()).
static tk_status stage_blob(tk_ctx* ctx, const Blob& blob, cudaStream_t s, unsigned char** dev) {
    void *d = nullptr, *h = nullptr;
    tk_status st;
    if ((st = ctx_dev_scratch(ctx, blob.device_size(), &d)) != TK_OK) return st;
    if ((st = ctx_host_stage(ctx, std::max<size_t>(blob.size(), 1), &h)) != TK_OK) return st;
    blob.copy_to(h);
    if (!(blob.size() == 0)) CK(cudaMemcpyAsync(d, h, blob.size(), cudaMemcpyHostToDevice, s));
    *dev = static_cast<unsigned char*>(d);
    return TK_OK;
}

tk_status tk_block_gemm_f64(tk_ctx* ctx, const tk_bst* a_abi, const tk_bst* b_abi, tk_bst_out* out) {
    if (!ctx || !a_abi || !b_abi || !out) {
        set_error("tk_block_gemm_f64: null argument");
        return TK_ERR_INVALID_ARG;
    }
    std::memset(out, 0, sizeof(*out));
    std::string err;
    Rank2 A, B;
    if (!rank2_from_abi(*a_abi, A, "A", err) || !rank2_from_abi(*b_abi, B, "B", err)) {
        set_error("tk_block_gemm_f64: " + err);
        return TK_ERR_INVALID_ARG;
    }
    BlockGemmPlan P;
    tk_status st = guard_host("tk_block_gemm_f64", err, [&] { return block_gemm_plan(A, B, P, err); });
    if (st != TK_OK) {
        set_error("tk_block_gemm_f64: " + err);
        return st;
    }
    if ((st = fill_out_header(a_abi, b_abi, A, B, P, out, true)) != TK_OK) return st;
    if (P.total == 0) return TK_OK;
    Guard gd(ctx->device);
    // one host-to-device copy: A, B and the tables; C is written on the device
    // and read back through the same staging buffer
    Blob blob;
    const size_t oa = blob.add(A.data, sizeof(double) * (size_t)A.total);
    const size_t ob = blob.add(B.data, sizeof(double) * (size_t)B.total);
    const TableBlob tb = add_tables(blob, P.g);
    const size_t oc = blob.reserve(sizeof(double) * (size_t)P.total);
    auto run = [&]() -> tk_status {
        void* sp = nullptr;
        tk_status s2;
        if ((s2 = ctx_stream(ctx, &sp)) != TK_OK) return s2;
        cudaStream_t s = (cudaStream_t)sp;
        unsigned char* d = nullptr;
        if ((s2 = ctx_host_stage(ctx, sizeof(double) * (size_t)P.total, &sp)) != TK_OK) return s2;
        if ((s2 = stage_blob(ctx, blob, s, &d)) != TK_OK) return s2;
        CK(launch_gemm_f64((const GemmTile*)(d + tb.tiles), (int)P.g.tiles.size(), (const GemmTask*)(d + tb.tasks),
                           (const GemmSeg*)(d + tb.segs), (const double*)(d + oa), (const double*)(d + ob),
                           (double*)(d + oc), s));
        CK(cudaMemcpyAsync(ctx->host_stage, d + oc, sizeof(double) * (size_t)P.total, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        std::memcpy(out->data, ctx->host_stage, sizeof(double) * (size_t)P.total);
        return TK_OK;
    };
    st = run();
    if (st != TK_OK) tk_bst_free(out);
    return st;
}

tk_status tk_block_gemm_f64_dev(tk_ctx* ctx, const tk_bst* a_abi, const tk_bst* b_abi, tk_bst_out* out,
                                double* c_dev, void* stream) {
    if (!ctx || !a_abi || !b_abi || !out) {
        set_error("tk_block_gemm_f64_dev: null argument");
        return TK_ERR_INVALID_ARG;
    }
    std::memset(out, 0, sizeof(*out));
    std::string err;
    Rank2 A, B;
    if (!rank2_from_abi(*a_abi, A, "A", err) || !rank2_from_abi(*b_abi, B, "B", err)) {
        set_error("tk_block_gemm_f64_dev: " + err);
        return TK_ERR_INVALID_ARG;
    }
    BlockGemmPlan P;
    tk_status st = guard_host("tk_block_gemm_f64_dev", err, [&] { return block_gemm_plan(A, B, P, err); });
    if (st != TK_OK) {
        set_error("tk_block_gemm_f64_dev: " + err);
        return st;
    }
    if ((st = fill_out_header(a_abi, b_abi, A, B, P, out, false)) != TK_OK) return st;
    if (!c_dev || P.total == 0) return TK_OK;
    Guard gd(ctx->device);
    Blob blob;
    const TableBlob tb = add_tables(blob, P.g);
    cudaStream_t s = (cudaStream_t)stream;
    auto run = [&]() -> tk_status {
        unsigned char* d = nullptr;
        tk_status s2 = stage_blob(ctx, blob, s, &d);
        if (s2 != TK_OK) return s2;
        CK(launch_gemm_f64((const GemmTile*)(d + tb.tiles), (int)P.g.tiles.size(), (const GemmTask*)(d + tb.tasks),
                           (const GemmSeg*)(d + tb.segs), A.data, B.data, c_dev, s));
        // the tables live in the context's shared scratch: finish before returning
        CK(cudaStreamSynchronize(s));
        return TK_OK;
    };
    st = run();
    if (st != TK_OK) tk_bst_free(out);
    return st;
}

void tk_bst_free(tk_bst_out* t) {
    if (!t) return;
    std::free(t->keys);
    std::free(t->block_offsets);
    std::free(t->data);
    std::free(t->owned_charges);
    std::free(t->owned_dims);
    t->keys = nullptr;
    t->block_offsets = nullptr;
    t->data = nullptr;
    t->owned_charges = nullptr;
    t->owned_dims = nullptr;
    t->n_blocks = 0;
    t->total = 0;
}

tk_status tk_spmv_f64(tk_ctx* ctx, const tk_bst* a_abi, const double* x, double* y) {
    if (!a_abi || !x || !y) {
        set_error("tk_spmv_f64: null argument");
        return TK_ERR_INVALID_ARG;
    }
    std::string err;
    Rank2 A;
    if (!rank2_from_abi(*a_abi, A, "A", err)) {
        set_error("tk_spmv_f64: " + err);
        return TK_ERR_INVALID_ARG;
    }
    const int64_t rows = A.legs[0].total, cols = A.legs[1].total;
    // One task per row sector (faer.rs:336-388: y zeroed, each block adds
    // its product into its row range); blocks of one row sector are K segments.
    GemmTable g;
    std::map<int, std::vector<int>> by_row;
    for (size_t b = 0; b < A.keys.size(); ++b) by_row[A.rs[b]].push_back((int)b);
    std::vector<char> covered((size_t)A.legs[0].n(), 0);
    for (auto& kv : by_row) {
        int r = kv.first;
        covered[r] = 1;
        GemmTask t{};
        t.M = (int32_t)A.legs[0].dim[r]; t.N = 1;
        t.c_off = A.legs[0].off[r]; t.c_rs = 1; t.c_cs = 1;
        t.alpha = 1.0; t.beta = 0.0;
        t.seg_begin = (int)g.segs.size();
        for (int b : kv.second) {
            int c = A.cs[b];
            GemmSeg s{};
            s.a_off = A.offs[b]; s.a_rs = (int32_t)A.legs[1].dim[c]; s.a_cs = 1;
            s.b_off = A.legs[1].off[c]; s.b_rs = 1; s.b_cs = 1;
            s.K = (int32_t)A.legs[1].dim[c];
            g.segs.push_back(s);
        }
        t.seg_end = (int)g.segs.size();
        g.tasks.push_back(t);
        gemm_add_tiles(g, (int)g.tasks.size() - 1);
    }
    // Row sectors without blocks are zero.
    for (int r = 0; r < A.legs[0].n(); ++r) {
        if (covered[r]) continue;
        GemmTask t{};
        t.M = (int32_t)A.legs[0].dim[r]; t.N = 1;
        t.c_off = A.legs[0].off[r]; t.c_rs = 1; t.c_cs = 1;
        t.alpha = 1.0; t.beta = 0.0;
        t.seg_begin = t.seg_end = (int)g.segs.size();
        g.tasks.push_back(t);
        gemm_add_tiles(g, (int)g.tasks.size() - 1);
    }
    if (rows == 0) return TK_OK;
    int dev = ctx ? ctx->device : 0;
    Guard gd(dev);
    Scratch sc;
    double *da, *dx, *dy;
    GemmTask* dt; GemmSeg* ds; GemmTile* dl;
    std::vector<double> ha(A.data, A.data + A.total), hx(x, x + cols);
    CK(sc.put(ha, &da));
    CK(sc.put(hx, &dx));
    CK(sc.make((size_t)rows, &dy));
    CK(sc.put(g.tasks, &dt));
    CK(sc.put(g.segs, &ds));
    CK(sc.put(g.tiles, &dl));
    CK(launch_gemm_f64(dl, (int)g.tiles.size(), dt, ds, da, dx, dy, nullptr));
    CK(cudaMemcpy(y, dy, sizeof(double) * (size_t)rows, cudaMemcpyDeviceToHost));
    return TK_OK;
}

}  // extern "C"
