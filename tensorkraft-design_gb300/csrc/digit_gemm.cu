// digit_gemm.cu -- FP64 products on the fp16 tensor cores.
//
// This GPU does 1.2 TFLOP/s in FP64 and 1.9 PFLOP/s in fp16, so an FP64
// product is cheaper as 28 exact fp16 ones.  The error-free splitting is the
// published one of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59, 2012):
// every operand row becomes seven integer digits (digit_gemm.cuh), and
//   sum_k x_k y_k = 2^(ea + eb - 66) sum_s 2^(8 (6 - s)) v_s,
//   v_s = sum over i + j = s <= 6 of sum_k d_i d'_j.
// Every v_s is an integer below 2^24 over 64 k (level s holds two products
// with a leading digit, at most 2^16 each, and s - 1 of at most 2^14; level 0
// one of 2^18), so fp32 accumulation is exact; after 64 k the seven sums are
// added to an integer sum per output, and the result is rounded to FP64
// once.  Left out are, of an element, what lies below half a unit of its row's
// grid, 2^(e - 58) (nothing for the elements within five binary orders of the
// row's largest), and the levels 7 and up, at most 6.03 x 2^-60 2^(ea + eb) a k.
// So an output's error goes by the largest elements of its row and column: by
// norm it is smaller than that of an FP64 chain, but an output that is small
// because its row and column are large at different k has fewer right digits.
// Dense products are checked output by output (digit_gate_kernel); the matvec
// scales its operands' k so that its result is held by norm (stack_f64.cu).
//
// The kernel is persistent and warp-specialised, one CTA per SM: one thread
// moves operands by TMA (32 k of all digits of 128 + 64 rows: 84 KB, a ring of
// two), one warp issues tcgen05.mma, sixteen warps drain the accumulators.  The
// digits of 32 B rows lie one after the other in shared memory and the levels
// 32 columns apart in TMEM, so digit i of A meets digits 0 .. 6 - i of B in
// ONE instruction (N = 32 (7 - i)) that lands on levels i .. 6: seven
// instructions per 16 k, and A is read once for each.  A tile's two column
// halves have accumulators of their own (2 x 224 columns): one is drained
// while the other is summed.
//
// Measured (2048^3, N(0, 1) operands): product 0.40 ms (1.2 PFLOP/s of fp16,
// 0.63 of the measured peak), the call 0.52 ms, against 14.6 ms for the FP64
// kernel, whose pipe is at its limit; relative error 4.9e-17 against 5.8e-16
// at K = 300.  The 28 instructions of a stage take 1935 clocks alone (1792
// ideal) and 2790 here; leaving the loads out changes nothing, leaving the
// drains out 50 us: what bounds it is the waits, two or three instructions
// deep in the tensor cores' queue, for stages and drained accumulators.
#include "digit_gemm.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

#include "tk_plan.cuh"

namespace tk {
namespace {

constexpr int KW = 32;                                // K of one ring stage
constexpr int HN = 32;                                // columns of a tile half
constexpr int A_BYTES = kDigits * kTcBM * KW * 2;     // 57344
constexpr int H_BYTES = kDigits * HN * KW * 2;        // 14336
constexpr int STAGE_BYTES = A_BYTES + 2 * H_BYTES;    // 86016
constexpr int EPI_WARPS = 16;
constexpr int WCOLS = 16;                             // columns a drain warp holds: half a tile half
constexpr int NTHREADS = 32 * (EPI_WARPS + 2);
constexpr int SCOLS = 8;                              // columns staged at a time for the stores
constexpr int ST_LD = SCOLS + 1;
constexpr int STORE_BYTES = 32 * ST_LD * 8;           // per drain warp
constexpr int TILE_CACHE = 64;                        // tiles of a CTA kept in shared memory
constexpr int SMEM_BYTES = 1024 + kDigitRing * STAGE_BYTES + EPI_WARPS * STORE_BYTES + TILE_CACHE * (int)sizeof(TcTile) + 256;
static_assert(sizeof(TcTile) % 8 == 0 && SMEM_BYTES <= 227 * 1024, "tiles are copied as 8-byte words");
constexpr int TMEM_ALLOC = 512, TMEM_HALF = 256;
constexpr long WAIT_LIMIT = 1L << 24;

constexpr int kExBias = 2110;  // 2 * 1022 + 114 - 48: V * 2^(exa + exb - kExBias)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// mbar_test without its suspension: 60 clocks less where nothing is to be waited for.
__device__ __forceinline__ bool mbar_done(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Once one wait of the CTA has run out (*stop), every later one
// returns at once, so that all roles leave together.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* stop, int* redo) {
    for (long i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_test(b, parity)) return true;
        if (*stop) return false;
    }
    *stop = 1;
    atomicExch(redo, kDigitWait);
    return false;
}
// Bounded wait for work already issued, whatever else went wrong.
__device__ __forceinline__ void mbar_drain(uint64_t* b, uint32_t parity) {
    for (long i = 0; i < WAIT_LIMIT; ++i)
        if (mbar_test(b, parity)) return;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(0), "r"(smem_u32(bar))
        : "memory");
}
// K-major rows of 64 bytes, 64-byte swizzle, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512u >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
// kind::f16: fp32 accumulate, fp16 A and B, both K-major, M = 128.
__device__ __forceinline__ uint32_t idesc_f16(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTcBM >> 4) << 24);
}
// Called by a whole warp with the same arguments; one lane issues.  (Under a
// branch on the lane the operands would be moved to uniform registers one by
// one for each instruction, which takes longer than the instruction.)
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld4(uint32_t t, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(t));
}

// One output's sum: s 2^24 + l, in units of 2^8 of level 6.
struct Sum {
    int64_t s;
    int32_t l;
    // += the seven level sums of 64 k.  An int32 conversion runs at a sixteenth
    // of the rate of an fp32 operation here, so levels 3 and 4 first hand
    // their upper parts to the level above (adding 1.5 * 2^23 leaves a rounded
    // integer in the low mantissa bits; every step is exact) and four
    // conversions are left.  The last one rounds at 2^-58 of row maximum times
    // column maximum.
    __device__ __forceinline__ void add(float v0, float v1, float v2, float v3, float v4, float v5, float v6) {
        const float M = 12582912.0f;
        const float h4 = fmaf(v4, 0x1p-8f, M) - M;
        const float l4 = fmaf(h4, -256.0f, v4);
        const float w3 = v3 + h4;
        const float h3 = fmaf(w3, 0x1p-8f, M) - M;
        const float l3 = fmaf(h3, -256.0f, w3);
        l += __float2int_rn(fmaf(l3, 65536.0f, fmaf(l4, 256.0f, fmaf(v6, 0x1p-8f, v5))));
        mad(__float2int_rz(v2 + h3), 1);
        mad(__float2int_rz(v1), 256);
        mad(__float2int_rz(v0), 65536);
    }
    // s += a * b as one wide multiply-add (a shift and a 64-bit addition take four instructions)
    __device__ __forceinline__ void mad(int a, int b) { asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s) : "r"(a), "r"(b)); }
    __device__ __forceinline__ void carry() {  // l back to 24 bits
        s += l >> 24;
        l &= 0xFFFFFF;
    }
    // (s 2^24 + l) 2^-u with m = 2^(24 - u)
    __device__ __forceinline__ int64_t whole(uint32_t m, int u) const {
        int64_t r = l >> u;
        asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(r) : "r"((uint32_t)s), "r"(m));
        return r + ((int64_t)(uint64_t)((uint32_t)((uint64_t)s >> 32) * m) << 32);
    }
};
constexpr int kCarryChunks = 64;  // chunks after which l is near its range

// x * 2^(e - kExpo) rounded to nearest, on the integer pipes (the FP64 pipe does
// two operations a clock).  Free of branches, so that the columns of a row
// overlap; *off is set where |x| < 2^32, which to_double_slow computes, as it
// does where a tile's exponents come near the ends of the range (to_double
// itself checks none).
constexpr int kExpo = 1084;
constexpr int kExpLow = 40, kExpHigh = 2040;  // for e in between it holds whatever x is
__device__ __forceinline__ double to_double(int64_t x, int e, uint32_t* off) {
    const int32_t neg = (int32_t)((uint64_t)x >> 32) >> 31;
    const uint64_t u = (uint64_t)((x ^ (int64_t)neg) - (int64_t)neg);
    const uint32_t h = (uint32_t)(u >> 32), l = (uint32_t)u;
    // the leading bit to bit 62, so that rounding at bit 10 cannot carry out
    const int z = __clz(h) - 1;
    uint64_t q = ((uint64_t)__funnelshift_l(l, h, z) << 32) | (l << (z & 31));
    q = (q + 0x200u) >> 10;
    const bool zero = h == 0;
    *off |= zero ? l : 0u;
    const uint32_t rh = ((uint32_t)(q >> 32) + ((uint32_t)(e - z) << 20)) | ((uint32_t)neg & 0x80000000u);
    return zero ? 0.0 : __hiloint2double((int)rh, (int)(uint32_t)q);
}
__device__ __noinline__ double to_double_slow(int64_t x, int e) {
    int t = e - kExpo;
    uint64_t u = x < 0 ? 0 - (uint64_t)x : (uint64_t)x;
    if (u == 0) return 0.0;
    // drop the bits below the result's last place, 2^-1074 at the least
    const int drop = max(11 - __clzll((long long)u), -1074 - t);
    if (drop > 0) {
        const int d = min(drop, 63);
        const uint64_t half = 1ull << (d - 1), rest = u & ((1ull << d) - 1);
        u = drop > 64 ? 0 : (u >> d) + (rest >= half);  // ties away from zero, as in to_double
        t += drop;
    }
    const double r = u == 0 ? 0.0 : t > 1000 ? INFINITY : ldexp((double)(long long)u, t);
    return x < 0 ? -r : r;
}

// Tile ti of a launch: from the table, or (mode 0) of the C grid, columns first.
template <int MODE>
__device__ __forceinline__ TcTile tile_of(const TcTile* __restrict__ tiles, const DigitOut& om, int ti) {
    if (MODE != 0) return tiles[ti];
    TcTile t;
    const int ntn = (om.n + kTcBN - 1) / kTcBN, m0 = ti / ntn * kTcBM, n0 = ti % ntn * kTcBN;
    t.a_row = t.ldc = m0;
    t.a_cs = om.m;
    t.b_row = t.n0 = n0;
    t.b_cs = om.n;
    t.k_valid = om.k;
    t.parts = 1;
    t.m_valid = min(kTcBM, om.m - m0);
    t.n_valid = min(kTcBN, om.n - n0);
    return t;
}

// The K of a tile: `parts` operands' K one after the other (two for complex
// products), each from a chunk of its own; ring steps of KW, drained after at
// most 64 k.
struct KSteps {
    int parts, per, kch;  // ring steps and chunks a part
    bool paired;          // two parts of one step each are drained together
    __device__ __forceinline__ KSteps(const TcTile& t)
        : parts(max(t.parts, 1)), per((t.k_valid + KW - 1) / KW), kch((t.k_valid + kTcBK - 1) / kTcBK), paired(per == 1) {}
    __device__ __forceinline__ int drains() const { return paired ? (parts + 1) >> 1 : parts * kch; }
    // whether step q of part p is the first, the last one between two drains
    __device__ __forceinline__ bool first(int p, int q) const { return ((paired ? p : q) & 1) == 0; }
    __device__ __forceinline__ bool last(int p, int q) const {
        return paired ? (p & 1) || p == parts - 1 : (q & 1) || q == per - 1;
    }
};

template <int MODE>
__global__ void __launch_bounds__(NTHREADS, 1) digit_gemm_kernel(const TcTile* __restrict__ tiles,
                                                                 const int32_t* __restrict__ begin,
                                                                 const __grid_constant__ DigitMaps maps,
                                                                 const int32_t* __restrict__ exa,
                                                                 const int32_t* __restrict__ exb, const DigitOut om,
                                                                 int* redo) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    double* store = (double*)(smem + kDigitRing * STAGE_BYTES);
    TcTile* cache = (TcTile*)(smem + kDigitRing * STAGE_BYTES + EPI_WARPS * STORE_BYTES);
    uint64_t* full = (uint64_t*)(cache + TILE_CACHE);
    uint64_t* empty = full + kDigitRing;
    uint64_t* acc_full = empty + kDigitRing;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* done = acc_empty + 2;
    uint32_t* tslot = (uint32_t*)(done + 1);
    volatile int* stop = (volatile int*)(tslot + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    dep_launch();
    if (threadIdx.x == 0) {
        for (int i = 0; i < kDigitRing; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], EPI_WARPS / 2);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPI_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(TMEM_ALLOC)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // this CTA's tiles: a run of the table, or every gridDim.x-th of the C grid.
    // Its first tiles are copied (the table is the plan's, no kernel writes it):
    // each role then starts a tile without waiting for its descriptor.
    const int t_begin = MODE == 0 ? (int)blockIdx.x : begin[blockIdx.x];
    const int t_end = MODE == 0 ? om.tiles : begin[blockIdx.x + 1];
    const int t_step = MODE == 0 ? (int)gridDim.x : 1;
    if (MODE != 0) {
        const int n = min(t_end - t_begin, TILE_CACHE) * (int)(sizeof(TcTile) / 8);
        for (int i = threadIdx.x; i < n; i += NTHREADS)
            reinterpret_cast<uint64_t*>(cache)[i] = reinterpret_cast<const uint64_t*>(tiles + t_begin)[i];
    }
    auto tile_at = [&](int ti) {
        return MODE != 0 && ti - t_begin < TILE_CACHE ? cache[ti - t_begin] : tile_of<MODE>(tiles, om, ti);
    };
    dep_wait();
    if (threadIdx.x == 0) *stop = *(volatile int*)redo;  // an operand held an infinity or a NaN: another kernel computes this product
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    const bool run = *stop == 0;  // written before the barrier; a wait can only run out after it
    __syncthreads();
    if (warp == EPI_WARPS) {
        if (lane == 0) {
            int it = 0;
            bool ok = run;
            for (int ti = t_begin; ti < t_end && ok; ti += t_step) {
                const TcTile t = tile_at(ti);
                const int halves = t.n_valid > HN ? 2 : 1;
                const int box = (t.m_valid + 31) >> 5;
                const uint32_t bytes = kDigits * KW * 2 * (32 * box + HN * halves);
                const KSteps ks(t);
                for (int part = 0; part < ks.parts && ok; ++part)
                for (int q = 0; q < ks.per && ok; ++q, ++it) {
                    const int st = it % kDigitRing;
                    uint8_t* base = smem + st * STAGE_BYTES;
                    if (it >= kDigitRing) ok = mbar_wait(&empty[st], (it / kDigitRing - 1) & 1, stop, redo);
                    if (!ok) break;
                    mbar_expect_tx(&full[st], bytes);
                    const int x = (q & 1) * KW, c = part * ks.kch + (q >> 1);
                    tma_load_3d(base, &maps.a[box - 1], x, t.a_row + c * t.a_cs, &full[st]);
                    for (int h = 0; h < halves; ++h)
                        tma_load_3d(base + A_BYTES + h * H_BYTES, &maps.b, x, t.b_row + c * t.b_cs + HN * h, &full[st]);
                }
            }
            // the loads in flight land before the CTA's shared memory goes
            for (int i = max(0, it - kDigitRing); i < it; ++i) mbar_drain(&full[i % kDigitRing], (i / kDigitRing) & 1);
        }
    } else if (warp == EPI_WARPS + 1) {
        int it = 0, unit = 0;
        uint32_t drained = 0, phase = 0;  // per accumulator: whether it was summed before, the parity to wait for
        bool ok = run;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            return __all_sync(0xffffffffu, mbar_done(bar, parity)) ||
                   __all_sync(0xffffffffu, mbar_wait(bar, parity, stop, redo));
        };
        for (int ti = t_begin; ti < t_end && ok; ti += t_step) {
            const TcTile t = tile_at(ti);
            const int halves = t.n_valid > HN ? 2 : 1;
            const uint32_t astep = (uint32_t)((((t.m_valid + 31) >> 5) * 32) * KW * 2) >> 4;
            const KSteps k(t);
            for (int part = 0; part < k.parts && ok; ++part)
            for (int q = 0; q < k.per && ok; ++q, ++it) {
                const int st = it % kDigitRing;
                const bool first = k.first(part, q), last = k.last(part, q);
                ok = wait(&full[st], (it / kDigitRing) & 1);
                const uint32_t sa = smem_u32(smem + st * STAGE_BYTES);
                const uint64_t a0 = sw64_desc(sa);
                const bool both = t.k_valid - q * KW > 16;  // 16-k steps of this stage
                for (int h = 0; h < halves && ok; ++h) {
                    const int buf = (unit + h) & 1;
                    if (first && ((drained >> buf) & 1)) {
                        ok = wait(&acc_empty[buf], (phase >> buf) & 1);
                        phase ^= 1u << buf;
                    }
                    if (!ok) break;
                    fence_after();
                    const uint64_t b0 = sw64_desc(sa + A_BYTES + h * H_BYTES);
                    const uint32_t d0 = tmem + buf * TMEM_HALF;
                    // the second step goes backwards, so that wide instructions are the
                    // ones in the queue (two or three deep) during the next wait
#pragma unroll
                    for (int kk = 0; kk < KW / 16; ++kk) {
                        if (kk > 0 && !both) break;
#pragma unroll
                        for (int j = 0; j < kDigits; ++j) {
                            const int i = kk == 0 ? j : kDigits - 1 - j;
                            mma_f16(d0 + i * HN, a0 + i * astep + kk * 2, b0 + kk * 2, idesc_f16((kDigits - i) * HN),
                                    i > 0 || kk > 0 || !first);
                        }
                    }
                    if (last) {
                        mma_commit(&acc_full[buf]);
                        drained |= 1u << buf;
                    }
                }
                mma_commit(&empty[st]);
            }
            unit += halves;
        }
        // no instruction is in flight when the accumulators are given back
        mma_commit(done);
        mbar_drain(done, 0);
    } else {
        // warps 0-7 drain accumulator 0, warps 8-15 accumulator 1; warp % 4 is
        // the TMEM lane quarter, (warp / 4) % 2 the 16 of the half's 32 columns:
        // a thread holds one row of 16 columns
        const int buf = warp >> 3, row0 = (warp & 3) * 32, col0 = ((warp >> 2) & 1) * WCOLS;
        const uint32_t tbase = tmem + buf * TMEM_HALF + col0 + ((uint32_t)row0 << 16);
        double* sw = store + warp * (STORE_BYTES / 8);
        int drains = 0, unit = 0;
        bool ok = run;
        for (int ti = t_begin; ti < t_end && ok; ti += t_step) {
            const TcTile t = tile_at(ti);
            const int halves = t.n_valid > HN ? 2 : 1;
            const int h = (buf - unit) & 1;
            unit += halves;
            if (h >= halves) continue;
            const int nc = min(WCOLS, t.n_valid - h * HN - col0);  // columns of this warp's that the tile has
            const bool mine = row0 < t.m_valid && nc > 0;
            // what the stores will need, on its way while the sums are drained:
            // exponents (a row of this thread, a column per lane), output offsets
            const int cl = lane & (SCOLS - 1), r0 = lane / SCOLS;
            int ea = 1, eb = 1;
            int64_t place[WCOLS / SCOLS] = {}, rows = 0;
            int32_t pitch[WCOLS / SCOLS] = {};
            if (mine) {
                if (row0 + lane < t.m_valid) {
                    ea = exa[t.a_row + row0 + lane];
                    if (MODE == 1) rows = om.rowtab[t.out_off + row0 + lane];
                }
                eb = exb[t.b_row + h * HN + col0 + min(lane, nc - 1)];  // (a column past the tile's takes the last one's)
                if (MODE == 2)
#pragma unroll
                    for (int g = 0; g < WCOLS / SCOLS; ++g)
                        if (g * SCOLS + cl < nc) {
                            place[g] = om.colbase[t.out_off + h * HN + col0 + g * SCOLS + cl];
                            pitch[g] = om.colstride[t.out_off + h * HN + col0 + g * SCOLS + cl];
                        }
            }
            Sum acc[WCOLS];
#pragma unroll
            for (int i = 0; i < WCOLS; ++i) acc[i] = {0, 0};
            const int chunks = KSteps(t).drains();
            for (int c = 0; c < chunks && ok; ++c) {
                ok = mbar_wait(&acc_full[buf], drains & 1, stop, redo);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                ++drains;
                fence_after();
                if (mine) {
#pragma unroll
                    for (int g = 0; g < WCOLS / 4; ++g) {
                        uint32_t v[kDigits][4];
#pragma unroll
                        for (int s = 0; s < kDigits; ++s) tmem_ld4(tbase + s * HN + g * 4, v[s]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            auto f = [&](int s) { return __uint_as_float(v[s][i]); };
                            acc[g * 4 + i].add(f(0), f(1), f(2), f(3), f(4), f(5), f(6));
                        }
                    }
                    if (c % kCarryChunks == kCarryChunks - 1) {
#pragma unroll
                        for (int i = 0; i < WCOLS; ++i) acc[i].carry();
                    }
                }
                fence_before();
                if (lane == 0) mbar_arrive(&acc_empty[buf]);
            }
            if (!ok || !mine) continue;
            // s 2^24 + l in 64 bits, for the whole row less the u low bits that the
            // row's largest sum leaves no room for (it then has 62 of its own); of the
            // tile's columns only: the others' operand rows belong to other tiles or to
            // nobody, and must not decide how these are rounded
            uint32_t bits = 0;
#pragma unroll
            for (int i = 0; i < WCOLS; ++i) {
                const int32_t hi = (int32_t)(acc[i].s >> 32);
                if (i < nc) bits |= (uint32_t)(hi ^ (hi >> 31));
            }
            const int u = max(0, 26 - __clz((int)bits));
            const uint32_t um = 1u << (24 - u);
            ea += u + 8 - kExBias + kExpo;
            const int eb_lo = __reduce_min_sync(0xffffffffu, eb), eb_hi = __reduce_max_sync(0xffffffffu, eb);
            const bool inside = ea + eb_lo >= kExpLow && ea + eb_hi <= kExpHigh;
            // eight columns at a time through shared memory: consecutive lanes
            // store consecutive columns
#pragma unroll
            for (int g = 0; g < WCOLS / SCOLS; ++g) {
                if (g * SCOLS >= nc) break;
                uint32_t off = inside ? 0u : 1u;
                __syncwarp();
#pragma unroll
                for (int i = 0; i < SCOLS; ++i)
                    sw[lane * ST_LD + i] =
                        to_double(acc[g * SCOLS + i].whole(um, u), ea + __shfl_sync(0xffffffffu, eb, g * SCOLS + i), &off);
                if (__any_sync(0xffffffffu, off != 0 && row0 + lane < t.m_valid)) {
#pragma unroll
                    for (int i = 0; i < SCOLS; ++i)
                        sw[lane * ST_LD + i] =
                            to_double_slow(acc[g * SCOLS + i].whole(um, u), ea + __shfl_sync(0xffffffffu, eb, g * SCOLS + i));
                }
                __syncwarp();
                const int col = h * HN + col0 + g * SCOLS + cl;
                if (MODE != 1 && g * SCOLS + cl >= nc) continue;
                double* o;
                int64_t step = 0;
                if (MODE == 2) {
                    step = pitch[g];
                    o = om.out + place[g] + (int64_t)(t.ldc + row0 + r0) * step;
                } else if (MODE == 1) {
                    // columns from `split` on are the imaginary part's
                    const int at = t.n0 + col;
                    o = t.split > 0 && at >= t.split ? om.out_im + (at - t.split) : om.out + at;
                } else {
                    step = om.c_rs;
                    o = om.out + (int64_t)(t.n0 + col) * om.c_cs + (int64_t)(t.ldc + row0 + r0) * step;
                }
                step *= 32 / SCOLS;
                const int last = t.m_valid - row0 - r0;  // rows of this lane's are 4 v < last
                if (MODE == 0 && (om.alpha != 1.0 || om.beta != 0.0)) {
                    for (int v = 0; v < SCOLS && v * (32 / SCOLS) < last; ++v, o += step) {
                        double x = om.alpha * sw[(v * (32 / SCOLS) + r0) * ST_LD + cl];
                        if (om.beta != 0.0) x += om.beta * *o;
                        *o = x;
                    }
                } else if (MODE == 1) {
#pragma unroll
                    for (int v = 0; v < SCOLS; ++v) {
                        const int64_t row = __shfl_sync(0xffffffffu, rows, v * (32 / SCOLS) + r0);
                        if (v * (32 / SCOLS) < last && g * SCOLS + cl < nc) o[row] = sw[(v * (32 / SCOLS) + r0) * ST_LD + cl];
                    }
                } else {
#pragma unroll
                    for (int v = 0; v < SCOLS; ++v, o += step) {
                        if (v * (32 / SCOLS) >= last) break;
                        *o = sw[(v * (32 / SCOLS) + r0) * ST_LD + cl];
                    }
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == EPI_WARPS) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_ALLOC) : "memory");
    }
}

// ---------------------------------------------------------------- digits

__device__ __forceinline__ uint32_t abs_hi(double x) { return (uint32_t)__double2hiint(x) & 0x7FFFFFFFu; }
// The high word of |x|, 1 for what has none of its own: zero only for zero.
__device__ __forceinline__ uint32_t abs_top(double x) {
    const uint32_t hi = abs_hi(x);
    return hi == 0 && __double2loint(x) != 0 ? 1u : hi;
}
// Biased exponent of a row whose largest element has these high bits (below 1
// for a row of subnormals).
__device__ __forceinline__ int row_exponent(uint32_t max_hi, int* redo) {
    const int e = (int)(max_hi >> 20);
    if (e == 2047) atomicExch(redo, kDigitValue);
    return e > 0 ? e : 12 - __clz((int)(max_hi | 1));
}
// x 2^k on its row's grid, rounded to nearest, plus 128 in each of the six
// low bytes: byte j is then digit 6 - j plus 128, the upper 16 bits digit 0.
__device__ __noinline__ uint64_t shifted_up(uint64_t m, int n) { return n > 63 ? 0 : m << n; }
__device__ __forceinline__ uint64_t on_grid(double x, int ex, int k = 0) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int e = (int)(b >> 52) & 0x7FF;
    uint64_t m = (b & 0xFFFFFFFFFFFFFull) << 5;  // one bit more than the grid has, for the rounding
    if (e) m |= 1ull << 57;
    const int s = min(ex - max(e, 1) - k, 63);
    if (__builtin_expect(s < 0, 0))  // (rows of subnormals or zeros alone)
        m = shifted_up(m, -s);
    else
        m >>= s;
    m = (m + 1) >> 1;
    const uint64_t neg = (uint64_t)((int64_t)b >> 63);
    return (m ^ neg) - neg + 0x0000808080808080ull;
}
// The digits of two neighbouring elements, as pairs of fp16.
__device__ __forceinline__ void digits2(double x, double y, int ex, uint32_t* d, int kx = 0, int ky = 0) {
    const uint64_t a = on_grid(x, ex, kx), b = on_grid(y, ex, ky);
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
    // 0x6400 | n is fp16 1024 + n
    auto half_of = [](uint32_t v, uint32_t bias) {
        const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&bias));
        return *reinterpret_cast<const uint32_t*>(&h);
    };
    auto bytes = [&](uint32_t u, uint32_t v, uint32_t sel) {
        return half_of((__byte_perm(u, v, sel) & 0x00FF00FFu) | 0x64006400u, 0x64806480u);  // minus 1152
    };
    d[6] = bytes(al, bl, 0x4400);
    d[5] = bytes(al, bl, 0x5511);
    d[4] = bytes(al, bl, 0x6622);
    d[3] = bytes(al, bl, 0x7733);
    d[2] = bytes(ah, bh, 0x4400);
    d[1] = bytes(ah, bh, 0x5511);
    const uint32_t top = ((uint32_t)((int)ah >> 16) + 512u) | (((uint32_t)((int)bh >> 16) + 512u) << 16);
    d[0] = half_of(top + 0x64006400u, 0x66006600u);  // minus 1536
}
__device__ __forceinline__ void put_digits(const DigitStack& o, int64_t row, int k, const uint32_t* d) {
    uint32_t* p = reinterpret_cast<uint32_t*>(o.q) + row * (kDigits * kTcBK / 2) + (k >> 1);
#pragma unroll
    for (int j = 0; j < kDigits; ++j) p[j * (kTcBK / 2)] = d[j];
}

// A complex operand's digits d + i f at chunk offsets c0 (first part) and c1.
template <bool DUAL>
__device__ __forceinline__ void put_complex(const DigitStack& o, int64_t row, int n_dual, int64_t c0, int64_t c1, int k,
                                            const uint32_t* d, const uint32_t* f) {
    put_digits(o, row + c0, k, d);
    if (!DUAL) {
        put_digits(o, row + c1, k, f);
        return;
    }
    put_digits(o, row + n_dual + c0, k, f);
    put_digits(o, row + n_dual + c1, k, d);
    uint32_t m[kDigits];
#pragma unroll
    for (int j = 0; j < kDigits; ++j) m[j] = f[j] ^ 0x80008000u;
    put_digits(o, row + c1, k, m);
}

// Exponent of x 2^k (below 1 for subnormals), kNoExponent for zero.
constexpr int kNoExponent = -(1 << 20);
__device__ __forceinline__ int exponent_of(double x, int k) {
    const uint32_t hi = abs_hi(x);
    const int e = (int)(hi >> 20);
    const bool zero = (hi | (uint32_t)__double2loint(x)) == 0;
    return zero ? kNoExponent : (e > 0 ? e : 12 - __clz((int)(hi | 1))) + k;
}

// A row's exponent; one with nothing but dead columns counts as zeros.
__device__ __forceinline__ int scaled_row_exponent(int mx) { return mx < kDeadColumn / 2 ? 1 : mx; }

// One CTA per 64-wide chunk of a stack (blockIdx.y, past the stack's last: nothing): the columns' exponents,
// sixteen rows at a time (a cylinder's L stack has thousands: with four, its plan took 0.4 ms more of 39).
constexpr int kColumnRows = 16;
__global__ void __launch_bounds__(kColumnRows * kTcBK) digit_columns_kernel(const DigitRows* __restrict__ jobs,
                                                                         const double* __restrict__ q64,
                                                                         const double* __restrict__ q64_im,
                                                                         const int32_t* __restrict__ ex,
                                                                         int32_t* __restrict__ kx) {
    __shared__ int top[kColumnRows][kTcBK];
    const DigitRows j = jobs[blockIdx.x];
    const int k = threadIdx.x & 63, w = threadIdx.x >> 6, c = blockIdx.y;
    if (c >= j.kch) return;
    int mx = kNoExponent;
#pragma unroll 4
    for (int r = w; r < j.n; r += kColumnRows) {
        const int64_t at = (((int64_t)j.row + (int64_t)c * j.cs + r) << 6) + k;
        const int unit = ex ? ex[j.ex0 + r] : 1023;
        if (unit == kNoGain) continue;
        mx = max(mx, exponent_of(q64[at], -unit));
        if (q64_im) mx = max(mx, exponent_of(q64_im[at], -unit));
    }
    top[w][k] = mx;
    __syncthreads();
    if (w != 0) return;
    for (int i = 1; i < kColumnRows; ++i) mx = max(mx, top[i][k]);
    kx[j.kx + c * kTcBK + k] = mx == kNoExponent ? kDeadColumn : mx;
}

// One warp per row of an FP64 stack (K-major 64-wide chunks): the row's
// largest exponent, then its digits; the first kKeep chunks stay in registers
// in between, the others are read again (from L1 or L2).
constexpr int kKeep = 3;
__global__ void __launch_bounds__(32 * kDigitRowsPerCta) digit_rows_kernel(const DigitRows* __restrict__ jobs,
                                                                           const double* __restrict__ q64,
                                                                           const int32_t* __restrict__ kx, int sign,
                                                                           const DigitStack out, int* redo) {
    const DigitRows j = jobs[blockIdx.x];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    dep_launch();
    if (w >= j.n) return;
    dep_wait();
    const int64_t row = (int64_t)j.row + w;
    auto at = [&](int c) { return reinterpret_cast<const double2*>(q64 + ((row + (int64_t)c * j.cs) << 6))[lane]; };
    auto scale = [&](int c) {
        if (j.kx < 0) return make_int2(0, 0);
        const int2 k = reinterpret_cast<const int2*>(kx + j.kx + c * kTcBK)[lane];
        return make_int2(sign * k.x, sign * k.y);
    };
    double2 v[kKeep];
    int mx = kNoExponent;
    uint32_t hi = 0, tiny = 0;  // tiny: whether there are subnormals
    auto top1 = [&](double x, int k) {
        const uint32_t h = abs_hi(x);
        const int e = (int)(h >> 20);
        hi = max(hi, h);
        tiny |= e > 0 ? 0u : h | (uint32_t)__double2loint(x);
        mx = max(mx, e > 0 ? e + k : kNoExponent);
    };
    auto top = [&](const double2& u, const int2& k) {
        top1(u.x, k.x);
        top1(u.y, k.y);
    };
#pragma unroll
    for (int c = 0; c < kKeep; ++c)
        if (c < j.kch) {
            v[c] = at(c);
            top(v[c], scale(c));
        }
#pragma unroll 4
    for (int c = kKeep; c < j.kch; ++c) top(at(c), scale(c));
    if (__any_sync(0xffffffffu, tiny != 0)) {
        for (int c = 0; c < j.kch; ++c) {
            const double2 u = at(c);
            const int2 k = scale(c);
            mx = max(mx, max(exponent_of(u.x, k.x), exponent_of(u.y, k.y)));
        }
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (hi >= 0x7FF00000u) atomicExch(redo, kDigitValue);
    const int ex = scaled_row_exponent(mx);
    if (lane == 0) out.ex[row] = ex;
    auto put = [&](int c, const double2& u) {
        const int2 k = scale(c);
        uint32_t d[kDigits];
        digits2(u.x, u.y, ex, d, k.x, k.y);
        put_digits(out, row + (int64_t)c * j.cs, 2 * lane, d);
    };
#pragma unroll
    for (int c = 0; c < kKeep; ++c)
        if (c < j.kch) put(c, v[c]);
#pragma unroll 2
    for (int c = kKeep; c < j.kch; ++c) put(c, at(c));
}

// The same for a complex operand (planar): the row's two parts on one grid, the
// real part's chunks first, out row `to` + r (chunks `cs_out` apart).  DUAL (the
// B operand of a product): row r holds (re | -im), row r + n_dual (im | re).
template <bool DUAL>
__global__ void __launch_bounds__(32 * kDigitRowsPerCta) digit_rows_complex_kernel(const DigitRowsC* __restrict__ jobs,
                                                                                   const double* __restrict__ re,
                                                                                   const double* __restrict__ im,
                                                                                   const int32_t* __restrict__ kx,
                                                                                   int sign, const DigitStack out,
                                                                                   int* redo) {
    const DigitRowsC j = jobs[blockIdx.x];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    dep_launch();
    if (w >= j.n) return;
    dep_wait();
    const int64_t row = (int64_t)j.row + w, to = (int64_t)j.to + w;
    auto at = [&](const double* q, int c) {
        return reinterpret_cast<const double2*>(q + ((row + (int64_t)c * j.cs) << 6))[lane];
    };
    auto scale = [&](int c) {
        if (j.kx < 0) return make_int2(0, 0);
        const int2 k = reinterpret_cast<const int2*>(kx + j.kx + c * kTcBK)[lane];
        return make_int2(sign * k.x, sign * k.y);
    };
    int mx = kNoExponent;
    uint32_t hi = 0;
#pragma unroll 2
    for (int c = 0; c < j.kch; ++c) {
        const double2 a = at(re, c), b = at(im, c);
        const int2 k = scale(c);
        hi = max(max(hi, max(abs_hi(a.x), abs_hi(a.y))), max(abs_hi(b.x), abs_hi(b.y)));
        mx = max(max(mx, max(exponent_of(a.x, k.x), exponent_of(a.y, k.y))),
                 max(exponent_of(b.x, k.x), exponent_of(b.y, k.y)));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (hi >= 0x7FF00000u) atomicExch(redo, kDigitValue);
    const int ex = scaled_row_exponent(mx);
    if (lane == 0) {
        out.ex[to] = ex;
        if (DUAL) out.ex[to + j.n_dual] = ex;
    }
    for (int c = 0; c < j.kch; ++c) {
        const double2 a = at(re, c), b = at(im, c);
        const int2 k = scale(c);
        uint32_t d[kDigits], f[kDigits];
        digits2(a.x, a.y, ex, d, k.x, k.y);
        digits2(b.x, b.y, ex, f, k.x, k.y);
        put_complex<DUAL>(out, to, j.n_dual, (int64_t)c * j.cs_out, (int64_t)(j.kch + c) * j.cs_out, 2 * lane, d, f);
    }
}

// psi sub-blocks: up to CW columns x all K rows by one CTA, lanes along the
// columns (CW = 8: four rows of them); a 64-wide chunk is turned in shared memory (`pitch` doubles a column,
// odd).  A K of one chunk is read once (a complex Hubbard D = 512 vector: 17 -> 6
// us against reading it twice).  CPLX: both parts of a complex vector, on one
// grid.
constexpr int PT = 256;
template <bool CPLX, int CW>
__global__ void __launch_bounds__(PT) digit_psi_kernel(const DigitPsi* __restrict__ jobs, const double* __restrict__ x,
                                                       const double* __restrict__ xi, const int32_t* __restrict__ kx,
                                                       int pitch, const DigitStack out, int* redo) {
    extern __shared__ double tile[];  // [CW][pitch], the imaginary part's behind it
    __shared__ int smax[32], scale[kTcBK];
    const DigitPsi j = jobs[blockIdx.x];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int nr = j.cols, K = j.rows, kch = (K + kTcBK - 1) / kTcBK;
    double* tile_im = tile + CW * pitch;
    const int col = lane % CW, kw = w * (32 / CW) + lane / CW;  // this thread's column, first k
    constexpr int KS = PT / CW;                                 // k step of the CTA
    const int64_t src = j.src + col;
    const int32_t* sk = kx + j.kx;  // (a plan constant)
    dep_launch();
    if (tid < 32) smax[tid] = kNoExponent;
    if (tid < kTcBK) scale[tid] = sk[tid];
    __syncthreads();
    dep_wait();
    int mx = kNoExponent;
    uint32_t hi = 0, tiny = 0;  // tiny: whether there are subnormals
    auto look = [&](double v, int s) {
        const uint32_t h = abs_hi(v);
        const int e = (int)(h >> 20);
        hi = max(hi, h);
        tiny |= e > 0 ? 0u : h | (uint32_t)__double2loint(v);
        mx = max(mx, e > 0 ? e + s : kNoExponent);
    };
    // chunk c into shared memory, zeros to a whole 16-wide step (they are multiplied)
    auto fetch = [&](int c) {
        const int k0 = c * kTcBK, kv = (min(kTcBK, K - k0) + 15) & ~15;
#pragma unroll 4
        for (int k = kw; k < kv; k += KS) {
            const bool in = col < nr && k0 + k < K;
            const int64_t o = src + (int64_t)(k0 + k) * j.pitch;
            const double v = in ? x[o] : 0.0;
            tile[col * pitch + k] = v;
            if (kch == 1) look(v, scale[k]);
            if (CPLX) {
                const double u = in ? xi[o] : 0.0;
                tile_im[col * pitch + k] = u;
                if (kch == 1) look(u, scale[k]);
            }
        }
        return kv;
    };
    if (kch == 1) {
        fetch(0);
    } else {
#pragma unroll 4
        for (int k = kw; k < K; k += KS)
            if (col < nr) {
                const int64_t o = src + (int64_t)k * j.pitch;
                const int s = sk[k];
                look(x[o], s);
                if (CPLX) look(xi[o], s);
            }
    }
    if (tiny) {
        for (int k = kw; k < K; k += KS) {  // (col < nr, or it would have seen zeros)
            const int64_t o = src + (int64_t)k * j.pitch;
            mx = max(mx, exponent_of(x[o], sk[k]));
            if (CPLX) mx = max(mx, exponent_of(xi[o], sk[k]));
        }
    }
    atomicMax(&smax[col], mx);
    if (hi >= 0x7FF00000u) atomicExch(redo, kDigitValue);
    __syncthreads();
    if (tid < nr) {
        const int ex = scaled_row_exponent(smax[tid]);
        out.ex[(int64_t)j.to + tid] = ex;
        if (CPLX) out.ex[(int64_t)j.to + j.n_dual + tid] = ex;
        smax[tid] = ex;
    }
    for (int c = 0; c < kch; ++c) {
        __syncthreads();
        const int kv = kch == 1 ? (K + 15) & ~15 : fetch(c);
        if (kch > 1) {
            if (tid < kTcBK) scale[tid] = sk[c * kTcBK + tid];
            __syncthreads();
        }
        // rows and pairs of k over the threads
        const int pairs = kv >> 1;
        for (int e = tid; e < nr * pairs; e += PT) {
            const int r = e / pairs, k = 2 * (e - r * pairs);
            const double* v = tile + r * pitch + k;
            uint32_t d[kDigits];
            digits2(v[0], v[1], smax[r], d, scale[k], scale[k + 1]);
            if (CPLX) {
                const double* u = tile_im + r * pitch + k;
                uint32_t f[kDigits];
                digits2(u[0], u[1], smax[r], f, scale[k], scale[k + 1]);
                put_complex<true>(out, (int64_t)j.to + r, j.n_dual, (int64_t)c * j.cs, (int64_t)(kch + c) * j.cs, k, d, f);
            } else {
                put_digits(out, (int64_t)j.to + r + (int64_t)c * j.cs, k, d);
            }
        }
    }
}

constexpr int BT = 256;
// Whether x lies on the grid of digits 0 .. 3 of a row with exponent ex: its lowest
// bit at 2^(ex - 1055) or above.
__device__ __forceinline__ bool in_four_digits(double x, int ex) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int e = (int)(b >> 52) & 0x7FF;
    const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | (e ? 1ull << 52 : 0);
    return m == 0 || max(e, 1) + __ffsll((long long)m) - 1 >= ex + 20;
}
// Whether x may have bits below its row's grid.
__device__ __forceinline__ bool below_grid(double x, int ex) {
    const uint32_t hi = abs_hi(x);
    return (int)(hi >> 20) < ex - 4 && (hi | (uint32_t)__double2loint(x)) != 0;
}
// |x| 2^-e in fp32, rounded down (e by its biased form ex: |x| < 2^(ex - 1022))
__device__ __forceinline__ float below_one(double x, int ex) {
    const uint32_t hi = abs_hi(x);
    const int e = (int)(hi >> 20) - ex + 126;
    const uint32_t m = ((hi & 0xFFFFFu) << 3) | ((uint32_t)__double2loint(x) >> 29);
    return hi >> 20 && e > 0 ? __uint_as_float(((uint32_t)e << 23) | m) : 0.0f;
}
// The k's of a product that digit_gate_kernel looks at: kGate of them, or all.
constexpr int kGate = kDigitSamples;
__host__ __device__ __forceinline__ int gate_k(int s, int K) { return K > kGate ? (int)((int64_t)s * K / kGate) : s; }
// The two operands of a dense product, 32 rows x 64 k a CTA (the rows of A,
// then those of B).  PASS 0 leaves every row's largest high word in top (zeroed
// before), PASS 1 writes the exponents, the digits and the gate's samples, and finds
// whether an element is not on the grid of four digits (*wide) and, for a K of one
// chunk, the most elements of a row that may be off its grid (*inexact, zeroed before);
// lanes walk along the shorter stride.
template <int PASS>
__global__ void __launch_bounds__(BT) digit_matrix_kernel(const DigitMatrix A, const DigitMatrix B, int K, int* wide,
                                                          int* redo) {
    __shared__ double tile[32][kTcBK + 1];
    __shared__ int sex[32];
    const int na = (A.rows + 31) / 32;
    const bool first = (int)blockIdx.x < na;
    const DigitMatrix& m = first ? A : B;
    const int r0 = ((int)blockIdx.x - (first ? 0 : na)) * 32, nr = min(32, m.rows - r0), k0 = (int)blockIdx.y * kTcBK;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const double* x = m.x + r0 * m.rs + k0 * m.ks;
    auto fetch = [&](int r, int k) { return r < nr && k0 + k < K ? x[r * m.rs + k * m.ks] : 0.0; };
    if (PASS == 1 && tid < nr) {
        sex[tid] = row_exponent(m.top[r0 + tid], redo);
        if (blockIdx.y == 0) m.out.ex[r0 + tid] = sex[tid];
    }
    if ((m.rs < 0 ? -m.rs : m.rs) < (m.ks < 0 ? -m.ks : m.ks)) {
#pragma unroll
        for (int i = 0; i < kTcBK / (BT / 32); ++i) tile[lane][w + i * (BT / 32)] = fetch(lane, w + i * (BT / 32));
    } else {
#pragma unroll
        for (int i = 0; i < 32 / (BT / 64); ++i) {
            const int r = (tid >> 6) + i * (BT / 64), k = tid & 63;
            tile[r][k] = fetch(r, k);
        }
    }
    __syncthreads();
    uint32_t off = 0;  // elements off the grid, a byte for each of the warp's four rows
    bool four = true, look = false;  // look: whether *wide is still open
    int at[2] = {-1, -1};            // which samples this lane's two k are (-1: none)
    if (PASS == 1) {
        look = *(volatile int*)wide == 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = k0 + 2 * lane + i, s = K > kGate ? (int)(((int64_t)k * kGate + K - 1) / K) : k;
            if (k < K && s < kGate && gate_k(s, K) == k) at[i] = s;
        }
    }
    for (int r = w; r < nr; r += BT / 32) {
        if (PASS == 0) {
            const uint32_t mx = __reduce_max_sync(0xffffffffu, max(abs_top(tile[r][lane]), abs_top(tile[r][lane + 32])));
            if (lane == 0) atomicMax(m.top + r0 + r, mx);
        } else {
            const double u = tile[r][2 * lane], v = tile[r][2 * lane + 1];
            uint32_t d[kDigits];
            digits2(u, v, sex[r], d);
            put_digits(m.out, r0 + r + (int64_t)blockIdx.y * m.rows, 2 * lane, d);
            if (look) four = four && in_four_digits(u, sex[r]) && in_four_digits(v, sex[r]);
            if (K <= kTcBK) off |= (uint32_t)(below_grid(u, sex[r]) + below_grid(v, sex[r])) << (r - w);
            if (at[0] >= 0) m.sample[(int64_t)at[0] * m.rows + r0 + r] = below_one(u, sex[r]);
            if (at[1] >= 0) m.sample[(int64_t)at[1] * m.rows + r0 + r] = below_one(v, sex[r]);
        }
    }
    if (PASS == 1) {
        if (__syncthreads_or(!four) && tid == 0) atomicExch(wide, 1);
        if (K <= kTcBK) {
            static_assert(32 / (BT / 32) == 4 && BT / 32 == 8, "rows w, w + 8, w + 16, w + 24: bytes 0 .. 3");
            off = __reduce_add_sync(0xffffffffu, off);
            if (lane == 0)
                atomicMax(m.inexact, (int)max(max(off & 255u, (off >> 8) & 255u), max((off >> 16) & 255u, off >> 24)));
        }
    }
}

// Whether the digits hold a dense product as exactly as an FP64 chain of K steps
// does, output by output.  They leave out half a unit, 2^(e - 58), of an element that
// is not on its row's grid (shares f_a and f_b of the two rows' k) and the products of
// digits i + j > 6, 6.03 x 2^-60 2^(ea + eb) a k:
//   |error| <= (2^-58 (f_a + f_b) + 0.052 x 2^-53) K 2^(ea + eb)
// with the roundings of the sums, where the chain's bound is K 2^-53 sum |a_k b_k|.  So
// an output with
//   sum |a_k b_k| >= ((f_a + f_b) / 32 + 0.052) 2^(ea + eb)
// has the smaller bound on digits (f = 1 where K is longer than a chunk: there the sums
// are far above it).  The sum over kGate of the k, evenly spaced, is a
// lower bound of it and enough for operands without structure (N(0, 1): about 0.6 at
// 64 k, the least of a million outputs 0.27); where one output falls below, *redo
// sends the product to the FP64 pipe.  Rows of zeros, and operands whose elements all
// lie in four digits, have no error at all.  (A statement on the rows alone will not
// do: sum |a_k b_k| depends on where the large elements of both meet.)
// 64 x 64 outputs a CTA in fp32; at 2048^3 it takes 21 us and the call 515 us (507 without).
__global__ void __launch_bounds__(BT) digit_gate_kernel(const DigitMatrix A, const DigitMatrix B, int K, const int* wide,
                                                        int* redo) {
    __shared__ __align__(16) float sa[kGate][64], sb[kGate][64];
    if (*wide == 0) return;
    const int tid = threadIdx.x, ks = min(K, kGate);
    const int m0 = (int)blockIdx.y * 64, n0 = (int)blockIdx.x * 64;
    for (int i = tid; i < 64 * ks; i += BT) {
        const int r = i & 63, k = i >> 6;
        sa[k][r] = m0 + r < A.rows ? A.sample[(int64_t)k * A.rows + m0 + r] : 0.0f;
        sb[k][r] = n0 + r < B.rows ? B.sample[(int64_t)k * B.rows + n0 + r] : 0.0f;
    }
    __syncthreads();
    const int tx = (tid & 15) * 4, ty = (tid >> 4) * 4;
    float acc[4][4] = {};
    for (int k = 0; k < ks; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(&sa[k][ty]), b = *reinterpret_cast<const float4*>(&sb[k][tx]);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    bool bad = false;
    const float least = (K <= kTcBK ? (float)(*A.inexact + *B.inexact) / (32.0f * (float)K) : 0.0625f) + 0.052f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            bad |= m0 + ty + i < A.rows && n0 + tx + j < B.rows && acc[i][j] < least && A.top[m0 + ty + i] != 0 &&
                   B.top[n0 + tx + j] != 0;
    if (__syncthreads_or(bad) && tid == 0) atomicExch(redo, kDigitValue);
}

}  // namespace

bool digit_maps(DigitMaps& m, const DigitStack& a, const DigitStack& b, std::string& err) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
        err = "cuTensorMapEncodeTiled entry point unavailable";
        return false;
    }
    std::memset(&m, 0, sizeof(m));
    auto make = [&](CUtensorMap* map, const DigitStack& s, int box_rows) {
        if (s.rows <= 0) return true;
        cuuint64_t dims[3] = {(cuuint64_t)kTcBK, (cuuint64_t)s.rows, (cuuint64_t)kDigits};
        cuuint64_t strides[2] = {(cuuint64_t)kTcBK * 2 * kDigits, (cuuint64_t)kTcBK * 2};
        cuuint32_t box[3] = {(cuuint32_t)KW, (cuuint32_t)box_rows, (cuuint32_t)kDigits};
        cuuint32_t estr[3] = {1, 1, 1};
        CUresult r = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn)(
            map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, s.q, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) err = "cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)r);
        return r == CUDA_SUCCESS;
    };
    for (int i = 0; i < 4; ++i)
        if (!make(&m.a[i], a, 32 * (i + 1))) return false;
    return make(&m.b, b, HN);
}

cudaError_t digit_setup() {
    cudaError_t e = cudaSuccess;
    for (const void* k : {(const void*)digit_gemm_kernel<0>, (const void*)digit_gemm_kernel<1>, (const void*)digit_gemm_kernel<2>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    return e;
}

cudaError_t launch_digit_gemm(int mode, const TcTile* tiles, const int32_t* begin, int ctas, const DigitMaps& maps,
                              const int32_t* exa, const int32_t* exb, const DigitOut& out, int* redo, cudaStream_t s) {
    if (ctas <= 0) return cudaSuccess;
    if (mode == 0) return launch_dependent(digit_gemm_kernel<0>, ctas, NTHREADS, SMEM_BYTES, s, tiles, begin, maps, exa, exb, out, redo);
    if (mode == 1) return launch_dependent(digit_gemm_kernel<1>, ctas, NTHREADS, SMEM_BYTES, s, tiles, begin, maps, exa, exb, out, redo);
    return launch_dependent(digit_gemm_kernel<2>, ctas, NTHREADS, SMEM_BYTES, s, tiles, begin, maps, exa, exb, out, redo);
}

void digit_schedule(const std::vector<TcTile>& in, int ctas, std::vector<TcTile>& out, std::vector<int32_t>& begin) {
    // microseconds a tile holds its SM: the product per 64 k, then the ends
    // (measured on Hubbard D = 2048 and on dense products)
    auto cost = [](const TcTile& t) {
        const double halves = t.n_valid > HN ? 2.0 : 1.0, k = std::ceil(t.k_valid / (double)KW) * 0.5 * std::max(t.parts, 1);
        return 1.0 + k * (0.8 + 1.4 * halves) + 4.0 * t.m_valid * t.n_valid / (kTcBM * (double)kTcBN);
    };
    auto pack = [&](const std::vector<TcTile>& v, std::vector<int>& cta) {
        std::vector<int> order(v.size());
        for (size_t i = 0; i < v.size(); ++i) order[i] = (int)i;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost(v[a]) > cost(v[b]); });
        std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>, std::greater<>> load;
        for (int c = 0; c < ctas; ++c) load.push({0.0, c});
        cta.assign(v.size(), 0);
        double top = 0.0;
        for (int i : order) {
            auto [t, c] = load.top();
            load.pop();
            cta[(size_t)i] = c;
            t += cost(v[(size_t)i]);
            top = std::max(top, t);
            load.push({t, c});
        }
        return top;
    };
    // half-wide tiles read A twice, but two SMs share what one would do
    // (with many tiles a CTA the whole ones come out as even)
    std::vector<TcTile> halves;
    const bool try_halves = in.size() < 4 * (size_t)ctas;
    for (const TcTile& t : in)
        for (int n = 0; try_halves && n < t.n_valid; n += HN) {
            TcTile q = t;
            q.b_row += n;
            q.n_valid = std::min(HN, t.n_valid - n);
            if (t.mode == 2) q.out_off += n;
            q.n0 += n;
            halves.push_back(q);
        }
    std::vector<int> whole_cta, half_cta;
    const double whole = pack(in, whole_cta), half = try_halves ? pack(halves, half_cta) : whole;
    const std::vector<TcTile>& v = half < whole ? halves : in;
    const std::vector<int>& cta = half < whole ? half_cta : whole_cta;
    std::vector<std::vector<int>> of((size_t)ctas);
    for (size_t i = 0; i < v.size(); ++i) of[(size_t)cta[i]].push_back((int)i);
    out.clear();
    begin.assign(1, 0);
    for (std::vector<int>& l : of) {
        std::stable_sort(l.begin(), l.end(), [&](int a, int b) { return cost(v[(size_t)a]) > cost(v[(size_t)b]); });
        for (int i : l) out.push_back(v[(size_t)i]);
        begin.push_back((int32_t)out.size());
    }
}

cudaError_t launch_digit_columns(const DigitRows* jobs, int n_jobs, int max_kch, const double* q64, const double* q64_im,
                                 const int32_t* ex, int32_t* kx, cudaStream_t s) {
    if (n_jobs <= 0 || max_kch <= 0) return cudaSuccess;
    digit_columns_kernel<<<dim3((unsigned)n_jobs, (unsigned)max_kch), kColumnRows * kTcBK, 0, s>>>(jobs, q64, q64_im, ex, kx);
    return cudaGetLastError();
}

cudaError_t launch_digit_rows(const DigitRows* jobs, int n_jobs, const double* q64, const int32_t* kx, int sign,
                              const DigitStack& out, int* redo, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    return launch_dependent(digit_rows_kernel, n_jobs, 32 * kDigitRowsPerCta, 0, s, jobs, q64, kx, sign, out, redo);
}

cudaError_t launch_digit_rows_complex(const DigitRowsC* jobs, int n_jobs, const double* re, const double* im,
                                      const int32_t* kx, int sign, bool dual, const DigitStack& out, int* redo,
                                      cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    return launch_dependent(dual ? digit_rows_complex_kernel<true> : digit_rows_complex_kernel<false>, n_jobs,
                            32 * kDigitRowsPerCta, 0, s, jobs, re, im, kx, sign, out, redo);
}

cudaError_t launch_digit_matrices(const DigitMatrix& a, const DigitMatrix& b, int K, int* wide, int* redo, cudaStream_t s) {
    const dim3 grid((unsigned)((a.rows + 31) / 32 + (b.rows + 31) / 32), (unsigned)((K + kTcBK - 1) / kTcBK));
    digit_matrix_kernel<0><<<grid, BT, 0, s>>>(a, b, K, wide, redo);
    digit_matrix_kernel<1><<<grid, BT, 0, s>>>(a, b, K, wide, redo);
    digit_gate_kernel<<<dim3((unsigned)((b.rows + 63) / 64), (unsigned)((a.rows + 63) / 64)), BT, 0, s>>>(a, b, K, wide, redo);
    return cudaGetLastError();
}

cudaError_t launch_digit_psi(const DigitPsi* jobs, int n_jobs, int cols, int max_k, const double* x, const double* x_im,
                             const int32_t* kx, const DigitStack& out, int* redo, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    const int pitch = ((std::min(max_k, kTcBK) + 15) & ~15) + 1;
    const size_t smem = sizeof(double) * cols * pitch * (x_im ? 2 : 1);
    auto* k = cols == 8 ? (x_im ? digit_psi_kernel<true, 8> : digit_psi_kernel<false, 8>)
                        : (x_im ? digit_psi_kernel<true, 32> : digit_psi_kernel<false, 32>);
    return launch_dependent(k, n_jobs, PT, smem, s, jobs, x, x_im, kx, pitch, out, redo);
}

}  // namespace tk
