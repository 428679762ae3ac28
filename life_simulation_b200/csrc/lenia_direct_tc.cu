// life_simulation_b200/csrc/lenia_direct_tc.cu -- the direct toroidal
// convolution as a banded GEMM on the tensor cores (tcgen05.mma kind::i8,
// exact 32-bit integer accumulators in tensor memory), fused with the growth
// epilogue: the same update as lenia_direct.cu (the work of leniaStep,
// Shaders/Field/Lenia.metal:63-128, for up to 4 kernel tables).
//
// Arithmetic. A field value a in [0, 2) is the 32-bit fixed-point number
// A = rint(a 2^31) = a0 2^24 + a1 2^16 + a2 2^8 + a3 (unsigned bytes), a weight
// w the number rint(w 2^e) = w0 2^16 + w1 2^8 + w2 (signed bytes; e the largest
// exponent that keeps the table in range). The products of byte i and byte j
// go to the integer sum of level i + j; levels 0 to 3 (nine of the twelve
// products) are summed exactly -- 3 * 4225 taps * 255 * 128 < 2^31 -- and
// combined in FP32 once: U = L0 2^(9-e) + (L1 + L2 / 2^8 + L3 / 2^16) 2^(1-e).
//
// Its error: a value of 2^-8 or more is exact, a fainter one off by up to 2^-32;
// the weights' rounding, half a unit of 2^-e a tap, is carried from tap to tap so
// that it cancels where the field is smooth; the levels left out weigh 2^-32 of
// a tap's share; the last combination rounds three times (two conversions, one
// FMA). The FP32 form rounds once per tap. U enters the growth as U - mu, which FP32
// rounds at 2^-25 |mu| or more away from mu, so that 2^-32 stays below the FP32
// form's own rounding for |mu| >= 2^-6, and kernels nearer zero run on the FP32
// form (direct_tc_holds). With 24-bit values, rint(a 2^23), a field of 1e-3
// had a potential off by 6e-5 of itself, two orders above the FP32 form's.
// An integer sum is the same in any order. A tile whose halo holds a value
// outside [0, 2) (an uploaded field may: infinities, NaN, negative values) takes
// the FP32 loop below, tap by tap in the order of lenia_direct.cu.
//
// The GEMM. A CTA owns 128 rows x 32 columns of output. Kernel row dy over a
// chunk of 32 input columns is D[128 x 32] += X[128 x 32] T[32 x 32]: X is the
// halo tile's rows dy .. dy + 127 (the accumulator's lanes are the output
// rows), T the Toeplitz block T[k][n] = w(dy, base + k - n) of the chunk that
// starts `base` columns beside the tile. A row of half width hw takes 1 + 2 Q
// / 32 chunks, Q = hw rounded up to 16, so the disc's corners cost less. The
// rows' shift by dy is 16 bytes in X's start address: both operands lie in
// shared memory in 16-byte rows (K-major core matrices without swizzle, rows
// evenly 16 bytes apart), so one staged tile serves every dy.
//
// What bounds it: the operands' shared-memory reads. A product of N columns
// takes max(46, 32 + N / 4) cycles (measured, N <= 128: 4 KB of X and 32 N
// bytes of T at 128 bytes a cycle, against N / 2 cycles of math), so small N
// is lost; T's byte planes are side by side in [0 | w0 | w1 | w2] rows, which makes
// the nine byte products four: X0 against [w0 | w1 | w2] (N = 96), X1 likewise,
// X2 against [w0 | w1] (N = 64), X3 against [0 | w0] (N = 64): 208 cycles a
// chunk, where nine products of N = 32 would take 414. X0, X1 and the pair X2,
// X3 add into accumulator columns of their own (levels 0..2, 1..3 and 2..3),
// summed in the epilogue: tcgen05.mma orders successive products only where
// accumulator and shape are the same, so windows of different products may not
// overlap. Wider tiles read X less often but clip
// T's window, and came out behind. The T blocks (4 KB a chunk) come through a
// ring of bulk copies from L2, requested by one warp and multiplied by another,
// whose loop is uniform over the warp.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "fft_fast_common.cuh"
#include "lenia_device.cuh"
#include "lenia_kernels.h"

namespace lenia {
namespace {

constexpr int kRows = 128;             // output rows of a tile (accumulator lanes)
constexpr int kTX = 32;                // output columns of a tile
constexpr int kPart = kTX / 2;         // output columns per epilogue thread
// Warps: 0..7 epilogue (tensor-memory lane quadrant warp % 4, half of the
// columns warp / 4), 8..15 stage the halo tiles, then kMmaWarps that issue the
// products of alternate T blocks into accumulators of their own, and one that
// requests the T blocks.
constexpr int kEpiWarps = 8, kStageWarps = 8, kMmaWarp = 16, kMmaWarps = 2, kLoadWarp = kMmaWarp + kMmaWarps;
constexpr int kThreads = 32 * (kLoadWarp + 1);
constexpr int kPlanes = 4;             // bytes of a value
// Tensor-memory columns of one issuing warp's accumulators: X0's levels 0..2
// from column 0, X1's 1..3 from 96, X2's and X3's 2..3 from 192. Sets: kMmaWarps for each
// of kBufs tiles (or kernels) in flight.
constexpr uint32_t kCols = 512, kAccX1 = 3 * kTX, kAccX2 = 6 * kTX, kAccCols = 8 * kTX;
constexpr uint32_t kBufs = kCols / (kAccCols * kMmaWarps);
constexpr uint32_t kChunk = 128u * 32u;  // bytes of one chunk's T: 128 rows (zeros, then three byte planes) of 32 k
constexpr uint32_t kZeros = kTX * 16u;   // bytes of a half chunk's zero rows
constexpr int kTurn = kPart + 4;       // pitch (floats) of the rows an epilogue warp turns A and A' in
constexpr uint32_t kPolls = 1u << 20;  // polls of a barrier before a CTA gives up (about a second)

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// Matrix descriptor (sm_100 format, no swizzle). Low word: start address and
// leading byte offset (between the two 16-byte halves of K = 32), high word:
// stride byte offset 128 (between groups of eight rows), all >> 4, and
// descriptor version 1.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo) { return (addr >> 4) | ((lbo >> 4) << 16); }
constexpr uint32_t kDescHi = (128u >> 4) | (1u << 14);
// kind::i8, S32 accumulator (2), A unsigned bytes (0), B signed bytes (1),
// both K-major, M = 128 (>> 4), N (>> 3).
constexpr uint32_t idesc(uint32_t n) {
    return (2u << 4) | (0u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// 1 in one lane of a converged warp: the one that issues (and so commits) its products.
__device__ __forceinline__ uint32_t elected() {
    uint32_t lead;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(lead));
    return lead;
}
// Issued by the one lane whose `lead` is set, in a converged warp: a
// predicate on the instruction, not a branch around it, so that the loop
// that computes the descriptors stays uniform and keeps them in uniform
// registers (in a one-lane branch they cost 20 to 60 cycles a product). a, b:
// low words of the operands' descriptors (their high words are constant).
__device__ __forceinline__ void mma_i8(uint32_t d, uint32_t a, uint32_t b, uint32_t id, uint32_t acc, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred p, q;\n .reg .b64 x, y;\n setp.ne.b32 p, %5, 0;\n setp.ne.b32 q, %6, 0;\n"
        " mov.b64 x, {%1, %4};\n mov.b64 y, {%2, %4};\n"
        " @q tcgen05.mma.cta_group::1.kind::i8 [%0], x, y, %3, p;\n}\n" ::"r"(d),
        "r"(a), "r"(b), "r"(id), "r"(kDescHi), "r"(acc), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void commit(uint64_t* bar, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(bar)),
        "r"(lead)
        : "memory");
}
// The products of one kernel row: NQ + 1 chunks from operand addresses a, b;
// PLANE: bytes of a byte plane, STEP: bytes of two granules (a chunk's 32
// columns). acc = 0: the first products of a kernel, which set all of the three
// accumulators' columns.
template <int NQ, uint32_t PLANE, uint32_t STEP>
__device__ __forceinline__ void mma_row(uint32_t tmem, uint32_t a, uint32_t b, uint32_t acc, uint32_t lead) {
#pragma unroll
    for (int c = 0; c <= NQ; ++c) {
        const uint32_t ac = a + uint32_t(c) * (STEP / 16), bc = b + uint32_t(c) * (kChunk / 16);
        const uint32_t add = c > 0 ? 1u : acc;
        mma_i8(tmem, ac, bc + kZeros / 16, idesc(96), add, lead);
        mma_i8(tmem + kAccX1, ac + PLANE / 16, bc + kZeros / 16, idesc(96), add, lead);
        mma_i8(tmem + kAccX2, ac + 2 * (PLANE / 16), bc + kZeros / 16, idesc(64), add, lead);
        mma_i8(tmem + kAccX2, ac + 3 * (PLANE / 16), bc, idesc(64), 1, lead);
    }
}
__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded, by a whole warp; false (for the whole warp) when the polls run out
// or another warp's have (`stop`).
__device__ __noinline__ bool bar_wait_slow(uint64_t* bar, uint32_t parity, volatile int* stop) {
    for (uint32_t i = 0; i < kPolls; ++i) {
        if (bar_try(bar, parity)) return true;
        if ((i & 255u) == 255u && *stop) return false;
    }
    *stop = 1;
    return false;
}
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, volatile int* stop) {
    bool ok = bar_try(bar, parity);
    if (!__all_sync(0xffffffffu, ok)) ok = bar_wait_slow(bar, parity, stop);
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// 4 consecutive accumulator columns of this warp's lane quadrant (not
// waited for).
__device__ __forceinline__ void tmem_ld4(uint32_t addr, int32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(addr));
}

__device__ __forceinline__ int wrap(int v, int n) {
    if (v >= 0 && v < n) return v;
    v %= n;
    return v < 0 ? v + n : v;
}

// 0 <= a < 2 exactly when the sign and the top exponent bit are clear; + 0
// makes -0 zero.
__device__ __forceinline__ bool out_of_range(const float4& a) {
    return (((__float_as_uint(a.x + 0.0f) | __float_as_uint(a.y + 0.0f)) |
             (__float_as_uint(a.z + 0.0f) | __float_as_uint(a.w + 0.0f))) &
            0xC0000000u) != 0u;
}
// Four values as the bytes of levels 0 to 3, value i in byte i.
__device__ __forceinline__ void pack_bytes(const float4& a, uint32_t (&w)[kPlanes]) {
    const uint32_t v0 = __float2uint_rn(a.x * 2147483648.0f), v1 = __float2uint_rn(a.y * 2147483648.0f);
    const uint32_t v2 = __float2uint_rn(a.z * 2147483648.0f), v3 = __float2uint_rn(a.w * 2147483648.0f);
    const uint32_t l01 = __byte_perm(v0, v1, 0x5140), l23 = __byte_perm(v2, v3, 0x5140);
    const uint32_t h01 = __byte_perm(v0, v1, 0x7362), h23 = __byte_perm(v2, v3, 0x7362);
    w[0] = __byte_perm(h01, h23, 0x7632);
    w[1] = __byte_perm(h01, h23, 0x5410);
    w[2] = __byte_perm(l01, l23, 0x7632);
    w[3] = __byte_perm(l01, l23, 0x5410);
}

// A warp's share of a tile with values that the byte form cannot hold, in the
// FP32 form: rows y0 .. y0 + 15, a column a lane, taps in the order of
// direct_tile, four rows at a time on the same weights. Out of line, with no
// state of the epilogue's alive, so that the tiles of the byte form pay nothing
// for it. First frames of uploads whose tiles all take it: 1920 x 1080 R = 13
// 810 us, 1280 x 720 R = 32 1800 us (one output and one tap a thread at a time,
// rows across the lanes: 7.5 and 19.7 ms; FP32 kernels 104 and 216 us). A step
// clips its field to [0, 1], so an upload has one such frame.
constexpr int kFpRows = 16;
__device__ __noinline__ void fp32_rows(const float* __restrict__ src, float* __restrict__ dst,
                                       const float* __restrict__ weights, const uint32_t* __restrict__ spans,
                                       const DirectGeometry& g, const StepParams& p, const GrowthExtras& ex, int nk,
                                       int x0, int y0) {
    constexpr int N = 4;
    const int W = int(p.width), H = int(p.height), x = x0 + int(threadIdx.x & 31u);
    const EulerStep euler(p);
#pragma unroll 1
    for (int y = y0; y < min(y0 + kFpRows, H); y += N) {
        float sum[N] = {};
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            float acc[N] = {};
#pragma unroll 1
            for (int dyi = 0; dyi < g.ksize; ++dyi) {
                const uint32_t sp = spans[k * g.ksize + dyi];
                const float* w = weights + size_t(k * g.ksize + dyi) * g.wp + g.xp;
                const float* row[N];
#pragma unroll
                for (int j = 0; j < N; ++j) row[j] = src + size_t(wrap(y + j + dyi - g.r, H)) * W;
                int d = int(sp & 0xFFFFu) - 128;
#pragma unroll 1
                for (int c = int(sp >> 16); c > 0; --c, d += 8) {
                    float a[8][N], t[8];
                    if (x0 + d >= 0 && x0 + 32 + d + 8 <= W) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
#pragma unroll
                            for (int j = 0; j < N; ++j) a[i][j] = __ldg(row[j] + x + d + i);
                    } else {
                        int at = wrap(x + d, W);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
#pragma unroll
                            for (int j = 0; j < N; ++j) a[i][j] = __ldg(row[j] + at);
                            at = at + 1 == W ? 0 : at + 1;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) t[i] = __ldg(w + d + i);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < N; ++j) acc[j] = fmaf(t[i], a[i][j], acc[j]);
                }
            }
            const float mu = k == 0 ? p.mu[0] : k == 1 ? p.mu[1] : k == 2 ? p.mu[2] : p.mu[3];
            const float sigma = k == 0 ? p.sigma[0] : k == 1 ? p.sigma[1] : k == 2 ? p.sigma[2] : p.sigma[3];
            const float h = k == 0 ? p.weight[0] : k == 1 ? p.weight[1] : k == 2 ? p.weight[2] : p.weight[3];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const float shift = p.mu_jitter > 0.0f
                                        ? mu_jitter_shift(p, uint32_t(x), rand_row(uint32_t(y + j), ex.jitter_base))
                                        : 0.0f;
                sum[j] = growth_add(sum[j], h, bell(acc[j], mu + shift, sigma), euler.asym);
            }
        }
        euler.divide(sum);
#pragma unroll 1
        for (int j = 0; j < N; ++j) {
            if (y + j >= H || x >= W) continue;
            const size_t at = size_t(y + j) * W + size_t(x);
            const float s = j == 0 ? sum[0] : j == 1 ? sum[1] : j == 2 ? sum[2] : sum[3];
            float v[1] = {euler(__ldg(src + at), s)};
            noise_inject_clip(p, ex, v, uint32_t(x), uint32_t(y + j));
            dst[at] = v[0];
        }
    }
}

// T blocks in flight: what the staged tiles leave room for.
template <int P>
constexpr int kStages = P == 16 ? 6 : 5;

// Barriers and flags of a CTA.
struct TcShared {
    uint64_t t_full[6], t_empty[6];              // T blocks
    uint64_t a_full[2], a_empty[2];              // staged halo tiles
    uint64_t d_full[kBufs], d_empty[kBufs];      // accumulators
    uint64_t drain[kMmaWarps];                   // products in flight when a wait ran out
    int bad[4];     // tile count + 1 of the last tile of slot (count % 4) with a value outside the byte form
    int stop;       // a wait ran out
    uint32_t tmem;  // tensor-memory address
    GrowthExtras ex;
};

// P: halo columns each side (16 for r <= 16, else 32); the staged planes have
// 128 + 2 P rows, of which 128 + 2 r are read. One CTA per SM loops
// over tiles; staging, products and epilogue of successive tiles overlap (two
// staged tiles, kBufs sets of accumulators).
template <int P>
__global__ void __launch_bounds__(kThreads, 1)
    direct_tc_kernel(const float* __restrict__ src, float* __restrict__ dst, const __grid_constant__ DirectTcPlan plan,
                     const float* __restrict__ weights, const uint32_t* __restrict__ spans,
                     const __grid_constant__ DirectGeometry g, const __grid_constant__ StepParams p, int nk,
                     int tiles_x, int tiles, int* err) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ TcShared sh;
    constexpr int RA = kRows + 2 * P, NG = (kTX + 2 * P) / 16;      // staged rows, 16-column granules
    constexpr uint32_t kPlane = uint32_t(RA) * 16u * uint32_t(NG);  // bytes of one staged byte plane
    constexpr uint32_t kStage = kChunk * uint32_t(1 + P / 16);
    const int tid = int(threadIdx.x), warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int W = int(p.width), H = int(p.height);
    unsigned char* ring = sm + 2u * kPlanes * kPlane;

    if (tid == 0) {
        sh.stop = 0;
        for (int i = 0; i < kStages<P>; ++i) {
            bar_init(&sh.t_full[i], 1);
            bar_init(&sh.t_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            bar_init(&sh.a_full[i], kStageWarps);
            bar_init(&sh.a_empty[i], kMmaWarps);
        }
        for (uint32_t i = 0; i < kBufs; ++i) {
            bar_init(&sh.d_full[i], kMmaWarps);
            bar_init(&sh.d_empty[i], kEpiWarps);
        }
        for (int i = 0; i < kMmaWarps; ++i) bar_init(&sh.drain[i], 1);
        for (int i = 0; i < 4; ++i) sh.bad[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sh.tmem)),
                     "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    growth_extras_init(sh.ex, p);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sh.tmem, 0);

    if (warp >= kEpiWarps && warp < kEpiWarps + kStageWarps) {
        // ---- Stage the halo tiles as byte planes, [16-column granule]
        // [row][16 bytes]: a warp access covers eight rows of a granule, four
        // lanes a row (64 bytes loaded; the 4-byte stores fill 128 contiguous
        // bytes), five or six accesses in flight.
        fastfft::grid_dependency_wait();
        constexpr int kGroups = RA / 8, kItems = kGroups * NG, kFlight = P == 16 ? 5 : 6;
        static_assert(kItems % (kFlight * kStageWarps) == 0, "whole batches of accesses");
        const int q = 4 * (lane & 3), rl = lane >> 2;
        uint32_t ai = 0;
        for (int tile = int(blockIdx.x); tile < tiles; tile += int(gridDim.x), ++ai) {
            const uint32_t buf = ai & 1u;
            if (ai >= 2 && !bar_wait(&sh.a_empty[buf], ((ai >> 1) - 1u) & 1u, &sh.stop)) break;
            const int ty = tile / tiles_x, x0 = (tile - ty * tiles_x) * kTX, y0 = ty * kRows;
            const bool inside = W % 4 == 0 && x0 >= P && x0 + kTX + P <= W;
            unsigned char* planes = sm + buf * kPlanes * kPlane;
            bool bad = false;
            if (W % 4 != 0 && x0 >= P && x0 + kTX + P + 3 <= W) {
                // Rows start anywhere in a 16-byte quad: the quads that hold the
                // tile's columns are loaded aligned, made bytes, and the bytes
                // shifted by the row's offset over the neighbouring lane's. (Four
                // loads a quad, and a row a thread in the epilogue's loads and
                // stores, at 1001 x 703, R = 9, two substeps: 28.7 -> 23.1 us.)
#pragma unroll 1
                for (int rg = warp - kEpiWarps; rg < kGroups; rg += kStageWarps) {
                    const int row = rg * 8 + rl;
                    const size_t at = size_t(wrap(y0 - g.r + row, H)) * W + size_t(x0 - P);
                    const uint32_t shift = uint32_t(at) & 3u;
                    const float4* quad = reinterpret_cast<const float4*>(src + (at - shift)) + (lane & 3);
                    float4 a[NG + 1];
#pragma unroll
                    for (int f = 0; f < NG; ++f) a[f] = __ldg(quad + 4 * f);
                    // The quad after the last granule's: the group's first lane reads it for the last.
                    a[NG] = (lane & 3) == 0 && shift != 0u ? __ldg(quad + 4 * NG) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    uint32_t w[NG + 1][kPlanes];
#pragma unroll
                    for (int f = 0; f <= NG; ++f) {
                        bad = bad || out_of_range(a[f]);
                        pack_bytes(a[f], w[f]);
                    }
                    const int from = (lane & 3) == 3 ? lane - 3 : lane + 1;
                    const uint32_t sel = 0x3210u + 0x1111u * shift;  // bytes shift .. shift + 3 of two words
#pragma unroll
                    for (int f = 0; f < NG; ++f)
#pragma unroll
                        for (int j = 0; j < kPlanes; ++j) {
                            const uint32_t next =
                                __shfl_sync(0xffffffffu, (lane & 3) == 0 ? w[f + 1][j] : w[f][j], from);
                            *reinterpret_cast<uint32_t*>(planes + uint32_t(j) * kPlane + (f * RA + row) * 16 + q) =
                                __byte_perm(w[f][j], next, sel);
                        }
                }
            } else {
#pragma unroll 1
                for (int i0 = warp - kEpiWarps; i0 < kItems; i0 += kFlight * kStageWarps) {
                    float4 a[kFlight];
#pragma unroll
                    for (int f = 0; f < kFlight; ++f) {
                        const int i = i0 + f * kStageWarps, gran = i / kGroups, row = (i - gran * kGroups) * 8 + rl;
                        const float* line = src + size_t(wrap(y0 - g.r + row, H)) * W;
                        const int x = x0 - P + 16 * gran + q;
                        if (inside) {
                            a[f] = __ldg(reinterpret_cast<const float4*>(line + x));
                        } else {
                            a[f].x = __ldg(line + wrap(x, W));
                            a[f].y = __ldg(line + wrap(x + 1, W));
                            a[f].z = __ldg(line + wrap(x + 2, W));
                            a[f].w = __ldg(line + wrap(x + 3, W));
                        }
                    }
#pragma unroll
                    for (int f = 0; f < kFlight; ++f) {
                        const int i = i0 + f * kStageWarps, gran = i / kGroups, row = (i - gran * kGroups) * 8 + rl;
                        bad = bad || out_of_range(a[f]);
                        uint32_t w[kPlanes];
                        pack_bytes(a[f], w);
                        unsigned char* o = planes + (gran * RA + row) * 16 + q;
#pragma unroll
                        for (int j = 0; j < kPlanes; ++j) *reinterpret_cast<uint32_t*>(o + uint32_t(j) * kPlane) = w[j];
                    }
                }
            }
            if (bad) *reinterpret_cast<volatile int*>(&sh.bad[ai & 3u]) = int(ai) + 1;
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(&sh.a_full[buf]);
        }
        fastfft::allow_dependents();
    } else if (warp == kLoadWarp) {
        // ---- T blocks (tables: they do not depend on the step before).
        uint32_t ti = 0;
        for (int tile = int(blockIdx.x); tile < tiles; tile += int(gridDim.x)) {
            uint32_t offset = 0;
#pragma unroll 1
            for (int r = 0; r < plan.first[nk]; ++r, ++ti) {
                const uint32_t st = ti % kStages<P>, bytes = kChunk * (1u + (uint32_t(plan.rows[r]) >> 14));
                if (ti >= kStages<P> && !bar_wait(&sh.t_empty[st], (ti / kStages<P> - 1u) & 1u, &sh.stop)) break;
                if (lane == 0) bulk_load(ring + st * kStage, plan.blocks + offset, bytes, &sh.t_full[st]);
                offset += bytes;
            }
            if (*reinterpret_cast<volatile int*>(&sh.stop)) break;
        }
        // After a wait ran out: the copies in flight get one more bounded wait.
        if (*reinterpret_cast<volatile int*>(&sh.stop)) {
            int never = 0;
            for (uint32_t i = ti > kStages<P> ? ti - kStages<P> : 0; i < ti; ++i)
                bar_wait_slow(&sh.t_full[i % kStages<P>], (i / kStages<P>) & 1u, &never);
        }
    } else if (warp >= kMmaWarp && warp < kMmaWarp + kMmaWarps) {
        // ---- Products of every kMmaWarps-th T block.
        const int m = warp - kMmaWarp;
        const uint32_t lead = elected();
        const uint32_t b_base = desc_lo(smem_u32(ring), kChunk / 2);
        uint32_t ai = 0, di = 0, st = 0, ph = 0;  // ring stage and its phase
        bool ok = true;
        for (int tile = int(blockIdx.x); tile < tiles && ok; tile += int(gridDim.x), ++ai) {
            const uint32_t buf = ai & 1u;
            const uint32_t a_base = desc_lo(smem_u32(sm) + buf * kPlanes * kPlane, RA * 16u) + uint32_t((P / 16) * RA);
            ok = bar_wait(&sh.a_full[buf], (ai >> 1) & 1u, &sh.stop);
#pragma unroll 1
            for (int k = 0; k < nk && ok; ++k, ++di) {
                const uint32_t db = di % kBufs, d = tmem + (db * kMmaWarps + uint32_t(m)) * kAccCols;
                if (di >= kBufs) ok = bar_wait(&sh.d_empty[db], (di / kBufs - 1u) & 1u, &sh.stop);
                fence_after();
                uint32_t acc = 0;  // the first products set the accumulators
                const int r0 = plan.first[k], r1 = plan.first[k + 1];
#pragma unroll 1
                for (int r = r0; r < r1 && ok; ++r) {
                    if ((r - r0) % kMmaWarps == m) {
                        const uint32_t row = plan.rows[r], nq = row >> 14;
                        const uint32_t a = a_base - nq * uint32_t(RA), b = b_base + st * (kStage / 16);
                        const uint32_t dy0 = row & 127u, dy1 = (row >> 7) & 127u;
                        ok = bar_wait(&sh.t_full[st], ph, &sh.stop);
                        if (!ok) break;
                        if (P == 32 && nq == 2) {
                            mma_row<2, kPlane, 32u * RA>(d, a + dy0, b, acc, lead);
                            if (dy1 != dy0) mma_row<2, kPlane, 32u * RA>(d, a + dy1, b, 1u, lead);
                        } else if (nq == 1) {
                            mma_row<1, kPlane, 32u * RA>(d, a + dy0, b, acc, lead);
                            if (dy1 != dy0) mma_row<1, kPlane, 32u * RA>(d, a + dy1, b, 1u, lead);
                        } else {
                            mma_row<0, kPlane, 32u * RA>(d, a + dy0, b, acc, lead);
                            if (dy1 != dy0) mma_row<0, kPlane, 32u * RA>(d, a + dy1, b, 1u, lead);
                        }
                        acc = 1;
                        commit(&sh.t_empty[st], lead);
                    }
                    if (++st == kStages<P>) st = 0, ph ^= 1u;
                }
                if (ok) commit(&sh.d_full[db], lead);
            }
            if (ok) commit(&sh.a_empty[buf], lead);
        }
    } else {
        // ---- Epilogue: growth sums of row y0 + 32 (warp % 4) + lane, columns
        // x0 + kPart (warp / 4) .. + kPart - 1, over the kernels; then A'.
        fastfft::grid_dependency_wait();
        const int quad = warp & 3, half = warp >> 2;
        const uint32_t mine = tmem + (uint32_t(32 * quad) << 16) + uint32_t(kPart * half);
        const EulerStep euler(p);
        const bool jitter = p.mu_jitter > 0.0f;
        // Selects instead of a dynamic index into the parameter block (which
        // would spill it to local memory).
        const auto pick = [](const float(&a)[kMaxKernels], int k) {
            return k == 0 ? a[0] : k == 1 ? a[1] : k == 2 ? a[2] : a[3];
        };
        uint32_t ai = 0, di = 0;
        bool ok = true;
        for (int tile = int(blockIdx.x); tile < tiles && ok; tile += int(gridDim.x), ++ai) {
            const int ty = tile / tiles_x, gx0 = (tile - ty * tiles_x) * kTX + kPart * half;
            const int gy = ty * kRows + 32 * quad + lane;
            // This thread's values of A, requested before the products are waited
            // for (rows past the field read its last one). Rows that start
            // anywhere in a quad are read two rows by 16 values an access and
            // turned to one row a thread below.
            const int gq = ty * kRows + 32 * quad;  // the warp's first row
            float av[kPart];
            const bool whole = W % 4 == 0 && gx0 + kPart <= W;
            if (whole) {
                const float4* arow = reinterpret_cast<const float4*>(src + size_t(min(gy, H - 1)) * W + gx0);
#pragma unroll
                for (int c = 0; c < kPart / 4; ++c) {
                    const float4 a = __ldg(arow + c);
                    av[4 * c] = a.x, av[4 * c + 1] = a.y, av[4 * c + 2] = a.z, av[4 * c + 3] = a.w;
                }
            } else {
                const int x = gx0 + (lane & 15);
#pragma unroll
                for (int c = 0; c < kPart; ++c)
                    av[c] = x < W ? __ldg(src + size_t(min(gq + 2 * c + (lane >> 4), H - 1)) * W + x) : 0.0f;
            }
            float sum[kPart] = {};  // growth sums
            bool bytes = true;      // no value of the tile's halo outside the byte form
#pragma unroll 1
            for (int k = 0; k < nk; ++k, ++di) {
                const uint32_t db = di % kBufs;
                if (!(ok = bar_wait(&sh.d_full[db], (di / kBufs) & 1u, &sh.stop))) break;
                fence_after();
                bytes = *reinterpret_cast<volatile int*>(&sh.bad[ai & 3u]) != int(ai) + 1;
                const float scale = pick(plan.scale, k);
                const float s0 = scale * 512.0f, s1 = scale * 2.0f;
                const float mu = pick(p.mu, k), sigma = pick(p.sigma, k), weight = pick(p.weight, k);
                // T blocks of kernel k: the issuing warps that had one.
                const int blocks = plan.first[k + 1] - plan.first[k];
                float u[kPart];
#pragma unroll
                for (int c = 0; c < kPart; c += 4) {
                    int32_t l0[4] = {}, l1[4] = {}, l2[4] = {}, l3[4] = {};
#pragma unroll
                    for (int m = 0; m < kMmaWarps; ++m) {
                        if (m >= blocks) break;
                        const uint32_t d = mine + (db * kMmaWarps + uint32_t(m)) * kAccCols + uint32_t(c);
                        int32_t x00[4], x01[4], x02[4], x11[4], x12[4], x13[4], x22[4], x23[4];  // X's byte, level
                        tmem_ld4(d, x00);
                        tmem_ld4(d + kTX, x01);
                        tmem_ld4(d + 2 * kTX, x02);
                        tmem_ld4(d + kAccX1, x11);
                        tmem_ld4(d + kAccX1 + kTX, x12);
                        tmem_ld4(d + kAccX1 + 2 * kTX, x13);
                        tmem_ld4(d + kAccX2, x22);
                        tmem_ld4(d + kAccX2 + kTX, x23);
                        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            l0[j] += x00[j];
                            l1[j] += x01[j] + x11[j];
                            l2[j] += x02[j] + x12[j] + x22[j];
                            l3[j] += x13[j] + x23[j];
                        }
                    }
                    // Levels 2 and 3 join level 1 as integers (rounded at 2^-31 of the sum).
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int32_t v2 = l2[j] + ((l3[j] + 128) >> 8);
                        const int32_t v1 = l1[j] + ((v2 + 128) >> 8);
                        u[c + j] = fmaf(float(l0[j]), s0, float(v1) * s1);
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) bar_arrive(&sh.d_empty[db]);
#pragma unroll
                for (int j = 0; j < kPart / 2; ++j) {
                    const float2 shift = jitter ? mu_jitter_pair(p, sh.ex, uint32_t(gx0 + 2 * j), uint32_t(gy))
                                                : make_float2(0.0f, 0.0f);
                    sum[2 * j] = growth_add(sum[2 * j], weight, bell(u[2 * j], mu + shift.x, sigma), euler.asym);
                    sum[2 * j + 1] =
                        growth_add(sum[2 * j + 1], weight, bell(u[2 * j + 1], mu + shift.y, sigma), euler.asym);
                }
            }
            if (!ok) break;  // its tile is left unwritten
            if (!bytes) {    // for every warp of the tile: the rows are shared out anew
                fp32_rows(src, dst, weights, spans, g, p, sh.ex, nk, gx0 - kPart * half, gq + kFpRows * half);
                continue;
            }
            float* rows = reinterpret_cast<float*>(ring + kStages<P> * kStage) + warp * (32 * kTurn);
            float4* own = reinterpret_cast<float4*>(rows + lane * kTurn);
            if (!whole) {
#pragma unroll
                for (int c = 0; c < kPart; ++c) rows[(2 * c + (lane >> 4)) * kTurn + (lane & 15)] = av[c];
                __syncwarp();
#pragma unroll
                for (int c = 0; c < kPart / 4; ++c) {
                    const float4 a = own[c];
                    av[4 * c] = a.x, av[4 * c + 1] = a.y, av[4 * c + 2] = a.z, av[4 * c + 3] = a.w;
                }
                __syncwarp();
            }
            euler.divide(sum);
            float4* orow = reinterpret_cast<float4*>(dst + size_t(min(gy, H - 1)) * W + gx0);
#pragma unroll
            for (int c = 0; c < kPart; c += 8) {
                float v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = euler(av[c + j], sum[c + j]);
                noise_inject_clip(p, sh.ex, v, uint32_t(gx0 + c), uint32_t(gy));
                const float4 lo = make_float4(v[0], v[1], v[2], v[3]), hi = make_float4(v[4], v[5], v[6], v[7]);
                if (!whole) {
                    own[c / 4] = lo;
                    own[c / 4 + 1] = hi;
                } else if (gy < H) {
                    orow[c / 4] = lo;
                    orow[c / 4 + 1] = hi;
                }
            }
            if (!whole) {
                const int x = gx0 + (lane & 15);
                __syncwarp();
#pragma unroll
                for (int c = 0; c < kPart; ++c) {
                    const int r = 2 * c + (lane >> 4);
                    if (gq + r < H && x < W) dst[size_t(gq + r) * W + x] = rows[r * kTurn + (lane & 15)];
                }
                __syncwarp();  // the rows are the next tile's
            }
        }
    }
    fence_before();
    __syncthreads();
    if (*reinterpret_cast<volatile int*>(&sh.stop)) {
        // A wait ran out: products still in flight get one more bounded wait
        // before their accumulators are freed.
        if (warp >= kMmaWarp && warp < kMmaWarp + kMmaWarps) {
            int never = 0;
            fence_after();
            commit(&sh.drain[warp - kMmaWarp], elected());
            bar_wait_slow(&sh.drain[warp - kMmaWarp], 0, &never);
        }
        __syncthreads();
    }
    if (warp == kMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols));
    if (tid == 0 && *reinterpret_cast<volatile int*>(&sh.stop) && err) atomicAdd(err, 1);
}

template <int P>
cudaError_t launch_t(int nk, const float* src, float* dst, const DirectTcPlan& plan, const float* weights,
                     const uint32_t* spans, const DirectGeometry& g, const StepParams& p, int* err, cudaStream_t s) {
    auto fn = direct_tc_kernel<P>;
    constexpr size_t smem = 2 * kPlanes * size_t(kRows + 2 * P) * (kTX + 2 * P) + size_t(kStages<P>) * kChunk * (1 + P / 16) +
                            sizeof(float) * kEpiWarps * 32 * kTurn;
    static fastfft::KernelState state;
    int per = 0;
    cudaError_t e = fastfft::prepare(state, fn, kThreads, smem, per);
    if (e != cudaSuccess) return e;
    const int tx = int((p.width + kTX - 1) / kTX), tiles = tx * int((p.height + kRows - 1) / kRows);
    return fastfft::launch_chained(fn, dim3(unsigned(std::min(tiles, fastfft::sms()))), kThreads, smem, s, src, dst,
                                   plan, weights, spans, g, p, nk, tx, tiles, err);
}

}  // namespace

// The T blocks of the kernel tables ((2r + 1)^2 weights each) in the order of
// the plan's rows: per kernel row with a nonzero weight and per chunk, two
// halves of k x 128 rows (32 of zeros, then byte plane j, output n) x 16 values
// of k.
bool direct_tc_tables(const std::vector<std::vector<float>>& luts, int r, DirectTcTables& out) {
    out = DirectTcTables();
    if (r < 0 || r > kMaxRadius || luts.empty() || luts.size() > size_t(kMaxKernels)) return false;
    const int ks = 2 * r + 1;
    int rows = 0;
    for (size_t k = 0; k < luts.size(); ++k) {
        const std::vector<float>& lut = luts[k];
        if (lut.size() != size_t(ks) * ks) return false;
        float top = 0.0f;
        for (float w : lut) {
            if (!std::isfinite(w)) return false;
            top = std::max(top, std::fabs(w));
        }
        // The largest e with top * 2^e within three signed bytes.
        if (!(top > 0.0f)) return false;
        int e = 0;
        std::frexp(8355711.0 / double(top), &e);
        e -= 1;  // 2^e <= 8355711 / top < 2^(e + 1)
        if (e > 100) return false;
        out.plan.scale[k] = float(std::ldexp(1.0, -e));
        out.plan.first[k] = rows;
        double carry = 0.0;
        int taps = 0;
        for (float w : lut) taps += w != 0.0f;
        out.min_taps = k == 0 ? taps : std::min(out.min_taps, taps);
        const auto row_at = [&](int dyi) { return lut.begin() + std::ptrdiff_t(dyi) * ks; };
        for (int dyi = 0; dyi < ks; ++dyi) {
            // Rows dy and -dy of a radial kernel are the same weights and share
            // one T block (the pair runs at the first of them).
            const int twin = 2 * r - dyi;
            const bool same = std::equal(row_at(dyi), row_at(dyi) + ks, row_at(twin));
            if (same && twin < dyi) continue;
            int hw = -1;
            std::vector<int32_t> wi(size_t(ks), 0);
            for (int dx = -r; dx <= r; ++dx) {
                // Rounded with the error of the weights before it, so that the
                // table's sum (1, or the scene's) is kept.
                const double w = std::ldexp(double(lut[size_t(dyi) * ks + size_t(dx + r)]), e);
                if (w == 0.0) continue;
                const double x = std::min(std::max(w + carry, -8355711.0), 8355711.0);
                const int32_t v = int32_t(std::llrint(x));
                carry += w - double(v);
                wi[size_t(dx + r)] = v;
                if (v != 0) hw = std::max(hw, std::abs(dx));
            }
            if (hw < 0) continue;
            const int nq = (hw + 15) / 16;
            const size_t at = out.blocks.size();
            out.blocks.resize(at + size_t(1 + nq) * kChunk, 0);
            for (int c = 0; c <= nq; ++c)
                for (int n = 0; n < kTX; ++n)
                    for (int kk = 0; kk < 32; ++kk) {
                        const int dx = 32 * c - 16 * nq + kk - n;
                        if (dx < -hw || dx > hw) continue;
                        const int32_t v = wi[size_t(dx + r)];
                        // Signed bytes: v = d0 2^16 + d1 2^8 + d2, each in [-128, 127].
                        const int32_t d2 = int32_t(int8_t(v & 0xFF)), v1 = (v - d2) / 256;
                        const int32_t d1 = int32_t(int8_t(v1 & 0xFF)), d0 = (v1 - d1) / 256;
                        const int32_t d[3] = {d0, d1, d2};
                        for (int j = 0; j < 3; ++j)
                            out.blocks[at + size_t(c) * kChunk + size_t(kk / 16) * (kChunk / 2) +
                                       kZeros + size_t(j * kTX + n) * 16 + size_t(kk % 16)] = uint8_t(int8_t(d[j]));
                    }
            out.chunks += (1 + nq) * (same && twin != dyi ? 2 : 1);
            out.plan.rows[rows++] = uint16_t(dyi | ((same ? twin : dyi) << 7) | (nq << 14));
        }
    }
    for (size_t k = luts.size(); k <= size_t(kMaxKernels); ++k) out.plan.first[k] = rows;
    return true;
}

// Frame times in us as measured back to back on a B200 (148 SMs), one kernel:
//                      R = 3        5        9        13       20       32
//   128 x 128   FP32    7.2      8.2      8.2      10.2     12.3     20.5
//               bytes   9.9     10.7     12.4      14.2     22.8     31.6
//   512 x 512   FP32    8.2     10.2     14.3      16.3     26.6     61.4
//               bytes  10.2     11.0     12.7      14.5     23.3     32.0
//   1001 x 703  FP32   12.2     15.3     25.0      38.7     63.5    133.1
//               bytes  15.2     16.0     19.1      22.6     37.1     55.4
//   1280 x 720  FP32   11.2     16.4     28.6      43.0     76.5    182.3
//               bytes  14.3     14.9     17.9      21.5     35.6     53.7
//   1920 x 1080 FP32   16.6     26.6     45.8      71.6    133.1    311.4
//               bytes  22.1     22.6     28.0      34.7     59.6     94.8
// (before the byte form the FP32 column was 205 us at 1280 x 720, R = 32 and 81
// at 1920 x 1080, R = 13). Both sides are modelled from them, within 10 % from R
// = 9 on: the byte form by a fixed 8.3 us (12 above R = 16, whose tiles stage a
// wider halo: launch, first tile's staging, last epilogue) and, per round of
// tiles over the SMs, the larger of the products (107 ns a chunk, and 0.9 us to
// read the sums, which the next products wait for) and the staging and epilogue
// (3.3 us); the FP32 form by its 8-tap multiply-adds (3.7e-8 us each on fields that
// fill the SMs evenly, from 2 million pixels on, up to 4.8e-8 below) and 5e-6 us a
// pixel. A CTA of the byte form holds its SM's tensor memory, so kernels of other
// contexts fill only the SMs it leaves free: the time a frame costs beside
// others (its share of the SMs, three quarters of it overlapped at best) counts
// as much as its own, and its own is at most a tenth longer. Two substeps of
// 1001 x 703, R = 9 with noise, jitter and blobs, FP32 / bytes: alone 57.8 / 48.8
// us, beside two others 33.8 / 32.9.
// Kernels of few taps stay on the FP32 form, whose rounding grows with the taps
// while the byte form's is fixed (they cross at R = 4, 49 taps).
bool direct_tc_faster(const DirectTcTables& t, uint64_t fp32_taps, int r, int w, int h, int sms) {
    if (t.min_taps < 60) return false;
    const double px = double(w) * h;
    const int tiles = ((w + kTX - 1) / kTX) * ((h + kRows - 1) / kRows), rounds = (tiles + sms - 1) / std::max(1, sms);
    const double bytes = (r <= 16 ? 8.3 : 12.0) + rounds * std::max(0.107 * t.chunks + 0.9, 3.3);
    const double share = 0.75 * bytes * std::min(1.0, double(tiles) / std::max(1, sms));
    const double work = px * (double(fp32_taps) * 3.7e-8 + 5e-6);  // of the FP32 form, the SMs full
    const double tap = 3.7e-8 + 1.1e-8 * std::min(1.0, std::max(0.0, (2.0e6 - px) / 1.1e6));
    const double fp32 = 7.0 + px * (double(fp32_taps) * tap + 5e-6);
    return bytes + share < fp32 + work && bytes < 1.1 * fp32;
}

// U is off by up to 2^-32 where FP32 values are fainter than 2^-8; FP32 rounds
// U - mu at 2^-25 |mu| or more there (at mu = 2^-6 twice the former).
bool direct_tc_holds(int nk, const StepParams& p) {
    for (int k = 0; k < nk; ++k)
        if (!(std::fabs(p.mu[k]) >= 0.015625f)) return false;
    return true;
}

cudaError_t launch_direct_tc(int nk, const float* src, float* dst, const DirectTcPlan& plan, const float* weights,
                             const uint32_t* spans, const DirectGeometry& g, const StepParams& p, int* err,
                             cudaStream_t s) {
    if (nk < 1 || nk > kMaxKernels) return cudaErrorInvalidValue;
    return g.r <= 16 ? launch_t<16>(nk, src, dst, plan, weights, spans, g, p, err, s)
                     : launch_t<32>(nk, src, dst, plan, weights, spans, g, p, err, s);
}

}  // namespace lenia
