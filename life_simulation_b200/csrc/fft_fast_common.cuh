// life_simulation_b200/csrc/fft_fast_common.cuh -- shared pieces of the
// compile-time-plan spectral kernels (forward step, adjoint step): the
// Stockham pass runner over a batch of transforms, the shared-memory pitch,
// table copies and 16-byte asynchronous copies.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "fft_ct.cuh"
#include "lenia_kernels.h"

namespace lenia {
namespace fastfft {

using namespace fftct;

constexpr int KB = kSpectralBlock;  // columns per block of the blocked layout

constexpr int roundup32(int x) { return (x + 31) / 32 * 32; }

// Blocks of a half spectrum of M columns (the last one padded when M is not
// a whole number of blocks), and the columns a plane then holds.
constexpr __host__ __device__ int blocks_of(int M) { return (M + KB - 1) / KB; }
constexpr __host__ __device__ int padded_columns(int M) { return blocks_of(M) * KB; }

// Row pitch of a batch of B transforms of n elements (float2), even. Shared
// memory serves an 8-byte access half a warp at a time: 16 / B consecutive
// elements of each of the B transforms, which cover the 32 banks once when
// transforms start 32 / B banks apart (an 8-bank start for every B left B = 2
// with two-way conflicts on every access: 4096 x 4096, three kernels, column
// pass of two columns 201 -> 184 us, row pass of two rows 194 -> 174 us).
constexpr int row_pitch(int n, int B = 4) {
    const int start = B == 2 ? 16 : B == 8 ? 4 : 8;
    int p = n + (n & 1);
    if (B == 1) return p;
    while ((2 * p) % 32 != start) ++p;
    return p;
}

// Element order of a first pass's output. Its items write R consecutive
// elements each in 16-byte pairs, eight lanes at a time, and when R is a
// multiple of 4 those lanes' pairs start on the same few bank quads: two-way
// conflicts at B = 4, four-way at B = 2, eight-way (R = 16) at one row. So
// element i goes to i ^ x(i), x a multiple of 2 that differs between the
// colliding lanes, and the pass that reads it applies the same: x(i) depends
// on i / R, which the reading items (i = j + t * N / R1, N / R1 a multiple of
// R) mostly know from j alone. Half-warps of 8-byte reads stay within runs
// that x permutes, so they are conflict-free as before.
template <class P, int B>
struct FirstPassOrder {
    static constexpr int R = P::radix(0);
    static constexpr int SHIFT = B == 1 ? 4 : R == 16 ? 4 : R == 8 ? 3 : 2;
    static constexpr int MASK = B == 1 ? 7 : B == 2 ? 3 : 1;
    static constexpr int N1 = P::n / P::radix(P::np > 1 ? 1 : 0);  // stride of the reading pass's inputs
    static constexpr bool on = P::np > 1 && (B == 1 || B == 2 || B == 4) && (R == 4 || R == 8 || R == 16) &&
                               N1 % (1 << SHIFT) == 0 && P::n % (2 * (MASK + 1)) == 0;  // x stays inside the row
    // Whether x is the same for all of a reading item's inputs.
    static constexpr bool fixed = on && (N1 >> SHIFT) % (MASK + 1) == 0;
    __device__ __forceinline__ static int x(int i) { return on ? ((i >> SHIFT) & MASK) << 1 : 0; }
};
// Input t of item j of pass PASS, in the order its buffer holds: pass 1 reads
// a first pass's output.
template <class P, int PASS, int B>
__device__ __forceinline__ int pass_in(int j, int t) {
    using I = PassIdx<P, PASS>;
    using O = FirstPassOrder<P, B>;
    if constexpr (PASS == 1 && O::on) {
        if constexpr (O::fixed) return (j ^ O::x(j)) + t * I::NR;
        const int i = j + t * I::NR;
        return i ^ O::x(i);
    }
    return I::in(j, t);
}

// One Stockham pass over a batch of B transforms: item q -> (b = q % B,
// j = q / B). All of a thread's items are loaded first, then twiddled,
// transformed and stored. src(b, i) / dst(b, i, v) address element i of
// transform b (of pass 1 in FirstPassOrder, i. e. of a buffer that store_run
// filled).
template <class P, int PASS, bool INV, int B, int T, class Src, class Dst>
__device__ __forceinline__ void pass_gen(Src&& src, Dst&& dst, const float2* __restrict__ tw, int cols) {
    using I = PassIdx<P, PASS>;
    constexpr int TOT = B * I::NR;
    constexpr int ITEMS = (TOT + T - 1) / T;
    float2 v[ITEMS][I::R];
    int jj[ITEMS], bi[ITEMS];
    bool ok[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const int q = int(threadIdx.x) + it * T;
        jj[it] = q / B;
        bi[it] = q - jj[it] * B;
        ok[it] = (TOT % T == 0 || q < TOT) && bi[it] < cols;
        if (ok[it]) {
#pragma unroll
            for (int t = 0; t < I::R; ++t) v[it][t] = src(bi[it], pass_in<P, PASS, B>(jj[it], t));
        }
    }
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        if (ok[it]) {
            I::template twiddle<INV>(v[it], jj[it], tw);
            Dft<I::R, INV>::run(v[it]);
            const int ob = I::out_base(jj[it]);
#pragma unroll
            for (int t = 0; t < I::R; ++t) dst(bi[it], ob + t * I::NS, v[it][t]);
        }
    }
}

// The R outputs of item j of plan P's first pass (span 1) are the R
// consecutive elements from j * R on: written two at a time (16-byte stores,
// half the store instructions and shared-memory wavefronts) when R is even, in
// FirstPassOrder. `row` must be 16-byte aligned when R is even (shared buffers
// at even float2 offsets, even pitches).
template <class P, int B>
__device__ __forceinline__ void store_run(float2* row, int j, const float2* v) {
    using O = FirstPassOrder<P, B>;
    constexpr int R = P::radix(0);
    if constexpr (R % 2 == 0) {
        // An item's R elements share x: 2t ^ x within its (aligned) run, or
        // the whole run moved when x reaches past it (R = 4 or 8 at one row).
        const int base = j * R, x = O::x(base);
#pragma unroll
        for (int t = 0; t < R / 2; ++t)
            *reinterpret_cast<float4*>(row + ((base + 2 * t) ^ x)) =
                make_float4(v[2 * t].x, v[2 * t].y, v[2 * t + 1].x, v[2 * t + 1].y);
    } else {
#pragma unroll
        for (int t = 0; t < R; ++t) row[j * R + t] = v[t];
    }
}

// Pass 0 (span 1) of plan P over a batch of B transforms into the shared
// buffer `buf` (row pitch PITCH, even): pass_gen with store_run's stores.
template <class P, bool INV, int B, int T, int PITCH, class Src>
__device__ __forceinline__ void pass0_buf(Src&& src, float2* buf, int cols) {
    using I = PassIdx<P, 0>;
    static_assert(I::NS == 1, "the first pass has span 1");
    constexpr int TOT = B * I::NR;
    constexpr int ITEMS = (TOT + T - 1) / T;
    float2 v[ITEMS][I::R];
    int jj[ITEMS], bi[ITEMS];
    bool ok[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const int q = int(threadIdx.x) + it * T;
        jj[it] = q / B;
        bi[it] = q - jj[it] * B;
        ok[it] = (TOT % T == 0 || q < TOT) && bi[it] < cols;
        if (ok[it]) {
#pragma unroll
            for (int t = 0; t < I::R; ++t) v[it][t] = src(bi[it], I::in(jj[it], t));
        }
    }
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        if (ok[it]) {
            Dft<I::R, INV>::run(v[it]);
            store_run<P, B>(buf + bi[it] * PITCH, jj[it], v[it]);
        }
    }
}

// Passes PASS..LAST-1 between two shared buffers (barrier after each);
// returns the buffer that holds the data afterwards.
template <class P, int PASS, int LAST, bool INV, int B, int T, int PITCH>
__device__ __forceinline__ float2* mid_passes(float2* a, float2* b, const float2* __restrict__ tw, int cols) {
    if constexpr (PASS < LAST) {
        pass_gen<P, PASS, INV, B, T>([&](int bb, int i) { return a[bb * PITCH + i]; },
                                     [&](int bb, int i, float2 v) { b[bb * PITCH + i] = v; }, tw, cols);
        __syncthreads();
        return mid_passes<P, PASS + 1, LAST, INV, B, T, PITCH>(b, a, tw, cols);
    } else {
        return a;
    }
}

__device__ __forceinline__ void copy_table(float2* dst, const float2* __restrict__ src, int n) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
}

// Asynchronous 16-byte global -> shared copy (completion: cp.async.wait_all,
// a hardware wait, then a block barrier).
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Launch geometry of a column pass over B columns per CTA iteration (forward
// plan PF; the inverse is PF reversed): T threads, ITL last-pass items per
// thread, shared buffers of pitch PITCH. S = 2 halves the thread count (each
// thread takes two last-pass items): fewer warps per CTA, twice the
// independent work per thread, and CTAs small enough for two per SM.
template <class PF, int B, int S = 1>
struct ColK {
    static_assert(KB % B == 0, "a column group lies inside one block");
    using PI = typename Reverse<PF>::type;
    static constexpr int H = PF::n;
    static constexpr int Hh = H / 2 + 1;
    static constexpr int RL = PF::last();
    static constexpr int NRL = H / RL;
    static constexpr int T = roundup32((B * NRL + S - 1) / S);
    static constexpr int ITL = (B * NRL + T - 1) / T;
    static constexpr int PITCH = row_pitch(H, B);
    // The work buffers start after the twiddle tables at an even float2
    // offset (16-byte aligned, for store_run's paired stores).
    static constexpr int BUF0 = (PF::tw_size() + PI::tw_size() + 1) / 2 * 2;
    static_assert(PITCH % 2 == 0, "column pitch must keep 16-byte alignment");
    static constexpr size_t smem() { return sizeof(float2) * (size_t(BUF0) + 2 * size_t(B) * PITCH + H); }
};

// Launch geometry of a row pass over RB rows per CTA iteration (inverse plan
// PI; the forward is PI reversed); S as for ColK.
template <class PI, int RB, int S = 1>
struct RowK {
    using PF = typename Reverse<PI>::type;
    static constexpr int M = PI::n;
    static constexpr int RC = PI::last();
    static constexpr int NRC = M / RC;
    static constexpr int T = roundup32((RB * NRC + S - 1) / S);
    static constexpr int ITL = (RB * NRC + T - 1) / T;
    static constexpr int PITCH = row_pitch(padded_columns(M), RB);  // even: rows start 16-byte aligned
    // Twiddle tables, then the buffers from an even float2 offset so the
    // 16-byte cp.async destinations are 16-byte aligned.
    static constexpr int TABLES = (M + 1) + PI::tw_size() + PF::tw_size();
    static constexpr int BUF0 = (TABLES + 1) / 2 * 2;
    static_assert(PITCH % 2 == 0, "row pitch must keep 16-byte alignment");
    // Tables plus `nbuf` buffers of RB rows.
    static constexpr size_t smem(int nbuf = 2) { return sizeof(float2) * (size_t(BUF0) + nbuf * size_t(RB) * PITCH); }
};

// Real rows of W = 2M values are transformed as M complex values
// z[n] = x[2n] + i x[2n+1]; the half spectrum X[0..M] is stored as M entries
// with X[0] + i X[M] in column 0 (both are real). twr[k] = exp(-2 pi i k / W).

// Stages rows y0..y0+rows-1 of a blocked-layout plane (H rows, M columns)
// into shared rows of pitch PITCH: per block, rows x 8 columns are
// contiguous (16-byte asynchronous copies, two columns each). The caller
// waits (cp_async_wait_all + barrier).
template <int M, int RB, int T, int PITCH>
__device__ __forceinline__ void stage_rows(float2* dst, const float2* __restrict__ plane, int H, int y0, int rows) {
    for (int q = threadIdx.x; q < blocks_of(M) * RB * (KB / 2); q += T) {
        const int c2 = q % (KB / 2);
        const int b = (q / (KB / 2)) % RB;
        const int kb = q / ((KB / 2) * RB);
        if (b < rows) cp_async16(dst + b * PITCH + kb * KB + 2 * c2, plane + (size_t(kb) * H + y0 + b) * KB + 2 * c2);
    }
}

// Stages rows y0..y0+rows-1 of a row-major real field (W = 2M floats per
// row) into shared rows of pitch PITCH, as M float2 pairs (x[2n], x[2n+1]):
// 16-byte asynchronous copies, or 8-byte ones when M is odd (rows then start
// 8 bytes off every other time). The caller waits.
template <int M, int RB, int T, int PITCH>
__device__ __forceinline__ void stage_field_rows(float2* dst, const float* __restrict__ field, int y0, int rows) {
    if constexpr (M % 2 != 0) {
        for (int q = threadIdx.x; q < RB * M; q += T) {
            const int c = q % M, b = q / M;
            if (b < rows) cp_async8(dst + b * PITCH + c, field + (size_t(y0 + b) * M + c) * 2);
        }
        return;
    }
    for (int q = threadIdx.x; q < RB * (M / 2); q += T) {
        const int c = q % (M / 2), b = q / (M / 2);
        if (b < rows) cp_async16(dst + b * PITCH + 2 * c, field + (size_t(y0 + b) * M + 2 * c) * 2);
    }
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// Waits until at most one committed group of this thread is still in flight.
__device__ __forceinline__ void cp_async_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// Inverse of the real-FFT split for element i of a staged half-spectrum row:
// Z'[k] = (X[k] + conj X[M-k]) + i exp(+2 pi i k/W) (X[k] - conj X[M-k]);
// the length-M inverse transform of Z' gives 2 z[n].
template <int M>
__device__ __forceinline__ float2 c2r_split(const float2* xr, const float2* twr, int i) {
    if (i == 0) {
        const float2 x0 = xr[0];
        return make_float2(x0.x + x0.y, x0.x - x0.y);
    }
    const float2 Xk = xr[i];
    const float2 Xm = fft::cconj(xr[M - i]);
    const float2 D = fft::cmul(fft::cconj(twr[i]), fft::csub(Xk, Xm));
    return fft::cadd(fft::cadd(Xk, Xm), make_float2(-D.y, D.x));
}

// Real-FFT split of the length-M forward transforms Z of `rows` packed real
// rows (shared, pitch PITCH) into half spectra, stored to rows y0.. of a
// blocked-layout plane two columns at a time.
template <int M, int RB, int T, int PITCH>
__device__ __forceinline__ void r2c_store_rows(const float2* Z, const float2* twr, float2* __restrict__ plane, int H,
                                               int y0, int rows) {
    for (int q = threadIdx.x; q < blocks_of(M) * RB * (KB / 2); q += T) {
        const int c2 = q % (KB / 2);
        const int b = (q / (KB / 2)) % RB;
        const int kb = q / ((KB / 2) * RB);
        if (b >= rows || (M % KB != 0 && kb * KB + 2 * c2 >= M)) continue;
        const float2* zr = Z + b * PITCH;
        float2 xv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int k = kb * KB + 2 * c2 + e;
            if (M % 2 != 0 && k >= M) {  // the padding column beside an odd M's last
                xv[e] = make_float2(0.0f, 0.0f);
                continue;
            }
            const float2 Zk = zr[k];
            if (k == 0) {
                xv[e] = make_float2(Zk.x + Zk.y, Zk.x - Zk.y);
            } else {
                const float2 Zc = fft::cconj(zr[M - k]);
                const float2 E = fft::cscale(fft::cadd(Zk, Zc), 0.5f);
                const float2 D = fft::csub(Zk, Zc);
                const float2 O = make_float2(0.5f * D.y, -0.5f * D.x);
                xv[e] = fft::cadd(E, fft::cmul(twr[k], O));
            }
        }
        *reinterpret_cast<float4*>(plane + (size_t(kb) * H + y0 + b) * KB + 2 * c2) =
            make_float4(xv[0].x, xv[0].y, xv[1].x, xv[1].y);
    }
}

// ------------------------------------------------------- launch helpers

inline int sms() {
    static int n = 0;
    if (!n) {
        int d = 0;
        cudaGetDevice(&d);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d);
        if (n <= 0) n = 148;
    }
    return n;
}

// The driver's number of the current CUDA context (0: none, or not told). No two
// contexts of a process share one, not even the primary contexts before and
// after a device reset, which have the same handle.
inline unsigned long long context_id() {
    struct Driver {
        CUresult (*current)(CUcontext*) = nullptr;
        CUresult (*id)(CUcontext, unsigned long long*) = nullptr;
        Driver() {
            void *c = nullptr, *i = nullptr;
            cudaDriverEntryPointQueryResult qc, qi;
            if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &c, cudaEnableDefault, &qc) != cudaSuccess ||
                cudaGetDriverEntryPoint("cuCtxGetId", &i, cudaEnableDefault, &qi) != cudaSuccess || !c || !i ||
                qc != cudaDriverEntryPointSuccess || qi != cudaDriverEntryPointSuccess) {
                cudaGetLastError();
                return;
            }
            current = reinterpret_cast<decltype(current)>(c);
            id = reinterpret_cast<decltype(id)>(i);
        }
    };
    static const Driver driver;
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!driver.id || driver.current(&ctx) != CUDA_SUCCESS || !ctx || driver.id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// Opts a kernel into `smem` (at least `limit`) bytes of dynamic shared memory
// and the largest shared-memory carveout, and gives its resident CTAs per SM at
// `threads` threads. Both belong to the CUDA context: `state` keeps the answer of
// the context that asked last, by its number, so that a context after a device
// reset, or a second one, opts in for itself. Asking the number takes 15 ns; the
// three calls made for every launch are host time that small calls wait for (an
// encode of one substep of 128 x 64 5.9 against 6.6 us, a gradient of four steps
// of 128 x 64 385 against 391 us). Each instantiation launches with one shape, or
// has a state for each and a common `limit`.
struct KernelState {
    std::atomic<unsigned long long> kept{0};  // context number << 8 | resident CTAs; 0: none
};
template <typename F>
cudaError_t prepare(KernelState& state, F fn, int threads, size_t smem, int& per_sm, size_t limit = 0) {
    const unsigned long long id = context_id(), kept = state.kept.load(std::memory_order_acquire);
    if (id != 0 && kept >> 8 == id) {
        per_sm = int(kept & 255u);
        return cudaSuccess;
    }
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(std::max(smem, limit)));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
    state.kept.store(id << 8 | (unsigned(per_sm) & 255u), std::memory_order_release);
    return cudaSuccess;
}

// Programmatic dependent launch. A kernel launched by `launch_chained` may
// start while the kernel before it in the stream is still running: it does
// its data-independent prologue (twiddle tables into shared memory), then
// `grid_dependency_wait` blocks until that kernel has completed and its
// writes are visible. `allow_dependents`, called when a CTA starts its last
// work item, lets the next chained kernel launch once every CTA of this one
// has called it (or exited): the next kernel's CTAs then do their prologue
// while this kernel's last items finish. Every CTA of a chained kernel
// waits before it touches data, so kernel completion stays transitive along
// the stream. Both instructions are no-ops in a kernel launched without the
// attribute.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// LENIA_CHAINED_LAUNCH=0 in the environment turns the attribute off (plain
// stream order), e.g. for tools that serialise launches anyway.
inline bool chained_launch_enabled() {
    static const bool on = [] {
        const char* v = std::getenv("LENIA_CHAINED_LAUNCH");
        return !(v && v[0] == '0' && v[1] == '\0');
    }();
    return on;
}

template <typename... KArgs, typename... Args>
cudaError_t launch_chained(void (*fn)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t s,
                           Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(unsigned(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = chained_launch_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

// Persistent grid over n worlds: grid.y = world, grid.x = CTAs per world
// (the resident CTAs of the device shared out, at most one per group).
// Rounded down: every CTA loops over its share of the pass, so a CTA beyond
// the resident slots would wait for a whole persistent CTA to finish -- a
// second wave as long as the first (e.g. 19 x 32 = 608 CTAs for 592 slots).
inline dim3 world_grid(int per_sm, int groups, int n) {
    const int resident = std::max(1, per_sm) * sms();
    const int x = std::max(1, std::min(groups, resident / std::max(1, n)));
    return dim3(unsigned(x), unsigned(n));
}

// Column plans (forward order) by transform length. The last radix is
// kept small: the column spectrum of the last pass lives in registers.
#define LENIA_COL_PLANS(X)     \
    X(1080, Plan<15, 9, 8>)    \
    X(512, Plan<8, 8, 8>)      \
    X(1024, Plan<16, 8, 8>)    \
    X(4096, Plan<16, 16, 16>)  \
    X(2048, Plan<16, 16, 8>)   \
    X(256, Plan<16, 16>)       \
    X(128, Plan<16, 8>)        \
    X(216, Plan<6, 6, 6>)      \
    X(64, Plan<8, 8>)
// Row plans (inverse order) by M = W/2 (a multiple of 8).
#define LENIA_ROW_PLANS(X)     \
    X(960, Plan<8, 15, 8>)     \
    X(512, Plan<8, 8, 8>)      \
    X(2048, Plan<16, 16, 8>)   \
    X(256, Plan<8, 4, 8>)      \
    X(192, Plan<8, 3, 8>)      \
    X(128, Plan<16, 8>)        \
    X(64, Plan<8, 8>)

}  // namespace fastfft
}  // namespace lenia
