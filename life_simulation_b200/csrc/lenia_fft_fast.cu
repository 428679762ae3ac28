// life_simulation_b200/csrc/lenia_fft_fast.cu -- the spectral path's column
// and row passes for field sizes with a compile-time FFT plan (the sizes of
// the benchmark configs and common sim resolutions; the other lengths with
// factors 2, 3 and 5 are lenia_fft_wide*.cu's, the rest lenia_fft.cu's).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "lenia_fft_wide.cuh"

namespace lenia {

bool fast_col_plan(int H, FastPlan& fwd) {
    switch (H) {
#define X(n, ...) \
    case n: plan_radices<__VA_ARGS__>(fwd); return true;
        LENIA_COL_PLANS(X)
#undef X
    default: return false;
    }
}

bool fast_row_plan(int M, FastPlan& inv) {
    switch (M) {
#define X(n, ...) \
    case n: plan_radices<__VA_ARGS__>(inv); return true;
        LENIA_ROW_PLANS(X)
#undef X
    default: return false;
    }
}

// Per-pass twiddles of a plan in the device layout: for pass p >= 1 with
// span Ns and radix R, entry [(t-1)*Ns + m] = exp(-2 pi i m t / (Ns R)).
void fast_plan_twiddles(const FastPlan& plan, std::vector<float2>& out) {
    out.clear();
    int ns = plan.radix[0];
    for (int p = 1; p < plan.np; ++p) {
        const int r = plan.radix[p];
        for (int t = 1; t < r; ++t)
            for (int m = 0; m < ns; ++m) {
                const double a = 2.0 * M_PI * double(m) * double(t) / double(ns * r);
                out.push_back(make_float2(float(std::cos(a)), float(-std::sin(a))));
            }
        ns *= r;
    }
}

bool fast_twiddle_tables(int H, int M, std::vector<float2> (&out)[4]) {
    FastPlan cf, ri;
    if (!fast_col_plan(H, cf) || !fast_row_plan(M, ri)) return false;
    FastPlan rcf = cf, rri = ri;
    for (int i = 0; i < cf.np; ++i) rcf.radix[i] = cf.radix[cf.np - 1 - i];
    for (int i = 0; i < ri.np; ++i) rri.radix[i] = ri.radix[ri.np - 1 - i];
    const FastPlan* plans[4] = {&cf, &rcf, &ri, &rri};
    for (int q = 0; q < 4; ++q) {
        fast_plan_twiddles(*plans[q], out[q]);
        if (out[q].empty()) out[q].push_back(make_float2(1.0f, 0.0f));
    }
    return true;
}

namespace {

cudaError_t col_dispatch(int H, int M, int batch, const SpectralWorld& w0, const SpectralWorld* worlds, int n,
                         const FastTables& t, cudaStream_t s) {
    switch (H) {
#define X(h, ...)                                                                                  \
    case h:                                                                                        \
        if (batch == (4 | kHalfThreads)) return launch_col_t<__VA_ARGS__, 4, 2>(w0, worlds, n, M, t, s); \
        if (batch == 8) return launch_col_t<__VA_ARGS__, 8>(w0, worlds, n, M, t, s);               \
        if (batch == 4) return launch_col_t<__VA_ARGS__, 4>(w0, worlds, n, M, t, s);               \
        return launch_col_t<__VA_ARGS__, 2>(w0, worlds, n, M, t, s);
        LENIA_COL_PLANS(X)
#undef X
    default: return cudaErrorNotSupported;
    }
}

// CM: the variant that also writes the colour layer (w0.rgba); the other
// launches use the one compiled without that store, which would otherwise
// cost every row pass a few per cent.
template <bool CM>
cudaError_t row_dispatch_t(int H, int M, int batch, const SpectralWorld& w0, const SpectralWorld* worlds, int n,
                           const float2* tw_r2c, const FastTables& t, cudaStream_t s) {
    const int rb = batch & 7;
    const bool pipe = (batch & kRowPipelined) != 0;
    if (batch & kHalfThreads) return cudaErrorInvalidConfiguration;  // columns only
    switch (M) {
#define X(m, ...)                                                                                      \
    case m:                                                                                            \
        if (pipe) {                                                                                    \
            if (rb == 4) return launch_row_t<__VA_ARGS__, 4, true, CM>(w0, worlds, n, H, tw_r2c, t, s); \
            if (rb == 2) return launch_row_t<__VA_ARGS__, 2, true, CM>(w0, worlds, n, H, tw_r2c, t, s); \
            return launch_row_t<__VA_ARGS__, 1, true, CM>(w0, worlds, n, H, tw_r2c, t, s);              \
        }                                                                                              \
        if (rb == 4) return launch_row_t<__VA_ARGS__, 4, false, CM>(w0, worlds, n, H, tw_r2c, t, s);    \
        if (rb == 2) return launch_row_t<__VA_ARGS__, 2, false, CM>(w0, worlds, n, H, tw_r2c, t, s);    \
        return launch_row_t<__VA_ARGS__, 1, false, CM>(w0, worlds, n, H, tw_r2c, t, s);
        LENIA_ROW_PLANS(X)
#undef X
    default: return cudaErrorNotSupported;
    }
}

cudaError_t row_dispatch(int H, int M, int batch, const SpectralWorld& w0, const SpectralWorld* worlds, int n,
                         const float2* tw_r2c, const FastTables& t, cudaStream_t s) {
    if (w0.rgba && !worlds) return row_dispatch_t<true>(H, M, batch, w0, worlds, n, tw_r2c, t, s);
    return row_dispatch_t<false>(H, M, batch, w0, worlds, n, tw_r2c, t, s);
}

template <class PF, int B, int S = 1>
bool col_shape_ok() {
    using K = ColK<PF, B, S>;
    return K::T <= 1024 && ColStage<PF, B, S>::smem() <= 227 * 1024;
}

template <class PI, int RB, bool PIPE, int S = 1>
bool row_shape_ok() {
    using K = RowK<PI, RB, S>;
    return K::T <= 1024 && K::smem(PIPE ? 3 : 2) <= 227 * 1024;
}

}  // namespace

bool fast_shapes_supported(int H, int M, int col_batch, int row_batch) {
    bool col = false, row = false;
    switch (H) {
#define X(h, ...)                                                        \
    case h:                                                              \
        col = col_batch == 8                    ? col_shape_ok<__VA_ARGS__, 8>()    \
              : col_batch == 4                  ? col_shape_ok<__VA_ARGS__, 4>()    \
              : col_batch == (4 | kHalfThreads) ? col_shape_ok<__VA_ARGS__, 4, 2>() \
              : col_batch == 2                  ? col_shape_ok<__VA_ARGS__, 2>() : false; \
        break;
        LENIA_COL_PLANS(X)
#undef X
    default: break;
    }
    const int rb = row_batch & 7;
    const bool pipe = (row_batch & kRowPipelined) != 0;
    if ((row_batch & ~(kRowPipelined | 7)) != 0) return false;
    switch (M) {
#define X(m, ...)                                                                                      \
    case m:                                                                                            \
        row = pipe ? (rb == 4   ? row_shape_ok<__VA_ARGS__, 4, true>()                                 \
                      : rb == 2 ? row_shape_ok<__VA_ARGS__, 2, true>()                                 \
                      : rb == 1 ? row_shape_ok<__VA_ARGS__, 1, true>() : false)                        \
                   : (rb == 4   ? row_shape_ok<__VA_ARGS__, 4, false>()                                \
                      : rb == 2 ? row_shape_ok<__VA_ARGS__, 2, false>()                                \
                      : rb == 1 ? row_shape_ok<__VA_ARGS__, 1, false>() : false);                      \
        break;
        LENIA_ROW_PLANS(X)
#undef X
    default: break;
    }
    return col && row;
}

namespace {

SpectralWorld col_world(const FftGeometry& g, const float2* S, float2* U) {
    SpectralWorld w{};
    w.S = S;
    w.U = U;
    w.khat = g.khat;
    w.M = g.M;
    w.nk = g.nk;
    return w;
}

SpectralWorld row_world(const FftGeometry& g, const float2* U, const float* A, float* A_out, float2* S_next,
                        const StepParams& p, int nk, void* rgba16f, const ColorMapParams* cm) {
    SpectralWorld w{};
    if (rgba16f && cm && nk > 0) {
        w.rgba = static_cast<uint2*>(rgba16f);
        w.cm = *cm;
    }
    w.U = const_cast<float2*>(U);  // read only by the row pass
    w.A = A;
    w.A_out = A_out;
    w.S_next = S_next;
    w.M = g.M;
    w.nk = nk;
    w.p = p;
    w.p.height = uint32_t(g.H);
    return w;
}

}  // namespace

cudaError_t launch_col_fast(const FftGeometry& g, const FastTables& t, int batch, const float2* S,
                            float2* U, cudaStream_t s) {
    return col_dispatch(g.H, g.M, batch, col_world(g, S, U), nullptr, 1, t, s);
}

cudaError_t launch_row_fast(const FftGeometry& g, const FastTables& t, int batch, const float2* U,
                            const float* A, float* A_out, float2* S_next, const StepParams& p,
                            int nk, cudaStream_t s, void* rgba16f, const ColorMapParams* cm) {
    return row_dispatch(g.H, g.M, batch, row_world(g, U, A, A_out, S_next, p, nk, rgba16f, cm), nullptr, 1, g.tw_r2c,
                        t, s);
}

bool spectral_col_plan(int H, FastPlan& fwd) {
    if (fast_col_plan(H, fwd)) return true;
#define F(p) \
    if (wide_col_plan_##p(H, fwd)) return true;
    LENIA_WIDE_EACH(F)
#undef F
    return false;
}

bool spectral_row_plan(int M, FastPlan& inv) {
    if (fast_row_plan(M, inv)) return true;
#define F(p) \
    if (wide_row_plan_##p(M, inv)) return true;
    LENIA_WIDE_EACH(F)
#undef F
    return false;
}

cudaError_t launch_col_wide(const FftGeometry& g, const FastTables& t, int shape, const float2* S, float2* U,
                            cudaStream_t s) {
    const SpectralWorld w = col_world(g, S, U);
    FastPlan catalogue;
    if (fast_col_plan(g.H, catalogue)) return col_dispatch(g.H, g.M, shape == 0 ? 4 : 2, w, nullptr, 1, t, s);
    cudaError_t e = cudaErrorNotSupported;
#define F(p) \
    if (e == cudaErrorNotSupported) e = wide_col_##p(g.H, shape, w, t, s);
    LENIA_WIDE_EACH(F)
#undef F
    return e;
}

cudaError_t launch_row_wide(const FftGeometry& g, const FastTables& t, int shape, const float2* U, const float* A,
                            float* A_out, float2* S_next, const StepParams& p, int nk, cudaStream_t s, void* rgba16f,
                            const ColorMapParams* cm) {
    const SpectralWorld w = row_world(g, U, A, A_out, S_next, p, nk, rgba16f, cm);
    FastPlan catalogue;
    if (fast_row_plan(g.M, catalogue)) return wide_row_mixed(g.M, g.H, shape, w, g.tw_r2c, t, s);
    cudaError_t e = cudaErrorNotSupported;
#define F(p_) \
    if (e == cudaErrorNotSupported) e = wide_row_##p_(g.M, g.H, shape, w, g.tw_r2c, t, s);
    LENIA_WIDE_EACH(F)
#undef F
    return e;
}

cudaError_t launch_col_fast_worlds(int H, int M, const FastTables& t, int batch, const SpectralWorld* worlds,
                                   int n, cudaStream_t s) {
    return col_dispatch(H, M, batch, SpectralWorld{}, worlds, n, t, s);
}

cudaError_t launch_row_fast_worlds(int H, int M, const FastTables& t, const float2* tw_r2c, int batch,
                                   const SpectralWorld* worlds, int n, cudaStream_t s) {
    return row_dispatch(H, M, batch, SpectralWorld{}, worlds, n, tw_r2c, t, s);
}

}  // namespace lenia
