// life_simulation_b200/csrc/lenia_fft_wide_part.cuh -- one part of the wide
// lengths: LENIA_WIDE_COLS / LENIA_WIDE_ROWS list its lengths and
// LENIA_WIDE_NAME(f) names its functions (see lenia_fft_wide.cuh).
#include "lenia_fft_wide.cuh"

namespace lenia {

bool LENIA_WIDE_NAME(wide_col_plan)(int H, FastPlan& fwd) {
    switch (H) {
#define X(n) \
    case n: plan_radices<WidePlan<n>>(fwd); return true;
        LENIA_WIDE_COLS(X)
#undef X
    default: return false;
    }
}

bool LENIA_WIDE_NAME(wide_row_plan)(int M, FastPlan& inv) {
    switch (M) {
#define X(n) \
    case n: plan_radices<WidePlan<n>>(inv); return true;
        LENIA_WIDE_ROWS(X)
#undef X
    default: return false;
    }
}

namespace {

template <class PF>
cudaError_t wide_col_shape(int shape, const SpectralWorld& w, const FastTables& t, cudaStream_t s) {
    constexpr int B = wide_cols<PF>();
    if (shape == 0) return launch_col_t<PF, B, wide_split<PF>()>(w, nullptr, 1, w.M, t, s);
    if constexpr (B > 2) return launch_col_t<PF, B / 2>(w, nullptr, 1, w.M, t, s);
    return cudaErrorNotSupported;
}

}  // namespace

cudaError_t LENIA_WIDE_NAME(wide_col)(int H, int shape, const SpectralWorld& w, const FastTables& t, cudaStream_t s) {
    switch (H) {
#define X(n) \
    case n: return wide_col_shape<WidePlan<n>>(shape, w, t, s);
        LENIA_WIDE_COLS(X)
#undef X
    default: return cudaErrorNotSupported;
    }
}

namespace {

template <class PI, bool CM>
cudaError_t wide_row_shape(int H, int shape, const SpectralWorld& w, const float2* tw_r2c, const FastTables& t,
                           cudaStream_t s) {
    constexpr int RB = wide_rows<PI>();
    if (shape == 0) return launch_row_t<PI, RB, true, CM, 1, true>(w, nullptr, 1, H, tw_r2c, t, s);
    if constexpr (RB > 1) return launch_row_t<PI, RB / 2, true, CM, 1, true>(w, nullptr, 1, H, tw_r2c, t, s);
    return cudaErrorNotSupported;
}

}  // namespace

cudaError_t LENIA_WIDE_NAME(wide_row)(int M, int H, int shape, const SpectralWorld& w, const float2* tw_r2c,
                                      const FastTables& t, cudaStream_t s) {
    switch (M) {
#define X(n)                                                                         \
    case n:                                                                          \
        return w.rgba ? wide_row_shape<WidePlan<n>, true>(H, shape, w, tw_r2c, t, s) \
                      : wide_row_shape<WidePlan<n>, false>(H, shape, w, tw_r2c, t, s);
        LENIA_WIDE_ROWS(X)
#undef X
    default: return cudaErrorNotSupported;
    }
}

}  // namespace lenia
