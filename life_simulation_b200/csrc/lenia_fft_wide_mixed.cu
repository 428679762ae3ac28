// life_simulation_b200/csrc/lenia_fft_wide_mixed.cu -- row passes of fields
// whose half row has a catalogue plan and whose column length is a wide one
// (lenia_fft_wide.cuh).
#include "lenia_fft_wide.cuh"

namespace lenia {
namespace {

template <class PI, bool CM>
cudaError_t mixed_shape(int H, int shape, const SpectralWorld& w, const float2* tw_r2c, const FastTables& t,
                        cudaStream_t s) {
    if (shape == 0) return launch_row_t<PI, 4, true, CM, 1, true>(w, nullptr, 1, H, tw_r2c, t, s);
    return launch_row_t<PI, 2, true, CM, 1, true>(w, nullptr, 1, H, tw_r2c, t, s);
}

}  // namespace

cudaError_t wide_row_mixed(int M, int H, int shape, const SpectralWorld& w, const float2* tw_r2c, const FastTables& t,
                           cudaStream_t s) {
    switch (M) {
#define X(m, ...)                                                                   \
    case m:                                                                         \
        return w.rgba ? mixed_shape<__VA_ARGS__, true>(H, shape, w, tw_r2c, t, s)   \
                      : mixed_shape<__VA_ARGS__, false>(H, shape, w, tw_r2c, t, s);
        LENIA_ROW_PLANS(X)
#undef X
    default: return cudaErrorNotSupported;
    }
}

}  // namespace lenia
