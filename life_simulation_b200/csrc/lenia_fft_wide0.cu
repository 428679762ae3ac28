// life_simulation_b200/csrc/lenia_fft_wide0.cu -- part 0 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_0
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_0
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_0
#include "lenia_fft_wide_part.cuh"
