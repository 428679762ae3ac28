// life_simulation_b200/csrc/lenia_fft_wide1.cu -- part 1 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_1
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_1
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_1
#include "lenia_fft_wide_part.cuh"
