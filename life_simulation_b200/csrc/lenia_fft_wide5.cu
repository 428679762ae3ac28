// life_simulation_b200/csrc/lenia_fft_wide5.cu -- part 5 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_5
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_5
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_5
#include "lenia_fft_wide_part.cuh"
