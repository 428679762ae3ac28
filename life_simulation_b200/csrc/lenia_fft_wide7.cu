// life_simulation_b200/csrc/lenia_fft_wide7.cu -- part 7 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_7
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_7
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_7
#include "lenia_fft_wide_part.cuh"
