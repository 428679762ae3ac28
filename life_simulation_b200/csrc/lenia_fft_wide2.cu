// life_simulation_b200/csrc/lenia_fft_wide2.cu -- part 2 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_2
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_2
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_2
#include "lenia_fft_wide_part.cuh"
