// life_simulation_b200/csrc/lenia_fft_wide3.cu -- part 3 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_3
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_3
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_3
#include "lenia_fft_wide_part.cuh"
