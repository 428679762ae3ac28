// life_simulation_b200/csrc/lenia_fft_wide4.cu -- part 4 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_4
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_4
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_4
#include "lenia_fft_wide_part.cuh"
