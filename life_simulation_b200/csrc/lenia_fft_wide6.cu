// life_simulation_b200/csrc/lenia_fft_wide6.cu -- part 6 of the wide lengths
// (lenia_fft_wide.cuh).
#define LENIA_WIDE_NAME(f) f##_6
#define LENIA_WIDE_COLS LENIA_WIDE_COLS_6
#define LENIA_WIDE_ROWS LENIA_WIDE_ROWS_6
#include "lenia_fft_wide_part.cuh"
