// fft_len1.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(25) X(42) X(63) X(90) X(125) X(160) X(200) X(250) X(315) X(378) X(448)
#define CRAVA_ROWS(X) \
  X(36) X(64) X(75) X(100) X(150) X(210) X(225) X(280) X(360) X(450)

CRAVA_LENGTHS(1)
