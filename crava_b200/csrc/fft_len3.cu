// fft_len3.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(28) X(48) X(70) X(98) X(128) X(168) X(216) X(256) X(324) X(392) X(480)
#define CRAVA_ROWS(X) \
  X(42) X(49) X(72) X(112) X(162) X(175) X(224) X(294) X(384) X(486)

CRAVA_LENGTHS(3)
