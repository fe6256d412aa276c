// fft_len2.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(27) X(45) X(64) X(96) X(126) X(162) X(210) X(252) X(320) X(384) X(450)
#define CRAVA_ROWS(X) \
  X(40) X(63) X(70) X(108) X(160) X(189) X(216) X(288) X(378) X(480)

CRAVA_LENGTHS(2)
