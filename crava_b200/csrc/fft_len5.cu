// fft_len5.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(32) X(50) X(75) X(105) X(140) X(180) X(225) X(280) X(343) X(405) X(490)
#define CRAVA_ROWS(X) \
  X(35) X(50) X(84) X(126) X(135) X(180) X(250) X(320) X(400) X(500)

CRAVA_LENGTHS(5)
