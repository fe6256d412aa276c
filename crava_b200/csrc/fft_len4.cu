// fft_len4.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(30) X(49) X(72) X(100) X(135) X(175) X(224) X(270) X(336) X(400) X(486)
#define CRAVA_ROWS(X) \
  X(45) X(48) X(80) X(120) X(147) X(168) X(240) X(300) X(392) X(490)

CRAVA_LENGTHS(4)
