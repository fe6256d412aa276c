// fft_len6.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(35) X(54) X(80) X(108) X(144) X(189) X(240) X(288) X(350) X(420) X(500)
#define CRAVA_ROWS(X) \
  X(27) X(54) X(90) X(125) X(128) X(192) X(252) X(324) X(420) X(504)

CRAVA_LENGTHS(6)
