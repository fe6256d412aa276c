// fft_len0.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(24) X(40) X(60) X(84) X(120) X(150) X(196) X(245) X(300) X(375) X(441) X(512)
#define CRAVA_ROWS(X) \
  X(32) X(60) X(81) X(98) X(144) X(200) X(243) X(270) X(350) X(448)

CRAVA_LENGTHS(0)
