// fft_len7.cu -- an eighth of the compiled lengths of the column passes and
// of the synthetic seismic, and row sizes of the x pass (fft_pass.cuh): all 2, 3, 5, 7-smooth column lengths
// 24 .. 512, even rows 32 .. 512 and odd rows 25 .. 255.
#include "fft_pass.cuh"

#define CRAVA_COLS(X) \
  X(36) X(56) X(81) X(112) X(147) X(192) X(243) X(294) X(360) X(432) X(504)
#define CRAVA_ROWS(X) \
  X(25) X(56) X(96) X(105) X(140) X(196) X(245) X(256) X(336) X(432) X(512)

CRAVA_LENGTHS(7)
