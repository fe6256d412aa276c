// fft_len.cu -- the kernels of one line length, CRAVA_LENGTH: its column passes
// and synthetic seismic, and the x pass of rows of that size.
//
// Compiled once per length.  A module is loaded whole when the first of its
// kernels is used, so a length that shares one with others makes the first call
// of a process wait for all of theirs: with the 89 lengths in 8 modules of 6 MB
// the first 96x200x300 transform took 9.5 ms and a graph over two surveys 20 ms
// to create, with a module each 1.3 and 6 ms.
#include "fft_pass.cuh"

#define CRAVA_JOIN_(a, b) a##b
#define CRAVA_JOIN(a, b) CRAVA_JOIN_(a, b)

namespace crava {

ColLaunch CRAVA_JOIN(col_launch_, CRAVA_LENGTH)() { return run_cols<CRAVA_LENGTH>; }
RowLaunch CRAVA_JOIN(row_launch_, CRAVA_LENGTH)() { return row_of<CRAVA_LENGTH>(); }
SyntLaunch CRAVA_JOIN(synt_launch_, CRAVA_LENGTH)() { return synt_of<CRAVA_LENGTH>(); }

}  // namespace crava
