// fft_banks.cuh -- shared-memory layout of the rows of the x pass.
//
// A row of N points in shared memory has its first digit's step padded to S
// and its pitch to P (8-byte elements).  The stages, the split and the
// pre-split walk a row by its digits, so which S and P keep the 16 lanes of an
// access in different banks depends on the radices: the pairs below minimise
// the accesses' wavefronts, summed over the phases of a pass (counted over 32
// rows, S up to 4 and P up to 15 above their least values, a tenth more memory
// weighed as 0.03 wavefronts).  On average 1.4 wavefronts per 1 that an ideal
// layout would need, where an odd S and the least P give 2.0.
#pragma once

namespace crava {

struct RowBanks {
  int n, sf, pf, si, pi;  // line length; S and P forward (radices ascending; 32: 8 x 4) and inverse (descending)
};
constexpr RowBanks kRowBanks[] = {
    {16, 5, 20, 5, 20}, {18, 7, 21, 5, 35}, {20, 5, 20, 5, 28}, {21, 7, 21, 5, 35},
    {24, 7, 28, 5, 36}, {25, 5, 25, 6, 37}, {27, 11, 33, 3, 35}, {28, 7, 28, 5, 36},
    {30, 7, 35, 6, 37}, {32, 5, 44, 5, 44}, {35, 11, 55, 6, 53}, {36, 9, 54, 9, 54},
    {40, 9, 45, 6, 53}, {42, 7, 42, 7, 54}, {45, 9, 45, 5, 53}, {48, 9, 54, 6, 54},
    {49, 9, 63, 9, 71}, {50, 13, 65, 5, 53}, {54, 9, 54, 6, 54}, {56, 9, 63, 10, 87},
    {60, 13, 78, 7, 70}, {63, 9, 63, 7, 71}, {64, 9, 72, 9, 72}, {70, 13, 91, 7, 71},
    {72, 10, 89, 9, 88}, {75, 19, 95, 5, 85}, {80, 10, 81, 9, 104}, {81, 9, 81, 9, 89},
    {84, 15, 105, 7, 87}, {90, 13, 117, 9, 105}, {96, 14, 113, 9, 120}, {98, 15, 105, 7, 103},
    {100, 11, 110, 10, 106}, {105, 15, 105, 9, 135}, {108, 13, 117, 9, 121}, {112, 14, 113, 9, 136},
    {120, 13, 130, 10, 122}, {125, 29, 149, 29, 149}, {126, 15, 135, 9, 137}, {128, 18, 145, 9, 152},
    {135, 15, 135, 9, 137}, {140, 15, 150, 11, 154}, {144, 13, 156, 13, 156}, {147, 53, 161, 21, 149},
    {150, 15, 150, 10, 154}, {160, 17, 170, 10, 170}, {162, 19, 171, 9, 169}, {168, 15, 180, 13, 188},
    {175, 38, 195, 25, 185}, {180, 15, 180, 13, 204}, {189, 67, 207, 25, 229}, {192, 17, 204, 13, 220},
    {196, 17, 238, 17, 238}, {200, 21, 210, 10, 202}, {210, 15, 210, 15, 238}, {216, 19, 228, 13, 236},
    {224, 17, 238, 14, 238}, {225, 17, 255, 17, 255}, {240, 17, 255, 15, 255}, {243, 83, 257, 27, 251},
    {245, 50, 257, 35, 259}, {250, 50, 258, 26, 265}, {252, 19, 266, 15, 270}, {256, 17, 272, 17, 272}};

constexpr RowBanks row_banks(int n) {
  for (const RowBanks &b : kRowBanks)
    if (b.n == n) return b;
  return RowBanks{n, 0, 0, 0, 0};
}

}  // namespace crava
