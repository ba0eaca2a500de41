// Rows of a complex 8 x 8 matrix as unevaluated sums of two doubles (about 106
// bits), on the host.
#pragma once

namespace qfbh {

struct alignas(64) Rows8 {
    double xh[8][8], xl[8][8], yh[8][8], yl[8][8];  // row, column: real and imaginary part
};

// This CPU has the instructions dd_mix is made of (AVX2 and FMA).
bool dd_available();

// Rows k[0 .. n) become the n x n complex matrix m (re, im pairs, row-major) times
// them (n = 1, 2 or 4), in the four columns from 4 where halves' bit 1 is set and
// from 0 where its bit 0 is.
void dd_mix(Rows8 &r, const int *k, int n, const double *m, unsigned halves);

}  // namespace qfbh
