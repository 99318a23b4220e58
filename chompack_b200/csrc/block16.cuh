// The 16 x 16 diagonal blocks of the tile and small-front tasks, factored and
// inverted by one warp.  Included by engine_kernel.cuh inside its namespace,
// after dmma8; the CPU test of the lanes' order (tests/test_block16_lanes.py)
// compiles it with a host dmma8.
#pragma once

// The pivots of an 8 x 8 block held by every lane (a, lower part), with the
// lane's row x beside them (row j of the block when own == j); r = 1 / L(j, j).
// Returns the first non-positive pivot, taken as 1, or -1.
__device__ __forceinline__ int potrf_pivots8(double (&a)[8][8], double (&x)[8], double (&r)[8], int own) {
  int bad = -1;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const bool np = !(a[j][j] > 0.0);
    if (np && bad < 0) bad = j;
    const double d = np ? 1.0 : a[j][j];
    r[j] = rsqrt(d);
    a[j][j] = d * r[j];
    x[j] = own == j ? a[j][j] : x[j] * r[j];
#pragma unroll
    for (int i = j + 1; i < 8; i++) a[j][i] *= r[j];
#pragma unroll
    for (int c = j + 1; c < 8; c++) {
#pragma unroll
      for (int i = c; i < 8; i++) a[c][i] = fma(-a[j][i], a[j][c], a[c][i]);
      x[c] = fma(-x[j], a[j][c], x[c]);
    }
  }
  return bad;
}

// Cholesky of a 16 x 16 diagonal block sL (factor; else the block already
// holds L) and its inverse sM (lower part written), by one warp, in two
// 8-column groups (only the first with cols <= 8, where the rest of the
// block is the identity).
// Every lane holds the group's 8 x 8 block and factors it for itself, so the
// chain from pivot to pivot is rsqrt -> multiply -> FMA with no exchange;
// beside it lane i reduces row i of the group's columns (the 8 rows of the
// block, then the 8 rows below) and lane c afterwards forms column c of the
// inverse by substitution, the first eight columns in two halves.  (As
// M21 = -M22 (L21 M11) the lower left block would lose what the conditions
// of both diagonal blocks multiply to.)  The second diagonal 8 x 8 block takes
// its rank-8 update, and the columns of the inverse the product between their
// halves, by MMAs.
// One lane per row with every pivot column broadcast through shared memory
// took 300 cycles a pivot on an idle SM: 19.2k for the 64 of a tile, and 6.4k
// for its four inverses; this takes 16.7k for both.
// Returns the block's first non-positive pivot (zero pivot when !factor), or
// -1; such a pivot is taken as 1.  Without factor, sM may be sL: the inverse
// takes the block's place.  !INV: no inverse, 1 / L(j, j) at sM[j] instead.
template <int LD, int LDM, bool INV = true>
__device__ __forceinline__ int potrf_block16(double* sL, double* sM, double* sTw, bool factor, int cols = 16) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, c8 = lane & 7;
  int first_bad = -1;
#pragma unroll 1
  for (int h = 0; h < (cols > 8 ? 2 : 1); h++) {
    const int b0 = 8 * h;
    double a[8][8], r[8];  // a[c][i]: entry (i, c), i >= c
    // row b0 + (lane mod 16): of the block, or below it (h = 0)
    const int row = b0 + (h == 0 ? (lane & 15) : c8);
    double x[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
#pragma unroll
      for (int i = c; i < 8; i++) a[c][i] = sL[(b0 + c) * LD + b0 + i];
      x[c] = sL[(b0 + c) * LD + row];
    }
    if (factor) {
      const int bad = potrf_pivots8(a, x, r, row - b0);
      if (bad >= 0 && first_bad < 0) first_bad = 8 * h + bad;
      __syncwarp();
      if (lane < (h == 0 ? 16 : 8)) {
#pragma unroll
        for (int c = 0; c < 8; c++)
          if (lane >= c) sL[(b0 + c) * LD + row] = x[c];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const bool bad = a[j][j] == 0.0;
        first_bad = (bad && first_bad < 0) ? 8 * h + j : first_bad;
        r[j] = 1.0 / (bad ? 1.0 : a[j][j]);
      }
      __syncwarp();  // in place: every lane has read the block
    }
    if (!INV) {
      if (lane == 0) {
#pragma unroll
        for (int j = 0; j < 8; j++) sM[b0 + j] = r[j];
      }
      __syncwarp();
    } else {
      // column b0 + first of the inverse, right-looking: as soon as M(l, c) is
      // known it is added into the partial sums of the later rows
      const int first = h == 0 ? c8 : (lane & 15) - 8;
      double m[8], t[8];
#pragma unroll
      for (int i = 0; i < 8; i++) t[i] = first < 0 ? sTw[8 * c8 + i] : 0.0;
#pragma unroll
      for (int l = 0; l < 8; l++) {
        m[l] = l == first ? r[l] : (l > first ? -r[l] * t[l] : 0.0);
#pragma unroll
        for (int i = l + 1; i < 8; i++) t[i] = fma(a[l][i], m[l], t[i]);
      }
      if (lane < (h == 0 ? 8 : 16)) {
#pragma unroll
        for (int i = 0; i < 8; i++)
          if (i >= first) sM[(b0 + first) * LDM + b0 + i] = m[i];
      }
      __syncwarp();
      if (h == 0 && cols > 8) {
        // what the first eight columns of the inverse start the second half
        // with: L21 M11, column-major
        double v[2] = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 8; k += 4) dmma8(v, sL[(k + q) * LD + 8 + g], sM[g * LDM + k + q]);
        sTw[16 * q + g] = v[0];
        sTw[16 * q + 8 + g] = v[1];
        __syncwarp();
      }
    }
    if (factor && h == 0) {
      // the second diagonal block: A(r, c) -= sum_k L(r, k) L(c, k), lower part
      const int rr = 8 + g, cc = 8 + 2 * q;
      double v[2] = {sL[cc * LD + rr], sL[(cc + 1) * LD + rr]};
#pragma unroll
      for (int k = 0; k < 8; k += 4) {
        const double w = sL[(k + q) * LD + rr];
        dmma8(v, -w, w);
      }
      if (rr >= cc) sL[cc * LD + rr] = v[0];
      if (rr >= cc + 1) sL[(cc + 1) * LD + rr] = v[1];
      __syncwarp();
    }
  }
  if (INV && cols <= 8 && lane < 8) sM[(8 + lane) * LDM + 8 + lane] = 1.0;  // the second half is the identity, as L's is
  return first_bad;
}
