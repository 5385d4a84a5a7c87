// pdt_rad_fast.cuh -- transform passes of the radial operators for grid lengths with a compiled split G = P Q.
//
// Every array between the passes has the coils innermost: T[image row][gx][c], F[gy][gx][c]. The gather kernels then
// read and write all coils of a cell or sample as one run, and a column pass is a pass over the M = G C columns of
// a row-major matrix. Image x sits on grid slot (x - N/2) mod G, so slot p holds image x = (p + N/2) mod G when
// that is < N (zero padding elsewhere); spectra are in natural order.
//   rl_rows_fwd   image rows . sens_c / deap -> FFT along x  -> T
//   rl_cols_fwd   FFT along y of each column of T             -> F
//   rl_cols_inv   IFFT along y of each column, keep the N image rows -> T
//   rl_rows_inv   IFFT along x, crop, / deap, conj(sens_c) . and the coil sum
// A transform is a P-point DFT per t < Q over p = t + Q j, a twiddle and a Q-point DFT per k1 < P (index k1 + P k2),
// both in registers, with one exchange through shared memory; global loads and stores belong to the two ends and
// run along whole rows of the coils-innermost arrays. Before (one lane group per sequence, coil planes, transposed
// stores in runs of four rows): 12 coils, G = 384, 62 us for the four passes.
#pragma once

#include <algorithm>

#include "pdt_cfft.cuh"
#include "pdt_internal.h"

namespace pdt {

constexpr int kRadT = 256;      // threads of a pass
constexpr int kRadCoils = 16;   // coils per block of the row passes
constexpr int kRadCols = 16;    // columns per block of the column passes: 128-byte rows

// Lengths: 16 k, and 12 k and 10 k between them (grids 2, 1.5 and 1.25 times an image of 8 k).
#define PDT_RAD_SIZES(X)                                                                                            \
  X(4, 8) X(6, 8) X(8, 8) X(10, 8) X(6, 16) X(7, 16) X(8, 16) X(9, 16) X(10, 16) X(11, 16) X(12, 16) X(13, 16)    \
  X(14, 16) X(15, 16) X(16, 16) X(18, 16) X(20, 16) X(21, 16) X(22, 16) X(23, 16) X(24, 16) X(25, 16) X(26, 16)   \
  X(27, 16) X(28, 16) X(30, 16) X(32, 16) X(6, 12) X(7, 12) X(9, 12) X(11, 12) X(13, 12) X(15, 12) X(18, 12)      \
  X(21, 12) X(22, 12) X(25, 12) X(26, 12) X(27, 12) X(30, 12) X(6, 10) X(7, 10) X(9, 10) X(10, 10) X(11, 10)      \
  X(13, 10) X(14, 10) X(15, 10) X(20, 10) X(22, 10) X(25, 10) X(26, 10) X(28, 10) X(20, 32) X(24, 32)

struct RadPass {
  int N, G, C, off;
  float scale;
  const float2* sens;  // (N, N, C) or null
  const float* deap;   // [N]
  const float2* tw;    // [Q][P] exp(-2 pi i t k1 / G)
};

struct RadRowKernels {
  void (*fwd)(RadPass, const float2*, float2*) = nullptr;
  void (*inv)(RadPass, const float2*, float2*) = nullptr;
  int P = 0, Q = 0;
  bool ok() const { return fwd != nullptr; }
};
struct RadColKernels {
  void (*fwd)(RadPass, const float2*, float2*) = nullptr;
  void (*inv)(RadPass, const float2*, float2*) = nullptr;
};
RadRowKernels find_rad_rows(int G);
RadColKernels find_rad_cols(int G);

inline int rad_cb(int C) { return std::min(C, kRadCoils); }
inline size_t rad_rows_fwd_smem(const RadRowKernels& k, int N, int C) {
  return sizeof(float2) * ((size_t)k.P * k.Q + N + (size_t)k.P * (k.Q + 1) * (rad_cb(C) | 1));
}
inline size_t rad_rows_inv_smem(const RadRowKernels& k, int N, int C) {
  return sizeof(float2) * ((size_t)k.P * k.Q + (size_t)k.P * (k.Q + 1) * (rad_cb(C) | 1) + (size_t)rad_cb(C) * N) +
         sizeof(float) * (size_t)N;
}
inline size_t rad_cols_smem(const RadRowKernels& k) {
  return sizeof(float2) * (size_t)k.P * k.Q * (1 + kRadCols);
}

}  // namespace pdt
