// pdt_cart_rows.h -- row passes of the Cartesian operators on register transforms: image rows . coil maps -> DFT along W
// -> sampled columns, and back with the coil sum, for the compiled row lengths.
#pragma once

#include <cstddef>

#include "pdt_internal.h"

namespace pdt {

struct RowFft {
  int W = 0, Hi = 0, C = 0, ns = 0;
  int mx = 0, ox = 0;            // forward slot x holds image column (x - mx) mod W; inverse slot x is column (x + ox) mod W
  const float2* sens = nullptr;  // coil 0, image row 0, or null
  size_t coil_stride = 0;        // elements between coils
  const float2* tw = nullptr;    // [W] exp(-2 pi i m / W)
  const int* fs2s = nullptr;     // [W] spectrum index -> sampled column or -1 (forward)
  const int* as2s = nullptr;     // the same for the inverse's input
};

// Whether rows of this length and number of sampled columns have kernels that fit into max_smem bytes of shared memory
// a block; sets these kernels' limit to it.
bool row_fft_ok(int W, int ns, bool sens, int max_smem);
// t[c][s][y] <- sampled columns of DFT(u . sens_c). `zero` (may be null): nzero values set to zero on the way.
void launch_row_fft_fwd(const RowFft& a, const float2* u, float2* t, int* tick, float2* zero, size_t nzero,
                        cudaStream_t st);
// out <- sum_c conj(sens_c) . IDFT of t[c][s][y]
void launch_row_fft_adj(const RowFft& a, const float2* t, float2* out, cudaStream_t st);

}  // namespace pdt
