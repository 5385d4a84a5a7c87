// pdt_rad_cols.cu -- the column passes of the radial operators (pdt_rad_fast.cuh).
#include "pdt_rad_fast.cuh"

namespace pdt {
namespace {

// Block: kRadCols columns m of the M = G C. Loads and stores are 128-byte rows straight from and to registers.
template <int P, int Q, bool INV>
__global__ void __launch_bounds__(kRadT) rl_cols(RadPass d, const float2* __restrict__ in, float2* __restrict__ out) {
  constexpr int G = P * Q, S = INV ? 1 : -1;
  extern __shared__ __align__(16) float2 rsm[];
  float2* tws = rsm;      // [Q][P]
  float2* Y = tws + G;    // [P][Q][kRadCols]
  const int tid = threadIdx.x, M = G * d.C, m = blockIdx.x * kRadCols + tid % kRadCols, q = tid % kRadCols;
  const bool ok = m < M;
  for (int i = tid; i < G; i += kRadT) tws[i] = d.tw[i];
  pdl_wait();  // `in` comes from the previous kernel
  pdl_trigger();
  for (int t = tid / kRadCols; t < Q; t += kRadT / kRadCols) {
    float2 v[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
      int p = t + Q * j;
      if (!INV) {
        p += d.off;
        if (p >= G) p -= G;
      }
      v[j] = ok && (INV || p < d.N) ? in[(size_t)p * M + m] : c2(0.f, 0.f);
    }
    cfft_out<P, S>(v, [&](auto K, float2 o) { Y[(decltype(K)::value * Q + t) * kRadCols + q] = o; });
  }
  __syncthreads();
  for (int k1 = tid / kRadCols; k1 < P; k1 += kRadT / kRadCols) {
    float2 v[Q];
#pragma unroll
    for (int t = 0; t < Q; ++t) v[t] = Y[(k1 * Q + t) * kRadCols + q];
#pragma unroll
    for (int t = 1; t < Q; ++t) v[t] = INV ? cmulc(v[t], tws[t * P + k1]) : cmul(v[t], tws[t * P + k1]);
    cfft<Q, S>(v);
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2) {
      int p = k1 + P * k2;
      if (INV) {
        p += d.off;
        if (p >= G) p -= G;
      }
      if (ok && (!INV || p < d.N)) out[(size_t)p * M + m] = v[k2];
    }
  }
}

}  // namespace

RadColKernels find_rad_cols(int G) {
#define PDT_RADCOL(P_, Q_)                \
  if (G == P_ * Q_) {                     \
    RadColKernels k;                      \
    k.fwd = rl_cols<P_, Q_, false>;       \
    k.inv = rl_cols<P_, Q_, true>;        \
    return k;                             \
  }
  PDT_RAD_SIZES(PDT_RADCOL)
#undef PDT_RADCOL
  return RadColKernels();
}

}  // namespace pdt
