// pdt_rad_rows.cu -- the row passes of the radial operators (pdt_rad_fast.cuh).
#include "pdt_rad_fast.cuh"

namespace pdt {
namespace {

// Block (row y, chunk of up to kRadCoils coils).
template <int P, int Q>
__global__ void __launch_bounds__(kRadT) rl_rows_fwd(RadPass d, const float2* __restrict__ u, float2* __restrict__ T) {
  constexpr int G = P * Q, LD = Q + 1;
  extern __shared__ __align__(16) float2 rsm[];
  const int tid = threadIdx.x, y = blockIdx.x, c0 = blockIdx.y * kRadCoils, N = d.N;
  const int nc = min(kRadCoils, d.C - c0), cp = min(kRadCoils, d.C) | 1;  // odd row length of Y: no bank conflicts
  float2* tws = rsm;       // [Q][P]
  float2* uw = tws + G;    // [N] the image row, scaled
  float2* Y = uw + N;      // [P][LD][cp]
  for (int i = tid; i < G; i += kRadT) tws[i] = d.tw[i];
  const float dy = d.deap[y];
  pdl_wait();  // u comes from the previous kernel
  pdl_trigger();
  for (int x = tid; x < N; x += kRadT) uw[x] = u[(size_t)y * N + x] * (d.scale / (d.deap[x] * dy));
  __syncthreads();
  for (int i = tid; i < nc * Q; i += kRadT) {
    const int c = i / Q, t = i % Q;
    const float2* s = d.sens ? d.sens + ((size_t)(c0 + c) * N + y) * N : nullptr;
    float2 v[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
      int x = t + Q * j + d.off;
      if (x >= G) x -= G;
      v[j] = c2(0.f, 0.f);
      if (x < N) v[j] = s ? cmul(uw[x], s[x]) : uw[x];
    }
    cfft_out<P, -1>(v, [&](auto K, float2 o) { Y[(decltype(K)::value * LD + t) * cp + c] = o; });
  }
  __syncthreads();
  for (int i = tid; i < nc * P; i += kRadT) {
    const int c = i % nc, k1 = i / nc;
    float2 v[Q];
#pragma unroll
    for (int t = 0; t < Q; ++t) v[t] = Y[(k1 * LD + t) * cp + c];
#pragma unroll
    for (int t = 1; t < Q; ++t) v[t] = cmul(v[t], tws[t * P + k1]);
    cfft<Q, -1>(v);
    float2* o = T + ((size_t)y * G + k1) * d.C + c0 + c;
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2) o[(size_t)(P * k2) * d.C] = v[k2];
  }
}

// Block: row y, all coils in chunks; the coils are summed in order.
template <int P, int Q>
__global__ void __launch_bounds__(kRadT) rl_rows_inv(RadPass d, const float2* __restrict__ T, float2* __restrict__ out) {
  constexpr int G = P * Q, LD = Q + 1, KX = (G + kRadT - 1) / kRadT;
  extern __shared__ __align__(16) float2 rsm[];
  const int tid = threadIdx.x, y = blockIdx.x, N = d.N, C = d.C;
  const int cb = min(kRadCoils, C), cp = cb | 1;
  float2* tws = rsm;                                          // [Q][P]
  float2* Y = tws + G;                                        // [P][LD][cp]
  float2* Z = Y + P * LD * cp;                                // [cb][N]
  float* w = reinterpret_cast<float*>(Z + (size_t)cb * N);    // [N]
  const float dy = d.deap[y];
  for (int i = tid; i < G; i += kRadT) tws[i] = d.tw[i];
  for (int x = tid; x < N; x += kRadT) w[x] = d.scale / (d.deap[x] * dy);
  pdl_wait();  // T comes from the previous kernel
  pdl_trigger();
  float2 acc[KX];
#pragma unroll
  for (int k = 0; k < KX; ++k) acc[k] = c2(0.f, 0.f);
  for (int c0 = 0; c0 < C; c0 += cb) {
    const int nc = min(cb, C - c0);
    for (int i = tid; i < nc * Q; i += kRadT) {
      const int c = i % nc, t = i / nc;
      const float2* src = T + ((size_t)y * G + t) * C + c0 + c;
      float2 v[P];
#pragma unroll
      for (int j = 0; j < P; ++j) v[j] = src[(size_t)(Q * j) * C];
      cfft_out<P, 1>(v, [&](auto K, float2 o) { Y[(decltype(K)::value * LD + t) * cp + c] = o; });
    }
    __syncthreads();
    for (int i = tid; i < nc * P; i += kRadT) {
      const int c = i / P, k1 = i % P;
      const float2* s = d.sens ? d.sens + ((size_t)(c0 + c) * N + y) * N : nullptr;
      float2 v[Q];
#pragma unroll
      for (int t = 0; t < Q; ++t) v[t] = Y[(k1 * LD + t) * cp + c];
#pragma unroll
      for (int t = 1; t < Q; ++t) v[t] = cmulc(v[t], tws[t * P + k1]);
      cfft<Q, 1>(v);
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) {
        int x = k1 + P * k2 + d.off;
        if (x >= G) x -= G;
        if (x < N) {
          const float2 val = v[k2] * w[x];
          Z[(size_t)c * N + x] = s ? cmulc(val, s[x]) : val;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KX; ++k) {
      const int x = tid + k * kRadT;
      if (x < N)
#pragma unroll 4
        for (int c = 0; c < nc; ++c) acc[k] += Z[(size_t)c * N + x];
    }
    // the next chunk writes Z after the barrier behind its first phase, and Y is free
  }
#pragma unroll
  for (int k = 0; k < KX; ++k) {
    const int x = tid + k * kRadT;
    if (x < N) out[(size_t)y * N + x] = acc[k];
  }
}

}  // namespace

RadRowKernels find_rad_rows(int G) {
#define PDT_RADROW(P_, Q_)                    \
  if (G == P_ * Q_) {                         \
    RadRowKernels k;                          \
    k.fwd = rl_rows_fwd<P_, Q_>;              \
    k.inv = rl_rows_inv<P_, Q_>;              \
    k.P = P_;                                 \
    k.Q = Q_;                                 \
    return k;                                 \
  }
  PDT_RAD_SIZES(PDT_RADROW)
#undef PDT_RADROW
  return RadRowKernels();
}

}  // namespace pdt
