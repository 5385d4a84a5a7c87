// pdt_cart_rows.cu -- row passes of the Cartesian operators on register transforms (pdt_cart_rows.h).
#include "pdt_cart_rows.h"

#include <cooperative_groups.h>

#include <algorithm>

#include "pdt_cfft.cuh"
#include "pdt_device.cuh"

namespace pdt {
namespace {

namespace cg = cooperative_groups;

// A block takes kRows rows: the sampled columns t[c][s][y] are read and written in runs of 64 bytes. Row n = P Q as in
// the solvers' row operator: P-point DFTs over x = t + Q j, twiddles, Q-point DFTs, spectrum index k1 + P k2, one
// exchange through shared memory between (rows of Q + 1 values: both directions without bank conflicts).
constexpr int kRows = 8;

// Rows of sampled columns in shared memory: [row][ns], the rows 2 modulo 16 values apart, so that eight rows of two
// neighbouring columns lie in different banks.
__host__ __device__ constexpr int row_ld(int ns) { return (ns + 13) / 16 * 16 + 2; }

__device__ __forceinline__ void load_tables(const RowFft& a, int P, int Q, const int* map, float2* tws, int* s2s) {
  for (int i = threadIdx.x; i < P * Q; i += blockDim.x) {
    tws[i] = a.tw[(i / P) * (i % P)];  // [t][k1]
    s2s[i] = map[i];
  }
}

// Block (row block, coil). Bound by latency: 15 coils, 320 x 368 rows are 600 blocks of 128 threads, all resident.
// The stores that clear the dense k-space (28 MB there, a pass of its own before) run in the shade of the loads: the
// operator's forward 40 us with lane-FFT rows and the separate pass, 33 with these.
template <int P, int Q>
__global__ void __launch_bounds__(kRows * Q) row_fft_fwd(RowFft a, const float2* __restrict__ u, float2* __restrict__ t1,
                                                         int* __restrict__ tick, float2* __restrict__ zero, size_t nzero) {
  constexpr int n = P * Q, LD = Q + 1, T = kRows * Q;
  extern __shared__ __align__(16) float2 rsm[];
  const int tid = threadIdx.x, LDs = row_ld(a.ns);
  float2* tws = rsm;                  // [Q][P]
  float2* Y = tws + n;                // [kRows][P][LD]
  float2* stage = Y + kRows * P * LD;  // [kRows][LDs]
  int* s2s = reinterpret_cast<int*>(stage + kRows * LDs);
  load_tables(a, P, Q, a.fs2s, tws, s2s);
  pdl_wait();  // u comes from the previous kernel; t1 and zero may still be read by it
  pdl_trigger();
  if (tick && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) atomicAdd(tick, 1);
  const int y0 = blockIdx.x * kRows, c = blockIdx.y, nr = min(kRows, a.Hi - y0);
  {
    const int r = tid / Q, t = tid % Q;
    const size_t row = y0 + (r < nr ? r : 0);  // rows past the last one transform the first and drop it
    const float2* ur = u + row * n;
    const float2* sr = a.sens ? a.sens + c * a.coil_stride + row * n : nullptr;
    float2 v[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
      int x = t + Q * j - a.mx;
      if (x < 0) x += n;
      v[j] = ur[x];
      if (sr) v[j] = cmul(v[j], sr[x]);
    }
    if (zero) {
      const size_t nb = (size_t)gridDim.x * gridDim.y, b = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
      const size_t head = (reinterpret_cast<size_t>(zero) & 15) ? 1 : 0, n4 = (nzero - head) / 2;
      float4* z4 = reinterpret_cast<float4*>(zero + head);
      const size_t e = (b + 1) * n4 / nb;
      for (size_t i = b * n4 / nb + tid; i < e; i += T) z4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (b == 0 && tid == 0 && head) zero[0] = c2(0.f, 0.f);
      if (b == 0 && tid == 0 && head + 2 * n4 < nzero) zero[nzero - 1] = c2(0.f, 0.f);
    }
    float2* yc = Y + r * (P * LD) + t;
    cfft_out<P, -1>(v, [&](auto K, float2 o) { yc[decltype(K)::value * LD] = o; });
  }
  __syncthreads();
  for (int i = tid; i < kRows * P; i += T) {
    const int r = i / P, k1 = i % P;
    const float2* yr = Y + i * LD;
    float2 v[Q];
    v[0] = yr[0];
#pragma unroll
    for (int t = 1; t < Q; ++t) v[t] = cmul(yr[t], tws[t * P + k1]);
    cfft_out<Q, -1>(v, [&](auto K, float2 o) {
      const int s = s2s[k1 + P * decltype(K)::value];
      if (s >= 0) stage[r * LDs + s] = o;
    });
  }
  __syncthreads();
  for (int i = tid; i < kRows * a.ns; i += T) {
    const int s = i / kRows, r = i % kRows;
    if (r < nr) t1[((size_t)c * a.ns + s) * a.Hi + y0 + r] = stage[r * LDs + s];
  }
}

// Block (row block, coil group); the coil groups of a row block form a cluster and add their sums through distributed
// shared memory in rank order. A thread owns the same P pixels of a row for every coil and sums them in registers.
// The next coil's columns arrive by asynchronous copies during this one, its map rows after the last use of this
// one's (the first coil's before the programmatic wait: maps are constant). The operator's adjoint at 15 coils,
// 640 x 368: 42 us with tensor-core rows (22-bit operands, 1.2e-6 off), 36 with these (1.3e-7); 12 coils, 256 x 256, all
// columns sampled: 50 us with lane-FFT rows, 21 with these.
template <int P, int Q>
__global__ void __launch_bounds__(kRows * Q) row_fft_adj(RowFft a, const float2* __restrict__ t2, float2* __restrict__ out) {
  constexpr int n = P * Q, LD = Q + 1, T = kRows * Q;
  extern __shared__ __align__(16) float2 rsm[];
  const int tid = threadIdx.x, LDs = row_ld(a.ns), G = gridDim.y, g = blockIdx.y;
  float2* tws = rsm;
  float2* Y = tws + n;                                  // [kRows][P][LD]; at the end the group's sums [kRows][n]
  float2* X = Y + kRows * P * LD;                       // two of [kRows][LDs]
  float2* S = X + 2 * kRows * LDs;                      // [kRows][n], with maps
  int* s2s = reinterpret_cast<int*>(S + (a.sens ? kRows * n : 0));
  const int y0 = blockIdx.x * kRows, nr = min(kRows, a.Hi - y0);
  const int cb = g * a.C / G, ce = (g + 1) * a.C / G;
  auto maps = [&](int c) {
    const float2* src = a.sens + c * a.coil_stride + (size_t)y0 * n;
    for (int i = tid; i < nr * n; i += T) cp_async8(S + i, src + i);
  };
  auto columns = [&](int c) {
    float2* dst = X + ((c - cb) & 1) * kRows * LDs;
    for (int i = tid; i < kRows * a.ns; i += T) {
      const int s = i / kRows, r = i % kRows;
      if (r < nr) cp_async8(dst + r * LDs + s, t2 + ((size_t)c * a.ns + s) * a.Hi + y0 + r);
    }
  };
  if (a.sens) maps(cb);
  cp_async_commit();
  load_tables(a, P, Q, a.as2s, tws, s2s);
  pdl_wait();  // t2 comes from the previous kernel; out may still be read by it
  pdl_trigger();
  columns(cb);
  cp_async_commit();
  const int r = tid / Q, t = tid % Q;
  float2 acc[P];
#pragma unroll
  for (int j = 0; j < P; ++j) acc[j] = c2(0.f, 0.f);
  for (int c = cb; c < ce; ++c) {
    if (c + 1 < ce) columns(c + 1);
    cp_async_commit();
    // pending in order: (maps and) columns of the first coil, the next columns; later columns, maps, next columns
    if (c == cb)
      cp_async_wait<1>();
    else
      cp_async_wait<2>();
    __syncthreads();
    const float2* xc = X + ((c - cb) & 1) * kRows * LDs;
    for (int i = tid; i < kRows * P; i += T) {
      const int k1 = i % P;
      const float2* xr = xc + (i / P) * LDs;
      float2* yr = Y + i * LD;
      float2 v[Q];
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) {
        const int s = s2s[k1 + P * k2];
        v[k2] = s >= 0 ? xr[s] : c2(0.f, 0.f);
      }
      cfft_out<Q, 1>(v, [&](auto K, float2 o) {
        constexpr int tt = decltype(K)::value;
        if constexpr (tt == 0)
          yr[0] = o;
        else
          yr[tt] = cmulc(o, tws[tt * P + k1]);
      });
    }
    cp_async_wait<1>();
    __syncthreads();
    float2* yc = Y + r * (P * LD) + t;
    float2 v[P];
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) v[k1] = yc[k1 * LD];
    const float2* sr = S + r * n;
    cfft_out<P, 1>(v, [&](auto J, float2 o) {
      constexpr int j = decltype(J)::value;
      int x = t + Q * j + a.ox;
      if (x >= n) x -= n;
      acc[j] += a.sens ? cmulc(o, sr[x]) : o;
    });
    __syncthreads();  // Y and S are free
    if (a.sens && c + 1 < ce) maps(c + 1);
    cp_async_commit();
  }
  cp_async_wait<0>();
#pragma unroll
  for (int j = 0; j < P; ++j) {
    int x = t + Q * j + a.ox;
    if (x >= n) x -= n;
    Y[r * n + x] = acc[j];
  }
  float2* o = out + (size_t)y0 * n;
  const int total = nr * n;
  if (G == 1) {
    __syncthreads();
    for (int i = tid; i < total; i += T) o[i] = Y[i];
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int i = g * total / G + tid; i < (g + 1) * total / G; i += T) {
    float2 z = c2(0.f, 0.f);
    for (int q = 0; q < G; ++q) z += cluster.map_shared_rank(Y, q)[i];
    o[i] = z;
  }
  cluster.sync();  // the other blocks have read this one's sums
}

typedef void (*RowFwdFn)(RowFft, const float2*, float2*, int*, float2*, size_t);
typedef void (*RowAdjFn)(RowFft, const float2*, float2*);

struct RowKernel {
  int P, Q;
  RowFwdFn fwd;
  RowAdjFn adj;
};

#define PDT_ROW_SIZES(X)                                                                                       \
  X(6, 8) X(8, 8) X(10, 8) X(6, 16) X(7, 16) X(8, 16) X(9, 16) X(10, 16) X(11, 16) X(12, 16) X(13, 16) X(14, 16) \
  X(15, 16) X(16, 16) X(17, 16) X(18, 16) X(19, 16) X(20, 16) X(21, 16) X(22, 16) X(23, 16) X(24, 16) X(26, 16)  \
  X(28, 16) X(30, 16) X(32, 16) X(24, 24) X(20, 32)

const RowKernel kRowKernels[] = {
#define PDT_ROW_ENTRY(P, Q) {P, Q, row_fft_fwd<P, Q>, row_fft_adj<P, Q>},
    PDT_ROW_SIZES(PDT_ROW_ENTRY)
#undef PDT_ROW_ENTRY
};

const RowKernel* find(int W) {
  for (const RowKernel& k : kRowKernels)
    if (k.P * k.Q == W) return &k;
  return nullptr;
}

size_t row_smem(const RowKernel& k, int ns, bool sens, bool adj) {
  const size_t n = (size_t)k.P * k.Q;
  return sizeof(float2) * (n + (size_t)kRows * (k.P * (k.Q + 1) + (adj ? 2 : 1) * row_ld(ns) + (adj && sens ? n : 0))) +
         sizeof(int) * n;
}

}  // namespace

bool row_fft_ok(int W, int ns, bool sens, int max_smem) {
  const RowKernel* k = find(W);
  if (!k || ns <= 0 || std::max(row_smem(*k, ns, sens, true), row_smem(*k, ns, sens, false)) > (size_t)max_smem) return false;
  PDT_CUDA_CHECK(cudaFuncSetAttribute(k->fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
  PDT_CUDA_CHECK(cudaFuncSetAttribute(k->adj, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
  return true;
}

void launch_row_fft_fwd(const RowFft& a, const float2* u, float2* t, int* tick, float2* zero, size_t nzero,
                        cudaStream_t st) {
  const RowKernel& k = *find(a.W);
  const size_t smem = row_smem(k, a.ns, a.sens != nullptr, false);
  LaunchEx lx(dim3((a.Hi + kRows - 1) / kRows, a.C), dim3(kRows * k.Q), smem, st);
  PDT_CUDA_CHECK(cudaLaunchKernelEx(&lx.cfg, k.fwd, a, u, t, tick, zero, nzero));
  count_launch();
}

void launch_row_fft_adj(const RowFft& a, const float2* t, float2* out, cudaStream_t st) {
  const RowKernel& k = *find(a.W);
  const size_t smem = row_smem(k, a.ns, a.sens != nullptr, true);
  const int G = std::min(8, a.C);  // portable cluster size
  LaunchEx lx(dim3((a.Hi + kRows - 1) / kRows, G), dim3(kRows * k.Q), smem, st, G > 1 ? G : 0);
  PDT_CUDA_CHECK(cudaLaunchKernelEx(&lx.cfg, k.adj, a, t, out));
  count_launch();
}

}  // namespace pdt
