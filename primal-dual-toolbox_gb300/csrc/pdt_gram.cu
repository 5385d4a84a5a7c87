// pdt_gram.cu -- the solvers' iterations with a line-sampled Cartesian operator (pdt_gram.h): the row
// operator K^H K, and the image side of an iteration in one tile pass.
#include "pdt_gram.h"

#include <algorithm>
#include <cmath>
#include <string>
#include <utility>

#include "pdt_cfft.cuh"
#include "pdt_primal.cuh"

namespace pdt {
namespace {

constexpr int kGramThreads = 128;

struct RowsArgs {
  int W, H, C, CB;  // CB: coils per pass
  const float2* sens;
  size_t coil_stride;
  const float2* tw;
  const float* spec;
  const float2* D;
  float2* part;
};

// Block (g, y): row y, coil group g, in passes of up to CB coils. Per pass, with a block barrier between,
//   1  per coil and t < Q: s_c . D at x = t + Q j (j < P), P-point DFT            -> Y[c][k1][t]
//   2  per coil and k1 < P: twiddle, Q-point DFT, times the spectrum of G, inverse -> Y[c][k1][t]
//   3  per coil and t: inverse P-point DFT, times conj(s_c)                         -> Y[c][j][t]
//   4  sum over the pass's coils in coil order
// Between DFT and inverse a spectrum value never leaves its thread, so a transform pair costs two exchanges
// through shared memory; rows of Y hold Q + 1 values so that both access directions are free of bank
// conflicts. A row shift commutes with G, so the shifts of the operator's transforms drop out and slot x holds
// image column x. The coil maps (used twice) arrive by asynchronous copies, the first pass's and the tables
// before the programmatic wait and each further pass's during the one before it. Bound by issue slots
// and barriers (15 coils, 320 x 368: 7.1 M warp instructions, 4.0 M of them on the FMA pipe) and by waves:
// 128 threads and five coils a block; with 96 or 64 threads and four or two coils 28.5 us an iteration.
template <int P, int Q, int MINB>
__global__ void __launch_bounds__(kGramThreads, MINB) gram_rows_kernel(RowsArgs a) {
  constexpr int n = P * Q, LD = Q + 1, KX = (n + kGramThreads - 1) / kGramThreads;
  extern __shared__ __align__(16) float2 gsm[];
  const int tid = threadIdx.x, y = blockIdx.y, W = a.W;
  const int cb = (int)((long long)blockIdx.x * a.C / gridDim.x), ce = (int)((long long)(blockIdx.x + 1) * a.C / gridDim.x);
  const bool two = ce - cb > a.CB;
  float2* tws = gsm;                                          // [Q][P]
  float2* Ds = tws + n;                                       // [n], zero past W
  float2* Y = Ds + n;                                         // [CB][P][LD]
  float2* S = Y + a.CB * (P * LD);                            // one or two of [CB][n], zero past W
  float* spec = reinterpret_cast<float*>(S + (a.sens ? (two ? 2 : 1) * a.CB * n : 0));  // [n]
  auto stage = [&](int c0, float2* dst) {
    const int nc = min(a.CB, ce - c0);
    const float2* src = a.sens + (size_t)c0 * a.coil_stride + (size_t)y * W;
    for (int c = 0; c < nc; ++c, src += a.coil_stride, dst += n)
      for (int x = tid; x < W; x += kGramThreads) cp_async8(dst + x, src + x);
  };
  if (a.sens) stage(cb, S);
  cp_async_commit();
  for (int i = tid; i < n; i += kGramThreads) {
    tws[i] = a.tw[i];
    spec[i] = a.spec[i];
  }
  if (W < n) {
    for (int x = W + tid; x < n; x += kGramThreads) Ds[x] = c2(0.f, 0.f);
    if (a.sens)
      for (int c = 0; c < (two ? 2 : 1) * a.CB; ++c)
        for (int x = W + tid; x < n; x += kGramThreads) S[c * n + x] = c2(0.f, 0.f);
  }
  pdl_wait();  // everything above is constant; D comes from the previous kernel
  pdl_trigger();
  for (int x = tid; x < W; x += kGramThreads) Ds[x] = a.D[(size_t)y * W + x];
  float2 z[KX];
#pragma unroll
  for (int k = 0; k < KX; ++k) z[k] = c2(0.f, 0.f);
  int pass = 0;
  for (int c0 = cb; c0 < ce; c0 += a.CB, ++pass) {
    const int nc = min(a.CB, ce - c0);
    const float2* sc = S + (size_t)(pass & 1) * a.CB * n;
    if (a.sens && c0 + a.CB < ce) stage(c0 + a.CB, S + (size_t)((pass + 1) & 1) * a.CB * n);
    cp_async_commit();
    cp_async_wait<1>();  // this pass's maps
    __syncthreads();
    for (int i = tid; i < nc * Q; i += kGramThreads) {
      const int c = i / Q, t = i % Q;
      float2 v[P];
      if (a.sens) {
        const float2* s = sc + c * n + t;
#pragma unroll
        for (int j = 0; j < P; ++j) v[j] = cmul(Ds[t + Q * j], s[Q * j]);
      } else {
#pragma unroll
        for (int j = 0; j < P; ++j) v[j] = Ds[t + Q * j];
      }
      float2* yc = Y + c * (P * LD) + t;
      cfft_out<P, -1>(v, [&](auto K, float2 o) { yc[decltype(K)::value * LD] = o; });
    }
    __syncthreads();
    for (int i = tid; i < nc * P; i += kGramThreads) {
      const int k1 = i % P;
      float2* yr = Y + i * LD;
      float2 v[Q];
      v[0] = yr[0];
#pragma unroll
      for (int t = 1; t < Q; ++t) v[t] = cmul(yr[t], tws[t * P + k1]);
      cfft<Q, -1>(v);
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) v[k2] = v[k2] * spec[k2 * P + k1];
      cfft<Q, 1>(v);
      yr[0] = v[0];
#pragma unroll
      for (int t = 1; t < Q; ++t) yr[t] = cmulc(v[t], tws[t * P + k1]);
    }
    __syncthreads();
    for (int i = tid; i < nc * Q; i += kGramThreads) {
      const int c = i / Q, t = i % Q;
      float2* yc = Y + c * (P * LD) + t;
      float2 v[P];
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) v[k1] = yc[k1 * LD];
      if (a.sens) {
        const float2* s = sc + c * n + t;
        cfft_out<P, 1>(v, [&](auto J, float2 o) {
          constexpr int j = decltype(J)::value;
          yc[j * LD] = cmulc(o, s[Q * j]);
        });
      } else {
        cfft_out<P, 1>(v, [&](auto J, float2 o) { yc[decltype(J)::value * LD] = o; });
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KX; ++k) {
      const int x = tid + k * kGramThreads;
      if (x >= W) continue;
      const float2* yx = Y + (x / Q) * LD + x % Q;
      for (int c = 0; c < nc; ++c) z[k] += yx[c * (P * LD)];
    }
    // the next pass's phase 1 overwrites Y after the barrier at its top
  }
  float2* out = a.part + ((size_t)blockIdx.x * a.H + y) * W;
#pragma unroll
  for (int k = 0; k < KX; ++k) {
    const int x = tid + k * kGramThreads;
    if (x < W) out[x] = z[k];
  }
}

// ------------------------------------------------------------------------------------------------
// Image side of an iteration for a 32 x 8 tile: the primal update on the tile and one column and row beyond
// it (the next dual update reads ubar and vbar at x + 1 and y + 1), from the p, q of the tile and its
// halo; then the dual update and D of the next iteration. Everything but K^H K D is complete before the
// row kernel starts, and nothing the row kernel reads is written here, so the divergences, the v update and
// the next q run before the programmatic wait (L2 loads: this SM may hold older lines). Bound by the latency
// of its load phases: four blocks an SM (48 registers, some spilled) make one wave of the 480 blocks of a
// 320 x 368 image and 17.6 us an iteration with the row kernel, solves one after the other; three blocks 21.2, two 19.7
// (in a form with U for D). D, its compensation and w are loaded together with the sums: before the wait they took
// registers (18.7 us an iteration against 17.9, set-up included).
// ------------------------------------------------------------------------------------------------
constexpr int GX = 32, GY = 8, GT = 320;  // (GX + 1) (GY + 1) = 297 primal pixels, one a thread

template <bool TGV, bool ROWS>
__global__ void __launch_bounds__(GT, 4) gram_image_kernel(GramImage s) {
  __shared__ float2 s_px[GY + 2][GX + 2], s_py[GY + 2][GX + 2];  // [x0 - 1, x0 + GX] x [y0 - 1, y0 + GY]
  __shared__ float2 s_qxx[TGV ? GY + 2 : 1][GX + 2], s_qyy[TGV ? GY + 2 : 1][GX + 2], s_qxy[TGV ? GY + 2 : 1][GX + 2];
  __shared__ float2 s_ub[GY + 1][GX + 1];  // [x0, x0 + GX] x [y0, y0 + GY]
  __shared__ float2 s_vx[TGV ? GY + 1 : 1][GX + 1], s_vy[TGV ? GY + 1 : 1][GX + 1];
  const int tid = threadIdx.x, W = s.W, H = s.H;
  const int x0 = blockIdx.x * GX, y0 = blockIdx.y * GY;
  auto ld = [](const void* p, size_t i) { return __ldcg(static_cast<const float2*>(p) + i); };
  const int it = __ldcg(s.header + 4 + s.par), last = __ldcg(s.header + 1) - 1;
  const float4 row = s.table[min(max(it, 0), last)];
  const float4 next = s.table[min(max(it + 1, 0), last)];
  for (int i = tid; i < (GX + 2) * (GY + 2); i += GT) {
    const int ly = i / (GX + 2), lx = i - ly * (GX + 2);
    const int gx = x0 - 1 + lx, gy = y0 - 1 + ly;
    if (gx >= 0 && gx < W && gy >= 0 && gy < H) {
      const size_t idx = (size_t)gy * W + gx;
      s_px[ly][lx] = ld(s.src.px, idx);
      s_py[ly][lx] = ld(s.src.py, idx);
      if constexpr (TGV) {
        s_qxx[ly][lx] = ld(s.src.qxx, idx);
        s_qyy[ly][lx] = ld(s.src.qyy, idx);
        s_qxy[ly][lx] = ld(s.src.qxy, idx);
      }
    }
  }
  const int ly = tid / (GX + 1), lx = tid - ly * (GX + 1);
  const int x = x0 + lx, y = y0 + ly;
  const bool in = tid < (GX + 1) * (GY + 1) && x < W && y < H;
  const bool own = in && lx < GX && ly < GY;
  const size_t idx = in ? (size_t)y * W + x : 0;
  float2 ou = c2(0.f, 0.f), kf = ou, ovx = ou, ovy = ou;
  if (in) {
    ou = ld(s.src.u, idx);
    if constexpr (ROWS) {
      kf = row.z * __ldcg(s.h + idx);
      if (s.z0) kf = kf + row.w * __ldcg(s.z0 + idx);
    }
    if constexpr (TGV) {
      ovx = ld(s.src.vx, idx);
      ovy = ld(s.src.vy, idx);
    }
  }
  __syncthreads();
  // div- along x and y with the reference's boundary rules: f(0) first, -f(n-2) last, f(i) - f(i-1) between
  auto dx = [&](const float2 (*e)[GX + 2]) {
    const float2 c = e[ly + 1][lx + 1], p = e[ly + 1][lx];
    return x > 0 ? (x < W - 1 ? c - p : -p) : c;
  };
  auto dy = [&](const float2 (*e)[GX + 2]) {
    const float2 c = e[ly + 1][lx + 1], p = e[ly][lx + 1];
    return y > 0 ? (y < H - 1 ? c - p : -p) : c;
  };
  bool finite = true;
  float2 dp = c2(0.f, 0.f);
  if (in) {
    dp = dx(s_px) + dy(s_py);
    if constexpr (TGV) {
      const float2 vxn = ovx + s.tau * ((dx(s_qxx) + dy(s_qxy)) + s_px[ly + 1][lx + 1]);
      const float2 vyn = ovy + s.tau * ((dy(s_qyy) + dx(s_qxy)) + s_py[ly + 1][lx + 1]);
      finite = isfinite(vxn.x) && isfinite(vxn.y) && isfinite(vyn.x) && isfinite(vyn.y);
      s_vx[ly][lx] = 2.0f * vxn - ovx;
      s_vy[ly][lx] = 2.0f * vyn - ovy;
      if (own) {
        static_cast<float2*>(s.dst.vx)[idx] = vxn;
        static_cast<float2*>(s.dst.vy)[idx] = vyn;
      }
    }
  }
  const int xp = lx + (x < W - 1), yp = ly + (y < H - 1);
  if constexpr (TGV) {
    __syncthreads();
    if (own && it >= last) {
      static_cast<float2*>(s.dst.vbx)[idx] = s_vx[ly][lx];
      static_cast<float2*>(s.dst.vby)[idx] = s_vy[ly][lx];
    } else if (own) {  // the next iteration's q (tgv_kernels.cuh:225-258)
      const float2 vx = s_vx[ly][lx], vy = s_vy[ly][lx];
      const float2 gxy = 0.5f * (s_vx[yp][lx] - vx + s_vy[ly][xp] - vy);
      const float2 qa = s_qxx[ly + 1][lx + 1] + s.sigma * (s_vx[ly][xp] - vx);
      const float2 qb = s_qyy[ly + 1][lx + 1] + s.sigma * (s_vy[yp][lx] - vy);
      const float2 qc = s_qxy[ly + 1][lx + 1] + s.sigma * gxy;
      const float sq = dual_proj_scale(sqrtf(abs2(qa) + abs2(qb) + 2.0f * abs2(qc)), next.x);
      static_cast<float2*>(s.dst.qxx)[idx] = qa * sq;
      static_cast<float2*>(s.dst.qyy)[idx] = qb * sq;
      static_cast<float2*>(s.dst.qxy)[idx] = qc * sq;
    }
  }
  pdl_wait();  // K^H K D comes from the row kernel
  pdl_trigger();
  if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) s.header[4 + (s.par ^ 1)] = it + 1;
  float2 Do = c2(0.f, 0.f), De = Do, w = Do;
  if (ROWS && own) {  // in flight together with the sums (earlier they would only hold registers)
    Do = __ldcg(s.D + idx);
    De = __ldcg(s.D + (size_t)W * H + idx);
    w = __ldcg(s.w + idx);
  }
  if (in) {
    float2 kh = s.part[idx];
    for (int g = 1; g < s.groups; ++g) kh += s.part[idx + (size_t)g * W * H];
    if constexpr (ROWS) kh = kh + kf;
    const float2 un = ou + s.tau * (dp - kh);
    s_ub[ly][lx] = 2.0f * un - ou;
    finite = finite && isfinite(un.x) && isfinite(un.y);
    if (own) static_cast<float2*>(s.dst.u)[idx] = un;
  }
  if (own && !finite) s.header[2] = 1;
  __syncthreads();
  if (!own) return;
  const float2 c = s_ub[ly][lx];
  if (!ROWS || it >= last) static_cast<float2*>(s.dst.ub)[idx] = c;
  if (it >= last) return;
  // the next iteration's p (tgv_kernels.cuh:260-292)
  float2 gx = s_ub[ly][xp] - c, gy = s_ub[yp][lx] - c;
  if constexpr (TGV) {
    gx = gx - s_vx[ly][lx];
    gy = gy - s_vy[ly][lx];
  }
  const float2 a = s_px[ly + 1][lx + 1] + s.sigma * gx, b = s_py[ly + 1][lx + 1] + s.sigma * gy;
  const float sp = dual_proj_scale(sqrtf(abs2(a) + abs2(b)), TGV ? next.y : 1.0f);
  static_cast<float2*>(s.dst.px)[idx] = a * sp;
  static_cast<float2*>(s.dst.py)[idx] = b * sp;
  if constexpr (!ROWS) return;
  // D + its compensation
  auto step = [&](float d, float e, float ub, float& nd, float& ne) {
    const float inc = __fadd_rn(e, s.k * ((ub - s.lambda * d) - s.lambda * e));
    nd = __fadd_rn(d, inc);
    ne = __fsub_rn(inc, __fsub_rn(nd, d));
  };
  float2 nd, ne;
  step(Do.x, De.x, c.x - w.x, nd.x, ne.x);
  step(Do.y, De.y, c.y - w.y, nd.y, ne.y);
  s.Dnext[idx] = nd;
  s.Dnext[(size_t)W * H + idx] = ne;
}

constexpr int kStartThreads = 256;

// dots[block] = {|w|^2, Re <w, K^H K w>} over every kGramDots-th run of pixels.
__global__ void __launch_bounds__(kStartThreads) gram_dots_kernel(size_t n, const float2* __restrict__ w,
                                                                  const float2* __restrict__ part, int groups,
                                                                  float2* __restrict__ dots) {
  __shared__ float2 sh[kStartThreads];
  float2 s = c2(0.f, 0.f);
  for (size_t i = blockIdx.x * (size_t)kStartThreads + threadIdx.x; i < n; i += (size_t)kGramDots * kStartThreads) {
    float2 g = part[i];
    for (int q = 1; q < groups; ++q) g += part[i + q * n];
    const float2 v = w[i];
    s += c2(abs2(v), v.x * g.x + v.y * g.y);
  }
  sh[threadIdx.x] = s;
  for (int o = kStartThreads / 2; o > 0; o >>= 1) {
    __syncthreads();
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
  }
  if (threadIdx.x == 0) dots[blockIdx.x] = sh[0];
}

__global__ void __launch_bounds__(kStartThreads) gram_start_kernel(size_t n, const float2* __restrict__ dots,
                                                                   const float2* __restrict__ ubar, float k,
                                                                   float2* __restrict__ w, float2* __restrict__ D) {
  __shared__ float2 sh[kGramDots];
  if (threadIdx.x < kGramDots) sh[threadIdx.x] = dots[threadIdx.x];
  for (int o = kGramDots / 2; o > 0; o >>= 1) {
    __syncthreads();
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
  }
  __syncthreads();
  float a = sh[0].x / sh[0].y;
  if (!isfinite(a)) a = 0.f;
  const size_t i = blockIdx.x * (size_t)kStartThreads + threadIdx.x;
  if (i >= n) return;
  const float2 v = a * w[i];
  w[i] = v;
  D[i] = k * (ubar[i] - v);
  D[n + i] = c2(0.f, 0.f);
}

__global__ void __launch_bounds__(kStartThreads) gram_total_kernel(size_t n, const float2* __restrict__ D,
                                                                   const float2* __restrict__ w, float c,
                                                                   float2* __restrict__ out) {
  const size_t i = blockIdx.x * (size_t)kStartThreads + threadIdx.x;
  if (i < n) out[i] = c2(fmaf(c, w[i].x, D[i].x), fmaf(c, w[i].y, D[i].y));
}

typedef void (*GramFn)(RowsArgs);

struct GramKernel {
  GramLength len;
  GramFn fn;
};

// Lengths n = P Q: the multiples of 16 that leave P values a thread, and larger ones for the padded rows.
#define PDT_GRAM_SIZES(X)                                                                                      \
  X(4, 8) X(6, 8) X(8, 8) X(10, 8) X(6, 16) X(7, 16) X(8, 16) X(9, 16) X(10, 16) X(11, 16) X(12, 16) X(13, 16) \
  X(14, 16) X(15, 16) X(16, 16) X(17, 16) X(18, 16) X(19, 16) X(20, 16) X(21, 16) X(22, 16) X(23, 16)          \
  X(24, 16) X(26, 16) X(28, 16) X(30, 16) X(32, 16) X(24, 24) X(20, 32) X(24, 32) X(32, 32)

constexpr int gram_minb(int P, int Q) { return P <= 24 && Q <= 16 ? 5 : 4; }

const GramKernel kGramKernels[] = {
#define PDT_GRAM_ROW(P, Q) {{P * Q, P, Q}, gram_rows_kernel<P, Q, gram_minb(P, Q)>},
    PDT_GRAM_SIZES(PDT_GRAM_ROW)
#undef PDT_GRAM_ROW
};

// Coils per pass: one transform task a thread in each phase.
int gram_pass(const GramLength& l) { return std::max(1, kGramThreads / std::max(l.P, l.Q)); }

size_t gram_smem(const GramLength& l, int CB, int stages) {
  return sizeof(float2) * ((size_t)2 * l.n + (size_t)CB * l.P * (l.Q + 1) + (size_t)stages * CB * l.n) +
         sizeof(float) * (size_t)l.n;
}

}  // namespace

GramLength gram_length(int W) {
  GramLength best{0, 0, 0};
  for (const auto& k : kGramKernels) {
    if (k.len.n == W) return k.len;
    if (k.len.n >= 2 * W - 1 && (best.n == 0 || k.len.n < best.n)) best = k.len;
  }
  return best;
}

int gram_groups(const GramLength& len, int H, int C, int sms) {
  const int passes = (C + gram_pass(len) - 1) / gram_pass(len);
  return std::max(1, std::min(passes, (6 * sms + H / 2) / std::max(H, 1)));
}

void gram_tables(int W, const GramLength& len, const std::vector<float>& m2, std::vector<float2>& tw,
                 std::vector<float>& spec) {
  const int n = len.n;
  auto roots = [](int N) {
    std::vector<double> c(N), s(N);
    for (int i = 0; i < N; ++i) {
      c[i] = std::cos(2.0 * M_PI * i / N);
      s[i] = std::sin(2.0 * M_PI * i / N);
    }
    return std::make_pair(c, s);
  };
  const auto rn = roots(n);
  tw.resize(n);
  for (int t = 0; t < len.Q; ++t)
    for (int k1 = 0; k1 < len.P; ++k1)
      tw[t * len.P + k1] = make_float2((float)rn.first[t * k1], (float)-rn.second[t * k1]);
  spec.assign(n, 0.f);
  if (n == W) {
    for (int k = 0; k < n; ++k) spec[k] = (float)((double)m2[k] / W);
    return;
  }
  // h[d] = (1 / W) sum_k m2[k] exp(2 pi i k d / W), |d| < W, laid out circularly in length n (h[-d] is the
  // conjugate of h[d], so the spectrum is real)
  const auto rw = roots(W);
  std::vector<double> hr(W, 0.0), hi(W, 0.0);
  for (int k = 0; k < W; ++k) {
    if (m2[k] == 0.f) continue;
    for (int d = 0, i = 0; d < W; ++d) {
      hr[d] += m2[k] * rw.first[i];
      hi[d] += m2[k] * rw.second[i];
      i += k;
      if (i >= W) i -= W;
    }
  }
  for (int k = 0; k < n; ++k) {
    double a = hr[0];
    for (int d = 1, i = k; d < W; ++d) {  // 2 Re(h[d] exp(-2 pi i k d / n)); i = k d mod n
      a += 2.0 * (hr[d] * rn.first[i] + hi[d] * rn.second[i]);
      i += k;
      if (i >= n) i -= n;
    }
    spec[k] = (float)(a / W / n);
  }
}

void launch_gram_rows(const GramRows& g, const float2* D, float2* part, cudaStream_t st) {
  for (const auto& k : kGramKernels) {
    if (k.len.n != g.len.n || k.len.P != g.len.P) continue;
    const int per = (g.C + g.groups - 1) / g.groups;  // coils of the largest group, in equal passes
    const int passes = (per + gram_pass(g.len) - 1) / gram_pass(g.len);
    const int CB = (per + passes - 1) / passes;
    const size_t smem = gram_smem(g.len, CB, g.sens ? (passes > 1 ? 2 : 1) : 0);
    const RowsArgs a{g.W, g.H, g.C, CB, g.sens, g.coil_stride, g.tw, g.spec, D, part};
    PDT_CUDA_CHECK(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    LaunchEx lx(dim3(g.groups, g.H), dim3(kGramThreads), smem, st);
    PDT_CUDA_CHECK(cudaLaunchKernelEx(&lx.cfg, k.fn, a));
    count_launch();
    return;
  }
  throw Error(PDT_ERR_STATE, "no row kernel for transform length " + std::to_string(g.len.n));
}

void launch_gram_image(bool tgv, bool rows, const GramImage& s, cudaStream_t st) {
  LaunchEx lx(dim3((s.W + GX - 1) / GX, (s.H + GY - 1) / GY), dim3(GT), 0, st);
  auto fn = tgv ? (rows ? gram_image_kernel<true, true> : gram_image_kernel<true, false>)
                : (rows ? gram_image_kernel<false, true> : gram_image_kernel<false, false>);
  PDT_CUDA_CHECK(cudaLaunchKernelEx(&lx.cfg, fn, s));
  count_launch();
}

void launch_gram_start(int W, int H, const float2* part, int groups, const float2* ubar, float k, float2* w, float2* D,
                       float2* dots, cudaStream_t st) {
  const size_t n = (size_t)W * H;
  gram_dots_kernel<<<kGramDots, kStartThreads, 0, st>>>(n, w, part, groups, dots);
  PDT_LAUNCH_CHECK();
  gram_start_kernel<<<(unsigned)((n + kStartThreads - 1) / kStartThreads), kStartThreads, 0, st>>>(n, dots, ubar, k, w, D);
  PDT_LAUNCH_CHECK();
  count_launch(2);
}

void launch_gram_total(int W, int H, const float2* D, const float2* w, float c, float2* out, cudaStream_t st) {
  const size_t n = (size_t)W * H;
  gram_total_kernel<<<(unsigned)((n + kStartThreads - 1) / kStartThreads), kStartThreads, 0, st>>>(n, D, w, c, out);
  PDT_LAUNCH_CHECK();
  count_launch();
}

}  // namespace pdt
