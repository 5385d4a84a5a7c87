// pdt_denoise.cu -- TV and TGV^2 denoising: several primal-dual iterations per launch (temporal blocking).
//
// A block holds a region of RX x RY pixels, each thread a vertical strip of SR of them with its state in
// registers. An iteration reads one pixel to the right and below (gradients) and one to the left and above
// (divergences), so a region whose outermost `halo` rings are recomputed by its neighbours too is exact inside
// them after `halo` iterations; a region that covers the image needs no halo and takes any number. Neighbours
// along x, and those above and below a strip, come from shared memory; the others from the thread's registers.
//
// Arithmetic follows the reference kernels element by element:
//   grad+  (dp,   tgv_kernels.cuh:40-50)   Neumann forward differences, zero at x = W-1 / y = H-1
//   eps(v) (dp_sym, :25-38)                [dx vx, 0.5 (dy vx + dx vy), dy vy]
//   div-   (dm,   :67-80)                  x==0: p(0); x==W-1: -p(W-2); else p(x) - p(x-1)
//   div_h- (dm_sym, :104-134)
//   projections 1 / max(1, |.| / alpha) with |q|^2 = |qxx|^2 + |qyy|^2 + 2 |qxy|^2 (:136-154)
//   over-relaxation theta = 1: bar = 2 new - old.
// TvOptimizer is dual first (tvoptimizer.cu:76-125), TgvOptimizer primal first (tgvoptimizer.cu:117-137).
#include <algorithm>

#include "pdt_device.cuh"
#include "pdt_internal.h"

namespace pdt {
namespace {

// 1 / max(1, sqrt(n2) / alpha). Below inside = alpha^2 (1 - 2^-20) the root is certainly at most alpha and the
// quotient at most one, so the root and both divisions are skipped with the same result.
__device__ __forceinline__ float proj(float n2, float alpha, float inside) {
  if (n2 <= inside) return 1.0f;
  return 1.0f / fmaxf(1.0f, sqrtf(n2) / alpha);
}

struct DenoiseArgs {
  int W, H, halo, steps, store_bar;
  ImgPtrs in, out;
  const void* f;
  float tau, sigma, lambda, alpha0, alpha1, inside0, inside1;  // see proj()
};

template <class P, bool TGV, int RX, int RY, int SR, int MINB>
__global__ void __launch_bounds__(RX* RY / SR, MINB) denoise_kernel(DenoiseArgs a) {
  constexpr int N = RX * RY, NS = RX * (RY / SR);
  extern __shared__ __align__(16) unsigned char dn_smem[];
  // one element before and after each plane: the x neighbours of the region's corners (values never used)
  P* sm = reinterpret_cast<P*>(dn_smem) + 1;
  P* s_ub = sm;                                // u-bar
  P* s_px = sm + (N + 2);                      // p_x
  P* s_py = sm + 2 * (N + 2);                  // p_y, last row of each strip
  P* s_vx = s_py + (NS + 2);                   // v-bar
  P* s_vy = s_vx + (N + 2);
  P* s_qxx = s_vy + (N + 2);
  P* s_qxy = s_qxx + (N + 2);
  P* s_qyy = s_qxy + (N + 2);                  // last row of each strip
  const int W = a.W, H = a.H, tid = threadIdx.x;
  const int lx = tid % RX, st = tid / RX, ly = st * SR;
  const int gx = blockIdx.x * (RX - 2 * a.halo) - a.halo + lx;
  const int gy = blockIdx.y * (RY - 2 * a.halo) - a.halo + ly;
  const bool inx = gx >= 0 && gx < W;
  const bool xl = gx > 0, xr = gx < W - 1;
  const int up = st > 0 ? (st - 1) * RX + lx : 0;                   // last row of the strip above
  const int dn = ly + SR < RY ? (ly + SR) * RX + lx : ly * RX + lx;  // first row of the strip below
  const P zero = pzero<P>();
  P u[SR], f[SR], px[SR], py[SR], ub[SR], vx[SR], vy[SR], vbx[SR], vby[SR], qxx[SR], qyy[SR], qxy[SR];
  auto ld = [](const void* p, size_t i) { return static_cast<const P*>(p)[i]; };
#pragma unroll
  for (int j = 0; j < SR; ++j) {
    const bool ok = inx && gy + j >= 0 && gy + j < H;
    f[j] = ok ? ld(a.f, (size_t)(gy + j) * W + gx) : zero;
  }
  pdl_wait();  // f is constant; the state comes from the previous launch
  pdl_trigger();
#pragma unroll
  for (int j = 0; j < SR; ++j) {
    const bool ok = inx && gy + j >= 0 && gy + j < H;
    const size_t i = ok ? (size_t)(gy + j) * W + gx : 0;
    u[j] = ok ? ld(a.in.u, i) : zero;
    px[j] = ok ? ld(a.in.px, i) : zero;
    py[j] = ok ? ld(a.in.py, i) : zero;
    if constexpr (TGV) {
      vx[j] = ok ? ld(a.in.vx, i) : zero;
      vy[j] = ok ? ld(a.in.vy, i) : zero;
      qxx[j] = ok ? ld(a.in.qxx, i) : zero;
      qyy[j] = ok ? ld(a.in.qyy, i) : zero;
      qxy[j] = ok ? ld(a.in.qxy, i) : zero;
    } else {
      ub[j] = ok ? ld(a.in.ub, i) : zero;
    }
  }
  const float inv = 1.0f / (1.0f + a.tau * a.lambda);
  const float a1 = TGV ? a.alpha1 : 1.0f;
  const float in0 = a.inside0, in1 = a.inside1;
  // div- along x of a plane at row j (its value c there) and along y from the value above
  auto dx = [&](P c, const P* s, int j) {
    const P l = s[(ly + j) * RX + lx - 1];
    return xl ? (xr ? c - l : -l) : c;
  };
  auto dy = [&](P c, P prev, int j) { return gy + j > 0 ? (gy + j < H - 1 ? c - prev : -prev) : c; };
  auto put_dual = [&]() {
#pragma unroll
    for (int j = 0; j < SR; ++j) {
      const int i = (ly + j) * RX + lx;
      s_px[i] = px[j];
      if constexpr (TGV) {
        s_qxx[i] = qxx[j];
        s_qxy[i] = qxy[j];
      }
    }
    s_py[st * RX + lx] = py[SR - 1];
    if constexpr (TGV) s_qyy[st * RX + lx] = qyy[SR - 1];
  };
  auto put_bar = [&]() {
#pragma unroll
    for (int j = 0; j < SR; ++j) {
      const int i = (ly + j) * RX + lx;
      s_ub[i] = ub[j];
      if constexpr (TGV) {
        s_vx[i] = vbx[j];
        s_vy[i] = vby[j];
      }
    }
  };
  auto dual = [&]() {  // tgv_kernels.cuh:225-324
#pragma unroll
    for (int j = 0; j < SR; ++j) {
      const int i = (ly + j) * RX + lx;
      const bool yn = gy + j < H - 1;
      const P c = ub[j];
      const P r = xr ? s_ub[i + 1] : c, d = yn ? (j + 1 < SR ? ub[j + 1 < SR ? j + 1 : j] : s_ub[dn]) : c;
      P ex = r - c, ey = d - c;
      if constexpr (TGV) {
        ex = ex - vbx[j];
        ey = ey - vby[j];
      }
      const P e = px[j] + a.sigma * ex, g = py[j] + a.sigma * ey;
      const float s = proj(abs2(e) + abs2(g), a1, in1);
      px[j] = e * s;
      py[j] = g * s;
      if constexpr (TGV) {
        const P wx = vbx[j], wy = vby[j];
        const P rx = xr ? s_vx[i + 1] : wx, ry = xr ? s_vy[i + 1] : wy;
        const P bx = yn ? (j + 1 < SR ? vbx[j + 1 < SR ? j + 1 : j] : s_vx[dn]) : wx;
        const P by = yn ? (j + 1 < SR ? vby[j + 1 < SR ? j + 1 : j] : s_vy[dn]) : wy;
        const P qa = qxx[j] + a.sigma * (rx - wx);
        const P qb = qyy[j] + a.sigma * (by - wy);
        const P qc = qxy[j] + a.sigma * (0.5f * (bx - wx + ry - wy));
        const float t = proj(abs2(qa) + abs2(qb) + 2.0f * abs2(qc), a.alpha0, in0);
        qxx[j] = qa * t;
        qyy[j] = qb * t;
        qxy[j] = qc * t;
      }
    }
  };
  auto primal = [&]() {  // tgv_kernels.cuh:568-605, 647-686
#pragma unroll
    for (int j = 0; j < SR; ++j) {
      const P pyu = j ? py[j ? j - 1 : 0] : s_py[up];
      P un = u[j] + a.tau * ((dx(px[j], s_px, j) + dy(py[j], pyu, j)) + a.lambda * f[j]);
      un = un * inv;
      ub[j] = 2.0f * un - u[j];
      u[j] = un;
      if constexpr (TGV) {
        const P qyu = j ? qyy[j ? j - 1 : 0] : s_qyy[up];
        const P qcu = j ? qxy[j ? j - 1 : 0] : s_qxy[ly > 0 ? (ly - 1) * RX + lx : 0];
        const P nx = vx[j] + a.tau * ((dx(qxx[j], s_qxx, j) + dy(qxy[j], qcu, j)) + px[j]);
        const P ny = vy[j] + a.tau * ((dy(qyy[j], qyu, j) + dx(qxy[j], s_qxy, j)) + py[j]);
        vbx[j] = 2.0f * nx - vx[j];
        vby[j] = 2.0f * ny - vy[j];
        vx[j] = nx;
        vy[j] = ny;
      }
    }
  };
  if constexpr (TGV) {
    put_dual();
    __syncthreads();
#pragma unroll 1
    for (int it = 0; it < a.steps; ++it) {
      primal();
      put_bar();
      __syncthreads();
      dual();
      put_dual();
      __syncthreads();
    }
  } else {
    put_bar();
    __syncthreads();
#pragma unroll 1
    for (int it = 0; it < a.steps; ++it) {
      dual();
      put_dual();
      __syncthreads();
      primal();
      put_bar();
      __syncthreads();
    }
  }
  if (!inx || lx < a.halo || lx >= RX - a.halo) return;
#pragma unroll
  for (int j = 0; j < SR; ++j) {
    if (ly + j < a.halo || ly + j >= RY - a.halo || gy + j >= H) continue;
    const size_t i = (size_t)(gy + j) * W + gx;
    auto put = [&](void* p, P v) { static_cast<P*>(p)[i] = v; };
    put(a.out.u, u[j]);
    put(a.out.px, px[j]);
    put(a.out.py, py[j]);
    if (!TGV || a.store_bar) put(a.out.ub, ub[j]);
    if constexpr (TGV) {
      put(a.out.vx, vx[j]);
      put(a.out.vy, vy[j]);
      put(a.out.qxx, qxx[j]);
      put(a.out.qyy, qyy[j]);
      put(a.out.qxy, qxy[j]);
      if (a.store_bar) {
        put(a.out.vbx, vbx[j]);
        put(a.out.vby, vby[j]);
      }
    }
  }
}

template <class P, bool TGV, int RX, int RY, int SR, int MINB>
void launch_region(DenoiseArgs a, cudaStream_t st) {
  constexpr size_t N = RX * RY + 2, NS = RX * (RY / SR) + 2;
  constexpr size_t smem = sizeof(P) * (TGV ? 6 * N + 2 * NS : 2 * N + NS) + 16;
  auto fn = denoise_kernel<P, TGV, RX, RY, SR, MINB>;
  PDT_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int cx = RX - 2 * a.halo, cy = RY - 2 * a.halo;
  LaunchEx lx(dim3((a.W + cx - 1) / cx, (a.H + cy - 1) / cy), dim3(RX * RY / SR), smem, st);
  PDT_CUDA_CHECK(cudaLaunchKernelEx(&lx.cfg, fn, a));
  count_launch();
}

// Regions: 0: 32 x 32 on 512 threads (two rows a thread), 1: 32 x 32 on 256 threads, 2: 32 x 24 on 192.
template <class P, bool TGV>
void launch_any(int region, const DenoiseArgs& a, cudaStream_t st) {
  if constexpr (TGV && sizeof(P) == 4) {
    if (region == 2) return launch_region<P, TGV, 32, 24, 4, 3>(a, st);
  }
  if (region == 0)
    launch_region<P, TGV, 32, 32, 2, sizeof(P) == 4 ? 2 : 1>(a, st);
  else
    launch_region<P, TGV, 32, 32, 4, sizeof(P) == 4 || !TGV ? 3 : 2>(a, st);
}

}  // namespace

// More iterations a launch save launches and passes over the state and cost recomputed rings: 8 rings leave a quarter
// of a 32 x 32 region, 3 two thirds. Measured (us an iteration; solves back to back / alone; before: one TGV and
// four TV iterations a launch, index arithmetic and every value in shared memory):
//   64 x 48 TV f32      8: 0.35 / 0.69   6: 0.39 / 0.76   4: 0.47 / 0.92   (before 0.94 / 2.9)
//   250 x 200 TGV f32   6: 0.90 / 1.36   4: 0.95 / 1.53   8: 1.04 / 1.77
//   512 x 512 TV f32    3: 1.20 / 1.82   4: 1.24 / 1.90   2: 1.30 / 2.5    (before 2.28 / 3.8)
//   512 x 512 TGV f32   3: 2.36 / 3.41   4: 2.48 / 3.49                    (before 3.91 / 6.2)
//   4096 x 4096 TGV c64 3: 250  2: 276   4: 268                           (before 484, HBM-bound at 5.7 TB/s)
// Large images run on regions with more pixels a thread and more blocks an SM (512 x 512 TV c64: region 1 1.59,
// region 0 1.73; 4096 x 4096 TGV f32: region 2 132, 1 134, 0 142); there the instructions bound it (square roots,
// divisions, neighbours), not the 17 planes a launch.
// The lines lie where a count of blocks passes a whole wave, which depends on the sides rather than the area. Both sides,
// us an iteration of 121 back to back, TV f32 / TGV f32 / TV c64 / TGV c64:
//   181^2  8: 0.77 1.19 0.88 1.56   6: 0.84 1.25 0.97 1.69      200^2  8: 0.97 1.66 1.19 2.76   6: 0.83 1.25 0.96 1.69
//   362^2  6: 1.37 2.58 1.90 4.49   3: 1.44 2.34 1.88 3.81      400^2  6: 1.40 2.62 1.95 4.56   3: 1.77 2.39 2.32 3.95
//   632^2  region 0, f32: 2.69 5.02   1 or 2: 2.62 4.84          720^2  region 0, f32: 3.14 5.98   1 or 2: 3.10 5.86
// Four iterations are faster than the rule's number in some waves between (256^2 TGV f32 1.45 against 1.78, 448^2 TV f32
// 1.59 against 1.83, 720^2 TGV f32 5.31 against 5.86): the rule does not count blocks.
int denoise_steps(bool complex_, bool tgv, int W, int H, int iters, int* region) {
  const size_t n = (size_t)W * H;
  *region = 0;
  if (W <= 32 && H <= 32) return iters;  // one block holds the image
  if (n < 32768) return std::min(8, iters);
  if (n < 131072) return std::min(6, iters);
  if (complex_ || n >= 400000) *region = tgv && !complex_ ? 2 : 1;
  return std::min(3, iters);
}

void launch_denoise(bool complex_, bool tgv, int W, int H, const ImgPtrs& in, const ImgPtrs& out, const void* f, float tau,
                    float sigma, float lambda, float alpha0, float alpha1, int region, int halo, int steps,
                    bool store_bar, cudaStream_t st) {
  // the shortcut of proj() only where alpha^2 neither overflows (with n2 = inf the result is 0) nor loses bits to underflow
  auto inside = [](float al) { return al >= 0x1p-60f && al <= 0x1p60f ? al * al * (1.0f - 0x1p-20f) : -1.0f; };
  const DenoiseArgs a{W,     H,      halo,   steps,  store_bar ? 1 : 0, in,
                      out,   f,      tau,    sigma,  lambda,            alpha0,
                      alpha1, inside(alpha0), inside(tgv ? alpha1 : 1.0f)};
  if (complex_)
    tgv ? launch_any<float2, true>(region, a, st) : launch_any<float2, false>(region, a, st);
  else
    tgv ? launch_any<float, true>(region, a, st) : launch_any<float, false>(region, a, st);
}

}  // namespace pdt
