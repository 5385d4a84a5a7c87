// pdt_image.cu -- the image side of the with-operator solvers (TV / TGV^2), as a dual and a primal kernel.
//
// Fields read at a neighbour (u-bar, v-bar, p, q) ping-pong between an `in` and an `out` buffer so that tiles
// never read a neighbour's freshly written values. The denoising solvers are in pdt_denoise.cu.
#include "pdt_device.cuh"
#include "pdt_internal.h"
#include "pdt_primal.cuh"

namespace pdt {
namespace {

constexpr int TX = 32;
constexpr int TY = 8;
constexpr int NT = TX * TY;

// ------------------------------------------------------------------------------------------------
// TgvMriOptimizer / TgvOptimizerWithOp / TvOptimizerWithOp image side (dual first, K^H r given), as two
// kernels: the dual one runs a solve's first dual update (the others belong to the image kernel of pdt_gram.cu, or to
// spare blocks of the operator's adjoint launch), the primal one every primal update of the latter route:
//   dual    p <- proj_a1(p + sigma (grad+ ub - vb)),  q <- proj_a0(q + sigma eps(vb))   (in -> out)
//   primal  u+ = u + tau (div- p - K^H r),            v+ = v + tau (div_h- q + p)       (p, q from out)
// u and v are read only at their own pixel and update in place; u-bar and v-bar go to `out`.
// iter[0] is the iteration index (incremented by the primal kernel, which runs after the dual kernel
// has read it), iter[1] the length of the alpha table, iter[2] the non-finite flag: the primal kernel
// sets it to 1 when a new u or v is not finite (NaN or infinite data or operator output propagate
// into u within an iteration or two); the host reads and clears it.
// ------------------------------------------------------------------------------------------------
template <bool TGV>
__global__ void __launch_bounds__(NT) mri_dual_kernel(int W, int H, ImgPtrs in, ImgPtrs out, float sigma,
                                                      const float* __restrict__ alpha_tab,
                                                      const int* __restrict__ iter) {
  const int x = blockIdx.x * TX + threadIdx.x % TX, y = blockIdx.y * TY + threadIdx.x / TX;
  if (x >= W || y >= H) return;
  float alpha0, alpha1;
  dual_alphas<TGV>(alpha_tab, iter, alpha0, alpha1);
  mri_dual_pixel<TGV>(W, H, in, out, sigma, alpha0, alpha1, x, y);
}

template <bool TGV>
__global__ void __launch_bounds__(NT) mri_primal_kernel(int W, int H, ImgPtrs out, const float2* __restrict__ khr,
                                                        int G, long long gstride, float tau, int* __restrict__ iter) {
  pdl_wait();  // K^H r comes from the previous kernel
  pdl_trigger();
  if (iter && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) atomicAdd(iter, 1);
  const int x = blockIdx.x * TX + threadIdx.x % TX, y = blockIdx.y * TY + threadIdx.x / TX;
  if (x >= W || y >= H) return;
  const size_t idx = (size_t)y * W + x;
  float2 kh = khr[idx];
  for (int g = 1; g < G; ++g) kh += khr[idx + (size_t)g * gstride];
  if (!mri_primal_pixel<TGV>(W, H, out, x, y, kh, tau) && iter) iter[2] = 1;
}

__global__ void tick_kernel(int* tick) { atomicAdd(tick, 1); }

inline dim3 tile_grid(int W, int H) { return dim3((W + TX - 1) / TX, (H + TY - 1) / TY); }

}  // namespace

void launch_mri_dual(bool tgv, int W, int H, const ImgPtrs& in, const ImgPtrs& out, float sigma,
                     const float* alpha_tab, const int* iter, cudaStream_t st) {
  if (tgv)
    mri_dual_kernel<true><<<tile_grid(W, H), NT, 0, st>>>(W, H, in, out, sigma, alpha_tab, iter);
  else
    mri_dual_kernel<false><<<tile_grid(W, H), NT, 0, st>>>(W, H, in, out, sigma, alpha_tab, iter);
  PDT_LAUNCH_CHECK();
  count_launch();
}

void launch_mri_primal(bool tgv, int W, int H, const ImgPtrs& out, const float2* khr, int G, long long gstride,
                       float tau, int* iter, cudaStream_t st) {
  LaunchEx lx(tile_grid(W, H), dim3(NT), 0, st);
  if (tgv)
    PDT_CUDA_CHECK(cudaLaunchKernelEx(&lx.cfg, mri_primal_kernel<true>, W, H, out, khr, G, gstride, tau, iter));
  else
    PDT_CUDA_CHECK(cudaLaunchKernelEx(&lx.cfg, mri_primal_kernel<false>, W, H, out, khr, G, gstride, tau, iter));
  count_launch();
}

void launch_tick(int* tick, cudaStream_t st) {
  tick_kernel<<<1, 1, 0, st>>>(tick);
  PDT_LAUNCH_CHECK();
  count_launch();
}

void launch_fill_zero(void* p, size_t bytes, cudaStream_t st) {
  if (bytes) PDT_CUDA_CHECK(cudaMemsetAsync(p, 0, bytes, st));
}

}  // namespace pdt
