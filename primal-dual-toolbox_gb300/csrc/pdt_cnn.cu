// pdt_cnn.cu -- the learned warm start: a small residual CNN with BF16 weights and activations and FP32
// accumulation, trained and run by the engine's own kernels.
//
// Network (fully convolutional, 3 x 3 convolutions, zero padding, channel-last BF16 activations):
//   x  = [Re u0, Im u0] / s                       (u0 = A^H f, s = max |u0|)
//   h1 = relu(conv_in(x))                          2 -> 32
//   h_{l+1} = h_l + relu(conv_l(h_l)), l = 1..6    32 -> 32
//   o  = conv_out(h7)                              32 -> 8 (6 used)
//   u  = u0 + s (o0 + i o1),  v = s (o2 + i o3, o4 + i o5)
// Eight convolutions in all. All but the first run as implicit GEMMs on the tensor cores (tcgen05, BF16 in, FP32
// accumulate): pixels are the M dimension, output channels N, and (tap, input channel) K. The data gradient is the
// same kernel with flipped taps and transposed channels; the weight gradient is a second implicit GEMM with pixels
// as K, reduced over blocks in block order.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <memory>
#include <vector>

#include "pdt_device.cuh"
#include "pdt_internal.h"
#include "pdt_tc.cuh"

namespace pdt {
namespace {

typedef __nv_bfloat16 bf16;

constexpr int CH = 32;    // hidden channels
constexpr int TW = 16;    // the weight gradients' pixel tile: K = TW pixels an MMA
constexpr int TH = 8;
constexpr int NTAP = 9;

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// The pair of BF16 values g where the pair z is positive, else zero.
__device__ __forceinline__ uint32_t relu_mask(uint32_t g, uint32_t z) {
  const __nv_bfloat162 zz = *reinterpret_cast<const __nv_bfloat162*>(&z);
  return (__bfloat162float(zz.x) > 0.f ? g & 0xFFFFu : 0u) | (__bfloat162float(zz.y) > 0.f ? g & 0xFFFF0000u : 0u);
}

enum Epi {
  EPI_RELU_RES = 2,  // zsave = z, out = in + relu(z)   (CIN == COUT)
  EPI_F32 = 3,       // out32 = z (FP32)
  EPI_ACC = 4,       // acc32 += bf16(z)  (a residual stream's FP32 gradient; the BF16 rounding of a stored z), and
                     // out = bf16(acc32) where zsave (read) > 0, else 0: the gradient at the layer below
  EPI_F32_BF16 = 5   // out32 = bf16(z), stored as FP32 (starts a residual stream's gradient), and out likewise
};

// 3 x 3 convolution of CIN = 32 or 16 to COUT = 32 or 8 channels on the fifth-generation tensor cores (tcgen05
// kind::f16, BF16 operands, FP32 accumulator in tensor memory), as an implicit GEMM without an im2col copy: the
// hidden layers, their data gradients, the output layer (its 8 channels padded to N = 16) and the output layer's data
// gradient (16 padded input channels). One CTA computes a tile of 8 x 16 pixels (x, y) = the 128 rows of one MMA tile,
// rows ordered y-major. The input tile with its one-pixel zero halo (10 x 18 pixels) sits in shared memory in the
// no-swizzle K-major layout: channel group g (8 channels, 16 bytes) of pixel p at byte g kGroup + 16 p, so eight
// consecutive pixels form a core matrix (four groups are two pixels further apart, which puts the groups of a pixel in
// different bank quarters, so the halo's 16-byte stores do not conflict); the 8-pixel groups of the M tile are one
// halo row (160 bytes) apart, and tap (ky, kx) is the same layout started 16 (10 ky + kx) bytes in. The weights sit
// the same way ([tap][g][co] x 16 bytes). K = (tap, channel) in MMAs of K = 16 (two channel groups). One thread issues
// the MMAs and commits them to an mbarrier; the epilogue reads pixel rows from tensor memory (warps q and q + 4 share
// lane quarter q, and half the output channels each).
constexpr int kConvTcThreads = 256;
constexpr int kConvTcTW = 8, kConvTcTH = 16;                      // tile: 8 pixels wide, 16 rows
constexpr int kConvTcHaloPix = (kConvTcTW + 2) * (kConvTcTH + 2);  // 180
constexpr int kConvTcBufs = 3;

template <int CIN, int COUT>
struct ConvTc {
  static constexpr int kGroups = CIN / 8, kN = COUT < 16 ? 16 : COUT;
  static constexpr uint32_t kGroup = 16 * (kConvTcHaloPix + (kGroups == 4 ? 2 : 0));  // one channel group of the tile
  static constexpr uint32_t kIn = kGroups * kGroup, kW = NTAP * kGroups * kN * 16;
  // The farthest operand byte an MMA reads: A at tap (2, 2), the last two channel groups: 16 (2 10 + 2) +
  // (kGroups - 1) kGroup + 15 160 (last 8-pixel group) + 128 = (kGroups - 1) kGroup + 2880 <= kIn; B at tap 8, the last
  // two groups: the end of its kN rows, kW. Two mbarriers, the tensor-memory slot and the kN biases (FP32) follow.
  static constexpr size_t kSmem = 1024 + kConvTcBufs * kIn + kW + 32 + 4 * kN;
  static constexpr int kItems = kConvTcHaloPix * kGroups;                             // 16-byte items per tile
  static constexpr int kPre = (kItems + kConvTcThreads - 1) / kConvTcThreads;  // per thread
  static constexpr uint32_t kCols = 2 * kN < 32 ? 32 : 2 * kN;                         // two accumulators
};

__device__ __forceinline__ void ld_shared_v4(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Persistent: a CTA loads the weights once and walks tiles t = blockIdx.x, + gridDim.x, ... of the
// (x tiles) x (y tiles) x B grid in a pipeline: while tile t's epilogue runs, tile t + 1's MMAs run (its halo was stored
// before tile t's wait, into the next of three buffers, and it has the other accumulator) and tile t + 2's halo is on
// its way into registers. Three buffers, because a slower warp may still read tile t - 1's residual input: one barrier
// a tile. Each accumulator has its mbarrier, whose phase alternates with its uses.
// The FP32 residual gradient acc32 belongs to these kernels alone: float4 ((tile 8 + (channel / 4)) 128 + pixel row m),
// so that a warp's accesses are contiguous (at [pixel][channel] they touched 32 lines each).
// 4 x 320 x 320, cold, before and after pipeline and layout: hidden layer 31.7 -> 29.3 us, data gradient 59.6 -> 41.0
// (184 MB: 27 at copy rate), output layer 32.3 -> 19.4 and its data gradient 38.1 -> 25.2 (warp MMAs before).
template <int EPI, int CIN, int COUT>
__global__ void __launch_bounds__(kConvTcThreads, 4) conv3x3_tc(const bf16* __restrict__ in, const bf16* __restrict__ w,
                                                            const float* __restrict__ bias, int B, int H, int W,
                                                            bf16* __restrict__ out, bf16* __restrict__ zsave,
                                                            int* __restrict__ err, float* __restrict__ f32) {
  using C = ConvTc<CIN, COUT>;
  static_assert(EPI == EPI_F32 ? COUT == 8 : COUT == 32, "epilogues");
  static_assert(EPI != EPI_RELU_RES || CIN == COUT, "residual layers");
  extern __shared__ unsigned char conv_smem_raw[];
  const uint32_t off = tc::smem_addr(conv_smem_raw);
  unsigned char* sm = conv_smem_raw + ((1024u - (off & 1023u)) & 1023u);
  const uint32_t in_base = tc::smem_addr(sm), w_base = in_base + kConvTcBufs * C::kIn;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kConvTcBufs * C::kIn + C::kW);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
  float* bias_s = reinterpret_cast<float*>(bar + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntx = (W + kConvTcTW - 1) / kConvTcTW, nty = (H + kConvTcTH - 1) / kConvTcTH;
  const int ntiles = ntx * nty * B;
  if (tid < COUT) bias_s[tid] = bias ? bias[tid] : 0.f;
  if (tid == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tslot, C::kCols);
  // weights: item (tap, group, co) at byte ((tap kGroups + g) kN + co) 16, zero past COUT
  for (int i = tid; i < NTAP * C::kGroups * C::kN; i += kConvTcThreads) {
    const int co = i % C::kN, g = (i / C::kN) % C::kGroups, tap = i / (C::kN * C::kGroups);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (co < COUT) v = __ldg(reinterpret_cast<const uint4*>(w + ((size_t)tap * COUT + co) * CIN) + g);
    st_shared_v4(w_base + 16 * i, v);
  }
  const int q = warp & 3, h = warp >> 2;
  // the halo of tile t: item i = (pixel, channel group) of 16 bytes, zero outside the image
  uint4 pre[C::kPre];
  auto fetch = [&](int t) {
    const int bx = t % ntx, by = (t / ntx) % nty, b = t / (ntx * nty);
    const int x0 = bx * kConvTcTW, y0 = by * kConvTcTH;
    const bf16* inb = in + (size_t)b * H * W * CIN;
#pragma unroll
    for (int j = 0; j < C::kPre; ++j) {
      const int i = tid + j * kConvTcThreads;
      const int g = i % C::kGroups, pix = i / C::kGroups;
      const int hy = pix / (kConvTcTW + 2), hx = pix - hy * (kConvTcTW + 2);
      const int gy = y0 + hy - 1, gx = x0 + hx - 1;
      pre[j] = make_uint4(0u, 0u, 0u, 0u);
      if (i < C::kItems && gy >= 0 && gy < H && gx >= 0 && gx < W)
        pre[j] = __ldg(reinterpret_cast<const uint4*>(inb + ((size_t)gy * W + gx) * CIN) + g);
    }
  };
  auto stage = [&](uint32_t buf) {
#pragma unroll
    for (int j = 0; j < C::kPre; ++j) {
      const int i = tid + j * kConvTcThreads;
      if (i < C::kItems) st_shared_v4(buf + (i % C::kGroups) * C::kGroup + 16 * (i / C::kGroups), pre[j]);
    }
    tc::fence_async_smem();
  };
  uint32_t tmem = 0;
  auto issue = [&](uint32_t buf, int s) {  // the MMAs of the CTA's tile number s, by one thread
    const uint32_t idesc = tc::idesc_bf16(128, C::kN), d = tmem + C::kN * (s & 1);
    for (int tap = 0; tap < NTAP; ++tap) {
      const uint32_t a0 = buf + 16 * ((tap / 3) * (kConvTcTW + 2) + tap % 3);
      for (int k = 0; k < C::kGroups / 2; ++k)  // channel groups 2k, 2k + 1
        tc::mma_bf16(d, tc::desc_interleave(a0 + 2 * k * C::kGroup, C::kGroup, 16 * (kConvTcTW + 2)),
                     tc::desc_interleave(w_base + (tap * C::kGroups + 2 * k) * (16 * C::kN), 16 * C::kN, 128), idesc,
                     (tap | k) ? 1u : 0u);
    }
    tc::mma_commit(&bar[s & 1]);
  };
  const int step = gridDim.x;
  uint32_t cur = in_base, nxt = in_base + C::kIn;  // buffers of this tile and the next
  if ((int)blockIdx.x < ntiles) {
    fetch(blockIdx.x);
    stage(cur);
  }
  if ((int)blockIdx.x + step < ntiles) fetch(blockIdx.x + step);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  tmem = *tslot;
  // (the test hook withholds block 0's first tile: no MMAs and no commit, so the wait below runs out)
  if (tid == 0 && (int)blockIdx.x < ntiles && !(blockIdx.x == 0 && tc::g_drop_arrival)) issue(cur, 0);
  bool ok = true;
  int it = 0;
  for (int t = blockIdx.x; t < ntiles; t += step, ++it) {
    if (t + step < ntiles) {  // tile it + 1 of the grid: its MMAs run while this tile's epilogue does
      stage(nxt);
      tc::fence_before_sync();
      ok = __syncthreads_and(ok);
      tc::fence_after_sync();
      if (!ok) break;  // an earlier wait gave up; this tile's MMAs may be in flight (waited for below)
      if (tid == 0) issue(nxt, it + 1);
      if (t + 2 * step < ntiles) fetch(t + 2 * step);
    }
    const int bx = t % ntx, by = (t / ntx) % nty, b = t / (ntx * nty);
    const int m = 32 * q + lane, gy = by * kConvTcTH + (m >> 3), gx = bx * kConvTcTW + (m & 7);  // row m = pixel (m % 8, m / 8)
    const bool inside = gy < H && gx < W;
    const size_t pix = ((size_t)b * H + gy) * W + gx;
    // the accumulated gradient and the layer below's pre-activation, loaded while the MMAs run
    float4* ap = reinterpret_cast<float4*>(f32) + ((size_t)t * 8 + 4 * h) * 128 + m;
    float4 acc_in[4];
    uint4 zin[2];
    if constexpr (EPI == EPI_ACC || EPI == EPI_F32_BF16) {
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) acc_in[q4] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (inside) {
        const uint4* zp = reinterpret_cast<const uint4*>(zsave + pix * CH + 16 * h);
        zin[0] = zp[0];
        zin[1] = zp[1];
        if (EPI == EPI_ACC)
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) acc_in[q4] = ap[128 * q4];
      }
    }
    const bool done = tc::mbar_wait(&bar[it & 1], (it >> 1) & 1);  // every thread waits each phase in turn
    // after a give-up, wait once more (bounded) for MMAs still in flight before the tile buffer, the
    // accumulator and finally the tensor memory are released
    if (!done) tc::mbar_wait(&bar[it & 1], (it >> 1) & 1);
    ok = ok && done;
    tc::fence_after_sync();
    float v[16];
    tc::tmem_ld16(tmem + C::kN * (it & 1) + ((uint32_t)(32 * q) << 16) + (C::kN == 32 ? 16 * h : 0), v);
    if (ok && inside) {
      if constexpr (EPI == EPI_F32) {  // channels 4 h .. 4 h + 3
        float4 y;
        y.x = (h ? v[4] : v[0]) + bias_s[4 * h];
        y.y = (h ? v[5] : v[1]) + bias_s[4 * h + 1];
        y.z = (h ? v[6] : v[2]) + bias_s[4 * h + 2];
        y.w = (h ? v[7] : v[3]) + bias_s[4 * h + 3];
        reinterpret_cast<float4*>(f32 + pix * 8)[h] = y;
      } else if constexpr (EPI == EPI_RELU_RES) {
        uint32_t o[8], zz[8], res[8];
        float bs[16];
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint32_t r[4];
          ld_shared_v4(tc::smem_addr(bias_s) + 64 * h + 16 * q4, r);
#pragma unroll
          for (int e = 0; e < 4; ++e) bs[4 * q4 + e] = __uint_as_float(r[e]);
        }
        // the residual input: this pixel's channels 16 h .. 16 h + 15 in the tile
        const uint32_t hp = cur + 16 * (((m >> 3) + 1) * (kConvTcTW + 2) + (m & 7) + 1);
        ld_shared_v4(hp + 2 * h * C::kGroup, *reinterpret_cast<uint32_t(*)[4]>(&res[0]));
        ld_shared_v4(hp + (2 * h + 1) * C::kGroup, *reinterpret_cast<uint32_t(*)[4]>(&res[4]));
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // output channels 16 h + 2 j, + 1
          const float z0 = v[2 * j] + bs[2 * j], z1 = v[2 * j + 1] + bs[2 * j + 1];
          zz[j] = pack_bf16(z0, z1);
          const __nv_bfloat162 hv = *reinterpret_cast<const __nv_bfloat162*>(&res[j]);
          o[j] = pack_bf16(__bfloat162float(hv.x) + fmaxf(z0, 0.f), __bfloat162float(hv.y) + fmaxf(z1, 0.f));
        }
        uint4* op = reinterpret_cast<uint4*>(out + pix * CH + 16 * h);
        op[0] = make_uint4(o[0], o[1], o[2], o[3]);
        op[1] = make_uint4(o[4], o[5], o[6], o[7]);
        if (zsave) {  // (inference keeps no pre-activations)
          uint4* zp = reinterpret_cast<uint4*>(zsave + pix * CH + 16 * h);
          zp[0] = make_uint4(zz[0], zz[1], zz[2], zz[3]);
          zp[1] = make_uint4(zz[4], zz[5], zz[6], zz[7]);
        }
      } else {
        uint32_t o[8];
        const uint32_t zi[8] = {zin[0].x, zin[0].y, zin[0].z, zin[0].w, zin[1].x, zin[1].y, zin[1].z, zin[1].w};
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          float4 a = acc_in[q4];
          const __nv_bfloat162 lo = __floats2bfloat162_rn(v[4 * q4], v[4 * q4 + 1]);
          const __nv_bfloat162 hi = __floats2bfloat162_rn(v[4 * q4 + 2], v[4 * q4 + 3]);
          a.x += __bfloat162float(lo.x);
          a.y += __bfloat162float(lo.y);
          a.z += __bfloat162float(hi.x);
          a.w += __bfloat162float(hi.y);
          ap[128 * q4] = a;
          // ReLU's derivative on the rounded gradient
          o[2 * q4] = relu_mask(pack_bf16(a.x, a.y), zi[2 * q4]);
          o[2 * q4 + 1] = relu_mask(pack_bf16(a.z, a.w), zi[2 * q4 + 1]);
        }
        uint4* gp = reinterpret_cast<uint4*>(out + pix * CH + 16 * h);
        gp[0] = make_uint4(o[0], o[1], o[2], o[3]);
        gp[1] = make_uint4(o[4], o[5], o[6], o[7]);
      }
    }
    cur = nxt;
    nxt = nxt + C::kIn < w_base ? nxt + C::kIn : in_base;
  }
  // left early: the tile whose turn it was has its MMAs in flight (bounded)
  if (!ok && (int)blockIdx.x + it * step < ntiles) tc::mbar_wait(&bar[it & 1], (it >> 1) & 1);
  if (!ok) atomicExch(err, 0x2000);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, C::kCols);
  }
}

// Weight and bias gradient of a layer with 32 input channels on the tensor cores (tcgen05, kind::f16 BF16, FP32 in TMEM):
//   dW[ky 3 + kx][co][ci] = sum_p x[p + (ky - 1, kx - 1)][ci] dy[p][co],   db[co] = sum_p dy[p][co]
// as D_ky[m = kx 32 + ci][n = co] = sum_k A[k][m] B[k][n] with K = the 16 pixels of one tile row: A is the input tile
// shifted by kx, B the output gradient, and row 96 of A is one everywhere, so that row 96 of D is the bias gradient
// (rows 97 .. 127 are not read). Per 16 x 8 tile and tile row py, three MMAs (ky = 0, 1, 2: A from halo row py + ky) of
// M = 128, N = NC, K = 16 into three accumulators (TMEM columns NC ky). Both operands are MN-major, as the
// activations lie in memory: a core matrix is 8 pixels (rows, 16 bytes each) x 8 channels, channel group after
// channel group kWgGroupA / kWgGroupB apart, pixels 16 bytes apart, so staging is 16-byte copies (the K-major form
// needed a 2-byte store per value: 57 us a layer at 4 x 320 x 320 against 25; the
// reduction 11 us against 9). The group strides put the four groups of a
// pixel in different banks. The next tile is loaded into registers while this tile's MMAs run. CTAs are persistent
// over tiles and accumulate in TMEM; each writes partial[block][tap][co < COUT][ci] and [co < COUT], which
// wgrad_sum adds in block order. dy holds NC channels a pixel (COUT of them used).
constexpr int kWgThreads = 256;
constexpr uint32_t kWgGroupA = 16 * (10 * 16 + 2);  // 2592
constexpr uint32_t kWgGroupB = 16 * (8 * 16 + 2);   // 2080
constexpr uint32_t kWgA = 13 * kWgGroupA;           // 12 groups of x, one of ones; groups 13 .. 15 are read past it:
constexpr uint32_t kWgEnd = 16 * kWgGroupA > kWgA + 4 * kWgGroupB ? 16 * kWgGroupA : kWgA + 4 * kWgGroupB;
constexpr size_t kWgSmem = 1024 + kWgEnd + 64;
constexpr int kWgPerSm = 4;  // CTAs per SM: 128 TMEM columns and 43 KB each

template <int NC, int COUT>
__global__ void __launch_bounds__(kWgThreads, kWgPerSm) wgrad_tc(const bf16* __restrict__ x, const bf16* __restrict__ dy, int B,
                                                       int H, int W, float* __restrict__ partial, int* __restrict__ err) {
  constexpr uint32_t kCols = NC == 32 ? 128 : 64;
  constexpr int kX = (TH + 2) * (TW + 2) * 4, kPreX = (kX + kWgThreads - 1) / kWgThreads;
  constexpr int kD = TH * TW * (NC / 8), kPreD = (kD + kWgThreads - 1) / kWgThreads;
  extern __shared__ unsigned char wg_smem_raw[];
  const uint32_t off = tc::smem_addr(wg_smem_raw);
  unsigned char* sm = wg_smem_raw + ((1024u - (off & 1023u)) & 1023u);
  const uint32_t a_base = tc::smem_addr(sm), b_base = a_base + kWgA;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kWgEnd);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntx = (W + TW - 1) / TW, nty = (H + TH - 1) / TH;
  const int ntiles = ntx * nty * B;
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tslot, kCols);
  for (int i = tid; i < (TH + 2) * TW; i += kWgThreads)  // the ones: BF16 1 in the group's first channel
    st_shared_v4(a_base + 12 * kWgGroupA + 16 * i, make_uint4(0x3F80u, 0u, 0u, 0u));
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  const bool drop = tc::g_drop_arrival != 0;
  uint4 px[kPreX], pd[kPreD];
  auto fetch = [&](int t) {
    const int bx = t % ntx, by = (t / ntx) % nty, b = t / (ntx * nty);
    const int x0 = bx * TW, y0 = by * TH;
#pragma unroll
    for (int j = 0; j < kPreX; ++j) {  // item (halo row, halo column, channel group)
      const int i = tid + j * kWgThreads, cg = i & 3, col = (i >> 2) % (TW + 2), hy = (i >> 2) / (TW + 2);
      const int gy = y0 + hy - 1, gx = x0 + col - 1;
      px[j] = make_uint4(0u, 0u, 0u, 0u);
      if (i < kX && gy >= 0 && gy < H && gx >= 0 && gx < W)
        px[j] = __ldg(reinterpret_cast<const uint4*>(x + (((size_t)b * H + gy) * W + gx) * CH) + cg);
    }
#pragma unroll
    for (int j = 0; j < kPreD; ++j) {  // item (tile row, pixel, channel group)
      const int i = tid + j * kWgThreads, cg = i % (NC / 8), p = i / (NC / 8);
      const int gy = y0 + p / TW, gx = x0 + p % TW;
      pd[j] = make_uint4(0u, 0u, 0u, 0u);
      if (i < kD && gy < H && gx < W)
        pd[j] = __ldg(reinterpret_cast<const uint4*>(dy + (((size_t)b * H + gy) * W + gx) * NC) + cg);
    }
  };
  bool ok = true;
  int it = 0;
  if ((int)blockIdx.x < ntiles) fetch(blockIdx.x);
  for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++it) {
    // the operand buffers are free (the previous tile's MMAs are done)
#pragma unroll
    for (int j = 0; j < kPreX; ++j) {
      const int i = tid + j * kWgThreads, cg = i & 3, col = (i >> 2) % (TW + 2), hy = (i >> 2) / (TW + 2);
      if (i < kX)
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const int p = col - kx;
          if (p >= 0 && p < TW) st_shared_v4(a_base + (kx * 4 + cg) * kWgGroupA + 16 * (hy * TW + p), px[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < kPreD; ++j) {
      const int i = tid + j * kWgThreads, cg = i % (NC / 8), p = i / (NC / 8);
      if (i < kD) st_shared_v4(b_base + cg * kWgGroupB + 16 * p, pd[j]);
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // (the test hook withholds block 0's first tile: no MMAs and no commit, so the wait below runs out)
    if (tid == 0 && !(it == 0 && blockIdx.x == 0 && drop)) {
      const uint32_t idesc = tc::idesc_bf16(128, NC) | (1u << 15) | (1u << 16);  // both operands MN-major
      for (int py = 0; py < TH; ++py)
        for (int ky = 0; ky < 3; ++ky)
          tc::mma_bf16(tmem + NC * ky, tc::desc_interleave(a_base + (py + ky) * (16 * TW), 128, kWgGroupA),
                       tc::desc_interleave(b_base + py * (16 * TW), 128, kWgGroupB), idesc, (it > 0 || py > 0) ? 1u : 0u);
      tc::mma_commit(bar);
    }
    if (t + (int)gridDim.x < ntiles) fetch(t + gridDim.x);
    ok = tc::mbar_wait(bar, it & 1);
    if (!ok) tc::mbar_wait(bar, it & 1);  // wait (bounded) for MMAs still in flight before the tiles are reused
    tc::fence_after_sync();
    ok = __syncthreads_and(ok);
  }
  // epilogue: TMEM lane m (warps 0..3 own lanes 32 w .. 32 w + 31), column NC ky + co
  if (ok && warp < 4) {
    const int m = 32 * warp + lane;
    const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16);
    float* pb = partial + (size_t)blockIdx.x * (NTAP * COUT * CH + COUT);
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      float v[16];
#pragma unroll
      for (int h = 0; h < NC / 16; ++h) {
        tc::tmem_ld16(taddr + NC * ky + 16 * h, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int co = 16 * h + j;
          if (co >= COUT) continue;
          if (m < 96) pb[((size_t)(ky * 3 + (m >> 5)) * COUT + co) * CH + (m & 31)] = v[j];
          if (m == 96 && ky == 0) pb[NTAP * COUT * CH + co] = v[j];
        }
      }
    }
  }
  if (!ok && tid == 0) atomicCAS(err, 0, 0x2100);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kCols);
  }
}

// grad[i] = sum over the blocks b of partial[b][i], in a fixed order: a block takes 32 outputs, each of its 32 warps
// a range of b in order, and the warps' sums are added in order. Bound by the loads' latency (a training step of
// 4 x 320 x 320, seven of these: 922 us with 32 warps, 940 with 16 or 8).
constexpr int kWgSumWarps = 32;
__global__ void __launch_bounds__(32 * kWgSumWarps) wgrad_sum(const float* __restrict__ partial, int nblocks, int n,
                                                              float* __restrict__ grad) {
  __shared__ float sh[kWgSumWarps][32];
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  const int b0 = r * nblocks / kWgSumWarps, b1 = (r + 1) * nblocks / kWgSumWarps;
  float s = 0.f;
  if (i < n) {
#pragma unroll 8
    for (int b = b0; b < b1; ++b) s += partial[(size_t)b * n + i];
  }
  sh[r][lane] = s;
  __syncthreads();
  if (r || i >= n) return;
  for (int q = 1; q < kWgSumWarps; ++q) s += sh[q][lane];
  grad[i] = s;
}

// out[i] = sum over blocks b of partial[b * stride + i], i < n: one CUDA block per output, its 128 threads
// sum fixed strided subsets of the partials, then a fixed-order tree (the same order on every run).
__global__ void __launch_bounds__(128) sum_partials(const float* __restrict__ partial, int nblocks, int stride, int n,
                                                   float* __restrict__ out) {
  __shared__ float sh[128];
  const int i = blockIdx.x;
  if (i >= n) return;
  float s = 0.f;
  for (int b = threadIdx.x; b < nblocks; b += 128) s += partial[(size_t)b * stride + i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = 64; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[i] = sh[0];
}

// The data gradients' weights of layers 1 .. 7 (blockIdx.y = layer - 1): w'[tap'][ci][co] = w[8 - tap'][co][ci], the
// output layer's 8 output channels padded to 16. w: the flat BF16 parameters, layer l's weights at at[l - 1].
struct LayerOffsets {
  int at[7];
};
__global__ void flip_transpose(const bf16* __restrict__ w, LayerOffsets o, bf16* __restrict__ wt) {
  const int l = blockIdx.y, cout = l == 6 ? 8 : CH, cop = l == 6 ? 16 : CH, n = NTAP * CH * cop;
  const bf16* wl = w + o.at[l];
  bf16* out = wt + (size_t)l * NTAP * CH * CH;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int tap = i / (CH * cop), r = i - tap * CH * cop;
    const int ci = r / cop, co = r - ci * cop;  // wt[tap][ci (as out)][co (as in)]
    bf16 v = __float2bfloat16(0.f);
    if (co < cout) v = wl[((size_t)(8 - tap) * cout + co) * CH + ci];
    out[i] = v;
  }
}

// First layer, 2 -> 32 channels (too narrow for the tensor cores): SIMT, relu, saves z (unless null). A thread takes a
// pixel and writes its channels in 16-byte pieces (4-byte stores at a 64-byte stride: 75 us for 4 x 320 x 320, now 28).
__global__ void __launch_bounds__(256) conv_in_fwd(const float* __restrict__ x, const float* __restrict__ w,
                                                   const float* __restrict__ bias, int B, int H, int W,
                                                   bf16* __restrict__ out, bf16* __restrict__ zsave) {
  __shared__ __align__(16) float sw[NTAP * CH * 2];  // [tap][channel pair][input channel][channel of the pair]
  __shared__ __align__(8) float sb[CH];
  for (int i = threadIdx.x; i < NTAP * CH * 2; i += blockDim.x) {
    const int ci = i & 1, co = (i >> 1) % CH, tap = i / (2 * CH);
    sw[((tap * (CH / 2) + (co >> 1)) * 2 + ci) * 2 + (co & 1)] = w[i];
  }
  if (threadIdx.x < CH) sb[threadIdx.x] = bias[threadIdx.x];
  __syncthreads();
  const size_t n = (size_t)B * H * W;
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const int xx = (int)(p % W), yy = (int)((p / W) % H), b = (int)(p / ((size_t)W * H));
    float2 in[NTAP];
#pragma unroll
    for (int tap = 0; tap < NTAP; ++tap) {
      const int gy = yy + tap / 3 - 1, gx = xx + tap % 3 - 1;
      const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
      in[tap] = ok ? reinterpret_cast<const float2*>(x)[((size_t)b * H + gy) * W + gx] : c2(0.f, 0.f);
    }
#pragma unroll 1
    for (int c8 = 0; c8 < CH; c8 += 8) {
      uint32_t zz[4], oo[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 z = *reinterpret_cast<const float2*>(&sb[c8 + 2 * q]);
#pragma unroll
        for (int tap = 0; tap < NTAP; ++tap) {
          const float4 wt = *reinterpret_cast<const float4*>(&sw[(tap * (CH / 2) + c8 / 2 + q) * 4]);
          const float2 v = __fmul2_rn(c2(wt.z, wt.w), c2(in[tap].y, in[tap].y));
          z = __fadd2_rn(z, __ffma2_rn(c2(wt.x, wt.y), c2(in[tap].x, in[tap].x), v));
        }
        zz[q] = pack_bf16(z.x, z.y);
        oo[q] = pack_bf16(fmaxf(z.x, 0.f), fmaxf(z.y, 0.f));
      }
      if (zsave) reinterpret_cast<uint4*>(zsave + p * CH)[c8 / 8] = make_uint4(zz[0], zz[1], zz[2], zz[3]);
      reinterpret_cast<uint4*>(out + p * CH)[c8 / 8] = make_uint4(oo[0], oo[1], oo[2], oo[3]);
    }
  }
}

// Weight and bias gradients of the 2 -> 32 input layer, stage 1: lane = output channel co; a warp takes row segments
// of kSeg pixels and keeps the 3 x 3 window of the two input channels in registers, so that a pixel costs three
// (broadcast) window loads, one 64-byte load of g[p][0..31] and the 19 accumulations (all nine taps loaded and bounds-
// checked per pixel: 134 us for 4 x 320 x 320, now 47). The warps' sums are added in warp order in shared memory:
// partial[b][(tap CH + co) 2 + ci] = sum x[p + d(tap)][ci] g[p][co], partial[b][NTAP CH 2 + co] = sum g[p][co].
// sum_partials adds the blocks in a fixed order.
constexpr int kConvInPartial = NTAP * CH * 2 + CH;
constexpr int kPartialBlocksPerSm = 4;  // what is resident
constexpr int kConvInWarps = 8;
constexpr int kSeg = 32;
__global__ void __launch_bounds__(32 * kConvInWarps, kPartialBlocksPerSm) conv_in_wgrad_partial(const float* __restrict__ x,
                                                                           const bf16* __restrict__ g, int B, int H,
                                                                           int W, float* __restrict__ partial) {
  __shared__ float sh[kConvInWarps][2 * NTAP + 1][CH];
  const int co = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float2* x2 = reinterpret_cast<const float2*>(x);
  float2 acc[NTAP];
  float sb = 0.f;
#pragma unroll
  for (int t = 0; t < NTAP; ++t) acc[t] = c2(0.f, 0.f);
  const int nseg = (W + kSeg - 1) / kSeg;
  const long long total = (long long)nseg * H * B, nw = (long long)gridDim.x * kConvInWarps;
  for (long long q = (long long)blockIdx.x * kConvInWarps + w; q < total; q += nw) {
    const int x0 = (int)(q % nseg) * kSeg, x1 = min(x0 + kSeg, W);
    const long long row = q / nseg;  // b H + y
    const int yy = (int)(row % H);
    const float2* c = x2 + row * W;
    const float2* up = yy > 0 ? c - W : nullptr;
    const float2* dn = yy < H - 1 ? c + W : nullptr;
    const bf16* gr = g + (size_t)row * W * CH + co;
    float2 win[3][3];  // [dy][dx]; dx = 0, 1 filled, 2 loaded per pixel
    auto col = [&](int gx, int k) {
      const bool ok = gx >= 0 && gx < W;
      win[0][k] = ok && up ? up[gx] : c2(0.f, 0.f);
      win[1][k] = ok ? c[gx] : c2(0.f, 0.f);
      win[2][k] = ok && dn ? dn[gx] : c2(0.f, 0.f);
    };
    col(x0 - 1, 0);
    col(x0, 1);
#pragma unroll 4
    for (int gx = x0; gx < x1; ++gx) {
      col(gx + 1, 2);
      const float gv = __bfloat162float(gr[(size_t)gx * CH]);
      sb += gv;
#pragma unroll
      for (int t = 0; t < NTAP; ++t) {
        acc[t] = __ffma2_rn(win[t / 3][t % 3], c2(gv, gv), acc[t]);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        win[k][0] = win[k][1];
        win[k][1] = win[k][2];
      }
    }
  }
#pragma unroll
  for (int t = 0; t < NTAP; ++t) {
    sh[w][2 * t][co] = acc[t].x;
    sh[w][2 * t + 1][co] = acc[t].y;
  }
  sh[w][2 * NTAP][co] = sb;
  __syncthreads();
  float* out = partial + (size_t)blockIdx.x * kConvInPartial;
  for (int i = threadIdx.x; i < (2 * NTAP + 1) * CH; i += blockDim.x) {
    const int j = i / CH, c = i - j * CH;  // j = 2 tap + ci, or 2 NTAP for the bias
    float s = 0.f;
    for (int ww = 0; ww < kConvInWarps; ++ww) s += sh[ww][j][c];
    if (j < 2 * NTAP)
      out[((j >> 1) * CH + c) * 2 + (j & 1)] = s;
    else
      out[NTAP * CH * 2 + c] = s;
  }
}

__global__ void to_bf16(const float* __restrict__ a, size_t n, bf16* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(a[i]);
}

// Mean squared error over the 6 used output channels and its gradient (BF16, padded to the 16 channels the
// tensor-core kernels take).
__global__ void mse_loss(const float* __restrict__ y, const float* __restrict__ t, size_t npix, float scale,
                         bf16* __restrict__ g, double* __restrict__ partial) {
  __shared__ double sh[256];
  double s = 0;
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < npix; p += (size_t)gridDim.x * blockDim.x) {
    float d[8];
    const float4 ya = reinterpret_cast<const float4*>(y)[2 * p], yb = reinterpret_cast<const float4*>(y)[2 * p + 1];
    const float2* tp = reinterpret_cast<const float2*>(t) + 3 * p;
    const float2 t0 = tp[0], t1 = tp[1], t2 = tp[2];
    d[0] = ya.x - t0.x;
    d[1] = ya.y - t0.y;
    d[2] = ya.z - t1.x;
    d[3] = ya.w - t1.y;
    d[4] = yb.x - t2.x;
    d[5] = yb.y - t2.y;
    d[6] = d[7] = 0.f;
#pragma unroll
    for (int c = 0; c < 6; ++c) s += (double)d[c] * d[c];
    uint4 o;
    o.x = pack_bf16(2.f * d[0] * scale, 2.f * d[1] * scale);
    o.y = pack_bf16(2.f * d[2] * scale, 2.f * d[3] * scale);
    o.z = pack_bf16(2.f * d[4] * scale, 2.f * d[5] * scale);
    o.w = 0u;
    reinterpret_cast<uint4*>(g)[2 * p] = o;
    reinterpret_cast<uint4*>(g)[2 * p + 1] = make_uint4(0u, 0u, 0u, 0u);
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// Adam on FP32 master weights, BF16 copy refreshed.
__global__ void adam_step(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                          float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2,
                          bf16* __restrict__ wb) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16(wi);
  }
}

// x = [Re, Im] of the complex input / s per image (s = max |u0| of that image, given).
__global__ void prep_input(const float2* __restrict__ u0, const float* __restrict__ inv_s, int B, size_t npix,
                           float* __restrict__ x) {
  const size_t n = (size_t)B * npix;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float s = inv_s[i / npix];
    x[2 * i] = u0[i].x * s;
    x[2 * i + 1] = u0[i].y * s;
  }
}

// u = u0 + s (o0 + i o1), vx = s (o2 + i o3), vy = s (o4 + i o5)
__global__ void assemble_output(const float2* __restrict__ u0, const float* __restrict__ o, const float* __restrict__ s,
                                int B, size_t npix, float2* __restrict__ u, float2* __restrict__ v) {
  const size_t n = (size_t)B * npix;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t b = i / npix, p = i - b * npix;
    const float sc = s[b];
    u[i] = u0[i] + sc * c2(o[i * 8], o[i * 8 + 1]);
    v[(2 * b) * npix + p] = sc * c2(o[i * 8 + 2], o[i * 8 + 3]);
    v[(2 * b + 1) * npix + p] = sc * c2(o[i * 8 + 4], o[i * 8 + 5]);
  }
}

// training target: t = [(u* - u0)/s, v*/s] in 6 channels
__global__ void prep_target(const float2* __restrict__ u0, const float2* __restrict__ ut, const float2* __restrict__ vt,
                            const float* __restrict__ inv_s, int B, size_t npix, float* __restrict__ t) {
  const size_t n = (size_t)B * npix;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t b = i / npix, p = i - b * npix;
    const float s = inv_s[b];
    const float2 du = (ut[i] - u0[i]) * s;
    const float2 vx = vt[(2 * b) * npix + p] * s, vy = vt[(2 * b + 1) * npix + p] * s;
    t[i * 6 + 0] = du.x;
    t[i * 6 + 1] = du.y;
    t[i * 6 + 2] = vx.x;
    t[i * 6 + 3] = vx.y;
    t[i * 6 + 4] = vy.x;
    t[i * 6 + 5] = vy.y;
  }
}

// s[b] = max |u0| over image b; inv_s[b] = 1 / s[b] (1 for an all-zero image). Block per image.
// max |u0| of image blockIdx.y over the pixels of block column blockIdx.x, combined across blocks with an
// integer atomicMax on the float's bits (non-negative floats order like their bit patterns, so the result
// does not depend on the order); image_scale_finish turns the maxima into the scale and its inverse.
__global__ void image_scale_max(const float2* __restrict__ u0, size_t npix, int* __restrict__ imax) {
  __shared__ float sh[256];
  const float2* img = u0 + (size_t)blockIdx.y * npix;
  float m = 0.f;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npix; i += (size_t)gridDim.x * blockDim.x)
    m = fmaxf(m, sqrtf(abs2(img[i])));
  sh[threadIdx.x] = m;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] = fmaxf(sh[threadIdx.x], sh[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicMax(imax + blockIdx.y, __float_as_int(sh[0]));
}

__global__ void image_scale_finish(const int* __restrict__ imax, int B, float* __restrict__ s,
                                   float* __restrict__ inv_s) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const float m = __int_as_float(imax[b]);
  const float v = m > 0.f ? m : 1.f;
  s[b] = v;
  inv_s[b] = 1.f / v;
}

inline int grid_for(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 4096); }

}  // namespace

// ------------------------------------------------------------------------------------------------
// Host side: parameters, activations for a batch, forward / backward / Adam.
// ------------------------------------------------------------------------------------------------
// One layer's weights or biases within the network's flat arrays (weights then biases per layer).
struct CnnParam {
  int n = 0;                            // elements
  float *w = nullptr, *g = nullptr;     // FP32 master, gradient
  bf16* wb = nullptr;                   // BF16 copy (the tensor-core kernels read the weights of layers 1 .. 7)
};

class WarmStartCnn {
 public:
  static constexpr int kLayers = 8;  // conv_in, 6 hidden, conv_out
  explicit WarmStartCnn(uint64_t seed) {
    std::mt19937_64 gen(seed);
    // conv_in: [9][32][2] + bias 32; hidden: [9][32][32] + 32; conv_out: [9][8][32] + 8
    const int sizes[kLayers] = {NTAP * CH * 2, NTAP * CH * CH, NTAP * CH * CH, NTAP * CH * CH, NTAP * CH * CH,
                                NTAP * CH * CH, NTAP * CH * CH, NTAP * 8 * CH};
    const int fan_in[kLayers] = {NTAP * 2, NTAP * CH, NTAP * CH, NTAP * CH, NTAP * CH, NTAP * CH, NTAP * CH, NTAP * CH};
    const int nb[kLayers] = {CH, CH, CH, CH, CH, CH, CH, 8};
    for (int l = 0; l < kLayers; ++l) total_ += sizes[l] + nb[l];
    for (DevBuf* d : {&pw_, &pg_, &pm_, &pv_}) {
      d->ensure(total_ * sizeof(float));
      PDT_CUDA_CHECK(cudaMemset(d->p, 0, d->bytes));
    }
    pb_.ensure(total_ * sizeof(bf16));
    size_t at = 0;
    auto take = [&](CnnParam& p, int n) {
      p.n = n;
      p.w = pw_.as<float>() + at;
      p.g = pg_.as<float>() + at;
      p.wb = pb_.as<bf16>() + at;
      at += n;
    };
    std::vector<float> all;
    for (int l = 0; l < kLayers; ++l) {
      std::vector<float> w(sizes[l]);
      // He initialisation; the hidden residual branches start small so the net begins near identity
      const float sd = std::sqrt(2.0f / fan_in[l]) * ((l >= 1 && l <= 6) ? 0.25f : (l == 7 ? 0.1f : 1.0f));
      std::normal_distribution<float> dis(0.f, sd);
      for (auto& x : w) x = dis(gen);
      if (l == 7)  // output channels 6, 7 are padding
        for (int tap = 0; tap < NTAP; ++tap)
          for (int co = 6; co < 8; ++co)
            for (int ci = 0; ci < CH; ++ci) w[((size_t)tap * 8 + co) * CH + ci] = 0.f;
      take(W_[l], sizes[l]);
      take(B_[l], nb[l]);
      all.insert(all.end(), w.begin(), w.end());
      all.resize(at, 0.f);
    }
    upload_params(all.data());
    const struct {
      decltype(&conv3x3_tc<EPI_ACC, CH, CH>) fn;
      int smem;
    } convs[] = {{conv3x3_tc<EPI_RELU_RES, CH, CH>, (int)ConvTc<CH, CH>::kSmem},
                 {conv3x3_tc<EPI_ACC, CH, CH>, (int)ConvTc<CH, CH>::kSmem},
                 {conv3x3_tc<EPI_F32, CH, 8>, (int)ConvTc<CH, 8>::kSmem},
                 {conv3x3_tc<EPI_F32_BF16, 16, CH>, (int)ConvTc<16, CH>::kSmem}};
    for (auto& c : convs) {
      auto fn = c.fn;
      PDT_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, c.smem));
      // all of the unified L1 / shared storage as shared memory, so that several CTAs fit on an SM
      PDT_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    }
    for (auto fn : {wgrad_tc<32, 32>, wgrad_tc<16, 8>}) {
      PDT_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgSmem));
      PDT_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    }
    err_.ensure(sizeof(int));
    PDT_CUDA_CHECK(cudaMemset(err_.p, 0, sizeof(int)));
    int dev = 0;
    PDT_CUDA_CHECK(cudaGetDevice(&dev));
    PDT_CUDA_CHECK(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
    // resident CTAs per SM from the register file, shared memory and thread limits (256-register allocation
    // granules per warp, the per-block shared memory reservation)
    int regs_sm = 0, smem_sm = 0, smem_rsv = 0, thr_sm = 0;
    PDT_CUDA_CHECK(cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev));
    PDT_CUDA_CHECK(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    PDT_CUDA_CHECK(cudaDeviceGetAttribute(&smem_rsv, cudaDevAttrReservedSharedMemoryPerBlock, dev));
    PDT_CUDA_CHECK(cudaDeviceGetAttribute(&thr_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev));
    for (auto& c : convs) {
      cudaFuncAttributes fa{};
      PDT_CUDA_CHECK(cudaFuncGetAttributes(&fa, c.fn));
      const int warp_regs = ((fa.numRegs * 32 + 255) / 256) * 256;
      const int by_regs = regs_sm / (warp_regs * (kConvTcThreads / 32));
      const int by_smem = smem_sm / (c.smem + (int)fa.sharedSizeBytes + smem_rsv);
      const int by_thr = thr_sm / kConvTcThreads;
      conv_tc_per_sm_ = std::min({conv_tc_per_sm_, by_regs, by_smem, by_thr});
    }
    conv_tc_per_sm_ = std::max(conv_tc_per_sm_, 1);
  }

  // Raises (and clears) the error word of the tensor-core convolutions: set when an MMA completion wait
  // gave up, after which that launch's output is not valid.
  void check_error() {
    int e = 0;
    PDT_CUDA_CHECK(cudaMemcpy(&e, err_.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) {
      PDT_CUDA_CHECK(cudaMemset(err_.p, 0, sizeof(int)));
      throw Error(PDT_ERR_TIMEOUT, "warm-start network: a tensor-core convolution gave up waiting for its MMAs");
    }
  }

  // Parameters as one flat FP32 vector (weights then biases per layer) for saving / loading.
  std::vector<float> get_params() const { return download(pw_); }
  void set_params(const float* src, size_t n) {
    if (n < total_) throw Error(PDT_ERR_SIZE, "parameter vector too short");
    if (n != total_) throw Error(PDT_ERR_SIZE, "parameter vector length mismatch");
    upload_params(src);
  }
  size_t num_params() const { return total_; }

  // Forward pass for B images of H x W; u0 complex [B][H][W], s = per-image scale. Writes o (FP32, 8 ch).
  // `keep`: also the pre-activations, for backward().
  void forward(const float2* u0, const float* inv_s, int B, int H, int W, bool keep, cudaStream_t st) {
    alloc(B, H, W);
    const size_t npix = (size_t)B * H * W;
    prep_input<<<grid_for(npix), 256, 0, st>>>(u0, inv_s, B, (size_t)H * W, x_.as<float>());
    PDT_LAUNCH_CHECK();
    conv_in_fwd<<<grid_for(npix), 256, 0, st>>>(x_.as<float>(), W_[0].w, B_[0].w, B, H, W, h_[0].as<bf16>(),
                                               keep ? z_[0].as<bf16>() : nullptr);
    PDT_LAUNCH_CHECK();
    count_launch(2);
    const int tgrid = conv_tc_grid(B, H, W);
    for (int l = 1; l <= 6; ++l) {
      conv3x3_tc<EPI_RELU_RES, CH, CH><<<tgrid, kConvTcThreads, ConvTc<CH, CH>::kSmem, st>>>(
          h_[l - 1].as<bf16>(), W_[l].wb, B_[l].w, B, H, W, h_[l].as<bf16>(), keep ? z_[l].as<bf16>() : nullptr,
          err_.as<int>(), nullptr);
      PDT_LAUNCH_CHECK();
      count_launch();
    }
    conv3x3_tc<EPI_F32, CH, 8><<<tgrid, kConvTcThreads, ConvTc<CH, 8>::kSmem, st>>>(
        h_[6].as<bf16>(), W_[7].wb, B_[7].w, B, H, W, nullptr, nullptr, err_.as<int>(), o_.as<float>());
    PDT_LAUNCH_CHECK();
    count_launch();
  }

  // Backward pass after forward(): loss = mean over pixels of sum_c (o_c - t_c)^2 (t: 6 channels FP32).
  double backward(const float* target, int B, int H, int W, cudaStream_t st) {
    const size_t npix = (size_t)B * H * W;
    const float scale = 1.0f / (float)npix;
    const int lb = grid_for(npix);
    part_.ensure(sizeof(double) * lb);
    mse_loss<<<lb, 256, 0, st>>>(o_.as<float>(), target, npix, scale, go_.as<bf16>(), part_.as<double>());
    LayerOffsets at;
    for (int l = 1; l <= 7; ++l) at.at[l - 1] = (int)(W_[l].wb - pb_.as<bf16>());
    flip_transpose<<<dim3(36, 7), 256, 0, st>>>(pb_.as<bf16>(), at, wt_.as<bf16>());
    auto wt = [&](int l) { return wt_.as<bf16>() + (size_t)(l - 1) * NTAP * CH * CH; };
    PDT_LAUNCH_CHECK();
    const int tgrid = conv_tc_grid(B, H, W);
    // conv_out: dW, db, and dh6 = conv(go, W7') (8 -> 32 channels, padded to 16 input channels), with which the
    // residual stream's FP32 gradient starts as G = dh6 (the BF16 rounding of the convolution's output)
    wgrad(8, h_[6].as<bf16>(), go_.as<bf16>(), B, H, W, W_[7].g, st);
    bf16* gz = gz_[0].as<bf16>();  // dz = G * relu'(z_l) of the layer at hand; the next layer's goes to the other buffer
    bf16* gn = gz_[1].as<bf16>();
    conv3x3_tc<EPI_F32_BF16, 16, CH><<<tgrid, kConvTcThreads, ConvTc<16, CH>::kSmem, st>>>(
        go_.as<bf16>(), wt(7), nullptr, B, H, W, gz, z_[6].as<bf16>(), err_.as<int>(), gacc_.as<float>());
    PDT_LAUNCH_CHECK();
    count_launch(3);  // mse_loss, flip_transpose, conv3x3_tc
    for (int l = 6; l >= 1; --l) {
      // h_l = h_{l-1} + relu(z_l), z_l = conv_l(h_{l-1}):  dh_{l-1} = G + conv_l^T(dz), added into the FP32 residual
      // gradient in the convolution's epilogue, which also masks it for the layer below
      wgrad(CH, h_[l - 1].as<bf16>(), gz, B, H, W, W_[l].g, st);
      conv3x3_tc<EPI_ACC, CH, CH><<<tgrid, kConvTcThreads, ConvTc<CH, CH>::kSmem, st>>>(
          gz, wt(l), nullptr, B, H, W, gn, z_[l - 1].as<bf16>(), err_.as<int>(), gacc_.as<float>());
      PDT_LAUNCH_CHECK();
      count_launch();
      std::swap(gz, gn);
    }
    // conv_in: h1 = relu(z_0)
    {
      const int nb = kPartialBlocksPerSm * sms_;
      bpart_.ensure(sizeof(float) * (size_t)nb * kConvInPartial);
      conv_in_wgrad_partial<<<nb, 32 * kConvInWarps, 0, st>>>(x_.as<float>(), gz, B, H, W, bpart_.as<float>());
      // the weights and, right behind them as in the flat gradient, the biases
      sum_partials<<<kConvInPartial, 128, 0, st>>>(bpart_.as<float>(), nb, kConvInPartial, kConvInPartial, W_[0].g);
      PDT_LAUNCH_CHECK();
    }
    count_launch(2);  // conv_in_wgrad_partial, sum_partials
    std::vector<double> h(lb);
    PDT_CUDA_CHECK(cudaMemcpyAsync(h.data(), part_.p, sizeof(double) * lb, cudaMemcpyDeviceToHost, st));
    PDT_CUDA_CHECK(cudaStreamSynchronize(st));
    check_error();
    double loss = 0;
    for (double v : h) loss += v;
    return loss / (double)npix;
  }

  void adam(float lr, cudaStream_t st) {
    ++step_;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.f - std::pow(b1, (float)step_), c2 = 1.f - std::pow(b2, (float)step_);
    adam_step<<<grid_for(total_), 256, 0, st>>>(pw_.as<float>(), pg_.as<float>(), pm_.as<float>(), pv_.as<float>(),
                                                (int)total_, lr, b1, b2, eps, c1, c2, pb_.as<bf16>());
    PDT_LAUNCH_CHECK();
    count_launch();
  }

  const float* output() const { return o_.as<float>(); }
  // per-image scales of u0 (device): s, 1/s
  void scales(const float2* u0, int B, size_t npix_img, cudaStream_t st) {
    sc_.ensure(3 * sizeof(float) * std::max(B, 1));  // scale [B], inverse [B], maxima as int bits [B]
    int* imax = reinterpret_cast<int*>(sc_.as<float>() + 2 * B);
    PDT_CUDA_CHECK(cudaMemsetAsync(imax, 0, sizeof(int) * B, st));
    const int nbx = (int)std::max<size_t>(1, std::min<size_t>((npix_img + 255) / 256, (size_t)sms_));
    image_scale_max<<<dim3(nbx, B), 256, 0, st>>>(u0, npix_img, imax);
    image_scale_finish<<<(B + 127) / 128, 128, 0, st>>>(imax, B, sc_.as<float>(), sc_.as<float>() + B);
    PDT_LAUNCH_CHECK();
    count_launch(2);
  }
  const float* scale_ptr() const { return sc_.as<float>(); }
  const float* inv_scale_ptr(int B) const { return sc_.as<float>() + B; }
  std::vector<float> get_grads() const { return download(pg_); }
  float* target_buf(size_t npix) {
    t_.ensure(npix * 6 * sizeof(float));
    return t_.as<float>();
  }

  void make_target(const float2* u0, const float2* ut, const float2* vt, const float* inv_s, int B, size_t npix_img,
                   cudaStream_t st) {
    float* t = target_buf((size_t)B * npix_img);
    prep_target<<<grid_for((size_t)B * npix_img), 256, 0, st>>>(u0, ut, vt, inv_s, B, npix_img, t);
    PDT_LAUNCH_CHECK();
    count_launch();
  }
  void assemble(const float2* u0, const float* s, int B, size_t npix_img, float2* u, float2* v, cudaStream_t st) {
    assemble_output<<<grid_for((size_t)B * npix_img), 256, 0, st>>>(u0, o_.as<float>(), s, B, npix_img, u, v);
    PDT_LAUNCH_CHECK();
    count_launch();
  }

 private:
  std::vector<float> download(const DevBuf& d) const {
    std::vector<float> out(total_);
    PDT_CUDA_CHECK(cudaMemcpy(out.data(), d.p, total_ * sizeof(float), cudaMemcpyDeviceToHost));
    return out;
  }
  void upload_params(const float* src) {
    PDT_CUDA_CHECK(cudaMemcpy(pw_.p, src, total_ * sizeof(float), cudaMemcpyHostToDevice));
    to_bf16<<<grid_for(total_), 256>>>(pw_.as<float>(), total_, pb_.as<bf16>());
    PDT_LAUNCH_CHECK();
    PDT_CUDA_CHECK(cudaDeviceSynchronize());
  }
  // persistent tensor-core convolutions: what is resident (four CTAs per SM by registers), at most one tile each
  int conv_tc_grid(int B, int H, int W) const {
    const long long tiles = (long long)((W + kConvTcTW - 1) / kConvTcTW) * ((H + kConvTcTH - 1) / kConvTcTH) * B;
    return (int)std::min<long long>(tiles, (long long)conv_tc_per_sm_ * sms_);
  }
  void alloc(int B, int H, int W) {
    if (B == B_n_ && H == H_n_ && W == W_n_) return;
    const size_t npix = (size_t)B * H * W;
    x_.ensure(npix * 2 * sizeof(float));
    for (int l = 0; l < 7; ++l) {
      h_[l].ensure(npix * CH * sizeof(bf16));
      z_[l].ensure(npix * CH * sizeof(bf16));
    }
    o_.ensure(npix * 8 * sizeof(float));
    go_.ensure(npix * 16 * sizeof(bf16));
    for (auto& g : gz_) g.ensure(npix * CH * sizeof(bf16));
    const size_t tiles = (size_t)B * ((W + kConvTcTW - 1) / kConvTcTW) * ((H + kConvTcTH - 1) / kConvTcTH);
    gacc_.ensure(tiles * kConvTcTW * kConvTcTH * CH * sizeof(float));
    wt_.ensure((size_t)7 * NTAP * CH * CH * sizeof(bf16));
    B_n_ = B;
    H_n_ = H;
    W_n_ = W;
  }
  // The weight gradient and, behind it in the flat array, the bias gradient of a layer.
  void wgrad(int cout, const bf16* x, const bf16* dy, int B, int H, int W, float* grad, cudaStream_t st) {
    const int tiles = B * ((W + TW - 1) / TW) * ((H + TH - 1) / TH);
    const int nb = std::max(1, std::min(sms_ * kWgPerSm, tiles));
    const int n = NTAP * cout * CH + cout;
    wpart_.ensure((size_t)nb * (NTAP * CH * CH + CH) * sizeof(float));
    if (cout == CH)
      wgrad_tc<32, 32><<<nb, kWgThreads, kWgSmem, st>>>(x, dy, B, H, W, wpart_.as<float>(), err_.as<int>());
    else
      wgrad_tc<16, 8><<<nb, kWgThreads, kWgSmem, st>>>(x, dy, B, H, W, wpart_.as<float>(), err_.as<int>());
    PDT_LAUNCH_CHECK();
    wgrad_sum<<<(n + 31) / 32, 32 * kWgSumWarps, 0, st>>>(wpart_.as<float>(), nb, n, grad);
    PDT_LAUNCH_CHECK();
    count_launch(2);
  }

  CnnParam W_[kLayers], B_[kLayers];
  size_t total_ = 0;
  DevBuf pw_, pg_, pm_, pv_, pb_;  // flat FP32 master weights, gradients, Adam moments; BF16 copy
  DevBuf x_, h_[7], z_[7], o_, go_, gz_[2], gacc_, wt_, wpart_, part_, t_, sc_, err_, bpart_;

  int sms_ = 1;
  int conv_tc_per_sm_ = 8;  // resident conv3x3_tc CTAs per SM (each holds 64 TMEM columns: 8 x 64 <= 512)
  int B_n_ = 0, H_n_ = 0, W_n_ = 0;
  long step_ = 0;
};

void cnn_set_drop_arrival(int on) { PDT_CUDA_CHECK(tc::set_drop_arrival(on)); }

}  // namespace pdt

// ==================================================================================================
// C ABI of the warm-start network
// ==================================================================================================
struct pdt_cnn {
  std::unique_ptr<pdt::WarmStartCnn> impl;
};

namespace {
template <class F>
pdt_status cnn_guard(F&& fn) {
  try {
    fn();
    return PDT_OK;
  } catch (const pdt::Error& e) {
    pdt::set_last_error(e.what());
    return e.code;
  } catch (const std::exception& e) {
    pdt::set_last_error(e.what());
    return PDT_ERR_INVALID_ARGUMENT;
  }
}
void cnn_check(pdt_cnn* c, int B, int H, int W) {
  if (!c) throw pdt::Error(PDT_ERR_INVALID_ARGUMENT, "null network");
  if (B < 1 || H < 1 || W < 1) throw pdt::Error(PDT_ERR_INVALID_ARGUMENT, "B, H and W must be positive");
}
}  // namespace

extern "C" {

pdt_status pdt_cnn_create(uint64_t seed, pdt_cnn** out) {
  return cnn_guard([&] {
    if (!out) throw pdt::Error(PDT_ERR_INVALID_ARGUMENT, "null out");
    auto h = std::make_unique<pdt_cnn>();
    h->impl = std::make_unique<pdt::WarmStartCnn>(seed);
    *out = h.release();
  });
}

pdt_status pdt_cnn_destroy(pdt_cnn* c) {
  return cnn_guard([&] { delete c; });
}

pdt_status pdt_cnn_num_params(pdt_cnn* c, size_t* n) {
  return cnn_guard([&] {
    cnn_check(c, 1, 1, 1);
    *n = c->impl->num_params();
  });
}

pdt_status pdt_cnn_get_params(pdt_cnn* c, float* dst, size_t n) {
  return cnn_guard([&] {
    cnn_check(c, 1, 1, 1);
    auto v = c->impl->get_params();
    if (n != v.size()) throw pdt::Error(PDT_ERR_SIZE, "parameter count mismatch");
    std::memcpy(dst, v.data(), n * sizeof(float));
  });
}

pdt_status pdt_cnn_set_params(pdt_cnn* c, const float* src, size_t n) {
  return cnn_guard([&] {
    cnn_check(c, 1, 1, 1);
    c->impl->set_params(src, n);
  });
}

pdt_status pdt_cnn_get_grads(pdt_cnn* c, float* dst, size_t n) {
  return cnn_guard([&] {
    cnn_check(c, 1, 1, 1);
    auto v = c->impl->get_grads();
    if (n != v.size()) throw pdt::Error(PDT_ERR_SIZE, "parameter count mismatch");
    std::memcpy(dst, v.data(), n * sizeof(float));
  });
}

pdt_status pdt_cnn_train_step(pdt_cnn* c, const void* u0, const void* ut, const void* vt, int B, int H, int W,
                              float lr, void* stream, double* loss) {
  return cnn_guard([&] {
    cnn_check(c, B, H, W);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto& n = *c->impl;
    const size_t np = (size_t)H * W;
    n.scales(static_cast<const float2*>(u0), B, np, st);
    n.make_target(static_cast<const float2*>(u0), static_cast<const float2*>(ut), static_cast<const float2*>(vt),
                  n.inv_scale_ptr(B), B, np, st);
    n.forward(static_cast<const float2*>(u0), n.inv_scale_ptr(B), B, H, W, true, st);
    const double l = n.backward(n.target_buf((size_t)B * np), B, H, W, st);
    if (lr > 0.f) n.adam(lr, st);
    if (loss) *loss = l;
  });
}

pdt_status pdt_cnn_predict(pdt_cnn* c, const void* u0, int B, int H, int W, void* u, void* v, void* stream) {
  return cnn_guard([&] {
    cnn_check(c, B, H, W);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto& n = *c->impl;
    const size_t np = (size_t)H * W;
    n.scales(static_cast<const float2*>(u0), B, np, st);
    n.forward(static_cast<const float2*>(u0), n.inv_scale_ptr(B), B, H, W, false, st);
    n.assemble(static_cast<const float2*>(u0), n.scale_ptr(), B, np, static_cast<float2*>(u), static_cast<float2*>(v),
               st);
    if (!stream) {
      PDT_CUDA_CHECK(cudaStreamSynchronize(st));
      n.check_error();
    }
  });
}

}  // extern "C"
