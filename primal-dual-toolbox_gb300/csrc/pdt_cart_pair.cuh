// pdt_cart_pair.cuh -- K^H f of a Cartesian operator in pairs of FP32 values (about 48 bits), once per long solve.
//
// A line-sampled solve subtracts c K^H f from K^H K U in every iteration. K^H f of FP32 transforms is 1.3e-7 off, also
// in the directions that the mask does not see, where nothing but the regularisation pulls it back: after 1001
// iterations the image was 2.2e-6 off the solution in 64 bits (15 coils, 640 x 368), 7.6e-7 with this K^H f and 6e-7 with
// the k-space dual.
// A generic mixed-radix transform in pairs of FP32 values (an FP64 one would take five times as long on this GPU's FP64
// units) removes that error. It takes 0.2 ms there, 4 % of 256 iterations: shorter solves, where the error has not
// built up, do without.
// Included by pdt_cartesian.cu after CartDev.
#pragma once

namespace pdt {
namespace {

constexpr int kPairThreads = 256;

// A complex pair: {re, im, re remainder, im remainder}.
struct PairSum {
  float h, l;
  // + x y, with x = xh + xl and y = yh + yl (explicit roundings: a fused product would lose its error term)
  __device__ __forceinline__ void mac(float xh, float xl, float yh, float yl) {
    const float p = __fmul_rn(xh, yh);
    const float e = __fmaf_rn(xl, yh, __fmaf_rn(xh, yl, __fmaf_rn(xh, yh, -p)));
    const float s = __fadd_rn(h, p), t = __fsub_rn(s, h);
    l = __fadd_rn(l, __fadd_rn(__fadd_rn(__fsub_rn(h, __fsub_rn(s, t)), __fsub_rn(p, t)), e));
    h = s;
  }
  __device__ __forceinline__ void norm() {
    const float s = __fadd_rn(h, l);
    l = __fsub_rn(l, __fsub_rn(s, h));
    h = s;
  }
};

// a += x y
__device__ __forceinline__ void pair_cmac(PairSum& re, PairSum& im, float4 x, float4 y) {
  re.mac(x.x, x.z, y.x, y.z);
  re.mac(-x.y, -x.w, y.y, y.w);
  im.mac(x.x, x.z, y.y, y.w);
  im.mac(x.y, x.w, y.x, y.z);
}

// nseq inverse transforms (unscaled) of plan.n values in shared memory, sequence b at a[b n]: Stockham passes, a thread
// per output. tw[m] = exp(2 pi i m / n). Returns the buffer that holds the result; ends with a barrier.
__device__ __noinline__ float4* pair_ifft(float4* a, float4* b, int nseq, const FftPlan& pl, const float4* tw) {
  const int n = pl.n;
  int Ns = 1;
  for (int st = 0; st < pl.nst; ++st) {
    const int R = pl.radix[st], nb = n / R, unit = n / (Ns * R);
    for (int t = threadIdx.x; t < n * nseq; t += blockDim.x) {
      const int sq = t / n, o = t - sq * n;  // output o = (j / Ns) Ns R + q Ns + k of butterfly j, k = j mod Ns
      const int blk = o / (Ns * R), in = o - blk * (Ns * R), k = in % Ns, j = blk * Ns + k;
      const float4* src = a + (size_t)sq * n + j;
      const int step = in * unit;  // input r enters with w^(r in unit)
      PairSum re{0.f, 0.f}, im{0.f, 0.f};
      for (int r = 0, m = 0; r < R; ++r) {
        pair_cmac(re, im, src[(size_t)r * nb], tw[m]);
        m += step;
        if (m >= n) m -= n;
      }
      re.norm();
      im.norm();
      b[(size_t)sq * n + o] = make_float4(re.h, im.h, re.l, im.l);
    }
    __syncthreads();
    float4* x = a;
    a = b;
    b = x;
    Ns *= R;
  }
  return a;
}

// Sampled columns of f . mask, inverse transform along Hf, image rows -> t[c][s][yi]. Block (column, coil).
__global__ void __launch_bounds__(kPairThreads) pair_cols(CartDev d, const float4* __restrict__ tw, const float2* __restrict__ fc,
                                                          float4* __restrict__ t) {
  extern __shared__ float4 psm[];
  const int n = d.Hf, s = blockIdx.x, c = blockIdx.y;
  float4 *w = psm, *A = w + n, *B = A + n;
  const size_t col = (size_t)c * d.ns + s;
  for (int P = threadIdx.x; P < n; P += blockDim.x) {
    w[P] = tw[P];
    const float2 f = fc[col * n + P];
    const float m = d.maskc[(size_t)s * n + P];
    PairSum re{0.f, 0.f}, im{0.f, 0.f};
    re.mac(f.x, 0.f, m, 0.f);
    im.mac(f.y, 0.f, m, 0.f);
    A[imod((d.kperm ? d.kperm[P] : P) + d.mxH, n)] = make_float4(re.h, im.h, re.l, im.l);
  }
  __syncthreads();
  const float4* Z = pair_ifft(A, B, 1, d.planH, w);
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const int yi = imod(j + d.oyH, n) - d.y0;
    if (yi >= 0 && yi < d.Hi) t[col * d.Hi + yi] = Z[j];
  }
}

// Image row y: inverse transforms along W of the coils' sampled columns (`nq` at a time), conj(sens_c), coil sum and scale.
__global__ void __launch_bounds__(kPairThreads) pair_rows(CartDev d, const float4* __restrict__ tw, const float4* __restrict__ t,
                                                          int nq, float2 scale, float2* __restrict__ out,
                                                          float2* __restrict__ out_lo) {
  extern __shared__ float4 psm[];
  const int n = d.W, y = blockIdx.x;
  float4 *w = psm, *sum = w + n, *A = sum + n, *B = A + (size_t)nq * n;
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    w[x] = tw[x];
    sum[x] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int c0 = 0; c0 < d.C; c0 += nq) {
    const int nc = min(nq, d.C - c0);
    for (int i = threadIdx.x; i < nc * n; i += blockDim.x) {
      const int q = i / n, s = d.slot2s[i - q * n];
      A[i] = s >= 0 ? t[((size_t)(c0 + q) * d.ns + s) * d.Hi + y] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const float4* Z = pair_ifft(A, B, nc, d.planW, w);
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      const int x = imod(j + d.oxW, n);
      PairSum re{sum[j].x, sum[j].z}, im{sum[j].y, sum[j].w};
      for (int q = 0; q < nc; ++q) {
        const float2 s = d.sens ? d.sens[((size_t)(c0 + q) * d.Hf + y + d.y0) * n + x] : c2(1.f, 0.f);
        pair_cmac(re, im, Z[q * n + j], make_float4(s.x, -s.y, 0.f, 0.f));
      }
      sum[j] = make_float4(re.h, im.h, re.l, im.l);
    }
    __syncthreads();
  }
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    PairSum re{0.f, 0.f}, im{0.f, 0.f};
    re.mac(sum[j].x, sum[j].z, scale.x, scale.y);
    im.mac(sum[j].y, sum[j].w, scale.x, scale.y);
    re.norm();
    im.norm();
    const size_t o = (size_t)y * n + imod(j + d.oxW, n);
    out[o] = c2(re.h, im.h);
    out_lo[o] = c2(re.l, im.l);
  }
}

inline size_t pair_cols_smem(int Hf) { return sizeof(float4) * 3 * (size_t)Hf; }
inline size_t pair_rows_smem(int W, int nq) { return sizeof(float4) * (2 + 2 * (size_t)nq) * W; }

// v as the sum of two FP32 values
inline float2 pair_of(double v) { return make_float2((float)v, (float)(v - (double)(float)v)); }

// exp(2 pi i m / n), m < n
inline void pair_twiddles(int n, std::vector<float4>& tw) {
  tw.resize(n);
  for (int m = 0; m < n; ++m) {
    const double a = 6.283185307179586476925286766559 * m / n;
    const float2 re = pair_of(std::cos(a)), im = pair_of(std::sin(a));
    tw[m] = make_float4(re.x, im.x, re.y, im.y);
  }
}

}  // namespace
}  // namespace pdt
