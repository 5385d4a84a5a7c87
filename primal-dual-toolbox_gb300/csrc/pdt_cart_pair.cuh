// pdt_cart_pair.cuh -- K^H (K u - f) of a line-sampled Cartesian operator in pairs of FP32 values (about 48 bits), once
// per solve with the row operator (pdt_gram.h).
//
// The solve adds c times this image to K^H K D in every iteration, so an error of it acts in every iteration, also in
// the directions that the mask does not see, where nothing but the regularisation pulls it back. FP32 transforms are
// 1.3e-7 off; with them a TGV-MRI solve (8 coils, 96 x 92, reduction 0.01) of 255 iterations ended 5.5e-7 off the
// solution in 64 bits, where the k-space dual ends 2.1e-7 off. Pairs rather than FP64, whose units have a sixtieth of the
// FP32 rate on this GPU.
//
// pair_cols   sampled columns of mask . f, inverse transform along Hf, image rows: t[row][coil][column]
// pair_rows   per image row: rows of the coil images, their spectra times the squared mask, minus the columns, inverse
//             transform, conj(sens) and coil sum. The readout transforms of K^H K cancel (whole lines).
// The transforms are Stockham passes over sequences in shared memory: odd radices R first, by the sums x_r +- x_(R - r)
// (a pass of their own, which applies the twiddles too) and a thread per pair of outputs q, R - q; then radix 4 and 2.
// Bound by issue slots (a sum of pairs is eight instructions, a product of complex pairs 32), hence divisions by
// multiplication in the index arithmetic. 15 coils, 640 x 368 (320 image rows, 92 columns): 35 + 131 + 4 us.
// Included by pdt_cartesian.cu after CartDev.
#pragma once

namespace pdt {
namespace {

constexpr int kPairThreads = 128;  // of a block of pair_cols
constexpr int kPairCoils = 4;      // most coils at a time in pair_rows, 64 threads each

// h + l, l the rounding errors so far (explicit roundings: a fused product would lose its error term).
struct PairSum {
  float h, l;
  // + x, x = xh + xl
  __device__ __forceinline__ void add(float xh, float xl) {
    const float s = __fadd_rn(h, xh), t = __fsub_rn(s, h);
    l = __fadd_rn(l, __fadd_rn(__fadd_rn(__fsub_rn(h, __fsub_rn(s, t)), __fsub_rn(xh, t)), xl));
    h = s;
  }
  // + x y
  __device__ __forceinline__ void mac(float xh, float xl, float yh, float yl) {
    const float p = __fmul_rn(xh, yh);
    add(p, __fmaf_rn(xl, yh, __fmaf_rn(xh, yl, __fmaf_rn(xh, yh, -p))));
  }
};
__device__ __forceinline__ PairSum pair_mul(float xh, float xl, float yh, float yl) {
  const float p = __fmul_rn(xh, yh);
  return {p, __fmaf_rn(xl, yh, __fmaf_rn(xh, yl, __fmaf_rn(xh, yh, -p)))};
}

// A complex pair: {re, im, re remainder, im remainder}.
__device__ __forceinline__ float4 pair4(PairSum re, PairSum im) { return make_float4(re.h, im.h, re.l, im.l); }
__device__ __forceinline__ float4 pair_zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float4 pair_conj(float4 a) { return make_float4(a.x, -a.y, a.z, -a.w); }
__device__ __forceinline__ float4 pair_i(float4 a) { return make_float4(-a.y, a.x, -a.w, a.z); }
__device__ __forceinline__ float4 pair_add(float4 a, float4 b) {
  PairSum re{a.x, a.z}, im{a.y, a.w};
  re.add(b.x, b.z);
  im.add(b.y, b.w);
  return pair4(re, im);
}
__device__ __forceinline__ float4 pair_sub(float4 a, float4 b) {
  return pair_add(a, make_float4(-b.x, -b.y, -b.z, -b.w));
}
__device__ __forceinline__ float4 pair_cmul(float4 x, float4 y) {
  PairSum re = pair_mul(x.x, x.z, y.x, y.z), im = pair_mul(x.x, x.z, y.y, y.w);
  re.mac(-x.y, -x.w, y.y, y.w);
  im.mac(x.y, x.w, y.x, y.z);
  return pair4(re, im);
}
// x times the real pair {y.x, y.y}
__device__ __forceinline__ float4 pair_scale(float4 x, float2 y) {
  return pair4(pair_mul(x.x, x.z, y.x, y.y), pair_mul(x.y, x.w, y.x, y.y));
}

// t / d for t d < 2^32
struct PairDiv {
  unsigned d, m;
  __device__ explicit PairDiv(int n) : d(n), m(0xFFFFFFFFu / n + 1) {}
  __device__ __forceinline__ int operator()(int t) const { return d == 1 ? t : (int)__umulhi((unsigned)t, m); }
};

// nseq inverse transforms (unscaled) of pl.n values in shared memory, sequence i at a[i n]; pl from pair_plan().
// tw[m] = exp(2 pi i m / n). Returns the buffer that holds the result; starts after and ends with a barrier.
__device__ __noinline__ float4* pair_ifft(float4* a, float4* b, int nseq, const FftPlan& pl, const float4* tw) {
  const int n = pl.n, nt = blockDim.x;
  int Ns = 1;
  for (int st = 0; st < pl.nst; ++st) {
    const int R = pl.radix[st], nb = n / R, unit = nb / Ns, h = R / 2;
    const PairDiv by_nb(nb), by_Ns(Ns);
    if (R & 1) {  // x_r, x_(R - r) <- their sum and difference
      const PairDiv by_sq(nb * h);
      for (int t = threadIdx.x; t < nb * h * nseq; t += nt) {
        const int sq = by_sq(t), i = t - sq * (nb * h), p = by_nb(i), r = p + 1, j = i - p * nb, k = j - by_Ns(j) * Ns;
        float4 *px = a + sq * n + j + r * nb, *py = a + sq * n + j + (R - r) * nb;
        float4 x = *px, y = *py;
        if (k) {
          x = pair_cmul(x, tw[r * k * unit]);
          y = pair_cmul(y, tw[(R - r) * k * unit]);
        }
        *px = pair_add(x, y);
        *py = pair_sub(x, y);
      }
      __syncthreads();
    }
    const int items = R & 1 ? nb * (h + 1) : nb;  // tasks a sequence: butterfly j, output pair q
    const PairDiv by_sq(items);
    for (int t = threadIdx.x; t < items * nseq; t += nt) {
      const int sq = by_sq(t), i = t - sq * items, q = by_nb(i), j = i - q * nb, blk = by_Ns(j), k = j - blk * Ns;
      const float4* src = a + sq * n + j;
      float4* dst = b + sq * n + blk * Ns * R + k;
      if (R & 1) {  // X_q, X_(R - q) = A +- i B
        const float4 x0 = src[0];
        PairSum ar{x0.x, x0.z}, ai{x0.y, x0.w}, br{0.f, 0.f}, bi{0.f, 0.f};
        if (q == 0) {
          for (int r = 1; r <= h; ++r) {
            const float4 s = src[r * nb];
            ar.add(s.x, s.z);
            ai.add(s.y, s.w);
          }
          dst[0] = pair4(ar, ai);
          continue;
        }
        for (int r = 1, m = q; r <= h; ++r) {
          const float4 s = src[r * nb], d = src[(R - r) * nb], w = tw[m * nb];  // cos, sin of 2 pi r q / R
          ar.mac(s.x, s.z, w.x, w.z);
          ai.mac(s.y, s.w, w.x, w.z);
          br.mac(d.x, d.z, w.y, w.w);
          bi.mac(d.y, d.w, w.y, w.w);
          m += q;
          if (m >= R) m -= R;
        }
        const float4 A = pair4(ar, ai), iB = pair_i(pair4(br, bi));
        dst[q * Ns] = pair_add(A, iB);
        dst[(R - q) * Ns] = pair_sub(A, iB);
        continue;
      }
      auto in = [&](int r) {  // input r with its twiddle
        const float4 x = src[r * nb];
        return k ? pair_cmul(x, tw[r * k * unit]) : x;
      };
      if (R == 4) {
        const float4 x0 = src[0], x1 = in(1), x2 = in(2), x3 = in(3);
        const float4 s02 = pair_add(x0, x2), d02 = pair_sub(x0, x2), s13 = pair_add(x1, x3), i13 = pair_i(pair_sub(x1, x3));
        dst[0] = pair_add(s02, s13);
        dst[Ns] = pair_add(d02, i13);
        dst[2 * Ns] = pair_sub(s02, s13);
        dst[3 * Ns] = pair_sub(d02, i13);
      } else {
        const float4 x0 = src[0], x1 = in(1);
        dst[0] = pair_add(x0, x1);
        dst[Ns] = pair_sub(x0, x1);
      }
    }
    __syncthreads();
    float4* x = a;
    a = b;
    b = x;
    Ns *= R;
  }
  return a;
}

// Block (column, coil).
__global__ void __launch_bounds__(kPairThreads) pair_cols(CartDev d, FftPlan pl, const float4* __restrict__ tw,
                                                          const float2* __restrict__ fc, float4* __restrict__ t) {
  extern __shared__ float4 psm[];
  const int n = d.Hf, s = blockIdx.x, c = blockIdx.y;
  float4 *w = psm, *A = w + n, *B = A + n;
  const size_t col = (size_t)c * d.ns + s;
  for (int P = threadIdx.x; P < n; P += kPairThreads) {
    w[P] = tw[P];
    const float2 f = fc[col * n + P];
    A[imod((d.kperm ? d.kperm[P] : P) + d.mxH, n)] =
        pair_scale(make_float4(f.x, f.y, 0.f, 0.f), c2(d.maskc[(size_t)s * n + P], 0.f));
  }
  __syncthreads();
  const float4* Z = pair_ifft(A, B, 1, pl, w);
  for (int j = threadIdx.x; j < n; j += kPairThreads) {
    const int yi = imod(j + d.oyH, n) - d.y0;
    if (yi >= 0 && yi < d.Hi) t[((size_t)yi * d.C + c) * d.ns + s] = Z[j];
  }
}

// Block (image row y, coil group) of 64 threads per coil of a pass (at least 128); part[group][y][x]. Slot j of both
// transforms is image column j + oxW, spectrum index k the sampled column slot2s[k]. `fwd` = sqrt(Hf / W): what K and the
// readout transforms leave.
__global__ void __launch_bounds__(64 * kPairCoils) pair_rows(CartDev d, FftPlan pl, const float4* __restrict__ tw,
                                                             const float4* __restrict__ t, const float2* __restrict__ u,
                                                             int nq, float2 fwd, float4* __restrict__ part) {
  extern __shared__ float4 psm[];
  const int n = d.W, nt = blockDim.x, y = blockIdx.x, g = blockIdx.y;
  const int cb = g * d.C / gridDim.y, ce = (g + 1) * d.C / gridDim.y;
  float4 *w = psm, *sum = w + n, *A = sum + n, *B = A + nq * n;
  const PairDiv by_n(n);
  auto col = [&](int j) { return j + d.oxW < n ? j + d.oxW : j + d.oxW - n; };
  auto sens = [&](int c, int x) {
    return d.sens ? d.sens[((size_t)c * d.Hf + y + d.y0) * n + x] : c2(1.f, 0.f);
  };
  for (int x = threadIdx.x; x < n; x += nt) {
    w[x] = tw[x];
    sum[x] = pair_zero();
  }
  for (int c0 = cb; c0 < ce; c0 += nq) {
    const int nc = min(nq, ce - c0);
    for (int i = threadIdx.x; i < nc * n; i += nt) {  // conjugates: the transform is an inverse one
      const int q = by_n(i), x = col(i - q * n);
      const float2 s = sens(c0 + q, x), v = u[(size_t)y * n + x];
      A[i] = pair_conj(pair_cmul(make_float4(s.x, s.y, 0.f, 0.f), make_float4(v.x, v.y, 0.f, 0.f)));
    }
    __syncthreads();
    float4* Z = pair_ifft(A, B, nc, pl, w);
    for (int i = threadIdx.x; i < nc * n; i += nt) {
      const int q = by_n(i), s = d.slot2s[i - q * n];
      if (s < 0) {
        Z[i] = pair_zero();
        continue;
      }
      const float m = d.maskc[(size_t)s * d.Hf], m2 = __fmul_rn(m, m);
      const float4 k = pair_scale(pair_scale(pair_conj(Z[i]), fwd), c2(m2, __fmaf_rn(m, m, -m2)));
      Z[i] = pair_sub(k, t[((size_t)y * d.C + c0 + q) * d.ns + s]);
    }
    __syncthreads();
    Z = pair_ifft(Z, Z == A ? B : A, nc, pl, w);
    for (int j = threadIdx.x; j < n; j += nt) {
      const int x = col(j);
      float4 z = sum[j];
      for (int q = 0; q < nc; ++q) {
        const float2 s = sens(c0 + q, x);
        z = pair_add(z, pair_cmul(Z[q * n + j], make_float4(s.x, -s.y, 0.f, 0.f)));
      }
      sum[j] = z;
    }
    __syncthreads();
  }
  for (int j = threadIdx.x; j < n; j += nt) part[((size_t)g * d.Hi + y) * n + col(j)] = sum[j];
}

// out <- scale . sum of the groups' images, scale = 1 / sqrt(W Hf).
__global__ void __launch_bounds__(256) pair_sum(size_t n, const float4* __restrict__ part, int G, float2 scale,
                                                float2* __restrict__ out) {
  const size_t i = blockIdx.x * (size_t)256 + threadIdx.x;
  if (i >= n) return;
  float4 z = part[i];
  for (int g = 1; g < G; ++g) z = pair_add(z, part[g * n + i]);
  z = pair_scale(z, scale);
  out[i] = c2(__fadd_rn(z.x, z.z), __fadd_rn(z.y, z.w));
}

inline size_t pair_cols_smem(int Hf) { return sizeof(float4) * 3 * (size_t)Hf; }
inline size_t pair_rows_smem(int W, int nq) { return sizeof(float4) * (2 + 2 * (size_t)nq) * W; }
// Coil groups of a row, of equal size: about eight blocks an SM in all; and their coils at a time.
inline int pair_groups(int C, int Hi, int sms) {
  const int most = std::max(1, std::min((C + 1) / 2, (8 * sms + Hi / 2) / Hi)), per = (C + most - 1) / most;
  return (C + per - 1) / per;
}
inline int pair_coils(int C, int G) {
  const int per = (C + G - 1) / G, passes = (per + kPairCoils - 1) / kPairCoils;
  return (per + passes - 1) / passes;
}

// v as the sum of two FP32 values
inline float2 pair_of(double v) { return make_float2((float)v, (float)(v - (double)(float)v)); }

// The radices of pair_ifft: odd primes, largest first, then 4 and 2.
inline bool pair_plan(int n, FftPlan* pl) {
  FftPlan p;
  if (!make_fft_plan(n, &p)) return false;
  pl->n = n;
  pl->nst = 0;
  for (int i = p.nst - 1; i >= 0; --i)
    if (p.radix[i] & 1) pl->radix[pl->nst++] = p.radix[i];
  int m = n;
  for (int i = 0; i < pl->nst; ++i) m /= pl->radix[i];
  for (; m > 1; m /= pl->radix[pl->nst - 1]) {
    if (pl->nst >= kMaxStages) return false;
    pl->radix[pl->nst++] = m % 4 == 0 ? 4 : 2;
  }
  return true;
}

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
