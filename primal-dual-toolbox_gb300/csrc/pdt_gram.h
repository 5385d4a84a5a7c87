// pdt_gram.h -- the iterations of the with-operator solvers for masks of whole phase-encode lines.
//
// When every sampled column of the mask is constant along the readout, the readout transforms of K and K^H
// cancel and K^H K acts on each image row by itself:
//   (K^H K u)(y, .) = sum_c conj(s_c) . G (s_c . u)(y, .),   G = (1 / W) IDFT diag(m^2) DFT along the row,
// and the k-space dual of r <- (r + sigma (K ubar - f)) / (1 + sigma lambda) stays in the span
//   r_n = K U_n - c_n f + d_n r_0,   U <- U + k (ubar - lambda U),  k = sigma / (1 + sigma lambda),
//   c <- c + k (1 - lambda c) from 0,   d <- d - k lambda d from 1,
// so that K^H r_n = K^H K U_n - c_n K^H f + d_n K^H r_0 needs one image U, two fixed images and the row
// operator G: no k-space array and no transform along the readout inside an iteration. K^H K U_n and c_n K^H f are far
// larger than their difference, and a rounding error of either acts in every iteration, so neither is formed: with a
// reference image w = a K^H f, a least-squares in |K w - f|, and D = U - c w,
//   K^H r_n = K^H K D_n + c_n h + d_n K^H r_0,   h = K^H (K w - f),   D <- D + k ((ubar - w) - lambda D),
// where D grows with ubar - w only and h is transformed once with twice the precision (pdt_cart_pair.cuh). D is carried
// with a compensation term (the rounding errors of its updates, as in Kahan's summation): without it an update
// below half a unit in the last place of D is lost, and D stops up to (1 + sigma lambda) / (2 sigma lambda)
// units away from its limit, which K^H K passes on to u in every iteration. The error of K^H K D still grows with c
// (to 1 / lambda), so the solvers use this form up to a bound on c.
//
// One iteration is two launches: launch_gram_rows (K^H K D in coil-group partial sums) and
// launch_gram_image (primal update, then the next iteration's dual update and D).
#pragma once

#include <cstddef>
#include <vector>

#include "pdt_internal.h"

namespace pdt {

// One compiled transform length n = P Q (P values per thread, then Q).
struct GramLength {
  int n, P, Q;
};

// What an operator with a line mask hands to the solvers.
struct GramRows {
  int W = 0, H = 0, C = 0;        // image and coils
  const float2* sens = nullptr;   // coil 0, image row 0, or null (one coil without a map)
  size_t coil_stride = 0;         // elements between coils
  GramLength len{0, 0, 0};
  const float2* tw = nullptr;     // [Q][P] exp(-2 pi i t k1 / n)
  const float* spec = nullptr;    // [n] spectrum of G in the natural order, scaled for an unscaled inverse
  int groups = 1;                 // coil-group partial sums of K^H K D
};

// The compiled length for rows of W: W itself, or the smallest one that holds the linear convolution
// (n >= 2 W - 1), in which G is embedded as a Toeplitz operator. n = 0: none.
GramLength gram_length(int W);

// Coil groups for an H-row image on a GPU of `sms` multiprocessors.
int gram_groups(const GramLength& len, int H, int C, int sms);

// Host tables (tw: n values, spec: n values) of the row operator. m2[k]: squared mask value at the DFT
// index k of a row (0 where not sampled).
void gram_tables(int W, const GramLength& len, const std::vector<float>& m2, std::vector<float2>& tw,
                 std::vector<float>& spec);

struct GramImage {
  int W, H;
  ImgPtrs src;           // u, v and the p, q of this iteration
  ImgPtrs dst;           // new u, v; ubar, vbar (last iteration only, see launch_gram_image); p, q of the next
  const float2* D;       // this iteration's D, then its compensation (W x H each)
  float2* Dnext;
  const float2* part;    // `groups` partial sums of K^H K D, W x H each
  int groups;
  const float2* w;       // reference image
  const float2* h;       // K^H (K w - f)
  const float2* z0;      // K^H r_0, or null when r_0 = 0
  const float4* table;   // per iteration {alpha0, alpha1, c, d}
  int* header;           // [1] table length, [2] non-finite flag, [4], [5] iteration counters (see par)
  int par;               // this iteration's counter is header[4 + par]; it sets header[4 + (par ^ 1)]
  float tau, sigma, lambda, k;
};

// part[g] <- sum of conj(s_c) . G (s_c . D) over the coils of group g.
void launch_gram_rows(const GramRows& g, const float2* D, float2* part, cudaStream_t st);
// u, v <- the primal update from part; then, unless this is the table's last iteration, p, q and D of the
// next one (the last iteration stores ubar and vbar instead). Raises header[2] on a non-finite u or v. Without
// `rows`, part holds K^H r itself: D, w, h, z0 are not used and every iteration stores ubar, which the next operator
// round reads.
void launch_gram_image(bool tgv, bool rows, const GramImage& s, cudaStream_t st);
// w <- a w for w = K^H f and part = K^H K w, a = |w|^2 / <w, K^H K w> (0 where that is not finite), and the first
// iteration's D <- k (ubar - w) with compensation 0 (from D_0 = 0). `dots`: kGramDots values of scratch.
constexpr int kGramDots = 128;
void launch_gram_start(int W, int H, const float2* part, int groups, const float2* ubar, float k, float2* w, float2* D,
                       float2* dots, cudaStream_t st);
// out <- U = D + c w.
void launch_gram_total(int W, int H, const float2* D, const float2* w, float c, float2* out, cudaStream_t st);

}  // namespace pdt
