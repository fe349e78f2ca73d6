// Device helpers of the FP64 matrix-instruction kernels (fgt_pw64.cu,
// fgt_pw64_2d.cu): the matrix instruction, the spreading kernel as
// polynomials, stencil cells.
#pragma once
#include "fgt_pw_dev.cuh"

namespace fgt {

namespace {

// C (8x8) += A (8x4) B (4x8): lane holds A[lane/4][lane%4], B[lane%4][lane/4]
// and C[lane/4][2 (lane%4) + {0,1}].
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}
// Spreading kernel of one stencil cell and its derivative, from the formula
// of es_kernel / kernel_val_d with one reciprocal square root and one
// reciprocal instead of a square root and two divisions.
__device__ __forceinline__ void es64_cell(const PWArgs<double>& a, double f, double& phi,
                                          double& dphi) {
  const double z = f * a.inv_hw, q = 1.0 - z * z;
  const double rq = q > 0.0 ? rsqrt(q) : 0.0;
  const double e = exp(-(a.beta * (z * z)) * __drcp_rn(1.0 + q * rq));
  phi = e;
  dphi = e * (a.beta * a.dscale) * z * rq;
}
// The kernel on the interior cells of a stencil as polynomials in the
// position t in [-1/2, 1/2] inside the cell (piecewise polynomial kernels as
// in Barnett, Magland and af Klinteberg 2019).  Cell W-1-j mirrors cell j, so
// the even and the odd half of one polynomial serve both; the derivative
// comes out of the same Horner steps.  The first and the last cell, where the
// kernel ends in a square root, keep the formula.
constexpr int ESN = 16;  // coefficients: errors at the rounding of the values
struct Es64 {
  double tc;         // t = f0 + tc
  double dt;         // derivative scale
  double c[7][ESN];  // cells 1 .. W/2 - 1
};
template <int W, bool DERIV, class F>
__device__ __forceinline__ void es64_row(const PWArgs<double>& a, const Es64& es, double f0,
                                         F&& put) {
  const double t = f0 + es.tc, s = t * t;
#pragma unroll
  for (int j = 1; j < W / 2; j++) {
    const double* c = es.c[j - 1];
    double E = c[ESN - 2], O = c[ESN - 1], Ed = 0.0, Od = 0.0;
#pragma unroll
    for (int i = ESN - 4; i >= 0; i -= 2) {
      if constexpr (DERIV) {
        Ed = fma(Ed, s, E);
        Od = fma(Od, s, O);
      }
      E = fma(E, s, c[i]);
      O = fma(O, s, c[i + 1]);
    }
    double d0 = 0.0, d1 = 0.0;
    if constexpr (DERIV) {
      const double de = 2.0 * t * Ed, dd = fma(2.0 * s, Od, O);
      d0 = (de + dd) * es.dt;
      d1 = (de - dd) * es.dt;
    }
    put(j, fma(t, O, E), d0);
    put(W - 1 - j, fma(-t, O, E), d1);
  }
#pragma unroll
  for (int j = 0; j < W; j += W - 1) {
    double f, d;
    es64_cell(a, f0 + (double)j, f, d);
    put(j, f, d);
  }
}
// First stencil cell, inside the sub-grid, of a coordinate (offset from the
// box centre) and the kernel argument f0 of that cell.  Explicitly rounded:
// the sort and the kernel rows must agree on the cell.
template <int W>
__device__ __forceinline__ int cell64(const PWArgs<double>& a, double off, double& f0) {
  const double x = __dmul_rn(off, a.scale_d);
  const double i0 = ceil(__dsub_rn(__dmul_rn(x, a.inv_dx_d), a.hwdx_d));
  f0 = __fma_rn(-x, a.inv_dx_d, i0);
  const int b = (int)i0 - a.g.l0;
  return b < 0 ? 0 : (b > a.g.G - W ? a.g.G - W : b);
}

// Polynomials of the kernel on the cells 1 .. W/2 - 1 of a stencil: Chebyshev
// interpolation in extended precision, as monomials in t.
static void es_polys(int W, const PWArgs<double>& a, Es64& es) {
  constexpr int N = ESN;
  const long double pi = acosl(-1.0L), beta = a.beta;
  es.tc = a.hwdx_d - 0.5;
  es.dt = -a.dscale / a.inv_hw;
  long double T[N][N] = {};  // monomials of the Chebyshev polynomials
  T[0][0] = T[1][1] = 1;
  for (int j = 2; j < N; j++)
    for (int i = 0; i < N; i++) T[j][i] = (i ? 2 * T[j - 1][i - 1] : 0) - T[j - 2][i];
  struct Polys {
    int W = 0;
    double beta, c[7][N];
  };
  static thread_local Polys made[17];  // by width
  Polys& last = made[W];
  if (last.W != W || last.beta != a.beta) {
    for (int cell = 1; cell < W / 2; cell++) {
      long double f[N], m[N] = {};
      for (int k = 0; k < N; k++) {
        const long double t = cosl(pi * (k + 0.5L) / N) / 2;
        const long double z = (-0.5L * W + cell + 0.5L + t) / (0.5L * W);
        f[k] = expl(-beta * z * z / (1 + sqrtl(1 - z * z)));
      }
      for (int j = 0; j < N; j++) {
        long double s = 0;
        for (int k = 0; k < N; k++) s += f[k] * cosl(pi * j * (k + 0.5L) / N);
        s *= (j ? 2.0L : 1.0L) / N;
        for (int i = 0; i < N; i++) m[i] += s * T[j][i];
      }
      for (int i = 0; i < N; i++) last.c[cell - 1][i] = (double)(m[i] * (1 << i));  // of 2t -> of t
    }
    last.W = W;
    last.beta = a.beta;
  }
  for (int c = 0; c < W / 2 - 1; c++)
    for (int i = 0; i < N; i++) es.c[c][i] = last.c[c][i];
}

}  // namespace

}  // namespace fgt
