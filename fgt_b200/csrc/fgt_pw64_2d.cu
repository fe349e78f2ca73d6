// FP64 form and evaluation of small 2D boxes (at most SMALL2_MAX points)
// without wrap-around on the FP64 matrix instructions, one warp per (box,
// density).  The box's grid and half-complex intermediate share one shared
// memory buffer per warp; spreading is one product of the points' kernel rows,
// G[x][y] = sum_p (q wx)[x][p] wy[p][y], in registers over all tiles of the
// grid (its zeros cost less than sorting a few hundred points), and the line
// transforms are as in fgt_pw64.cu.  The SIMT warp-per-box kernels that these
// replace were bound by latency: 120-instruction kernel values one point at a
// time (spreading) and eight lone warps per SM on unblocked transforms.
// Two densities, 4e5 curve points in 2,300 boxes, K = 20: form 1.27 -> 0.44 ms,
// evaluation 1.43 -> 0.46 ms (phases, with their small launches).
#include <stdlib.h>

#include "fgt_pw64.cuh"
#include "fgt_pw64_dev.cuh"

namespace fgt {

namespace {

constexpr int W2D = 8;         // warps per CTA (fewer where their grids do not fit)
constexpr int T2D = 32 * W2D;
constexpr int PB2D = 16;       // points per batch of kernel rows

// Per warp: GP = 8 GT rows of S doubles; a kernel-row batch (2 x 16 rows of
// GP + 4) fits in the same space.  Row strides are 4 or 12 modulo 16: operand
// fragments (4 rows of 4) fall on distinct banks.
struct Lay2D {
  int S, buf;
  __host__ __device__ Lay2D(int GT, int MT) {
    S = (8 * GT > 16 * MT ? 8 * GT : 16 * MT) + 4;
    const int rows = 2 * PB2D * (8 * GT + 4), grid = 8 * GT * S;
    buf = rows > grid ? rows : grid;
  }
};
// doubles of the tables: cos and sin fragments, then the last dimension's
__host__ __device__ constexpr int tabs_form(int MT, int ksg) { return 32 * ksg * (2 * MT + 2 * MT); }
__host__ __device__ constexpr int tabs_eval(int GT, int K) {
  return 32 * GT * (2 * ((K + 4) / 4) + (2 * (K + 1) + 3) / 4);
}

template <int W, int GT, int MT>
__global__ void __launch_bounds__(T2D, 1)
    k_form2d64(const __grid_constant__ PWArgs<double> a, const __grid_constant__ Es64 es,
               const __grid_constant__ Form64 io, const int* __restrict__ first,
               int* __restrict__ next) {
  extern __shared__ __align__(16) double sm2[];
  const Geo& g = a.g;
  const int K = g.K, NH = K + 1, G = g.G, ksg = (G + 3) / 4;
  const int NFp = pad4(2 * K + 1), NHp = pad4(NH);
  const Lay2D lay(GT, MT);
  const int S = lay.S;
  constexpr int RS = 8 * GT + 4;
  double *re = sm2, *im = re + 32 * MT * ksg, *zt = im + 32 * MT * ksg;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l4 = lane & 3, r8 = lane >> 2;
  double* B = sm2 + tabs_form(MT, ksg) + (size_t)warp * lay.buf;
  for (int i = threadIdx.x; i < MT * ksg * 32; i += blockDim.x) {
    const int ln = i & 31, mt = (i >> 5) % MT, ks = (i >> 5) / MT;
    const int k = 8 * mt + (ln >> 2), l = 4 * ks + (ln & 3);
    const bool ok = k <= K && l < G;
    re[i] = ok ? a.twf[(size_t)l * 2 * NFp + K + k] : 0.0;
    im[i] = ok ? a.twf[(size_t)l * 2 * NFp + NFp + K + k] : 0.0;
  }
  for (int i = threadIdx.x; i < ksg * 2 * MT * 32; i += blockDim.x) {
    const int ln = i & 31, nt = (i >> 5) % (2 * MT), ks = (i >> 5) / (2 * MT);
    const int l = 4 * ks + (ln & 3), c = 8 * nt + (ln >> 2);
    zt[i] = l < G && c < 2 * NH ? a.twh[(size_t)l * 2 * NHp + (c & 1) * NHp + (c >> 1)] : 0.0;
  }
  __syncthreads();
  const int f0 = *first, nwork = (io.n_form - f0) * io.nd;
  for (;;) {
    int w = 0;
    if (lane == 0) w = atomicAdd(next, 1);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= nwork) break;
    const int fb = (int)io.order[f0 + w / io.nd], id = w % io.nd;
    if (!FGT_DCHECK(fb >= 0 && fb < io.n_form, 620)) continue;
    const int box = io.form_box[fb], p0 = io.s_lo[box], p1 = io.s_hi[box];
    if (!FGT_DCHECK(p0 >= 0 && p0 <= p1 && p1 <= io.ns, 621)) continue;
    double2* mp = reinterpret_cast<double2*>(io.mp + ((size_t)fb * io.nd + id) * 2 * g.nexp);
    for (int comp = 0; comp < io.ncomp; comp++) {
      const bool is_q = io.has_q && comp == 0;
      const int dd = comp - io.has_q;
      const double* sq = (is_q ? io.q : io.ds) + (size_t)id * io.ns;
      const double* sr = is_q ? nullptr : io.rn + (size_t)dd * io.ns;
      double acc[GT][GT][2];
#pragma unroll
      for (int m = 0; m < GT; m++)
#pragma unroll
        for (int n = 0; n < GT; n++) acc[m][n][0] = acc[m][n][1] = 0.0;
      for (int c0 = p0; c0 < p1; c0 += PB2D) {
        const int np = min(PB2D, p1 - c0);
        // kernel rows: lane (point, dimension), zero outside the stencil
        {
          const int p = lane & 15, d = lane >> 4;
          double* row = B + (d * PB2D + p) * RS;
          for (int j = 0; j < RS; j++) row[j] = 0.0;
          if (p < np) {
            const int pt = c0 + p;
            const double sc = d ? 1.0 : (sr ? sq[pt] * sr[pt] : sq[pt]);
            double f;
            const int o = cell64<W>(a, io.off[(size_t)d * io.ns + pt], f);
            es64_row<W, false>(a, es, f, [&](int j, double v, double) { row[o + j] = v * sc; });
          }
        }
        __syncwarp();
        for (int k = 0; k < np; k += 4) {
          const double *X = B + (k + l4) * RS + r8, *Y = X + PB2D * RS;
          double x[GT], y[GT];
#pragma unroll
          for (int m = 0; m < GT; m++) {
            x[m] = X[8 * m];
            y[m] = Y[8 * m];
          }
#pragma unroll
          for (int m = 0; m < GT; m++)
#pragma unroll
            for (int n = 0; n < GT; n++) dmma(acc[m][n][0], acc[m][n][1], x[m], y[n]);
        }
        __syncwarp();
      }
      // grid, then real -> ky in place, eight rows at a time
#pragma unroll
      for (int m = 0; m < GT; m++)
#pragma unroll
        for (int n = 0; n < GT; n++)
          *reinterpret_cast<double2*>(B + (8 * m + r8) * S + 8 * n + 2 * l4) =
              make_double2(acc[m][n][0], acc[m][n][1]);
      __syncwarp();
      for (int m = 0; m < GT; m++) {
        double in[2 * GT], c[2 * MT][2];
        double* row = B + (8 * m + r8) * S;
#pragma unroll
        for (int ks = 0; ks < 2 * GT; ks++) in[ks] = row[4 * ks + l4];
#pragma unroll
        for (int n = 0; n < 2 * MT; n++) c[n][0] = c[n][1] = 0.0;
#pragma unroll
        for (int ks = 0; ks < 2 * GT; ks++) {
          if (ks >= ksg) break;
#pragma unroll
          for (int n = 0; n < 2 * MT; n++)
            dmma(c[n][0], c[n][1], in[ks], zt[(ks * 2 * MT + n) * 32 + lane]);
        }
        __syncwarp();
#pragma unroll
        for (int n = 0; n < 2 * MT; n++)
          *reinterpret_cast<double2*>(row + 8 * n + 2 * l4) = make_double2(c[n][0], c[n][1]);
        __syncwarp();
      }
      // x: out(+-k) = p +- i q, into the expansion
      for (int nt = 0; nt < (2 * NH + 7) / 8; nt++) {
        double in[2 * GT], p[MT][2], q[MT][2];
#pragma unroll
        for (int ks = 0; ks < 2 * GT; ks++) in[ks] = B[(4 * ks + l4) * S + 8 * nt + r8];
#pragma unroll
        for (int m = 0; m < MT; m++) p[m][0] = p[m][1] = q[m][0] = q[m][1] = 0.0;
#pragma unroll
        for (int ks = 0; ks < 2 * GT; ks++) {
          if (ks >= ksg) break;
#pragma unroll
          for (int m = 0; m < MT; m++) {
            dmma(p[m][0], p[m][1], re[(ks * MT + m) * 32 + lane], in[ks]);
            dmma(q[m][0], q[m][1], im[(ks * MT + m) * 32 + lane], in[ks]);
          }
        }
        const int ky = 4 * nt + l4;
        if (ky < NH) {
#pragma unroll
          for (int m = 0; m < MT; m++) {
            const int k = 8 * m + r8;
            if (k > K) continue;
#pragma unroll
            for (int sg = 1; sg >= -1; sg -= 2) {
              if (sg < 0 && k == 0) continue;
              const int ki[3] = {K + sg * k, K + ky, 0};
              const double f = a.facf[ki[0]] * a.facf[ki[1]];
              double vr = (p[m][0] - sg * q[m][1]) * f, vi = (p[m][1] + sg * q[m][0]) * f;
              if (!is_q) {  // * (-i) ts(k_d) / sqrt(delta0)
                const double cc = a.ts[sel3(ki, dd)] * a.inv_sqd0, tr = vi * cc, ti = -vr * cc;
                vr = tr;
                vi = ti;
              }
              double2* o = mp + (size_t)ki[0] * NH + ky;
              if (comp > 0) {
                const double2 v = *o;
                vr += v.x;
                vi += v.y;
              }
              *o = make_double2(vr, vi);
            }
          }
        }
      }
      __syncwarp();
    }
  }
}

template <int W, bool DERIV, int GT, int MT>
__global__ void __launch_bounds__(T2D, 1)
    k_eval2d64(const __grid_constant__ PWArgs<double> a, const __grid_constant__ Es64 es,
               const __grid_constant__ Eval64 io, const int* __restrict__ first,
               int* __restrict__ next) {
  extern __shared__ __align__(16) double sm2[];
  const Geo& g = a.g;
  const int K = g.K, NH = K + 1, G = g.G, Gp = pad4(G), ksk = (NH + 3) / 4, ksz = (2 * NH + 3) / 4;
  const Lay2D lay(GT, MT);
  const int S = lay.S;
  double *re = sm2, *im = re + 32 * GT * ksk, *zt = im + 32 * GT * ksk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l4 = lane & 3, r8 = lane >> 2;
  double* B = sm2 + tabs_eval(GT, K) + (size_t)warp * lay.buf;
  for (int i = threadIdx.x; i < GT * ksk * 32; i += blockDim.x) {
    const int ln = i & 31, mt = (i >> 5) % GT, ks = (i >> 5) / GT;
    const int l = 8 * mt + (ln >> 2), k = 4 * ks + (ln & 3);
    const bool ok = l < G && k <= K;
    const double f = ok ? a.faci[K + k] : 0.0;
    re[i] = ok ? a.tif[(size_t)(K + k) * 2 * Gp + l] * f : 0.0;
    im[i] = ok ? a.tif[(size_t)(K + k) * 2 * Gp + Gp + l] * f : 0.0;
  }
  for (int i = threadIdx.x; i < ksz * GT * 32; i += blockDim.x) {
    const int ln = i & 31, nt = (i >> 5) % GT, ks = (i >> 5) / GT;
    const int c = 4 * ks + (ln & 3), l = 8 * nt + (ln >> 2), ky = c >> 1;
    double v = 0.0;
    if (c < 2 * NH && l < G) {
      v = a.tih[(size_t)ky * 2 * Gp + (c & 1) * Gp + l] * a.faci[K + ky];
      if (c & 1) v = -v;
    }
    zt[i] = v;
  }
  __syncthreads();
  const int f0 = *first, nwork = (*io.nbox_dev - f0) * io.nd;
  for (;;) {
    int w = 0;
    if (lane == 0) w = atomicAdd(next, 1);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= nwork) break;
    const int e = io.boxes[f0 + w / io.nd], id = w % io.nd;
    if (!FGT_DCHECK(e >= 0 && e < io.nbox, 622)) continue;
    const int box = io.eval_box[e];
    const double* L = io.loc + ((size_t)e * io.nd + id) * 2 * g.nexp;
    // x: modes +-k of four ky columns -> rows x
    for (int nt = 0; nt < 2 * MT; nt++) {
      double v0[2 * MT], v1[2 * MT], p[GT][2], q[GT][2];
      const int col = 8 * nt + r8;
#pragma unroll
      for (int ks = 0; ks < 2 * MT; ks++) {
        const int k = 4 * ks + l4;
        v0[ks] = v1[ks] = 0.0;
        if (k <= K && col < 2 * NH) {
          v0[ks] = __ldg(L + 2 * (size_t)(K + k) * NH + col);
          if (k > 0) v1[ks] = __ldg(L + 2 * (size_t)(K - k) * NH + col);
        }
      }
#pragma unroll
      for (int m = 0; m < GT; m++) p[m][0] = p[m][1] = q[m][0] = q[m][1] = 0.0;
#pragma unroll
      for (int ks = 0; ks < 2 * MT; ks++) {
        if (ks >= ksk) break;
        const double ev = v0[ks] + v1[ks], od = v0[ks] - v1[ks];
#pragma unroll
        for (int m = 0; m < GT; m++) {
          dmma(p[m][0], p[m][1], re[(ks * GT + m) * 32 + lane], ev);
          dmma(q[m][0], q[m][1], im[(ks * GT + m) * 32 + lane], od);
        }
      }
#pragma unroll
      for (int m = 0; m < GT; m++)
        *reinterpret_cast<double2*>(B + (8 * m + r8) * S + 8 * nt + 2 * l4) =
            make_double2(p[m][0] - q[m][1], p[m][1] + q[m][0]);
    }
    __syncwarp();
    // y, in place, eight rows at a time
    for (int m = 0; m < GT; m++) {
      double in[4 * MT], c[GT][2];
      double* row = B + (8 * m + r8) * S;
#pragma unroll
      for (int ks = 0; ks < 4 * MT; ks++) in[ks] = row[4 * ks + l4];
#pragma unroll
      for (int n = 0; n < GT; n++) c[n][0] = c[n][1] = 0.0;
#pragma unroll
      for (int ks = 0; ks < 4 * MT; ks++) {
        if (ks >= ksz) break;
#pragma unroll
        for (int n = 0; n < GT; n++) dmma(c[n][0], c[n][1], in[ks], zt[(ks * GT + n) * 32 + lane]);
      }
      __syncwarp();
#pragma unroll
      for (int n = 0; n < GT; n++)
        *reinterpret_cast<double2*>(row + 8 * n + 2 * l4) = make_double2(c[n][0], c[n][1]);
      __syncwarp();
    }
    // one point per lane
    for (int set = 0; set < 2; set++) {
      const int ne = set ? io.n[1] : io.n[0], nc = set ? io.ncomp[1] : io.ncomp[0];
      if (nc == 0 || ne == 0) continue;
      const double* off = set ? io.off[1] : io.off[0];
      double* out = set ? io.out[1] : io.out[0];
      const int q0 = set ? io.lo[1][box] : io.lo[0][box], q1 = set ? io.hi[1][box] : io.hi[0][box];
      if (!FGT_DCHECK(q0 >= 0 && q0 <= q1 && q1 <= ne, 623)) continue;
      for (int q = q0 + lane; q < q1; q += 32) {
        double fx, fy, py[W], dy[DERIV ? W : 1], px[W], dx[DERIV ? W : 1];
        const int ox = cell64<W>(a, off[q], fx), oy = cell64<W>(a, off[(size_t)ne + q], fy);
        es64_row<W, DERIV>(a, es, fx, [&](int j, double v, double d) {
          px[j] = v;
          if constexpr (DERIV) dx[j] = d;
        });
        es64_row<W, DERIV>(a, es, fy, [&](int j, double v, double d) {
          py[j] = v;
          if constexpr (DERIV) dy[j] = d;
        });
        const double* b = B + ox * S + oy;
        double pot = 0.0, gx = 0.0, gy = 0.0;
#pragma unroll
        for (int j = 0; j < W; j++) {
          double s0 = 0.0, s1 = 0.0;
#pragma unroll
          for (int i = 0; i < W; i++) {
            const double v = b[j * S + i];
            s0 = fma(v, py[i], s0);
            if constexpr (DERIV) s1 = fma(v, dy[i], s1);
          }
          pot = fma(px[j], s0, pot);
          if constexpr (DERIV) {
            gx = fma(dx[j], s0, gx);
            gy = fma(px[j], s1, gy);
          }
        }
        out[(size_t)id * ne + q] += pot;
        if constexpr (DERIV) {
          if (nc > 1) {
            // without the reference cell's derivative terms (interp_grad_cells)
            double kx = 0.0, ky = 0.0, sx = 0.0, sy = 0.0;
#pragma unroll
            for (int j = 0; j < W; j++) {
              kx += px[j];
              ky += py[j];
              sx += dx[j];
              sy += dy[j];
            }
            const double ref = b[(W / 2) * S + W / 2];
            out[((size_t)io.nd + id) * ne + q] += gx - ref * (sx * ky);
            out[((size_t)2 * io.nd + id) * ne + q] += gy - ref * (kx * sy);
          }
        }
      }
    }
    __syncwarp();
  }
}

// Warps of a CTA: W2D, or as many as their buffers leave room for.
int warps2d(int tabs, int buf) {
  return std::min(W2D, (int)((MAXSMEM / sizeof(double) - tabs) / buf));
}

// Calls f(GT, MT) for the tile counts of a grid of G cells and modes 0 .. K.
template <class F>
void tiles2d(int G, int K, F&& f) {
  const int gt = ceil_div(G, 8), mt = ceil_div(K + 1, 8);
  auto m = [&](auto gtc) {
    if (mt <= 2) f(gtc, std::integral_constant<int, 2>{});
    else if (mt == 3) f(gtc, std::integral_constant<int, 3>{});
    else f(gtc, std::integral_constant<int, 4>{});
  };
  if (gt <= 4) m(std::integral_constant<int, 4>{});
  else if (gt == 5) m(std::integral_constant<int, 5>{});
  else if (gt == 6) m(std::integral_constant<int, 6>{});
  else m(std::integral_constant<int, 7>{});
}

}  // namespace

bool small2d64_takes(int w, int K, int G, bool wrap) {
  return !wrap && w >= 6 && w <= 16 && w % 2 == 0 && K <= 31 && G <= 56;
}

void form2d64_launch(int w, const void* av, const Form64& io, const int* first, int* next,
                     cudaStream_t s) {
  const PWArgs<double>& a = *static_cast<const PWArgs<double>*>(av);
  Es64 es;
  es_polys(w, a, es);
  tiles2d(a.g.G, a.g.K, [&](auto gtc, auto mtc) {
    constexpr int GT = decltype(gtc)::value, MT = decltype(mtc)::value;
    const int nw = warps2d(tabs_form(MT, ceil_div(a.g.G, 4)), Lay2D(GT, MT).buf);
    const size_t sm = sizeof(double) * (tabs_form(MT, ceil_div(a.g.G, 4)) + (size_t)nw * Lay2D(GT, MT).buf);
    auto go = [&](auto kern) {
      set_smem(kern, sm);
      kern<<<kSMs, 32 * nw, sm, s>>>(a, es, io, first, next);
      FGT_LAUNCH_CHECK();
    };
    switch (w) {
      case 6: return go(k_form2d64<6, GT, MT>);
      case 8: return go(k_form2d64<8, GT, MT>);
      case 10: return go(k_form2d64<10, GT, MT>);
      case 12: return go(k_form2d64<12, GT, MT>);
      case 14: return go(k_form2d64<14, GT, MT>);
      default: return go(k_form2d64<16, GT, MT>);
    }
  });
}
void eval2d64_launch(int w, bool deriv, const void* av, const Eval64& io, const int* first,
                     int* next, cudaStream_t s) {
  const PWArgs<double>& a = *static_cast<const PWArgs<double>*>(av);
  Es64 es;
  es_polys(w, a, es);
  tiles2d(a.g.G, a.g.K, [&](auto gtc, auto mtc) {
    constexpr int GT = decltype(gtc)::value, MT = decltype(mtc)::value;
    const int nw = warps2d(tabs_eval(GT, a.g.K), Lay2D(GT, MT).buf);
    const size_t sm = sizeof(double) * (tabs_eval(GT, a.g.K) + (size_t)nw * Lay2D(GT, MT).buf);
    auto go = [&](auto kern) {
      set_smem(kern, sm);
      kern<<<kSMs, 32 * nw, sm, s>>>(a, es, io, first, next);
      FGT_LAUNCH_CHECK();
    };
    if (!deriv) {
      switch (w) {
        case 6: return go(k_eval2d64<6, false, GT, MT>);
        case 8: return go(k_eval2d64<8, false, GT, MT>);
        case 10: return go(k_eval2d64<10, false, GT, MT>);
        case 12: return go(k_eval2d64<12, false, GT, MT>);
        case 14: return go(k_eval2d64<14, false, GT, MT>);
        default: return go(k_eval2d64<16, false, GT, MT>);
      }
    }
    switch (w) {
      case 8: return go(k_eval2d64<8, true, GT, MT>);
      case 10: return go(k_eval2d64<10, true, GT, MT>);
      case 12: return go(k_eval2d64<12, true, GT, MT>);
      case 14: return go(k_eval2d64<14, true, GT, MT>);
      case 16: return go(k_eval2d64<16, true, GT, MT>);
      default: FGT_REQUIRE(false, FGT_ERR_UNSUPPORTED, "no evaluation kernel for this width");
    }
  });
}

}  // namespace fgt
