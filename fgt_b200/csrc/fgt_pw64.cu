// FP64 3D plane-wave form and evaluation on the FP64 matrix instructions
// (mma m8n8k4: 37 TFLOP/s measured, the rate of the FP64 FMA pipe, at one
// operand load per 256 FMAs instead of one per FMA).  Spreading, line
// transforms and interpolation are products of small matrices over blocks of
// points or lines:
//   spread       G[x][y,z] += sum_p (q wx wy)[y][p] wz[p][z], per x
//   transforms   out[+-k][c] = sum_l e^{-+ikl} in[l][c]; cos and sin sums are
//                kept apart, so +k and -k come from one pair of sums
//   interpolate  S[y][p] = sum_z G[x][y][z] wz[z][p], then over y and x
// Every box has its grid in global memory; a form is spread -> (z, y) per
// slab of x-planes -> x, an evaluation x, y, z per slab -> interpolate.
//
// FP64 pipe 42-64% busy (1e6 points on a sphere, eps = 1e-9), the rest waits
// for operands at one or two CTAs per SM.  Against W^3 atomics per point into a global grid,
// SIMT line transforms on one CTA per box and one stencil load per FMA
// (N = M = 4e6 on a sphere, pot + grad, delta = 1e-4, eps = 1e-9): form 39.6
// -> 3.9 ms, evaluation 37.2 -> 11.2 ms; N = M = 1.5e6, delta = 1e-2, eps =
// 1e-12: 33.7 -> 1.6 and 21.1 -> 5.0 ms.  One fused kernel per direction
// (spreading and transforms of a box in one 256-thread CTA) took 4.9 and
// 15.6 ms: the transforms want the 16 warps of two CTAs to hide their loads,
// the spreading and the interpolation 200+ registers per thread.  Grids that
// fit in shared memory gain too (N = M = 2e6, eps = 1e-6: form 3.2 -> 1.9,
// evaluation 7.8 -> 4.0 ms against a 200 KB grid and a SIMT stencil per CTA;
// N = 1e5, eps = 1e-3: 0.43 -> 0.22 and 0.37 -> 0.17).
#include <limits.h>
#include <stdlib.h>

#include <mutex>

#include "fgt_pw64.cuh"
#include "fgt_pw64_dev.cuh"

namespace fgt {

namespace {

constexpr int T64 = 256;
constexpr int W64 = T64 / 32;
constexpr int NBLK64 = 4096;  // blocks of base cells per box

// Grid of one box: plane x of rows (y or ky) of `rowp` doubles (z, or
// kz as (re, im)); rows start on whole 32-byte sectors.
struct Lay64 {
  int rowp, planep;
  __host__ __device__ Lay64(int G, int K) {
    const int c = G > 2 * (K + 1) ? G : 2 * (K + 1);
    rowp = (c + 3) & ~3;
    planep = rowp * (G > 2 * K + 1 ? G : 2 * K + 1);
  }
  __host__ __device__ size_t grid(int G) const { return (size_t)planep * G; }
};

// Barrier of one pair of warps (ids 1.. ; 0 is __syncthreads).
__device__ __forceinline__ void pair_sync(int pair) {
  asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
}

// ------------------------------------------------------------ point blocks
// Counting sort of a chunk of points by block of base cells and the list of
// its units: up to UP points of one block each, blocks in ascending order.
template <int CH, int UP>
struct Sort64 {
  int cnt[NBLK64];               // per block: count, then first point
  int tmp[CH];                   // rank << 12 | block
  unsigned ustart[NBLK64 + CH / UP];  // start << 7 | points
  unsigned short ublk[NBLK64 + CH / UP];
  unsigned short perm[CH];       // chunk index of every sorted point
  int ws[W64];
  int n_units, next;
};

template <int CH, int UP, class BlockOf>
__device__ void sort64(Sort64<CH, UP>& s, int n, int nblk, BlockOf&& block_of) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int i = t; i < nblk; i += T64) s.cnt[i] = 0;
  __syncthreads();
  for (int i = t; i < n; i += T64) {
    int b = block_of(i);
    if (!FGT_DCHECK(b >= 0 && b < nblk, 601)) b = 0;
    s.tmp[i] = (atomicAdd(&s.cnt[b], 1) << 12) | b;
  }
  __syncthreads();
  // exclusive scan of points (low 16 bits) and units (high 16 bits)
  const int per = (nblk + T64 - 1) / T64, b0 = min(nblk, t * per), b1 = min(nblk, b0 + per);
  int sum = 0;
  for (int b = b0; b < b1; b++) sum += s.cnt[b] + (((s.cnt[b] + UP - 1) / UP) << 16);
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) s.ws[warp] = inc;
  __syncthreads();
  int ex = inc - sum;
#pragma unroll
  for (int w = 0; w < W64; w++) ex += w < warp ? s.ws[w] : 0;
  if (t == T64 - 1) {
    s.n_units = (ex + sum) >> 16;
    s.next = 0;
  }
  for (int b = b0; b < b1; b++) {
    const int c = s.cnt[b], p0 = ex & 0xffff;
    int u = ex >> 16;
    s.cnt[b] = p0;
    for (int k = 0; k < c; k += UP, u++) {
      s.ustart[u] = ((unsigned)(p0 + k) << 7) | (unsigned)min(UP, c - k);
      s.ublk[u] = (unsigned short)b;
    }
    ex += c + (((c + UP - 1) / UP) << 16);
  }
  __syncthreads();
  for (int i = t; i < n; i += T64) {
    const int v = s.tmp[i], pos = s.cnt[v & 4095] + (v >> 12);
    if (FGT_DCHECK(pos >= 0 && pos < n, 602)) s.perm[pos] = (unsigned short)i;
  }
  __syncthreads();
}

// --------------------------------------------------------- line transforms
// Sums over ksn (<= KSM) steps of 4 inputs each for units of eight columns,
// one unit per warp at a time: p = re x e, q = im x o with MT tiles of eight
// outputs.  load(u, ks, e, o) gives the lane's operands, store(u, mt, p, q)
// takes the lane's outputs after every input of the unit has been read, so a
// unit may be transformed in place.  The 16 warps of an SM's two CTAs hide
// the loads of one another.
constexpr int TT64 = 256;  // threads of a transform CTA, two per SM
template <int MT, int KSM, class LD, class ST>
__device__ __forceinline__ void cs_units(int u0, int u1, int ksn, const double* re,
                                         const double* im, LD&& load, ST&& store) {
  const int lane = threadIdx.x & 31;
  for (int u = u0 + (threadIdx.x >> 5); u < u1; u += TT64 / 32) {
    double e[KSM], o[KSM], p[MT][2], q[MT][2];
#pragma unroll
    for (int ks = 0; ks < KSM; ks++) {
      e[ks] = o[ks] = 0.0;
      if (ks < ksn) load(u, ks, e[ks], o[ks]);
    }
#pragma unroll
    for (int m = 0; m < MT; m++) p[m][0] = p[m][1] = q[m][0] = q[m][1] = 0.0;
#pragma unroll
    for (int ks = 0; ks < KSM; ks++) {
      if (ks >= ksn) break;
#pragma unroll
      for (int m = 0; m < MT; m++) {
        dmma(p[m][0], p[m][1], re[(ks * MT + m) * 32 + lane], e[ks]);
        dmma(q[m][0], q[m][1], im[(ks * MT + m) * 32 + lane], o[ks]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < MT; m++) store(u, m, p[m], q[m]);
  }
}
// Eight lines per warp, nin (<= 64) inputs and NT tiles of eight outputs per
// line, in place: row(line) is the start of a line.
template <int NT, class ROW, class ST>
__device__ __forceinline__ void z_lines(int nl, int nin, const double* tab, ROW&& row, ST&& store) {
  const int lane = threadIdx.x & 31, l4 = lane & 3, r8 = lane >> 2, ksn = (nin + 3) / 4;
  for (int g = threadIdx.x >> 5; g < (nl + 7) / 8; g += TT64 / 32) {
    const int line = 8 * g + r8;
    double* b = row(line < nl ? line : 0);
    double in[16], c[NT][2];
#pragma unroll
    for (int ks = 0; ks < 16; ks++) in[ks] = ks < ksn && 4 * ks + l4 < nin ? b[4 * ks + l4] : 0.0;
#pragma unroll
    for (int n = 0; n < NT; n++) c[n][0] = c[n][1] = 0.0;
#pragma unroll
    for (int ks = 0; ks < 16; ks++) {
      if (ks >= ksn) break;
#pragma unroll
      for (int n = 0; n < NT; n++) dmma(c[n][0], c[n][1], in[ks], tab[(ks * NT + n) * 32 + lane]);
    }
    __syncwarp();
    if (line < nl)
#pragma unroll
      for (int n = 0; n < NT; n++) store(b, n, c[n]);
  }
}

// ------------------------------------------------------------------- form
// Tiles of 16^3 cells: whole matrix tiles in y and z, 12^3 / 16^3 of the FMAs
// useful at eps = 1e-9, and one 16^3-cell flush per block instead of W^3
// atomics per point (66 against 1728 where a block holds 62 points).
constexpr int FCH64 = 8192;  // points sorted at a time
constexpr int FUP64 = 64;    // points per unit
constexpr int FPB64 = 16;    // points per batch of kernel rows
constexpr int FRS64 = 20;    // kernel row stride: 4 rows of 4 fall on distinct banks
struct FormSmem64 {
  Sort64<FCH64, FUP64> s;
  alignas(16) double rows[W64 / 2][3][FPB64][FRS64];
  int unit[W64 / 2];
  int item;
};

// One pair of warps takes a unit, 64 points of one block of (17-W)^3 base
// cells whose stencils lie in a tile of 16^3 cells: warp h holds the tile's
// x planes 8h..8h+7 as 8 x (16 x 16) accumulators (64 doubles per lane) and
// the tile is added to the grid once per unit.  z cells sit in the column
// order that gives the four lanes of a row four consecutive cells per store.
template <int W>
__device__ void spread64(const PWArgs<double>& a, const Es64& es, const Lay64& lay, double* B, FormSmem64& sm,
                         const double* __restrict__ off, int ns, const double* __restrict__ sq,
                         const double* __restrict__ sr, int c0, int nbd) {
  constexpr int TB = 17 - W;
  const int G = a.g.G, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pair = warp >> 1, h = warp & 1, t = threadIdx.x & 63;
  double(*R)[FPB64][FRS64] = sm.rows[pair];
  for (;;) {
    if (t == 0) sm.unit[pair] = atomicAdd(&sm.s.next, 1);
    pair_sync(pair);
    const int u = sm.unit[pair];
    if (u >= sm.s.n_units) break;
    const int blk = sm.s.ublk[u], start = (int)(sm.s.ustart[u] >> 7),
              cnt = (int)(sm.s.ustart[u] & 127u);
    const int org[3] = {blk / (nbd * nbd) * TB, blk / nbd % nbd * TB, blk % nbd * TB};
    double acc[8][2][2][2];
#pragma unroll
    for (int x = 0; x < 8; x++)
#pragma unroll
      for (int j = 0; j < 8; j++) acc[x][j >> 2][(j >> 1) & 1][j & 1] = 0.0;
    for (int k0 = 0; k0 < cnt; k0 += FPB64) {
      const int np = min(FPB64, cnt - k0);
      // kernel rows: thread (point, dimension); z cells in column order
      const int p = t & 15, d = t >> 4;
      if (d < 3 && p < ((np + 3) & ~3)) {
        double* row = R[d][p];
        auto col = [&](int pos) { return d == 2 ? (pos & 8) + 2 * (pos & 3) + ((pos >> 2) & 1) : pos; };
        int o = 0;
        if (p < np) {
          const int pt = c0 + sm.s.perm[start + k0 + p];
          double f0;
          o = cell64<W>(a, off[(size_t)d * ns + pt], f0) - (d == 0 ? org[0] : (d == 1 ? org[1] : org[2]));
          const double sc = d == 0 ? (sr ? sq[pt] * sr[pt] : sq[pt]) : 1.0;
          es64_row<W, false>(a, es, f0, [&](int j, double v, double) { row[col((o + j) & 15)] = v * sc; });
        } else {
#pragma unroll
          for (int j = 0; j < W; j++) row[j] = 0.0;
        }
#pragma unroll
        for (int j = W; j < 16; j++) row[p < np ? col((o + j) & 15) : j] = 0.0;
      }
      pair_sync(pair);
      for (int k = 0; k < np; k += 4) {
        const int pk = k + (lane & 3), r = lane >> 2;
        const double y0 = R[1][pk][r], y1 = R[1][pk][8 + r];
        const double z0 = R[2][pk][r], z1 = R[2][pk][8 + r];
        const double2* rx = reinterpret_cast<const double2*>(&R[0][pk][8 * h]);
#pragma unroll
        for (int x2 = 0; x2 < 4; x2++) {
          const double2 wx = rx[x2];
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const double w = i ? wx.y : wx.x, a0 = w * y0, a1 = w * y1;
            double(*c)[2][2] = acc[2 * x2 + i];
            dmma(c[0][0][0], c[0][0][1], a0, z0);
            dmma(c[0][1][0], c[0][1][1], a0, z1);
            dmma(c[1][0][0], c[1][0][1], a1, z0);
            dmma(c[1][1][0], c[1][1][1], a1, z1);
          }
        }
      }
      pair_sync(pair);
    }
    const int y = org[1] + (lane >> 2), z = org[2] + (lane & 3);
    double* col = B + (size_t)(org[0] + 8 * h) * lay.planep + y * lay.rowp + z;
#pragma unroll
    for (int x = 0; x < 8; x++) {
      if (org[0] + 8 * h + x >= G) break;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int yh = j >> 2, dz = 8 * ((j >> 1) & 1) + 4 * (j & 1);
        const double v = acc[x][yh][(j >> 1) & 1][j & 1];
        if (y + 8 * yh < G && z + dz < G && v != 0.0)
          atomicAdd(col + x * lay.planep + 8 * yh * lay.rowp + dz, v);
      }
    }
  }
}

// Spreads component ic (density-major) of the items of boxes [i0, i1) of the
// order into the boxes' zeroed grids.
template <int W>
__global__ void __launch_bounds__(T64, 1)
    k_spread64(const __grid_constant__ PWArgs<double> a, const __grid_constant__ Es64 es,
               const __grid_constant__ Form64 io, int ic, int i0, int i1, int* __restrict__ next,
               double* __restrict__ grids) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FormSmem64& sm = *reinterpret_cast<FormSmem64*>(smem_raw);
  constexpr int TB = 17 - W;
  const int G = a.g.G, nbd = (G - W + TB) / TB, nblk = nbd * nbd * nbd;
  const Lay64 lay(G, a.g.K);
  const WorkItem* items = static_cast<const WorkItem*>(io.items);
  const int first = io.item_off[i0], last = i1 < io.n_form ? io.item_off[i1] : *io.n_items;
  const int id = ic / io.ncomp, comp = ic - id * io.ncomp;
  const bool is_q = io.has_q && comp == 0;
  const double* sq = (is_q ? io.q : io.ds) + (size_t)id * io.ns;
  const double* sr = is_q ? nullptr : io.rn + (size_t)(comp - io.has_q) * io.ns;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) sm.item = first + atomicAdd(next, 1);
    __syncthreads();
    if (sm.item >= last) break;
    const WorkItem it = items[sm.item];
    if (!FGT_DCHECK(it.slot >= 0 && it.slot < io.n_form && it.pslot >= i0 && it.pslot < i1, 603))
      continue;
    const int box = io.form_box[it.slot];
    int p0, p1;
    part_range(io.s_lo[box], io.s_hi[box], it.part, it.nparts, p0, p1);
    if (!FGT_DCHECK(p0 >= 0 && p0 <= p1 && p1 <= io.ns, 604)) continue;
    double* B = grids + (size_t)(it.pslot - i0) * lay.grid(G);
    for (int c0 = p0; c0 < p1; c0 += FCH64) {
      sort64(sm.s, min(FCH64, p1 - c0), nblk, [&](int i) {
        int b = 0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
          double f0;
          b = b * nbd + cell64<W>(a, io.off[(size_t)d * io.ns + c0 + i], f0) / TB;
        }
        return b;
      });
      spread64<W>(a, es, lay, B, sm, io.off, io.ns, sq, sr, c0, nbd);
      __syncthreads();
    }
  }
}

// cos and -sin fragments of the forward transforms; MT tiles of modes 0 .. K
template <int MT>
__device__ void form_tabs64(const PWArgs<double>& a, double* re, double* im) {
  const int K = a.g.K, G = a.g.G, NFp = pad4(2 * K + 1), ksg = (G + 3) / 4;
  for (int i = threadIdx.x; i < MT * ksg * 32; i += TT64) {
    const int ln = i & 31, mt = (i >> 5) % MT, ks = (i >> 5) / MT;
    const int k = 8 * mt + (ln >> 2), l = 4 * ks + (ln & 3);
    const bool ok = k <= K && l < G;
    re[i] = ok ? a.twf[(size_t)l * 2 * NFp + K + k] : 0.0;
    im[i] = ok ? a.twf[(size_t)l * 2 * NFp + NFp + K + k] : 0.0;
  }
}
// z (real -> kz) and y transforms of the planes of one (box, slab), in place.
template <int MT>
__global__ void __launch_bounds__(TT64, 2)
    k_form_zy64(const __grid_constant__ PWArgs<double> a, int nbox, double* __restrict__ grids) {
  extern __shared__ __align__(16) double tabs[];
  const Geo& g = a.g;
  const int K = g.K, NH = K + 1, G = g.G, NHp = pad4(NH), ksg = (G + 3) / 4;
  const int ntz = (2 * NH + 7) / 8, nslab = (G + SLAB64 - 1) / SLAB64;
  const int l4 = threadIdx.x & 3, r8 = (threadIdx.x & 31) >> 2;
  const Lay64 lay(G, K);
  double *re = tabs, *im = re + MT * ksg * 32, *zt = im + MT * ksg * 32;
  form_tabs64<MT>(a, re, im);
  for (int i = threadIdx.x; i < ksg * 2 * MT * 32; i += TT64) {
    const int ln = i & 31, nt = (i >> 5) % (2 * MT), ks = (i >> 5) / (2 * MT);
    const int l = 4 * ks + (ln & 3), c = 8 * nt + (ln >> 2);
    zt[i] = l < G && c < 2 * NH ? a.twh[(size_t)l * 2 * NHp + (c & 1) * NHp + (c >> 1)] : 0.0;
  }
  __syncthreads();
  for (int w = blockIdx.x; w < nbox * nslab; w += gridDim.x) {
    const int x0 = w % nslab * SLAB64, x1 = min(G, x0 + SLAB64);
    double* B = grids + (size_t)(w / nslab) * lay.grid(G) + (size_t)x0 * lay.planep;
    z_lines<2 * MT>(
        (x1 - x0) * G, G, zt,
        [&](int line) { return B + (size_t)(line / G) * lay.planep + line % G * lay.rowp; },
        [&](double* row, int nt, const double* c) {
          if (4 * nt + l4 < NH) reinterpret_cast<double2*>(row)[4 * nt + l4] = make_double2(c[0], c[1]);
        });
    __syncthreads();
    cs_units<MT, 16>(
        0, (x1 - x0) * ntz, ksg, re, im,
        [&](int u, int ks, double& e, double& o) {
          const int x = u / ntz, col = 8 * (u - x * ntz) + r8, l = 4 * ks + l4;
          e = o = l < G && col < 2 * NH ? B[(size_t)x * lay.planep + l * lay.rowp + col] : 0.0;
        },
        [&](int u, int mt, const double* p, const double* q) {
          const int x = u / ntz, kz = 4 * (u - x * ntz) + l4, k = 8 * mt + r8;
          if (kz >= NH || k > K) return;
          double2* row = reinterpret_cast<double2*>(B + (size_t)x * lay.planep) + kz;
          row[(K + k) * (lay.rowp / 2)] = make_double2(p[0] - q[1], p[1] + q[0]);
          if (k > 0) row[(K - k) * (lay.rowp / 2)] = make_double2(p[0] + q[1], p[1] - q[0]);
        });
  }
}
// x transform of eight ky rows of one box into its expansion, with weights
// and deconvolution (as k_form's expansion step).
constexpr int KYG64 = 8;
template <int MT>
__global__ void __launch_bounds__(TT64, 2)
    k_form_x64(const __grid_constant__ PWArgs<double> a, const __grid_constant__ Form64 io, int ic,
               int i0, int nbox, const double* __restrict__ grids) {
  extern __shared__ __align__(16) double tabs[];
  const Geo& g = a.g;
  const int K = g.K, NF = 2 * K + 1, NH = K + 1, G = g.G, nline = NF * NH, ksg = (G + 3) / 4;
  const int ntz = (2 * NH + 7) / 8, ngrp = (NF + KYG64 - 1) / KYG64;
  const int l4 = threadIdx.x & 3, r8 = (threadIdx.x & 31) >> 2;
  const Lay64 lay(G, K);
  const int id = ic / io.ncomp, comp = ic - id * io.ncomp;
  const bool is_q = io.has_q && comp == 0;
  const int dd = comp - io.has_q;
  double *re = tabs, *im = re + MT * ksg * 32;
  form_tabs64<MT>(a, re, im);
  __syncthreads();
  for (int w = blockIdx.x; w < nbox * ngrp; w += gridDim.x) {
    const int ky0 = w % ngrp * KYG64, ky1 = min(NF, ky0 + KYG64), i = w / ngrp;
    const double* B = grids + (size_t)i * lay.grid(G);
    const int fb = (int)io.order[i0 + i];
    if (!FGT_DCHECK(fb >= 0 && fb < io.n_form, 608)) continue;
    double2* mp = reinterpret_cast<double2*>(io.mp + ((size_t)fb * io.nd + id) * 2 * g.nexp);
    cs_units<MT, 16>(
        ky0 * ntz, ky1 * ntz, ksg, re, im,
        [&](int u, int ks, double& e, double& o) {
          const int ky = u / ntz, col = 8 * (u - ky * ntz) + r8, l = 4 * ks + l4;
          e = o = l < G && col < 2 * NH ? __ldg(B + (size_t)l * lay.planep + ky * lay.rowp + col) : 0.0;
        },
        [&](int u, int mt, const double* p, const double* q) {
          const int ky = u / ntz, kz = 4 * (u - ky * ntz) + l4, k = 8 * mt + r8;
          if (kz >= NH || k > K) return;
          const double fyz = a.facf[ky] * a.facf[K + kz];
#pragma unroll
          for (int sg = 1; sg >= -1; sg -= 2) {
            if (sg < 0 && k == 0) continue;
            const int ki[3] = {K + sg * k, ky, K + kz};
            const double f = a.facf[ki[0]] * fyz;
            double vr = (p[0] - sg * q[1]) * f, vi = (p[1] + sg * q[0]) * f;
            if (!is_q) {  // * (-i) ts(k_d) / sqrt(delta0)
              const double cc = a.ts[sel3(ki, dd)] * a.inv_sqd0, tr = vi * cc, ti = -vr * cc;
              vr = tr;
              vi = ti;
            }
            double2* m = mp + (size_t)ki[0] * nline + ky * NH + kz;
            if (comp > 0) {
              const double2 v = *m;
              vr += v.x;
              vi += v.y;
            }
            *m = make_double2(vr, vi);
          }
        });
  }
}

// ------------------------------------------------------------- evaluation
// Block of base cells (TBX, TBY, TBZ) of the interpolation and its tile:
// TX x-planes, 8 MY rows, 4 KZ cells.
template <int W>
struct Tile64;
template <>
struct Tile64<6> { static constexpr int TBX = 3, TBY = 3, TBZ = 3; };
template <>
struct Tile64<8> { static constexpr int TBX = 3, TBY = 1, TBZ = 5; };
template <>
struct Tile64<10> { static constexpr int TBX = 3, TBY = 7, TBZ = 3; };
template <>
struct Tile64<12> { static constexpr int TBX = 3, TBY = 5, TBZ = 5; };
template <>
struct Tile64<14> { static constexpr int TBX = 3, TBY = 3, TBZ = 3; };
template <>
struct Tile64<16> { static constexpr int TBX = 5, TBY = 1, TBZ = 5; };

constexpr int ECH64 = 4096;  // points sorted at a time
constexpr int EUP64 = 16;    // points per unit
template <int W, bool DERIV>
struct EvalSmem64 {
  using TL = Tile64<W>;
  static constexpr int TX = W + TL::TBX - 1, TY = W + TL::TBY - 1, TZ = W + TL::TBZ - 1;
  static constexpr int MY = TY / 8, KZ = TZ / 4, ND = DERIV ? 2 : 1;
  static constexpr int YS = TY == 8 ? 10 : 18, ZS = TZ % 8 == 4 ? TZ : TZ + 4;  // row strides
  static_assert(TY % 8 == 0 && TZ % 4 == 0 && ZS % 8 == 4, "whole matrix tiles");
  struct alignas(16) Rows {  // values (0) and derivatives (1) of a unit's kernel rows
    double x[ND][TX][EUP64];
    double y[ND][EUP64][YS];
    double z[ND][EUP64][ZS];
  };
  Sort64<ECH64, EUP64> s;
  Rows rows[W64];
  // a unit's kernel and derivative sums and its points' cells in the tile
  double ksum[W64][ND == 2 ? EUP64 : 1][3][2];
  int cell[W64][ND == 2 ? EUP64 : 1][3];
  int item;
};

// Powers of ts(k) along each dimension of evaluation component c (i ts per
// derivative, as eval_factor).
__device__ __forceinline__ void comp_powers(int c, int* n) {
  n[0] = n[1] = n[2] = 0;
  if (c == 0) return;
  if (c <= 3) {
    n[c - 1] = 1;
  } else {
    const int m = c - 4, p = m < 3 ? m : (m < 5 ? 0 : 1), q = m < 3 ? m : (m == 3 ? 1 : 2);
    n[p]++;
    n[q]++;
  }
}
__device__ __forceinline__ double ipow(double t, int n) { return n == 0 ? 1.0 : (n == 1 ? t : t * t); }

// cos / sin fragments of the x and y transforms with the deconvolution and
// ts(k)^n; the mode pair +-k enters as L(k) + L(-k) and L(k) - L(-k), the two
// swapped when n is odd.
template <int GT>
__device__ void tabs_xy64(const PWArgs<double>& a, double* re, double* im, int n) {
  const int K = a.g.K, G = a.g.G, Gp = pad4(G), ksk = (K + 4) / 4;
  for (int i = threadIdx.x; i < GT * ksk * 32; i += TT64) {
    const int ln = i & 31, mt = (i >> 5) % GT, ks = (i >> 5) / GT;
    const int l = 8 * mt + (ln >> 2), k = 4 * ks + (ln & 3);
    double r = 0.0, s = 0.0;
    if (l < G && k <= K) {
      const double f = a.faci[K + k] * ipow(a.ts[K + k], n);
      r = a.tif[(size_t)(K + k) * 2 * Gp + l] * f;
      s = a.tif[(size_t)(K + k) * 2 * Gp + Gp + l] * f;
    }
    re[i] = r;
    im[i] = s;
  }
}
// kz -> real fragments, with i^m of the component's m derivatives.
template <int GT>
__device__ void tabs_z64(const PWArgs<double>& a, double* zt, int n, int m) {
  const int K = a.g.K, NH = K + 1, G = a.g.G, Gp = pad4(G), ksz = (2 * NH + 3) / 4;
  const double sc = ipow(a.inv_sqd0, m);
  for (int i = threadIdx.x; i < ksz * GT * 32; i += TT64) {
    const int ln = i & 31, nt = (i >> 5) % GT, ks = (i >> 5) / GT;
    const int c = 4 * ks + (ln & 3), l = 8 * nt + (ln >> 2), kz = c >> 1;
    double v = 0.0;
    if (c < 2 * NH && l < G) {
      const double co = a.tih[(size_t)kz * 2 * Gp + l], si = a.tih[(size_t)kz * 2 * Gp + Gp + l];
      // Re(i^m (Cr + i Ci)(co + i si)) = Cr u + Ci w
      const double u = m == 0 ? co : (m == 1 ? -si : -co), w = m == 0 ? -si : (m == 1 ? -co : si);
      v = ((c & 1) ? w : u) * (a.faci[K + kz] * ipow(a.ts[K + kz], n) * sc);
    }
    zt[i] = v;
  }
}
// The planes of one (box, slab) of component c's grid from the box's
// expansion: x transform into the slab, then y and z in place.
template <int GT>
__global__ void __launch_bounds__(TT64, 2)
    k_planes64(const __grid_constant__ PWArgs<double> a, const __grid_constant__ Eval64 io, int id,
               int c, int i0, int i1, double* __restrict__ grids) {
  extern __shared__ __align__(16) double tabs[];
  const Geo& g = a.g;
  const int K = g.K, NF = 2 * K + 1, NH = K + 1, G = g.G, nline = NF * NH, ksk = (NH + 3) / 4;
  const int ntz = (2 * NH + 7) / 8, nslab = (G + SLAB64 - 1) / SLAB64;
  const int l4 = threadIdx.x & 3, r8 = (threadIdx.x & 31) >> 2;
  const Lay64 lay(G, K);
  double *re = tabs, *im = re + GT * ksk * 32, *zt = im + GT * ksk * 32;
  int n[3];
  comp_powers(c, n);
  tabs_xy64<GT>(a, re, im, n[0]);
  tabs_z64<GT>(a, zt, n[2], n[0] + n[1] + n[2]);
  __syncthreads();
  const int nbox = min(i1, *io.nbox_dev) - i0;
  for (int w = blockIdx.x; w < nbox * nslab; w += gridDim.x) {
    const int x0 = w % nslab * SLAB64, x1 = min(G, x0 + SLAB64), i = w / nslab;
    const int e = io.boxes[i0 + i];
    if (!FGT_DCHECK(e >= 0 && e < io.nbox, 605)) continue;
    const double* L = io.loc + ((size_t)e * io.nd + id) * 2 * g.nexp;
    double* B = grids + (size_t)i * lay.grid(G) + (size_t)x0 * lay.planep;
    if (n[1] != n[0]) {  // x and y tables differ
      __syncthreads();
      tabs_xy64<GT>(a, re, im, n[0]);
      __syncthreads();
    }
    // the slab's two row tiles of the x transform
    const double *rx = re + x0 / 8 * 32, *ix = im + x0 / 8 * 32;
    const bool two = x0 / 8 + 1 < GT;
    for (int u = threadIdx.x >> 5; u < NF * ntz; u += TT64 / 32) {
      const int ky = u / ntz, nt = u - ky * ntz, col = 8 * nt + r8, lane = threadIdx.x & 31;
      double v0[8], v1[8], p[2][2] = {}, q[2][2] = {};
#pragma unroll
      for (int ks = 0; ks < 8; ks++) {
        const int k = 4 * ks + l4;
        v0[ks] = v1[ks] = 0.0;
        if (ks < ksk && k <= K && col < 2 * NH) {
          const double* m = L + 2 * (size_t)(ky * NH) + col;
          v0[ks] = __ldg(m + 2 * (size_t)(K + k) * nline);
          if (k > 0) v1[ks] = __ldg(m + 2 * (size_t)(K - k) * nline);
        }
      }
#pragma unroll
      for (int ks = 0; ks < 8; ks++) {
        if (ks >= ksk) break;
        const double sm = v0[ks] + v1[ks], df = v0[ks] - v1[ks];
        const double ev = (n[0] & 1) ? df : sm, od = (n[0] & 1) ? sm : df;
        dmma(p[0][0], p[0][1], rx[ks * GT * 32 + lane], ev);
        dmma(q[0][0], q[0][1], ix[ks * GT * 32 + lane], od);
        if (two) {
          dmma(p[1][0], p[1][1], rx[(ks * GT + 1) * 32 + lane], ev);
          dmma(q[1][0], q[1][1], ix[(ks * GT + 1) * 32 + lane], od);
        }
      }
      const int kz = 4 * nt + l4;
#pragma unroll
      for (int m = 0; m < 2; m++) {
        const int xl = 8 * m + r8;
        if (x0 + xl < x1 && kz < NH)
          reinterpret_cast<double2*>(B + (size_t)xl * lay.planep + ky * lay.rowp)[kz] =
              make_double2(p[m][0] - q[m][1], p[m][1] + q[m][0]);
      }
    }
    __syncthreads();
    if (n[1] != n[0]) {
      tabs_xy64<GT>(a, re, im, n[1]);
      __syncthreads();
    }
    cs_units<GT, 8>(
        0, (x1 - x0) * ntz, ksk, re, im,
        [&](int u, int ks, double& e, double& o) {
          const int xl = u / ntz, col = 8 * (u - xl * ntz) + r8, k = 4 * ks + l4;
          if (k > K || col >= 2 * NH) return;
          const double* b = B + (size_t)xl * lay.planep + col;
          const double v0 = b[(K + k) * lay.rowp], v1 = k > 0 ? b[(K - k) * lay.rowp] : 0.0;
          e = (n[1] & 1) ? v0 - v1 : v0 + v1;
          o = (n[1] & 1) ? v0 + v1 : v0 - v1;
        },
        [&](int u, int mt, const double* p, const double* q) {
          const int xl = u / ntz, kz = 4 * (u - xl * ntz) + l4, y = 8 * mt + r8;
          if (y < G && kz < NH)
            reinterpret_cast<double2*>(B + (size_t)xl * lay.planep + y * lay.rowp)[kz] =
                make_double2(p[0] - q[1], p[1] + q[0]);
        });
    __syncthreads();
    z_lines<GT>(
        (x1 - x0) * G, 2 * NH, zt,
        [&](int line) { return B + (size_t)(line / G) * lay.planep + line % G * lay.rowp; },
        [&](double* row, int nt, const double* v) {
          if (8 * nt + 2 * l4 < G) reinterpret_cast<double2*>(row)[4 * nt + l4] = make_double2(v[0], v[1]);
        });
  }
}

// Interpolation of one unit (8 NT points at most) by one warp.  Per x plane
// of the tile: S = G wz and G dwz as matrix products (rows y, columns points),
// summed over the lane's rows y with wy, dwy and over x with wx, dwx.
template <int W, bool DERIV, int NT>
__device__ __forceinline__ void interp64(const Lay64& lay, const double* B, int G,
                                         const typename EvalSmem64<W, DERIV>::Rows& R,
                                         const int* org, double (*v)[2][4]) {
  using SM = EvalSmem64<W, DERIV>;
  constexpr int MY = SM::MY, KZ = SM::KZ, ND = SM::ND, TX = SM::TX;
  const int lane = threadIdx.x & 31, l4 = lane & 3, r8 = lane >> 2;
  double bz[NT][ND][KZ], wy[NT][2][ND][MY];
#pragma unroll
  for (int nt = 0; nt < NT; nt++)
#pragma unroll
    for (int d = 0; d < ND; d++) {
#pragma unroll
      for (int ks = 0; ks < KZ; ks++) bz[nt][d][ks] = R.z[d][8 * nt + r8][4 * ks + l4];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int m = 0; m < MY; m++) wy[nt][i][d][m] = R.y[d][8 * nt + 2 * l4 + i][8 * m + r8];
    }
  // cells past the grid carry zero weights: read the last one instead
  int oy[MY], oz[KZ];
#pragma unroll
  for (int m = 0; m < MY; m++) oy[m] = min(org[1] + 8 * m + r8, G - 1) * lay.rowp;
#pragma unroll
  for (int ks = 0; ks < KZ; ks++) oz[ks] = min(org[2] + 4 * ks + l4, G - 1);
  const int xmax = G - 1 - org[0];
  const double* P = B + (size_t)org[0] * lay.planep;
#pragma unroll
  for (int nt = 0; nt < NT; nt++)
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int k = 0; k < 4; k++) v[nt][i][k] = 0.0;
  double nx[MY][KZ];  // the next plane's cells, in flight
#pragma unroll
  for (int m = 0; m < MY; m++)
#pragma unroll
    for (int ks = 0; ks < KZ; ks++) nx[m][ks] = P[oy[m] + oz[ks]];
#pragma unroll 1
  for (int x = 0; x < TX; x++) {
    double cell[MY][KZ];
    const double* Pn = P + (size_t)min(x + 1, xmax) * lay.planep;
#pragma unroll
    for (int m = 0; m < MY; m++)
#pragma unroll
      for (int ks = 0; ks < KZ; ks++) {
        cell[m][ks] = nx[m][ks];
        nx[m][ks] = Pn[oy[m] + oz[ks]];
      }
    double t[NT][2][3];
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int i = 0; i < 2; i++) t[nt][i][0] = t[nt][i][1] = t[nt][i][2] = 0.0;
#pragma unroll
    for (int m = 0; m < MY; m++) {
      double s[NT][ND][2];
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int d = 0; d < ND; d++) s[nt][d][0] = s[nt][d][1] = 0.0;
#pragma unroll
      for (int ks = 0; ks < KZ; ks++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int d = 0; d < ND; d++)
            dmma(s[nt][d][0], s[nt][d][1], cell[m][ks], bz[nt][d][ks]);
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          t[nt][i][0] += wy[nt][i][0][m] * s[nt][0][i];
          if constexpr (DERIV) {
            t[nt][i][1] += wy[nt][i][1][m] * s[nt][0][i];
            t[nt][i][2] += wy[nt][i][0][m] * s[nt][1][i];
          }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      const double2 px = *reinterpret_cast<const double2*>(&R.x[0][x][8 * nt + 2 * l4]);
      double2 dx = px;
      if constexpr (DERIV) dx = *reinterpret_cast<const double2*>(&R.x[1][x][8 * nt + 2 * l4]);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const double wx = i ? px.y : px.x, dwx = i ? dx.y : dx.x;
        v[nt][i][0] += wx * t[nt][i][0];
        if constexpr (DERIV) {
          v[nt][i][1] += dwx * t[nt][i][0];
          v[nt][i][2] += wx * t[nt][i][1];
          v[nt][i][3] += wx * t[nt][i][2];
        }
      }
    }
  }
  // over the eight row lanes
#pragma unroll
  for (int o = 4; o < 32; o <<= 1)
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int k = 0; k < (DERIV ? 4 : 1); k++)
          v[nt][i][k] += __shfl_xor_sync(0xffffffffu, v[nt][i][k], o);
}

// Interpolates the items of boxes [i0, i1) of the order from the boxes'
// grids: density id, component c (0 and, with DERIV, the gradient).
template <int W, bool DERIV>
__global__ void __launch_bounds__(T64, 1)
    k_eval64(const __grid_constant__ PWArgs<double> a, const __grid_constant__ Es64 es,
             const __grid_constant__ Eval64 p, int id, int c, int i0, int i1,
             int* __restrict__ next, const double* __restrict__ grids) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using SM = EvalSmem64<W, DERIV>;
  using TL = Tile64<W>;
  SM& sm = *reinterpret_cast<SM*>(smem_raw);
  const int G = a.g.G, nb = G - W + 1;
  const int nbx = (nb + TL::TBX - 1) / TL::TBX, nby = (nb + TL::TBY - 1) / TL::TBY,
            nbz = (nb + TL::TBZ - 1) / TL::TBZ;
  const Lay64 lay(G, a.g.K);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const WorkItem* items = static_cast<const WorkItem*>(p.items);
  const int nbig = *p.nbox_dev;
  if (i0 >= nbig) return;
  const int first = p.item_off[i0], last = i1 < nbig ? p.item_off[i1] : *p.n_items;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) sm.item = first + atomicAdd(next, 1);
    __syncthreads();
    if (sm.item >= last) break;
    const WorkItem it = items[sm.item];
    const int e = it.slot;
    if (!FGT_DCHECK(e >= 0 && e < p.nbox && it.pslot >= i0 && it.pslot < i1, 609)) continue;
    const int box = p.eval_box[e];
    const double* B = grids + (size_t)(it.pslot - i0) * lay.grid(G);
    // the item's points: its share of both sets, sources first
    int q0[2], m[2];
#pragma unroll
    for (int set = 0; set < 2; set++) {
      q0[set] = m[set] = 0;
      if (c >= p.ncomp[set] || p.n[set] == 0) continue;
      int q1;
      part_range(p.lo[set][box], p.hi[set][box], it.part, it.nparts, q0[set], q1);
      if (FGT_DCHECK(q0[set] >= 0 && q0[set] <= q1 && q1 <= p.n[set], 606)) m[set] = q1 - q0[set];
    }
    const int np = m[0] + m[1];
    for (int c0 = 0; c0 < np; c0 += ECH64) {
      sort64(sm.s, min(ECH64, np - c0), nbx * nby * nbz, [&](int i) {
        const int set = c0 + i >= m[0] ? 1 : 0;
        const int pt = set ? q0[1] + c0 + i - m[0] : q0[0] + c0 + i;
        const double* off = set ? p.off[1] : p.off[0];
        const int ne = set ? p.n[1] : p.n[0];
        double f0;
        const int bx = cell64<W>(a, off[pt], f0) / TL::TBX;
        const int by = cell64<W>(a, off[(size_t)ne + pt], f0) / TL::TBY;
        const int bz = cell64<W>(a, off[2 * (size_t)ne + pt], f0) / TL::TBZ;
        return (bx * nby + by) * nbz + bz;
      });
      for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(&sm.s.next, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= sm.s.n_units) break;
        const int blk = sm.s.ublk[u], start = (int)(sm.s.ustart[u] >> 7),
                cnt = (int)(sm.s.ustart[u] & 127u);
      const int org[3] = {blk / (nby * nbz) * TL::TBX, blk / nbz % nby * TL::TBY,
                          blk % nbz * TL::TBZ};
      typename SM::Rows& R = sm.rows[warp];
      // kernel rows (point, dimension), one per lane at a time
      const int npad = cnt <= 8 ? 8 : 16;
      for (int r = lane; r < 3 * npad; r += 32) {
        const int d = r / npad, pi = r - d * npad;
        const int TD = d == 0 ? SM::TX : (d == 1 ? SM::TY : SM::TZ);
        double* w = d == 0 ? &R.x[0][0][pi] : (d == 1 ? &R.y[0][pi][0] : &R.z[0][pi][0]);
        const int st = d == 0 ? EUP64 : 1;
        const int dv = d == 0 ? SM::TX * EUP64 : (d == 1 ? EUP64 * SM::YS : EUP64 * SM::ZS);
        int o = 0;
        if (pi < cnt) {
          const int i = c0 + sm.s.perm[start + pi];
          const int set = i >= m[0] ? 1 : 0, pt = set ? q0[1] + i - m[0] : q0[0] + i;
          const double* off = (set ? p.off[1] : p.off[0]) + (size_t)d * (set ? p.n[1] : p.n[0]);
          double f0;
          o = cell64<W>(a, off[pt], f0) - (d == 0 ? org[0] : (d == 1 ? org[1] : org[2]));
          if (!FGT_DCHECK(o >= 0 && o + W <= TD, 607)) o = 0;
          double ks = 0.0, kd = 0.0;
          es64_row<W, DERIV>(a, es, f0, [&](int j, double f, double df) {
            w[(o + j) * st] = f;
            if constexpr (DERIV) {
              w[dv + (o + j) * st] = df;
              ks += f;
              kd += df;
            }
          });
          if constexpr (DERIV) {
            sm.ksum[warp][pi][d][0] = ks;
            sm.ksum[warp][pi][d][1] = kd;
            sm.cell[warp][pi][d] = o;
          }
        }
        // zero outside the stencil, and rows of no point
        for (int k = pi < cnt ? W : 0; k < TD; k++) {
          const int pos = o + k < TD ? o + k : o + k - TD;
          w[pos * st] = 0.0;
          if constexpr (DERIV) w[dv + pos * st] = 0.0;
        }
      }
      __syncwarp();
      double v[2][2][4];
      const int nt_n = cnt <= 8 ? 1 : 2;
      if (nt_n == 1) interp64<W, DERIV, 1>(lay, B, G, R, org, v);
      else interp64<W, DERIV, 2>(lay, B, G, R, org, v);
      __syncwarp();
      // lane row k writes component k of its two columns
      const int k = lane >> 2;
      if (k < (DERIV ? 4 : 1)) {
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
          if (nt >= nt_n) break;
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int pj = 8 * nt + 2 * (lane & 3) + i;
            if (pj >= cnt) continue;
            const int ii = c0 + sm.s.perm[start + pj];
            const int st = ii >= m[0] ? 1 : 0;
            const int q = st ? q0[1] + ii - m[0] : q0[0] + ii;
            const int comp = DERIV ? k : c;
            if (comp >= (st ? p.ncomp[1] : p.ncomp[0])) continue;
            double r = k == 0 ? v[nt][i][0]
                              : (k == 1 ? v[nt][i][1] : (k == 2 ? v[nt][i][2] : v[nt][i][3]));
            if constexpr (DERIV) {
              if (p.drop_ref && k > 0) {
                const auto& S = sm.ksum[warp][pj];
                const int* o = sm.cell[warp][pj];
                const int x = org[0] + o[0] + W / 2, y = org[1] + o[1] + W / 2,
                          z = org[2] + o[2] + W / 2;
                if (FGT_DCHECK(x >= 0 && x < G && y >= 0 && y < G && z >= 0 && z < G, 612))
                  r -= B[(size_t)x * lay.planep + y * lay.rowp + z] *
                       (S[0][k == 1] * S[1][k == 2] * S[2][k == 3]);
              }
            }
            double* out = st ? p.out[1] : p.out[0];
            atomicAdd(out + ((size_t)comp * p.nd + id) * (st ? p.n[1] : p.n[0]) + q, r);
          }
        }
      }
      // the next unit's kernel sums and cells take the place of those just read:
      // the shuffle that hands out the unit orders no memory
      __syncwarp();
      }
      __syncthreads();
    }
  }
}

// -------------------------------------------------------- few points a box
// Direct modal sums (k_eval_modal's) of boxes with at most pmax points,
// potential or potential + gradient, one CTA per box: per row (kx, ky) the
// sums over kz of eight points are one matrix product of the stored
// expansion, A[row][kz, part], with the points' phases, B[kz, part][point,
// (re, im)]; the gradient's ts(kz)-weighted sums are a second one.  Rows go
// round the warps.  KS: steps of four (kz, part), 2K+2 <= 4 KS.  36,000
// points in 2,672 boxes (K = 20): 7.2 ms by SIMT sums, 1.6 ms here.
template <int KS, bool GRAD>
__global__ void __launch_bounds__(T64, 1)
    k_modal64(const __grid_constant__ PWArgs<double> a, const __grid_constant__ Eval64 io, int pmax) {
  constexpr int NC = GRAD ? 4 : 1, ND = GRAD ? 2 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Geo& g = a.g;
  const int K = g.K, NF = 2 * K + 1, NH = K + 1, nrows = NF * NF;
  double2* E = reinterpret_cast<double2*>(smem_raw);  // [3][NF][pmax] (cos, sin)(k x_d)
  double* ts = reinterpret_cast<double*>(E + (size_t)3 * NF * pmax);  // [NF]
  double* red = ts + NF;                                              // [W64][8][NC]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l4 = lane & 3, r8 = lane >> 2;
  for (int k = threadIdx.x; k < NF; k += T64) ts[k] = a.ts[k];
  const int nbox = *io.nbox_dev;
  for (int bi = blockIdx.x; bi < nbox; bi += gridDim.x) {
    const int e = io.boxes[bi];
    if (!FGT_DCHECK(e >= 0 && e < io.nbox, 610)) continue;
    const int box = io.eval_box[e];
    const int n0 = io.n[0] > 0 && io.ncomp[0] > 0 ? io.hi[0][box] - io.lo[0][box] : 0;
    const int n1 = io.n[1] > 0 && io.ncomp[1] > 0 ? io.hi[1][box] - io.lo[1][box] : 0;
    const int np = n0 + n1;
    if (!FGT_DCHECK(np <= pmax, 611)) continue;
    __syncthreads();
    for (int i = threadIdx.x; i < np * 3 * NF; i += T64) {
      const int r = i / np, pi = i - r * np, d = r / NF, k = r - d * NF - K;
      const int set = pi < n0 ? 0 : 1;
      const int pt = set ? io.lo[1][box] + pi - n0 : io.lo[0][box] + pi;
      const double x = (set ? io.off[1] : io.off[0])[(size_t)d * (set ? io.n[1] : io.n[0]) + pt] * a.scale_d;
      double sn, cs;
      sincos(x * (double)k, &sn, &cs);
      E[(size_t)r * pmax + pi] = make_double2(cs, sn);
    }
    __syncthreads();
    for (int id = 0; id < io.nd; id++) {
      const double* L = io.loc + ((size_t)e * io.nd + id) * 2 * g.nexp;
      for (int p0 = 0; p0 < np; p0 += 8) {
        // phases: column r8 is (re, im)[r8 & 1] of point r8 / 2
        double b[2][ND][KS], v[2][NC];
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
          const int p = p0 + 4 * nt + (r8 >> 1);
#pragma unroll
          for (int ks = 0; ks < KS; ks++) {
            const int kz = 2 * ks + (l4 >> 1);
            double x = 0.0, t = 0.0;
            if (p < np && kz < NH) {
              const double2 z = E[(size_t)(2 * NF + K + kz) * pmax + p];
              const bool im = r8 & 1, part = l4 & 1;
              x = (kz ? 2.0 : 1.0) * (im == part ? z.x : (part ? -z.y : z.y));
              t = ts[K + kz];
            }
            b[nt][0][ks] = x;
            if constexpr (GRAD) b[nt][1][ks] = x * t;
          }
#pragma unroll
          for (int c = 0; c < NC; c++) v[nt][c] = 0.0;
        }
        const int nt_n = np - p0 > 4 ? 2 : 1;
        double in[KS];
        auto fetch = [&](int mt) {
          const int row = 8 * mt + r8;
          const double* m = L + 2 * (size_t)row * NH + l4;
#pragma unroll
          for (int ks = 0; ks < KS; ks++)
            in[ks] = row < nrows && 4 * ks + l4 < 2 * NH ? __ldg(m + 4 * ks) : 0.0;
        };
        const int nmt = (nrows + 7) / 8;
        if (warp < nmt) fetch(warp);
        for (int mt = warp; mt < nmt; mt += W64) {
          double s[2][ND][2] = {};
#pragma unroll
          for (int ks = 0; ks < KS; ks++)
#pragma unroll
            for (int d = 0; d < ND; d++) dmma(s[0][d][0], s[0][d][1], in[ks], b[0][d][ks]);
          if (nt_n > 1)
#pragma unroll
            for (int ks = 0; ks < KS; ks++)
#pragma unroll
              for (int d = 0; d < ND; d++) dmma(s[1][d][0], s[1][d][1], in[ks], b[1][d][ks]);
          if (mt + W64 < nmt) fetch(mt + W64);
          const int row = 8 * mt + r8;
          if (row < nrows) {
            const int kx = row / NF, ky = row - kx * NF;
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {
              const int p = p0 + 4 * nt + l4;
              if (p >= np) continue;
              const double2 ex = E[(size_t)kx * pmax + p], ey = E[(size_t)(NF + ky) * pmax + p];
              const double pr = ex.x * ey.x - ex.y * ey.y, pi = ex.x * ey.y + ex.y * ey.x;
              v[nt][0] += pr * s[nt][0][0] - pi * s[nt][0][1];
              if constexpr (GRAD) {
                const double ti = pr * s[nt][0][1] + pi * s[nt][0][0];
                v[nt][1] -= ts[kx] * ti;
                v[nt][2] -= ts[ky] * ti;
                v[nt][3] -= pr * s[nt][1][1] + pi * s[nt][1][0];
              }
            }
          }
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1)
#pragma unroll
          for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int c = 0; c < NC; c++) v[nt][c] += __shfl_xor_sync(0xffffffffu, v[nt][c], o);
        if (r8 == 0)
#pragma unroll
          for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int c = 0; c < NC; c++) red[(warp * 8 + 4 * nt + l4) * NC + c] = v[nt][c];
        __syncthreads();
        const int q = threadIdx.x / NC, c = threadIdx.x - q * NC, pj = p0 + q;
        if (q < 8 && pj < np) {
          double r = 0.0;
#pragma unroll
          for (int w = 0; w < W64; w++) r += red[(w * 8 + q) * NC + c];
          const int set = pj < n0 ? 0 : 1;
          if (c < (set ? io.ncomp[1] : io.ncomp[0])) {
            const int pt = set ? io.lo[1][box] + pj - n0 : io.lo[0][box] + pj;
            double* out = (set ? io.out[1] : io.out[0]) +
                          ((size_t)c * io.nd + id) * (set ? io.n[1] : io.n[0]) + pt;
            *out += c == 0 ? r : r * a.inv_sqd0;
          }
        }
        __syncthreads();
      }
    }
  }
}

}  // namespace

bool form64_takes(int w, int K, int G, bool wrap) {
  if (wrap || w < 6 || w > 14 || (w & 1) || K > 31 || G > 64) return false;
  const int tb = 17 - w, nbd = (G - w + tb) / tb;
  return nbd * nbd * nbd <= NBLK64;
}
template <int W>
static bool eval_blocks_fit(int G) {
  using TL = Tile64<W>;
  const int nb = G - W + 1;
  return (long)ceil_div(nb, TL::TBX) * ceil_div(nb, TL::TBY) * ceil_div(nb, TL::TBZ) <= NBLK64;
}
bool eval64_takes(int w, int K, int G, bool wrap) {
  if (wrap || K > 31 || G > 64) return false;
  switch (w) {
    case 6: return eval_blocks_fit<6>(G);
    case 8: return eval_blocks_fit<8>(G);
    case 10: return eval_blocks_fit<10>(G);
    case 12: return eval_blocks_fit<12>(G);
    case 14: return eval_blocks_fit<14>(G);
    case 16: return eval_blocks_fit<16>(G);
    default: return false;
  }
}

// Boxes whose grids may be held at a time: a 128th of the device's memory
// (1.4 GB, 2,700 boxes at eps = 1e-9) of the thread's workspace, which the
// form and the evaluations of a call use one after the other.  Fewer cost the
// ends of the runs: 2,265 boxes of 64 clusters, N = M = 2e6, evaluation 9.6 ms
// at once, 9.8 in runs of 1,184 and 2,000, 10.1 of 592, 13.6 of 148.
// FGT_GRID64_BOXES (a box count) lowers it, to test the loop over the runs.
static int grids_fit(const Lay64& lay, int G) {
  static std::mutex mu;
  static size_t budget[64] = {0};
  int dev = 0;
  FGT_CUDA(cudaGetDevice(&dev));
  size_t bytes;
  {
    std::lock_guard<std::mutex> lk(mu);
    size_t& b = budget[dev & 63];
    if (b == 0) {
      size_t free_b = 0, total_b = 0;
      FGT_CUDA(cudaMemGetInfo(&free_b, &total_b));
      b = total_b / 128;
    }
    bytes = b;
  }
  size_t held = std::max<size_t>(bytes / (sizeof(double) * lay.grid(G)), 1);
  if (const char* e = getenv("FGT_GRID64_BOXES")) {
    const long v = strtol(e, nullptr, 10);
    if (v > 0) held = std::min<size_t>(held, (size_t)v);
  }
  return (int)std::min<size_t>(held, INT_MAX);
}
// Buffer of the grids of `nbox` boxes in as few runs as fit, all of one
// length; shorter ones where the device has no room.  Returns their length.
static int alloc_grids(DBuf<double>& grids, const Lay64& lay, int G, int nbox, cudaStream_t s) {
  for (int fit = grids_fit(lay, G);; fit = (fit + 1) / 2) {
    const int held = ceil_div(nbox, ceil_div(nbox, fit));
    if (grids.try_alloc((size_t)held * lay.grid(G), s)) return held;
    FGT_REQUIRE(held > 1, FGT_ERR_NOMEM, "device workspace allocation failed");
  }
}
// The workspace a form or an evaluation takes is free again after it (its
// kernels run before any later ones on the stream).
struct ArenaMark {
  Arena* a = thread_arena();
  std::vector<size_t> m = a->mark();
  ~ArenaMark() { a->rewind(m); }
};

template <int W>
static void launch_form64(const PWArgs<double>& a, const Form64& io, cudaStream_t s) {
  const int G = a.g.G, K = a.g.K, NF = 2 * K + 1, ksg = (G + 3) / 4;
  if (io.n_form <= 0) return;
  const Lay64 lay(G, K);
  const ArenaMark mark;
  DBuf<double> grids;
  const int held = alloc_grids(grids, lay, G, io.n_form, s);
  const int runs = ceil_div(io.n_form, held) * io.nd * io.ncomp;
  DBuf<int> next;
  next.alloc_zeroed(runs, s);
  Es64 es;
  es_polys(W, a, es);
  set_smem(k_spread64<W>, sizeof(FormSmem64));
  int run = 0;
  for (int ic = 0; ic < io.nd * io.ncomp; ic++)
    for (int i0 = 0; i0 < io.n_form; i0 += held, run++) {
      const int n = std::min(held, io.n_form - i0);
      FGT_CUDA(cudaMemsetAsync(grids.get(), 0, sizeof(double) * n * lay.grid(G), s));
      k_spread64<W><<<kSMs, T64, sizeof(FormSmem64), s>>>(a, es, io, ic, i0, i0 + n,
                                                          next.get() + run, grids);
      FGT_LAUNCH_CHECK();
      auto transforms = [&](auto mtc) {
        constexpr int MT = decltype(mtc)::value;
        const size_t xy = sizeof(double) * 2 * MT * ksg * 32, z = sizeof(double) * 2 * MT * ksg * 32;
        set_smem(k_form_zy64<MT>, xy + z);
        k_form_zy64<MT><<<std::min(2 * kSMs, n * ceil_div(G, SLAB64)), TT64, xy + z, s>>>(a, n, grids);
        FGT_LAUNCH_CHECK();
        set_smem(k_form_x64<MT>, xy);
        k_form_x64<MT><<<std::min(2 * kSMs, n * ceil_div(NF, KYG64)), TT64, xy, s>>>(a, io, ic, i0, n,
                                                                                   grids);
        FGT_LAUNCH_CHECK();
      };
      const int mt = (K + 8) / 8;  // tiles of eight modes 0 .. K
      if (mt <= 2) transforms(std::integral_constant<int, 2>{});
      else if (mt == 3) transforms(std::integral_constant<int, 3>{});
      else transforms(std::integral_constant<int, 4>{});
    }
}
void form64_launch(int w, const void* av, const Form64& io, cudaStream_t s) {
  const PWArgs<double>& a = *static_cast<const PWArgs<double>*>(av);
  switch (w) {
    case 6: return launch_form64<6>(a, io, s);
    case 8: return launch_form64<8>(a, io, s);
    case 10: return launch_form64<10>(a, io, s);
    case 12: return launch_form64<12>(a, io, s);
    case 14: return launch_form64<14>(a, io, s);
    default: FGT_REQUIRE(false, FGT_ERR_UNSUPPORTED, "no FP64 form kernel for this width");
  }
}

template <int W, bool DERIV>
static void launch_eval64(const PWArgs<double>& a, const Eval64& io, cudaStream_t s) {
  const int G = a.g.G, K = a.g.K;
  const Lay64 lay(G, K);
  const ArenaMark mark;
  // the count of boxes with a grid is read back only where the bound asks for
  // several runs (~15 us against the empty ones and the memory)
  int nbox = io.nbox;
  if (nbox > grids_fit(lay, G)) nbox = fetch_int(io.nbox_dev, s);
  if (nbox <= 0) return;
  DBuf<double> grids;
  const int nc = DERIV ? 1 : io.ncomp_max, held = alloc_grids(grids, lay, G, nbox, s);
  const int runs = ceil_div(nbox, held) * io.nd * nc;
  DBuf<int> next;
  next.alloc_zeroed(runs, s);
  const size_t sm = sizeof(EvalSmem64<W, DERIV>);
  static_assert(sizeof(EvalSmem64<W, DERIV>) <= MAXSMEM, "shared memory of a CTA");
  Es64 es;
  es_polys(W, a, es);
  set_smem(k_eval64<W, DERIV>, sm);
  int run = 0;
  for (int id = 0; id < io.nd; id++)
    for (int c = 0; c < nc; c++)
      for (int i0 = 0; i0 < nbox; i0 += held, run++) {
        const int i1 = std::min(nbox, i0 + held);
        auto planes = [&](auto gtc) {
          constexpr int GT = decltype(gtc)::value;
          const size_t tb = sizeof(double) * 32 * GT * (2 * ceil_div(K + 1, 4) + ceil_div(2 * (K + 1), 4));
          set_smem(k_planes64<GT>, tb);
          k_planes64<GT><<<2 * kSMs, TT64, tb, s>>>(a, io, id, c, i0, i1, grids);
          FGT_LAUNCH_CHECK();
        };
        switch (ceil_div(G, 8)) {
          case 5: planes(std::integral_constant<int, 5>{}); break;
          case 6: planes(std::integral_constant<int, 6>{}); break;
          case 7: planes(std::integral_constant<int, 7>{}); break;
          case 8: planes(std::integral_constant<int, 8>{}); break;
          default: planes(std::integral_constant<int, 4>{});
        }
        k_eval64<W, DERIV><<<kSMs, T64, sm, s>>>(a, es, io, id, c, i0, i1, next.get() + run, grids);
        FGT_LAUNCH_CHECK();
      }
}
void eval64_launch(int w, bool deriv, const void* av, const Eval64& io, cudaStream_t s) {
  const PWArgs<double>& a = *static_cast<const PWArgs<double>*>(av);
#define FGT_E64(WW)                                                \
  case WW:                                                         \
    return deriv ? launch_eval64<WW, true>(a, io, s) : launch_eval64<WW, false>(a, io, s);
  switch (w) {
    case 6:
      FGT_REQUIRE(!deriv, FGT_ERR_UNSUPPORTED, "derivative evaluation needs a kernel width >= 7");
      return launch_eval64<6, false>(a, io, s);
    FGT_E64(8) FGT_E64(10) FGT_E64(12) FGT_E64(14) FGT_E64(16)
    default: FGT_REQUIRE(false, FGT_ERR_UNSUPPORTED, "no FP64 evaluation kernel for this width");
  }
#undef FGT_E64
}

bool modal64_launch(const void* av, const Eval64& io, int pmax, size_t smem, cudaStream_t s) {
  const PWArgs<double>& a = *static_cast<const PWArgs<double>*>(av);
  const int ks = ceil_div(2 * (a.g.K + 1), 4);
  if (ks > 16 || io.ncomp_max > 4) return false;
  auto go = [&](auto kern) {
    set_smem(kern, smem);
    kern<<<std::max(1, std::min(io.nbox, kSMs * 4)), T64, smem, s>>>(a, io, pmax);
  };
  const bool grad = io.ncomp_max > 1;
  if (ks <= 8) grad ? go(k_modal64<8, true>) : go(k_modal64<8, false>);
  else if (ks <= 11) grad ? go(k_modal64<11, true>) : go(k_modal64<11, false>);
  else if (ks <= 14) grad ? go(k_modal64<14, true>) : go(k_modal64<14, false>);
  else grad ? go(k_modal64<16, true>) : go(k_modal64<16, false>);
  return true;
}

}  // namespace fgt
