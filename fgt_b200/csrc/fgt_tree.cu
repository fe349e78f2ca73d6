// Device tree build: bounding box, path keys, level-synchronous refinement,
// 2:1 level restriction, box tables, sorted point ranges.
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <type_traits>

#include "fgt_tree.cuh"

namespace fgt {

namespace {

struct KeyParams {
  int dim, D;
  double cen0[FGT_MAXDIM];
  double bsh[64];  // bsh[l] = boxsize(l+1)/2: child-centre offset below level l
};

// Bounding box of both point sets: block partials [block][lo, hi][DIM], the
// last block to finish (ticket, zero at launch) reduces them into out[lo, hi].
template <int DIM>
__global__ void __launch_bounds__(256)
    k_bbox(const double* __restrict__ xs, int ns, const double* __restrict__ xt, int nt,
           double* __restrict__ part, unsigned* __restrict__ ticket, double* __restrict__ out) {
  double lo[DIM], hi[DIM];
#pragma unroll
  for (int k = 0; k < DIM; k++) { lo[k] = INFINITY; hi[k] = -INFINITY; }
  const long long n = (long long)ns + nt;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double* x = i < ns ? xs + (size_t)i * DIM : xt + (size_t)(i - ns) * DIM;
#pragma unroll
    for (int k = 0; k < DIM; k++) {
      lo[k] = fmin(lo[k], x[k]);
      hi[k] = fmax(hi[k], x[k]);
    }
  }
  __shared__ double slo[DIM][8], shi[DIM][8];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto reduce = [&](double* o) {
#pragma unroll
    for (int k = 0; k < DIM; k++) {
      double a = lo[k], b = hi[k];
      for (int q = 16; q; q >>= 1) {
        a = fmin(a, __shfl_xor_sync(0xffffffffu, a, q));
        b = fmax(b, __shfl_xor_sync(0xffffffffu, b, q));
      }
      if (lane == 0) { slo[k][w] = a; shi[k][w] = b; }
    }
    __syncthreads();
    if (threadIdx.x < DIM) {
      const int k = threadIdx.x;
      double a = INFINITY, b = -INFINITY;
      for (int q = 0; q < 8; q++) { a = fmin(a, slo[k][q]); b = fmax(b, shi[k][q]); }
      o[k] = a;
      o[DIM + k] = b;
    }
  };
  reduce(part + (size_t)blockIdx.x * 2 * DIM);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < DIM; k++) { lo[k] = INFINITY; hi[k] = -INFINITY; }
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < DIM; k++) {
      lo[k] = fmin(lo[k], __ldcg(part + (size_t)b * 2 * DIM + k));
      hi[k] = fmax(hi[k], __ldcg(part + (size_t)b * 2 * DIM + DIM + k));
    }
  reduce(out);
}

// Full path key of every point (D levels).  The centre recursion
// c_child = c_parent + sign*boxsize(l+1)/2 and the test x - c >= 0 are those
// of tree_refine_boxes (src/common/tree_routs_nd.f:42-45) and
// find_childbox_ind (src/common/pts_tree_nd.f:733-737), so box membership is
// bit-identical to the reference.
template <int DIM>
__global__ void k_point_keys(const double* __restrict__ x, int n, KeyParams p,
                             uint64_t* __restrict__ keys) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double c[DIM], xi[DIM];
#pragma unroll
    for (int k = 0; k < DIM; k++) { c[k] = p.cen0[k]; xi[k] = x[(size_t)i * DIM + k]; }
    uint64_t key = 0;
    for (int l = 0; l < p.D; l++) {
      int dig = 0;
      const double h = p.bsh[l];
#pragma unroll
      for (int k = 0; k < DIM; k++) {
        bool up = (xi[k] - c[k] >= 0);
        dig |= (up ? 1 : 0) << k;
        c[k] = c[k] + (up ? h : -h);
      }
      key = (key << DIM) | (uint64_t)dig;
    }
    keys[i] = key;
  }
}
void launch_point_keys(int dim, const double* x, int n, const KeyParams& p, uint64_t* keys,
                       cudaStream_t s) {
  if (dim == 1) k_point_keys<1><<<grid_for(n, 256), 256, 0, s>>>(x, n, p, keys);
  else if (dim == 2) k_point_keys<2><<<grid_for(n, 256), 256, 0, s>>>(x, n, p, keys);
  else k_point_keys<3><<<grid_for(n, 256), 256, 0, s>>>(x, n, p, keys);
  FGT_LAUNCH_CHECK();
}
// Source count of each box of level l from the sorted full keys.
__global__ void k_box_counts(const uint64_t* __restrict__ bk, int nb, int shift,
                             const uint64_t* __restrict__ sk, int ns, int* __restrict__ cnt) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) {
    uint64_t lo = bk[i] << shift, hi = (bk[i] + 1) << shift;
    cnt[i] = dev_lower_bound(sk, ns, hi) - dev_lower_bound(sk, ns, lo);
  }
}

__global__ void k_flag_gt(const int* __restrict__ cnt, int n, int ndiv, int* __restrict__ f) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    f[i] = cnt[i] > ndiv ? 1 : 0;
}

__global__ void k_compact_u64(const uint64_t* __restrict__ in, const int* __restrict__ flag,
                              const int* __restrict__ pos, int n, uint64_t* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (flag[i]) out[pos[i]] = in[i];
}

__global__ void k_children(const uint64_t* __restrict__ par, int n, int dim,
                           uint64_t* __restrict__ out) {
  int mc = 1 << dim;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * mc; i += gridDim.x * blockDim.x)
    out[i] = (par[i / mc] << dim) | (uint64_t)(i % mc);
}

__device__ __forceinline__ void key_to_coords(uint64_t key, int l, int dim, uint32_t* c) {
  for (int k = 0; k < dim; k++) c[k] = 0;
  for (int j = 0; j < l; j++) {
    int dig = (int)((key >> (dim * (l - 1 - j))) & ((1u << dim) - 1));
    for (int k = 0; k < dim; k++) c[k] = (c[k] << 1) | ((dig >> k) & 1);
  }
}
__device__ __forceinline__ uint64_t coords_to_key(const uint32_t* c, int l, int dim) {
  uint64_t key = 0;
  for (int j = 0; j < l; j++) {
    int dig = 0;
    for (int k = 0; k < dim; k++) dig |= ((c[k] >> (l - 1 - j)) & 1) << k;
    key = (key << dim) | (uint64_t)dig;
  }
  return key;
}

// Level restriction: every level-(l-1) position whose closure touches a
// non-leaf level-l box must itself be non-leaf (free-space adjacency, as the
// distance tests of pts_tree_fix_lr, src/common/pts_tree_nd.f:783-1035).
// Emits, per non-leaf box, the 2^dim touching level-(l-1) positions (out of
// range positions are replaced by the parent, removed later as duplicates).
__global__ void k_touching_parents(const uint64_t* __restrict__ nl, int n, int l, int dim,
                                   uint64_t* __restrict__ out) {
  int mc = 1 << dim;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * mc; i += gridDim.x * blockDim.x) {
    int b = i / mc, j = i % mc;
    uint32_t c[FGT_MAXDIM], q[FGT_MAXDIM];
    key_to_coords(nl[b], l, dim, c);
    uint32_t lim = 1u << (l - 1);
    for (int k = 0; k < dim; k++) {
      uint32_t m = c[k] >> 1;
      if ((j >> k) & 1) {
        // the other touching position: m-1 if c even, m+1 if c odd
        long long o = (c[k] & 1) ? (long long)m + 1 : (long long)m - 1;
        q[k] = (o >= 0 && o < (long long)lim) ? (uint32_t)o : m;
      } else {
        q[k] = m;
      }
    }
    out[i] = coords_to_key(q, l - 1, dim);
  }
}

__global__ void k_member(const uint64_t* __restrict__ a, int n, const uint64_t* __restrict__ set,
                         int m, int* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = dev_find(set, m, a[i]) >= 0 ? 1 : 0;
}

struct LevelTables {
  const uint64_t* keys[64];
  int n[64];
  int start[65];
};

__global__ void k_box_tables(int nboxes, int nlevels, int dim, LevelTables lt, KeyParams kp,
                             const uint64_t* __restrict__ key, const int* __restrict__ level,
                             const int* __restrict__ nonleaf, int* __restrict__ parent,
                             int* __restrict__ child0, double* __restrict__ center) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nboxes; b += gridDim.x * blockDim.x) {
    int l = level[b];
    uint64_t k = key[b];
    parent[b] = (l == 0) ? -1 : lt.start[l - 1] + dev_find(lt.keys[l - 1], lt.n[l - 1], k >> dim);
    child0[b] = (nonleaf[b] && l < nlevels)
                    ? lt.start[l + 1] + dev_find(lt.keys[l + 1], lt.n[l + 1], k << dim)
                    : -1;
    double c[FGT_MAXDIM];
    for (int d = 0; d < dim; d++) c[d] = kp.cen0[d];
    for (int j = 0; j < l; j++) {
      int dig = (int)((k >> (dim * (l - 1 - j))) & ((1u << dim) - 1));
      for (int d = 0; d < dim; d++) c[d] = c[d] + (((dig >> d) & 1) ? kp.bsh[j] : -kp.bsh[j]);
    }
    for (int d = 0; d < dim; d++) center[(size_t)b * dim + d] = c[d];
  }
}

__global__ void k_leaf_flags(const int* __restrict__ nonleaf, int n, int* __restrict__ f) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    f[i] = nonleaf[i] ? 0 : 1;
}
__global__ void k_leaf_starts(const uint64_t* __restrict__ key, const int* __restrict__ level,
                              const int* __restrict__ f, const int* __restrict__ pos, int n,
                              int dim, int D, uint64_t* __restrict__ ls,
                              uint32_t* __restrict__ lbox) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (f[i]) {
      ls[pos[i]] = key[i] << (dim * (D - level[i]));
      lbox[pos[i]] = (uint32_t)i;
    }
}

// Reference box of every leaf (by leaf ordinal): the leaf itself when it
// lies at or above the cut-off level, else its ancestor at that level.
__global__ void k_leaf_ref(const uint32_t* __restrict__ lbox, int nl, const int* __restrict__ level,
                           const int* __restrict__ parent, int ncutoff, int* __restrict__ lref) {
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < nl; o += gridDim.x * blockDim.x) {
    int b = (int)lbox[o];
    while (level[b] > ncutoff && FGT_DCHECK(parent[b] >= 0, 502)) b = parent[b];
    lref[o] = b;
  }
}
// ref[p] = lref[ordinal of sorted point p]
__global__ void k_point_ref(const uint32_t* __restrict__ ord, int n, const int* __restrict__ lref,
                            int* __restrict__ ref) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    ref[i] = lref[ord[i]];
}

// Leaf ordinal of each point (upper_bound - 1 over sorted leaf start keys);
// doubles as the radix key, the value is the original index.
__global__ void k_point_leaf(const uint64_t* __restrict__ pk, int n,
                             const uint64_t* __restrict__ ls, int nl,
                             uint32_t* __restrict__ ord, uint32_t* __restrict__ idx) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint64_t v = pk[i];
    int lo = 0, hi = nl;  // first start > v
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if (ls[mid] <= v) lo = mid + 1; else hi = mid;
    }
    if (!FGT_DCHECK(lo >= 1, 501)) lo = 1;  // every key lies at or after the first leaf
    ord[i] = (uint32_t)(lo - 1);
    idx[i] = (uint32_t)i;
  }
}

// leaf_lo[o] = first sorted position with ordinal >= o, o = 0..nl
__global__ void k_leaf_point_lo(const uint32_t* __restrict__ ord, int n, int nl,
                                int* __restrict__ lo) {
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o <= nl; o += gridDim.x * blockDim.x) {
    int a = 0, b = n;
    while (a < b) {
      int m = (a + b) >> 1;
      if (ord[m] < (uint32_t)o) a = m + 1; else b = m;
    }
    lo[o] = a;
  }
}

__global__ void k_box_ranges(const uint64_t* __restrict__ key, const int* __restrict__ level,
                             int nboxes, int dim, int D, const uint64_t* __restrict__ ls, int nl,
                             const int* __restrict__ slo, const int* __restrict__ tlo,
                             int* __restrict__ s0, int* __restrict__ s1, int* __restrict__ t0,
                             int* __restrict__ t1) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nboxes; b += gridDim.x * blockDim.x) {
    int sh = dim * (D - level[b]);
    uint64_t lo = key[b] << sh, hi = (key[b] + 1) << sh;
    int a = dev_lower_bound(ls, nl, lo), c = dev_lower_bound(ls, nl, hi);
    s0[b] = slo[a]; s1[b] = slo[c];
    t0[b] = tlo[a]; t1[b] = tlo[c];
  }
}

int bits_for(long long n) {
  int b = 0;
  while ((1ll << b) < n) b++;
  return b;
}

}  // namespace

void tree_setup_scalars(int dim, double delta, double eps, int iperiod, const double* d_src,
                        int ns, const double* d_trg, int nt, int* levcut, double* bs0,
                        double* cen0, cudaStream_t s) {
  if (iperiod != 1) {
    const long long n = (long long)ns + nt;
    const int gb = grid_for(n, 256, 4);
    DBuf<double> part((size_t)(gb + 1) * 2 * dim, s);
    DBuf<unsigned> ticket;
    ticket.alloc_zeroed(1, s);
    double* out = part.get() + (size_t)gb * 2 * dim;
    if (dim == 1) k_bbox<1><<<gb, 256, 0, s>>>(d_src, ns, d_trg, nt, part, ticket, out);
    else if (dim == 2) k_bbox<2><<<gb, 256, 0, s>>>(d_src, ns, d_trg, nt, part, ticket, out);
    else k_bbox<3><<<gb, 256, 0, s>>>(d_src, ns, d_trg, nt, part, ticket, out);
    FGT_LAUNCH_CHECK();
    double h[2 * FGT_MAXDIM];
    fetch_span(reinterpret_cast<const int*>(out), 4 * dim, reinterpret_cast<int*>(h), s);
    double lo[FGT_MAXDIM], hi[FGT_MAXDIM];
    for (int k = 0; k < dim; k++) {
      lo[k] = h[k];
      hi[k] = h[dim + k];
    }
    // pts_tree_nd.f:1390-1398
    *bs0 = hi[0] - lo[0];
    for (int k = 1; k < dim; k++)
      if (hi[k] - lo[k] > *bs0) *bs0 = hi[k] - lo[k];
    for (int k = 0; k < dim; k++) cen0[k] = (lo[k] + hi[k]) / 2;
  }
  // pts_tree_nd.f:1399-1410
  double dc = sqrt(delta * log(1.0 / eps));
  double dl = log(*bs0 / dc) / log(2.0);
  *levcut = (int)dl;
  if (iperiod == 1) return;
  if (*bs0 < dc) return;
  *levcut = *levcut + 1;
  *bs0 = ldexp(1.0, *levcut) * dc;
}

namespace {
// ------------------------------------------------------------- dense tree
// Tree over dense tables of the key space above the finest level: cell c of
// level l is key c, the cells of level l start at lev_off(l) of tables that
// hold all levels 0 .. D-1 one after the other.  A box exists where its
// parent's cell is flagged non-leaf, so the rank R of a flagged cell among
// all flagged cells numbers its children: box 1 + mc R + digit (level-major,
// keys ascending), and every step runs over cells without knowing a level's
// box count on the host.
struct CellLevels {
  int dim, D;
  __host__ __device__ long long cells(int l) const { return 1ll << (dim * l); }
  __host__ __device__ long long off(int l) const {
    return ((1ll << (dim * l)) - 1) / ((1 << dim) - 1);
  }
};

// Keys of sources and targets (one launch) and the source counts of the
// cells of level D-1.  Few cells: counted per block in shared memory first;
// lanes of a warp that hit the same cell add once.
constexpr int HIST_SMEM = 4096;
template <int DIM, bool SMEM>
__global__ void __launch_bounds__(256)
    k_keys_hist(const double* __restrict__ xs, int ns, const double* __restrict__ xt, int nt,
                KeyParams p, uint32_t* __restrict__ ks, uint32_t* __restrict__ kt,
                int* __restrict__ hist, int ncell) {
  __shared__ int sh[SMEM ? HIST_SMEM : 1];
  if (SMEM) {
    for (int i = threadIdx.x; i < ncell; i += blockDim.x) sh[i] = 0;
    __syncthreads();
  }
  const long long n = (long long)ns + nt;
  for (long long i0 = (long long)blockIdx.x * blockDim.x; i0 < n;
       i0 += (long long)gridDim.x * blockDim.x) {
    const long long i = i0 + threadIdx.x;
    uint32_t key = 0;
    const bool src = i < ns;
    if (i < n) {
      const double* x = src ? xs + (size_t)i * DIM : xt + (size_t)(i - ns) * DIM;
      double c[DIM], xi[DIM];
#pragma unroll
      for (int k = 0; k < DIM; k++) {
        c[k] = p.cen0[k];
        xi[k] = x[k];
      }
      for (int l = 0; l < p.D; l++) {
        uint32_t dig = 0;
        const double h = p.bsh[l];
#pragma unroll
        for (int k = 0; k < DIM; k++) {
          const bool up = (xi[k] - c[k] >= 0);
          dig |= (up ? 1u : 0u) << k;
          c[k] = c[k] + (up ? h : -h);
        }
        key = (key << DIM) | dig;
      }
      if (src) ks[i] = key;
      else kt[i - ns] = key;
    }
    const uint32_t cell = src ? key >> DIM : 0xffffffffu;
    const unsigned peers = __match_any_sync(0xffffffffu, cell);
    if (src && (__ffs(peers) - 1) == (int)(threadIdx.x & 31)) {
      if (SMEM) atomicAdd(&sh[cell], __popc(peers));
      else atomicAdd(&hist[cell], __popc(peers));
    }
  }
  if (SMEM) {
    __syncthreads();
    for (int i = threadIdx.x; i < ncell; i += blockDim.x)
      if (sh[i]) atomicAdd(&hist[i], sh[i]);
  }
}

// Counts and non-leaf flags of levels lhi .. lhi-q from the counts of level
// lhi: one block per cell of level lhi-q sums its subtree in shared memory.
constexpr int PYR_CELLS = 4096, PYR_T = 512;
__global__ void __launch_bounds__(PYR_T)
    k_pyramid(CellLevels cl, int lhi, int q, int ndiv, int* __restrict__ cnt,
              unsigned char* __restrict__ flag) {
  __shared__ int sc[PYR_CELLS];
  int n = 1 << (cl.dim * q);
  {
    const long long o = cl.off(lhi) + (long long)blockIdx.x * n;
    int v[PYR_CELLS / PYR_T];
#pragma unroll
    for (int k = 0; k < PYR_CELLS / PYR_T; k++) {
      const int i = threadIdx.x + k * PYR_T;
      v[k] = i < n ? cnt[o + i] : 0;
    }
#pragma unroll
    for (int k = 0; k < PYR_CELLS / PYR_T; k++) {
      const int i = threadIdx.x + k * PYR_T;
      if (i < n) {
        sc[i] = v[k];
        flag[o + i] = v[k] > ndiv ? 1 : 0;
      }
    }
  }
  __syncthreads();
  const int mc = 1 << cl.dim;
  for (int l = lhi - 1; l >= lhi - q; l--) {
    const int m = n >> cl.dim;
    int v[PYR_CELLS / 2 / PYR_T];
#pragma unroll
    for (int k = 0; k < PYR_CELLS / 2 / PYR_T; k++) {
      const int i = threadIdx.x + k * PYR_T;
      int a = 0;
      if (i < m)
        for (int j = 0; j < mc; j++) a += sc[i * mc + j];
      v[k] = a;
    }
    __syncthreads();
    const long long o = cl.off(l) + (long long)blockIdx.x * m;
#pragma unroll
    for (int k = 0; k < PYR_CELLS / 2 / PYR_T; k++) {
      const int i = threadIdx.x + k * PYR_T;
      if (i < m) {
        sc[i] = v[k];
        flag[o + i] = v[k] > ndiv ? 1 : 0;
        if (l == lhi - q) cnt[o + i] = v[k];
      }
    }
    __syncthreads();
    n = m;
  }
}

// Level restriction (k_touching_parents) on the flags: every level-(l-1)
// cell whose closure touches a non-leaf cell of level l becomes non-leaf.
__device__ __forceinline__ void touch_parents(const CellLevels& cl, int l, uint32_t cell,
                                              unsigned char* flag) {
  // coordinate k of a key is its bits k, k + dim, ..: neighbours by adding
  // and subtracting inside that bit field
  const int dim = cl.dim, mc = 1 << dim;
  const uint32_t par = cell >> dim, all = (uint32_t)(cl.cells(l - 1) - 1);
  const uint32_t field = (dim == 1 ? 0xffffffffu : (dim == 2 ? 0x55555555u : 0x49249249u));
  const long long o = cl.off(l - 1);
  uint32_t nb[FGT_MAXDIM];  // the other touching position of the coordinate, or its own
  for (int k = 0; k < dim; k++) {
    const uint32_t m = (field << k) & all, x = par & m;
    if ((cell >> k) & 1u) nb[k] = x == m ? x : (((x | ~m) + (1u << k)) & m);
    else nb[k] = x == 0 ? x : ((x - (1u << k)) & m);
  }
  for (int j = 0; j < mc; j++) {
    uint32_t q = 0;
    for (int k = 0; k < dim; k++) q |= ((j >> k) & 1) ? nb[k] : (par & (field << k) & all);
    flag[o + q] = 1;
  }
}
__global__ void k_restrict(CellLevels cl, int l, unsigned char* __restrict__ flag) {
  const long long n = cl.cells(l), o = cl.off(l);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    if (flag[o + i]) touch_parents(cl, l, (uint32_t)i, flag);
}
// levels lmax .. 2 in one block (few cells)
__global__ void __launch_bounds__(1024)
    k_restrict_rest(CellLevels cl, int lmax, unsigned char* flag) {
  for (int l = lmax; l >= 2; l--) {
    const int n = (int)cl.cells(l);
    const long long o = cl.off(l);
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      if (flag[o + i]) touch_parents(cl, l, (uint32_t)i, flag);
    __syncthreads();
  }
}

// Exclusive scans over cells in two launches: block sums, then every block
// adds the sums before it and writes its cells.  OP gives a cell's value
// (value() from the tables, stored() what the first launch kept of it) and
// takes its exclusive prefix.  CI cells per thread: 4, to have many blocks in
// flight on small tables, 16 where the sums of that many blocks would cost.
constexpr int CS_T = 256;
__device__ __forceinline__ int block_sum(int v, int* ws) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  int r = 0;
#pragma unroll
  for (int w = 0; w < CS_T / 32; w++) r += ws[w];
  __syncthreads();
  return r;
}
template <int CI, class OP>
__global__ void __launch_bounds__(CS_T) k_cells_sum(OP op, long long n, int* __restrict__ part) {
  __shared__ int ws[CS_T / 32];
  const long long b = (long long)blockIdx.x * CS_T * CI + threadIdx.x;
  int v = 0;
#pragma unroll
  for (int j = 0; j < CI; j++)
    if (b + j * CS_T < n) v += op.value(b + j * CS_T);
  v = block_sum(v, ws);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}
template <int CI, class OP>
__global__ void __launch_bounds__(CS_T) k_cells_scan(OP op, long long n, const int* __restrict__ part) {
  __shared__ int ws[CS_T / 32];
  int before = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += CS_T) before += part[i];
  before = block_sum(before, ws);
  const long long b = (long long)blockIdx.x * CS_T * CI + threadIdx.x * CI;
  int v[CI], s = 0;
#pragma unroll
  for (int j = 0; j < CI; j++) {
    v[j] = b + j < n ? op.stored(b + j) : 0;
    s += v[j];
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int inc = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  int ex = before + inc - s;
#pragma unroll
  for (int k = 0; k < CS_T / 32; k++) ex += k < w ? ws[k] : 0;
#pragma unroll
  for (int j = 0; j < CI; j++) {
    if (b + j < n) op.put(b + j, ex, v[j]);
    ex += v[j];
    if (b + j == n - 1) op.total(ex);
  }
}

// Rank of every flagged cell, and the ranks at which the levels start.
struct RankOp {
  CellLevels cl;
  const unsigned char* flag;
  int *rank, *lev;  // lev: D+1 entries, the last is the total
  __device__ int value(long long i) const { return flag[i]; }
  __device__ int stored(long long i) const { return flag[i]; }
  __device__ void put(long long i, int ex, int) const {
    rank[i] = ex;
    // starts of levels: i = (2^(dim l) - 1) / (2^dim - 1)
    const unsigned long long c = (unsigned long long)i * ((1 << cl.dim) - 1) + 1;
    if ((c & (c - 1)) == 0) {
      const int b = 63 - __clzll((long long)c);
      if (b % cl.dim == 0 && b / cl.dim < cl.D) lev[b / cl.dim] = ex;
    }
  }
  __device__ void total(int t) const { lev[cl.D] = t; }
};
// Leaves that start at a cell of level D-1, in key order: the mc children of
// a flagged cell, else one where the cell is the first of its leaf.
struct LeafOp {
  CellLevels cl;
  const unsigned char* flag;
  int* base;        // exclusive leaf count; total at [cells(D-1)]
  uint32_t* table;  // flagged: base | 2^31, else the ordinal of the cell's leaf
  __device__ int value(long long i) const {
    const int L = cl.D - 1;
    // a flag implies those above it: the level of the cell's leaf is the
    // number of flags on its path (independent loads)
    int l = 0;
    for (int k = 0; k < L; k++) l += flag[cl.off(k) + (i >> (cl.dim * (L - k)))];
    const int v = flag[cl.off(L) + i]
                      ? 1 << cl.dim
                      : ((i & ((1ll << (cl.dim * (L - l))) - 1)) == 0 ? 1 : 0);
    base[i] = v;
    return v;
  }
  __device__ int stored(long long i) const { return base[i]; }
  __device__ void put(long long i, int ex, int v) const {
    base[i] = ex;
    table[i] = v > 1 ? ((uint32_t)ex | 0x80000000u) : (uint32_t)(ex + v - 1);
  }
  __device__ void total(int t) const { base[cl.cells(cl.D - 1)] = t; }
};

// Steps 2-4 of a tree whose tables (all levels above the finest) fit in one
// block's shared memory: counts and flags up the levels, restriction down,
// ranks and leaf ordinals, in one launch instead of seven to ten.
// With 37,449 cells (3D, D = 6) one block took 0.2 ms against 0.08 of the
// launches it replaces.
constexpr int TREE_ONE = 5461;  // cells: 3D D <= 5, 2D D <= 7, 1D D <= 12
__global__ void __launch_bounds__(1024, 1)
    k_tree_one(CellLevels cl, int ndiv, const int* __restrict__ hist, unsigned char* __restrict__ gflag,
               int* __restrict__ grank, int* __restrict__ lev, int* __restrict__ base,
               uint32_t* __restrict__ table) {
  extern __shared__ __align__(16) int sc[];  // counts, then ranks
  const int T = (int)cl.off(cl.D), L = cl.D - 1, C1 = (int)cl.cells(L), mc = 1 << cl.dim;
  unsigned char* f = reinterpret_cast<unsigned char*>(sc + T);
  __shared__ int ws[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < C1; i += 1024) {
    const int c = hist[i];
    sc[cl.off(L) + i] = c;
    f[cl.off(L) + i] = c > ndiv ? 1 : 0;
  }
  __syncthreads();
  for (int l = L - 1; l >= 0; l--) {
    const int o = (int)cl.off(l), oc = (int)cl.off(l + 1), n = (int)cl.cells(l);
    for (int i = threadIdx.x; i < n; i += 1024) {
      int a = 0;
      for (int j = 0; j < mc; j++) a += sc[oc + i * mc + j];
      sc[o + i] = a;
      f[o + i] = a > ndiv ? 1 : 0;
    }
    __syncthreads();
  }
  for (int l = L; l >= 2; l--) {
    const int o = (int)cl.off(l), n = (int)cl.cells(l);
    for (int i = threadIdx.x; i < n; i += 1024)
      if (f[o + i]) touch_parents(cl, l, (uint32_t)i, f);
    __syncthreads();
  }
  // exclusive scan of a thread's run sum over the block
  auto scan = [&](int s, int* tot) {
    int inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    __syncthreads();
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    int b = 0, t = 0;
    for (int k = 0; k < 32; k++) {
      b += k < w ? ws[k] : 0;
      t += ws[k];
    }
    *tot = t;
    return b + inc - s;
  };
  {
    const int per = (T + 1023) / 1024, i0 = min(T, (int)threadIdx.x * per), i1 = min(T, i0 + per);
    int s = 0, tot;
    for (int i = i0; i < i1; i++) s += f[i];
    int ex = scan(s, &tot);
    for (int i = i0; i < i1; i++) {
      sc[i] = ex;
      ex += f[i];
    }
    __syncthreads();
    if (threadIdx.x <= cl.D) lev[threadIdx.x] = (int)threadIdx.x < cl.D ? sc[cl.off(threadIdx.x)] : tot;
    for (int i = threadIdx.x; i < T; i += 1024) {
      grank[i] = sc[i];
      gflag[i] = f[i];
    }
  }
  auto leaves = [&](int i) {  // leaves that start at cell i (LeafOp::value)
    int l = 0;
    for (int k = 0; k < L; k++) l += f[cl.off(k) + (i >> (cl.dim * (L - k)))];
    return f[cl.off(L) + i] ? mc : ((i & ((1 << (cl.dim * (L - l))) - 1)) == 0 ? 1 : 0);
  };
  __syncthreads();
  for (int i = threadIdx.x; i < C1; i += 1024) sc[i] = leaves(i);
  __syncthreads();
  const int per = (C1 + 1023) / 1024, i0 = min(C1, (int)threadIdx.x * per), i1 = min(C1, i0 + per);
  int s = 0, tot;
  for (int i = i0; i < i1; i++) s += sc[i];
  int ex = scan(s, &tot);
  for (int i = i0; i < i1; i++) {
    const int v = sc[i];
    sc[i] = ex;
    ex += v;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C1; i += 1024) {
    const int b = sc[i], e = i + 1 < C1 ? sc[i + 1] : tot;
    base[i] = b;
    table[i] = f[cl.off(L) + i] ? ((uint32_t)b | 0x80000000u) : (uint32_t)(e - 1);
  }
  if (threadIdx.x == 0) base[C1] = tot;
}

// Box tables: the children of every flagged cell (and the root); lref: the
// reference box of every leaf by ordinal (itself, or its parent at level D-1,
// the cut-off level).
__global__ void k_dense_boxes(CellLevels cl, KeyParams kp, const unsigned char* __restrict__ flag,
                              const int* __restrict__ rank, const int* __restrict__ base,
                              uint64_t* __restrict__ key, int* __restrict__ level,
                              int* __restrict__ nonleaf, int* __restrict__ parent,
                              int* __restrict__ child0, double* __restrict__ center,
                              int* __restrict__ lref, int nboxes, int nleaves) {
  const int dim = cl.dim, mc = 1 << dim, L = cl.D - 1;
  const long long T = cl.off(cl.D);
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < T * mc + 1;
       g += (long long)gridDim.x * blockDim.x) {
    int b, l, par;
    uint32_t k;
    if (g == T * mc) {  // the root
      b = 0;
      l = 0;
      k = 0;
      par = -1;
    } else {
      const long long i = g / mc;
      const int j = (int)(g - i * mc);
      if (!flag[i]) continue;
      int pl = 0;
      while (pl < L && i >= cl.off(pl + 1)) pl++;
      const uint32_t c = (uint32_t)(i - cl.off(pl));
      b = 1 + mc * rank[i] + j;
      l = pl + 1;
      k = (c << dim) | (uint32_t)j;
      par = pl == 0 ? 0 : 1 + mc * rank[cl.off(pl - 1) + (c >> dim)] + (int)(c & (mc - 1));
    }
    if (!FGT_DCHECK(b < nboxes, 503)) continue;
    const bool nl = l <= L && flag[cl.off(l) + k];
    key[b] = k;
    level[b] = l;
    nonleaf[b] = nl ? 1 : 0;
    parent[b] = par;
    child0[b] = nl ? 1 + mc * rank[cl.off(l) + k] : -1;
    double c[FGT_MAXDIM];
    for (int d = 0; d < dim; d++) c[d] = kp.cen0[d];
    for (int j = 0; j < l; j++) {
      const int dig = (int)((k >> (dim * (l - 1 - j))) & (uint32_t)(mc - 1));
      for (int d = 0; d < dim; d++) c[d] = c[d] + (((dig >> d) & 1) ? kp.bsh[j] : -kp.bsh[j]);
    }
    for (int d = 0; d < dim; d++) center[(size_t)b * dim + d] = c[d];
    if (!nl) {
      const int o = l <= L ? base[(long long)k << (dim * (L - l))] : base[k >> dim] + (int)(k & (mc - 1));
      if (FGT_DCHECK(o < nleaves, 504)) lref[o] = l <= L ? b : par;
    }
  }
}

// Leaf ordinal of every point of both sets.
__global__ void k_dense_ordinals(int dim, const uint32_t* __restrict__ ks, int ns,
                                 const uint32_t* __restrict__ kt, int nt,
                                 const uint32_t* __restrict__ table, uint32_t* __restrict__ os,
                                 uint32_t* __restrict__ is, uint32_t* __restrict__ ot,
                                 uint32_t* __restrict__ it) {
  const long long n = (long long)ns + nt;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const bool src = i < ns;
    const uint32_t j = (uint32_t)(src ? i : i - ns), k = src ? ks[j] : kt[j], t = table[k >> dim];
    const uint32_t o = (t >> 31) ? (t & 0x7fffffffu) + (k & ((1u << dim) - 1)) : t;
    (src ? os : ot)[j] = o;
    (src ? is : it)[j] = j;
  }
}
// First sorted point of every leaf, both sets (k_leaf_point_lo), and the
// reference box of every sorted point (k_point_ref).
__global__ void k_dense_leaf_points(const uint32_t* __restrict__ os, int ns,
                                    const uint32_t* __restrict__ ot, int nt, int nl,
                                    const int* __restrict__ lref, int* __restrict__ slo,
                                    int* __restrict__ tlo, int* __restrict__ sref,
                                    int* __restrict__ tref) {
  const long long np = (long long)ns + nt, n = np + 2 * ((long long)nl + 1);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    if (i < np) {
      if (i < ns) sref[i] = lref[os[i]];
      else tref[i - ns] = lref[ot[i - ns]];
      continue;
    }
    const bool src = i - np <= nl;
    const uint32_t o = (uint32_t)(src ? i - np : i - np - nl - 1);
    const uint32_t* ord = src ? os : ot;
    int a = 0, b = src ? ns : nt;
    while (a < b) {
      const int m = (a + b) >> 1;
      if (ord[m] < o) a = m + 1; else b = m;
    }
    (src ? slo : tlo)[o] = a;
  }
}
__global__ void k_dense_ranges(CellLevels cl, int nboxes, const uint64_t* __restrict__ key,
                               const int* __restrict__ level, const int* __restrict__ base,
                               const int* __restrict__ slo, const int* __restrict__ tlo,
                               int* __restrict__ s0, int* __restrict__ s1, int* __restrict__ t0,
                               int* __restrict__ t1) {
  const int L = cl.D - 1;
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nboxes; b += gridDim.x * blockDim.x) {
    const int l = level[b];
    const long long k = (long long)key[b];
    int a, c;
    if (l <= L) {
      const int sh = cl.dim * (L - l);
      a = base[k << sh];
      c = base[(k + 1) << sh];
    } else {
      a = base[k >> cl.dim] + (int)(k & ((1 << cl.dim) - 1));
      c = a + 1;
    }
    s0[b] = slo[a];
    s1[b] = slo[c];
    t0[b] = tlo[a];
    t1[b] = tlo[c];
  }
}

// The dense tables hold 2^(dim (D-1)) cells at the finest level they cover:
// taken when clearing and scanning them (about 20 bytes a cell) stays small
// against the points, up to 2^21 cells always.  Bound by launches for few
// points and by HBM for many.  Tree phase against sorted keys, level by level
// with a read-back each, as both were at first and as it is now: uniform N = 1e5
// (D = 6) 0.64 -> 0.16 ms, N = 3e3 (D = 5) 0.43 -> 0.12, clusters N + M = 4e6
// (D = 8) 1.76 -> 0.59, 2D periodic N = 1e7 2.14 -> 0.83.  At the line, 2^21
// cells in 3D, a whole call takes 0.44 ms against 0.38 by sorted keys for N =
// 500, the same for 3e3 to 1e4 points, 0.47 / 0.56 for 3e4 and 0.55 / 0.75 for
// 1e5; with 2^18 cells 0.27 / 0.36 for N = 500 and 0.41 / 0.79 for 1e5; with 2^20
// in 2D 0.35 / 0.41 and 0.42 / 0.89.  FGT_TREE_SORTED=1 takes the sorted keys,
// to compare the two.
bool dense_tree_takes(int dim, int D, int ns, int nt) {
  if (D < 1 || dim * (D - 1) > 24 || ns < 1) return false;
  const char* e = getenv("FGT_TREE_SORTED");
  if (e && e[0] == '1') return false;
  return (1ll << (dim * (D - 1))) <= 4 * ((long long)ns + nt) + (1ll << 21);
}

void tree_build_dense(Tree& t, const KeyParams& kp, const double* d_src, const double* d_trg,
                      cudaStream_t s) {
  const int dim = t.dim, D = t.D, mc = t.mc, ns = t.ns, nt = t.nt;
  const CellLevels cl{dim, D};
  const long long C1 = cl.cells(D - 1), T = cl.off(D), np = (long long)ns + nt;
  DBuf<uint32_t> ks(ns, s), kt(std::max(nt, 1), s), table((size_t)C1, s);
  DBuf<int> cnt((size_t)T, s), rank((size_t)T, s), base((size_t)C1 + 1, s), lev(D + 1, s);
  DBuf<unsigned char> flag((size_t)T, s);
  // 1. keys and source counts of the cells
  int* hist = cnt.get() + cl.off(D - 1);
  FGT_CUDA(cudaMemsetAsync(hist, 0, sizeof(int) * C1, s));
  auto keys = [&](auto d) {
    constexpr int DIM = decltype(d)::value;
    if (C1 <= HIST_SMEM)
      k_keys_hist<DIM, true><<<grid_for(np, 256, 8), 256, 0, s>>>(d_src, ns, d_trg, nt, kp, ks, kt,
                                                                  hist, (int)C1);
    else
      k_keys_hist<DIM, false><<<grid_for(np, 256), 256, 0, s>>>(d_src, ns, d_trg, nt, kp, ks, kt,
                                                               hist, (int)C1);
    FGT_LAUNCH_CHECK();
  };
  if (dim == 1) keys(std::integral_constant<int, 1>{});
  else if (dim == 2) keys(std::integral_constant<int, 2>{});
  else keys(std::integral_constant<int, 3>{});
  if (T <= TREE_ONE) {  // steps 2-4 in one block
    const size_t sm = 5 * (size_t)T + 16;  // 27 KB at most
    k_tree_one<<<1, 1024, sm, s>>>(cl, t.ndiv, hist, flag, rank, lev, base, table);
    FGT_LAUNCH_CHECK();
  } else {
  // 2. refinement on source counts (pts_tree_build, pts_tree_nd.f:520-590)
  for (int lhi = D - 1;;) {
    const int q = std::min(lhi, 12 / dim);
    k_pyramid<<<(unsigned)cl.cells(lhi - q), PYR_T, 0, s>>>(cl, lhi, q, t.ndiv, cnt, flag);
    FGT_LAUNCH_CHECK();
    lhi -= q;
    if (lhi == 0) break;
  }
  // 3. level restriction (minimal 2:1 balanced refinement)
  int l = D - 1;
  for (; l >= 2 && cl.cells(l) > 1024; l--) {
    k_restrict<<<grid_for(cl.cells(l), 256), 256, 0, s>>>(cl, l, flag);
    FGT_LAUNCH_CHECK();
  }
  if (l >= 2) {
    k_restrict_rest<<<1, 1024, 0, s>>>(cl, l, flag);
    FGT_LAUNCH_CHECK();
  }
  // 4. box numbers and leaf ordinals
  auto scan = [&](const auto& op, long long n) {
    auto go = [&](auto cells) {
      constexpr int CI = decltype(cells)::value;
      const int nb = ceil_div(n, CS_T * CI);
      DBuf<int> part(nb, s);
      k_cells_sum<CI><<<nb, CS_T, 0, s>>>(op, n, part.get());
      FGT_LAUNCH_CHECK();
      k_cells_scan<CI><<<nb, CS_T, 0, s>>>(op, n, part.get());
      FGT_LAUNCH_CHECK();
    };
    if (n <= (1ll << 20)) go(std::integral_constant<int, 4>{});
    else go(std::integral_constant<int, 16>{});
  };
  scan(RankOp{cl, flag, rank, lev}, T);
  scan(LeafOp{cl, flag, base, table}, C1);
  }
  DBuf<uint32_t> os(ns, s), ot(std::max(nt, 1), s);
  t.isrc.alloc(ns, s);
  t.itrg.alloc(std::max(nt, 1), s);
  k_dense_ordinals<<<grid_for(np, 256), 256, 0, s>>>(dim, ks, ns, kt, nt, table, os, t.isrc, ot,
                                                     t.itrg);
  FGT_LAUNCH_CHECK();
  int h[66];
  fetch_span(lev, D + 1, h, s);
  int nlevels = 0;
  while (nlevels < D && h[nlevels + 1] > h[nlevels]) nlevels++;
  t.nlevels = nlevels;
  t.lev_start.assign(nlevels + 2, 0);
  t.lev_start[1] = 1;
  for (int k = 1; k <= nlevels; k++) t.lev_start[k + 1] = 1 + mc * h[k];
  const int nboxes = t.nboxes = 1 + mc * h[D], nl = t.nleaves = nboxes - h[D];
  t.boxsize.resize(nlevels + 1);
  t.boxsize[0] = t.bs0;
  for (int k = 1; k <= nlevels; k++) t.boxsize[k] = t.boxsize[k - 1] / 2;
  // 5. box tables
  t.key.alloc(nboxes, s);
  t.level.alloc(nboxes, s);
  t.nonleaf.alloc(nboxes, s);
  t.parent.alloc(nboxes, s);
  t.child0.alloc(nboxes, s);
  t.center.alloc((size_t)nboxes * dim, s);
  DBuf<int> lref(nl, s), slo(nl + 1, s), tlo(nl + 1, s);
  k_dense_boxes<<<grid_for(T * mc + 1, 256), 256, 0, s>>>(cl, kp, flag, rank, base, t.key, t.level,
                                                         t.nonleaf, t.parent, t.child0, t.center,
                                                         lref, nboxes, nl);
  FGT_LAUNCH_CHECK();
  // 6. leaf order of the points (stable by original index)
  const int obits = bits_for(nl);
  DBuf<uint32_t> otmp(std::max(ns, nt), s), vtmp(std::max(ns, nt), s);
  radix_sort_u32(os, t.isrc, otmp, vtmp, ns, obits, s);
  if (nt > 0) radix_sort_u32(ot, t.itrg, otmp, vtmp, nt, obits, s);
  t.src_ref.alloc(ns, s);
  t.trg_ref.alloc(std::max(nt, 1), s);
  k_dense_leaf_points<<<grid_for(np + 2 * ((long long)nl + 1), 256), 256, 0, s>>>(
      os, ns, ot, nt, nl, lref, slo, tlo, t.src_ref, t.trg_ref);
  FGT_LAUNCH_CHECK();
  t.src_lo.alloc(nboxes, s);
  t.src_hi.alloc(nboxes, s);
  t.trg_lo.alloc(nboxes, s);
  t.trg_hi.alloc(nboxes, s);
  k_dense_ranges<<<grid_for(nboxes, 256), 256, 0, s>>>(cl, nboxes, t.key, t.level, base, slo, tlo,
                                                      t.src_lo, t.src_hi, t.trg_lo, t.trg_hi);
  FGT_LAUNCH_CHECK();
}

}  // namespace

namespace {
__global__ void k_fill_int(int* __restrict__ a, int n, int v) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = v;
}
}  // namespace

void tree_build(Tree& t, int dim, int iperiod, int npwlevel, int ndiv, double bs0,
                const double* cen0, const double* d_src, int ns, const double* d_trg, int nt,
                cudaStream_t s) {
  t.dim = dim;
  t.mc = 1 << dim;
  t.iperiod = iperiod;
  t.npwlevel = npwlevel;
  t.ncutoff = npwlevel > 0 ? npwlevel : 0;
  t.ndiv = ndiv;
  t.ns = ns;
  t.nt = nt;
  t.bs0 = bs0;
  for (int k = 0; k < dim; k++) t.cen0[k] = cen0[k];
  int D = npwlevel >= 0 ? npwlevel + 1 : 0;  // nlmax of pfgt.f:136-140
  FGT_REQUIRE(D * dim <= 63 && D < 63, FGT_ERR_UNSUPPORTED,
              "tree depth exceeds the 63-bit path key (delta too small for the data extent)");
  t.D = D;
  KeyParams kp;
  kp.dim = dim;
  kp.D = D;
  for (int k = 0; k < FGT_MAXDIM; k++) kp.cen0[k] = k < dim ? cen0[k] : 0.0;
  {
    double bs = bs0;
    for (int l = 0; l < 64; l++) {
      double bsc = bs / 2;  // boxsize(l+1)
      kp.bsh[l] = bsc / 2;
      bs = bsc;
    }
  }
  if (dense_tree_takes(dim, D, ns, nt)) {
    tree_build_dense(t, kp, d_src, d_trg, s);
    return;
  }
  // 1. full keys of sources and targets
  DBuf<uint64_t> skey(ns, s), tkey(nt, s), ksorted, ktmp(std::max(ns, nt), s);
  if (ns > 0) launch_point_keys(dim, d_src, ns, kp, skey, s);
  if (nt > 0) launch_point_keys(dim, d_trg, nt, kp, tkey, s);
  ksorted.alloc(std::max(ns, 1), s);
  if (ns > 0)
    FGT_CUDA(cudaMemcpyAsync(ksorted.get(), skey.get(), sizeof(uint64_t) * ns,
                             cudaMemcpyDeviceToDevice, s));
  radix_sort(ksorted, nullptr, ktmp, nullptr, ns, dim * D, s);

  // 2. refinement on source counts (pts_tree_build, pts_tree_nd.f:520-590)
  std::vector<DBuf<uint64_t>> lk;   // keys of each level
  std::vector<DBuf<uint64_t>> NL;   // non-leaf keys of each level
  std::vector<int> nlk, nnl;
  lk.emplace_back(1, s);
  FGT_CUDA(cudaMemsetAsync(lk[0].get(), 0, sizeof(uint64_t), s));
  nlk.push_back(1);
  int nlevels = 0;
  for (int l = 0; l < D; l++) {
    int nb = nlk[l];
    DBuf<int> cnt(nb, s), flag(nb, s), pos(nb, s), tot(1, s);
    k_box_counts<<<grid_for(nb, 256), 256, 0, s>>>(lk[l], nb, dim * (D - l), ksorted, ns, cnt);
    FGT_LAUNCH_CHECK();
    k_flag_gt<<<grid_for(nb, 256), 256, 0, s>>>(cnt, nb, ndiv, flag);
    FGT_LAUNCH_CHECK();
    exclusive_scan_i32(flag, pos, nb, tot, s);
    int nref = fetch_int(tot, s);
    if (nref == 0) break;
    NL.emplace_back(nref, s);
    nnl.push_back(nref);
    k_compact_u64<<<grid_for(nb, 256), 256, 0, s>>>(lk[l], flag, pos, nb, NL[l]);
    FGT_LAUNCH_CHECK();
    lk.emplace_back((size_t)nref * t.mc, s);
    nlk.push_back(nref * t.mc);
    k_children<<<grid_for((long long)nref * t.mc, 256), 256, 0, s>>>(NL[l], nref, dim, lk[l + 1]);
    FGT_LAUNCH_CHECK();
    nlevels = l + 1;
  }
  t.nlevels = nlevels;

  // 3. level restriction (minimal 2:1 balanced refinement)
  for (int l = nlevels - 1; l >= 2; l--) {
    int n = nnl[l], m = nnl[l - 1];
    int tot = n * t.mc + m;
    DBuf<uint64_t> cand(tot, s), ctmp(tot, s);
    k_touching_parents<<<grid_for((long long)n * t.mc, 256), 256, 0, s>>>(NL[l], n, l, dim, cand);
    FGT_LAUNCH_CHECK();
    FGT_CUDA(cudaMemcpyAsync(cand.get() + (size_t)n * t.mc, NL[l - 1].get(),
                             sizeof(uint64_t) * m, cudaMemcpyDeviceToDevice, s));
    radix_sort(cand, nullptr, ctmp, nullptr, tot, dim * (l - 1), s);
    DBuf<uint64_t> uniq(tot, s);
    int nu = unique_sorted_u64(cand, tot, uniq, s);
    NL[l - 1] = std::move(uniq);
    nnl[l - 1] = nu;
  }
  // final level key arrays: children of the (updated) non-leaf sets
  for (int l = 1; l <= nlevels; l++) {
    int n = nnl[l - 1];
    lk[l].alloc((size_t)n * t.mc, s);
    nlk[l] = n * t.mc;
    k_children<<<grid_for((long long)n * t.mc, 256), 256, 0, s>>>(NL[l - 1], n, dim, lk[l]);
    FGT_LAUNCH_CHECK();
  }

  // 4. global box tables
  t.lev_start.assign(nlevels + 2, 0);
  for (int l = 0; l <= nlevels; l++) t.lev_start[l + 1] = t.lev_start[l] + nlk[l];
  int nboxes = t.lev_start[nlevels + 1];
  t.nboxes = nboxes;
  t.boxsize.resize(nlevels + 1);
  t.boxsize[0] = bs0;
  for (int l = 1; l <= nlevels; l++) t.boxsize[l] = t.boxsize[l - 1] / 2;
  t.key.alloc(nboxes, s);
  t.level.alloc(nboxes, s);
  t.nonleaf.alloc(nboxes, s);
  t.parent.alloc(nboxes, s);
  t.child0.alloc(nboxes, s);
  t.center.alloc((size_t)nboxes * dim, s);
  for (int l = 0; l <= nlevels; l++) {
    const int n = t.lev_start[l + 1] - t.lev_start[l];
    if (n > 0) {
      k_fill_int<<<grid_for(n, 256), 256, 0, s>>>(t.level.get() + t.lev_start[l], n, l);
      FGT_LAUNCH_CHECK();
    }
  }
  for (int l = 0; l <= nlevels; l++) {
    FGT_CUDA(cudaMemcpyAsync(t.key.get() + t.lev_start[l], lk[l].get(),
                             sizeof(uint64_t) * nlk[l], cudaMemcpyDeviceToDevice, s));
    if (l < nlevels) {
      k_member<<<grid_for(nlk[l], 256), 256, 0, s>>>(lk[l], nlk[l], NL[l], nnl[l],
                                                      t.nonleaf.get() + t.lev_start[l]);
      FGT_LAUNCH_CHECK();
    } else {
      FGT_CUDA(cudaMemsetAsync(t.nonleaf.get() + t.lev_start[l], 0, sizeof(int) * nlk[l], s));
    }
  }
  FGT_REQUIRE(nlevels < 64, FGT_ERR_UNSUPPORTED, "too many levels");
  LevelTables lt;
  for (int l = 0; l <= nlevels; l++) {
    lt.keys[l] = lk[l].get();
    lt.n[l] = nlk[l];
    lt.start[l] = t.lev_start[l];
  }
  lt.start[nlevels + 1] = t.lev_start[nlevels + 1];
  k_box_tables<<<grid_for(nboxes, 256), 256, 0, s>>>(nboxes, nlevels, dim, lt, kp, t.key,
                                                      t.level, t.nonleaf, t.parent, t.child0,
                                                      t.center);
  FGT_LAUNCH_CHECK();

  // 5. leaves and the final point order (stable by original index)
  DBuf<int> lf(nboxes, s), lpos(nboxes, s), ltot(1, s);
  k_leaf_flags<<<grid_for(nboxes, 256), 256, 0, s>>>(t.nonleaf, nboxes, lf);
  FGT_LAUNCH_CHECK();
  exclusive_scan_i32(lf, lpos, nboxes, ltot, s);
  int nl = fetch_int(ltot, s);
  t.nleaves = nl;
  DBuf<uint64_t> ls(nl, s), lstmp(nl, s);
  DBuf<uint32_t> lbox(nl, s), lbtmp(nl, s);
  k_leaf_starts<<<grid_for(nboxes, 256), 256, 0, s>>>(t.key, t.level, lf, lpos, nboxes, dim, D,
                                                       ls, lbox);
  FGT_LAUNCH_CHECK();
  radix_sort(ls, lbox, lstmp, lbtmp, nl, dim * D, s);
  DBuf<int> lref(std::max(nl, 1), s);
  k_leaf_ref<<<grid_for(nl, 256), 256, 0, s>>>(lbox, nl, t.level, t.parent, t.ncutoff, lref);
  FGT_LAUNCH_CHECK();
  int obits = bits_for(nl);
  DBuf<int> slo(nl + 1, s), tlo(nl + 1, s);
  t.src_ref.alloc(std::max(ns, 1), s);
  t.trg_ref.alloc(std::max(nt, 1), s);
  {
    // leaf ordinals as 32-bit keys (half the key traffic of the sort)
    DBuf<uint32_t> ord(std::max(ns, 1), s);
    DBuf<uint32_t> vtmp(std::max(std::max(ns, nt), 1), s);
    uint32_t* otmp = reinterpret_cast<uint32_t*>(ktmp.get());  // >= max(ns, nt) u32
    t.isrc.alloc(std::max(ns, 1), s);
    auto point_leaf = [&](const uint64_t* keys, int n, uint32_t* o, uint32_t* idx) {
      k_point_leaf<<<grid_for(n, 256), 256, 0, s>>>(keys, n, ls, nl, o, idx);
      FGT_LAUNCH_CHECK();
    };
    if (ns > 0) {
      point_leaf(skey, ns, ord, t.isrc);
      radix_sort_u32(ord, t.isrc, otmp, vtmp, ns, obits, s);
    }
    k_leaf_point_lo<<<grid_for(nl + 1, 256), 256, 0, s>>>(ord, ns, nl, slo);
    FGT_LAUNCH_CHECK();
    if (ns > 0) {
      k_point_ref<<<grid_for(ns, 256), 256, 0, s>>>(ord, ns, lref, t.src_ref);
      FGT_LAUNCH_CHECK();
    }
    DBuf<uint32_t> tord(std::max(nt, 1), s);
    t.itrg.alloc(std::max(nt, 1), s);
    if (nt > 0) {
      point_leaf(tkey, nt, tord, t.itrg);
      radix_sort_u32(tord, t.itrg, otmp, vtmp, nt, obits, s);
    }
    k_leaf_point_lo<<<grid_for(nl + 1, 256), 256, 0, s>>>(tord, nt, nl, tlo);
    FGT_LAUNCH_CHECK();
    if (nt > 0) {
      k_point_ref<<<grid_for(nt, 256), 256, 0, s>>>(tord, nt, lref, t.trg_ref);
      FGT_LAUNCH_CHECK();
    }
  }
  t.src_lo.alloc(nboxes, s);
  t.src_hi.alloc(nboxes, s);
  t.trg_lo.alloc(nboxes, s);
  t.trg_hi.alloc(nboxes, s);
  k_box_ranges<<<grid_for(nboxes, 256), 256, 0, s>>>(t.key, t.level, nboxes, dim, D, ls, nl, slo,
                                                      tlo, t.src_lo, t.src_hi, t.trg_lo,
                                                      t.trg_hi);
  FGT_LAUNCH_CHECK();
}

void tree_download(const Tree& t, TreeHost& h, cudaStream_t s) {
  int nb = t.nboxes;
  auto dl = [&](auto& vec, const auto& buf, size_t n) {
    vec.resize(n);
    if (n) FGT_CUDA(cudaMemcpyAsync(vec.data(), buf.get(), sizeof(vec[0]) * n,
                                    cudaMemcpyDeviceToHost, s));
  };
  dl(h.key, t.key, nb);
  dl(h.level, t.level, nb);
  dl(h.nonleaf, t.nonleaf, nb);
  dl(h.parent, t.parent, nb);
  dl(h.child0, t.child0, nb);
  dl(h.src_lo, t.src_lo, nb);
  dl(h.src_hi, t.src_hi, nb);
  dl(h.trg_lo, t.trg_lo, nb);
  dl(h.trg_hi, t.trg_hi, nb);
  dl(h.center, t.center, (size_t)nb * t.dim);
  dl(h.isrc, t.isrc, t.ns);
  dl(h.itrg, t.itrg, t.nt);
  FGT_CUDA(cudaStreamSynchronize(s));
}

}  // namespace fgt
