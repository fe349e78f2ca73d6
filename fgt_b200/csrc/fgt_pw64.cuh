// FP64 3D plane-wave form and evaluation on the FP64 matrix instructions,
// for box sub-grids without wrap-around (fgt_pw64.cu).
#pragma once
#include "fgt_pw_dev.cuh"

namespace fgt {

// Arguments of a form / evaluation: those of the work-item kernels (FormIO,
// EvalPtrs), device pointers unless noted.  Items are in the order of the
// boxes and carry their box's place in it (WorkItem::pslot).
struct Form64 {
  const int *form_box, *s_lo, *s_hi;
  const uint32_t* order;  // form slots, most sources first
  const void* items;      // WorkItem[]
  const int *n_items, *item_off;  // item count, first item of every box
  int n_form, ns, nd, ncomp, has_q;
  const double *off, *q, *ds, *rn;
  double* mp;
};
struct Eval64 {
  const double* loc;
  const int *eval_box, *boxes;  // boxes: eval slots, most points first
  const int* nbox_dev;          // their count
  const void* items;
  const int *n_items, *item_off;
  int nbox;  // bound of the count
  const double* off[2];
  const int *lo[2], *hi[2];
  double* out[2];
  int n[2], ncomp[2];
  int nd, ncomp_max;
  // gradients without the terms of the stencil's centre cell (as
  // interp_grad_cells, which the grids that fit in shared memory had)
  int drop_ref;
};

// x-planes of a grid transformed by one CTA.
constexpr int SLAB64 = 16;

// Whether the kernels take this grid (kernel width, extents, block count).
bool form64_takes(int w, int K, int G, bool wrap);
bool eval64_takes(int w, int K, int G, bool wrap);
// Launches on stream s, grids from the call's workspace; `a`: the launch's
// PWArgs<double> (host pointer).
void form64_launch(int w, const void* a, const Form64& io, cudaStream_t s);
// Modal sums of the boxes with at most pmax points (3D; smem: dynamic shared
// memory, at least 3 (2K+1) pmax complex + (2K+1) + 256 doubles); false: not
// taken (hessians, expansions too long).  The caller checks the launch.
bool modal64_launch(const void* a, const Eval64& io, int pmax, size_t smem, cudaStream_t s);
void eval64_launch(int w, bool deriv, const void* a, const Eval64& io, cudaStream_t s);

// Small 2D boxes (fgt_pw64_2d.cu): the boxes from *first on of the order, one
// warp per (box, density); next: work counter, zero.
bool small2d64_takes(int w, int K, int G, bool wrap);
void form2d64_launch(int w, const void* a, const Form64& io, const int* first, int* next,
                     cudaStream_t s);
void eval2d64_launch(int w, bool deriv, const void* a, const Eval64& io, const int* first,
                     int* next, cudaStream_t s);

}  // namespace fgt
