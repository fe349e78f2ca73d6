// Interaction lists of the point FGT on the device: colleagues, plane-wave
// boxes and lists, and the modified list 1 of the direct near field.
#pragma once
#include "fgt_tree.cuh"

namespace fgt {

struct Lists {
  // plane-wave part (boxes at the cutoff level)
  int n_form = 0, n_eval = 0, n_trans = 0;
  DBuf<int> form_box;    // boxes that form a PW expansion (npts > ndiv)
  DBuf<int> eval_box;    // boxes with ifpwexp = 1
  DBuf<int> eval_self;   // per eval box: its own form slot or -1
  DBuf<int> trans_ptr;   // per eval box: CSR offsets into trans_src/trans_w (n_eval+1)
  DBuf<int> trans_src;   // form slot of the source expansion
  DBuf<int> trans_w;     // shift-table index 0..3^dim-1
  // translation by sibling groups: the 2^dim children of one parent at the
  // cut-off level, their eval slots (-1: none) and the form slots (-1: none)
  // of the 4^dim boxes around them, first coordinate fastest; in 3D only those
  // present, as slot * 64 + position, closed by a -1 where there are fewer
  int n_grp = 0;
  DBuf<int> grp_src, grp_trg;
  // direct part: CSR over all boxes (targets), sources are box ids
  DBuf<int> l1_ptr, l1_src;
  DBuf<int> l1_trg;  // target box of every list entry
  int n_l1 = 0;
};

// Whether the translation goes by sibling groups.  FP64 and 2D read memory less
// often so: 10^7 points in a periodic square 2.1 -> 0.78 ms, spheres of 4e6
// points at 1e-9 2.7 -> 1.9 and of 2e6 at 1e-6 1.2 -> 1.0.  In FP32 3D the
// expansions fit the L2 and the kernel by lists is as fast (0.56 / 0.57 ms at
// 1e6 points, 0.74 / 0.71 at 10^7).
inline bool translates_by_groups(int dim, bool fp64) { return dim < 3 || fp64; }

// nlevend / iperiod0 follow pfgtmain (src/pfgt/pfgt.f:618-650); groups: build
// the sibling groups too.
void build_lists(const Tree& t, int npwlevel, int iperiod0, int nlevend, bool do_pw, bool groups,
                 Lists& L, cudaStream_t s);

struct ListsHost {
  std::vector<int> form_box, eval_box, eval_self, trans_ptr, trans_src, trans_w, l1_ptr, l1_src;
};
void lists_download(const Lists& L, int nboxes, ListsHost& h, cudaStream_t s);

}  // namespace fgt
