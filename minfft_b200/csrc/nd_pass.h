// Small multi-dimensional transforms in one launch (nd_pass.cu): a cluster of
// CTAs per array transforms one axis after the other.
#pragma once

#include "axis_pass.cuh"

namespace mb {

constexpr int kNdMaxAxes = 4;
constexpr int kNdCluster = 8;     // CTAs per array
constexpr int kNdMaxThreads = 256;
constexpr int kNdMaxLog2L = 7;    // in-CTA DFTs of an axis: up to 128 points

// One axis step, in execution order: nb transforms, transform b = b0 + inner*b1
// starting at b0 + b1*in_row (out_row), elements inner apart.
struct NdAxis {
  int log2L;
  int nb, inner, in_row, out_row;
  int flags;
  const cpx *tw, *t1, *t2;  // root tables of n_tw, n_t1, n_t2 entries
  int n_tw, n_t1, n_t2;
};

struct NdParams {
  const void* in;
  void* mid;  // the steps between the first's input and the last's output
  void* out;
  int64_t in_stride, mid_stride, out_stride;  // elements between arrays, each of its own type
  int naxes;
  int table_elems;  // entries of all root tables
  int flags;        // F_VEC: real rows read (written) as complex pairs are aligned
  NdAxis ax[kNdMaxAxes];
};

// Kernel for the family of steps (first step's and last step's combo), and
// its dynamic shared memory for CTAs of `threads` and table_elems entries.
const void* nd_kernel(int first_combo, int last_combo);
size_t nd_smem(int threads, int table_elems);

}  // namespace mb
