// Instantiations of the one-tile-per-CTA axis-pass kernel for the first and
// last passes of the 1-D chains of long real lines (the type-2 permutation,
// the type-3 pre-rotation and the inverse real DFT's packing fused into the
// first pass's load; the real DFT's unpacking, the type-2 rotation and the
// type-3 de-interleave into the last pass's store): pass lengths 2^4 .. 2^10,
// radix 16.
#include "axis_pass.cuh"

namespace mb {

namespace {
template <class Ld, class St>
const void* line_pass(int log2L, int radix16) {
  static const void* const table[7] = {
      (const void*)axis_pass_kernel<16, 16, Ld, St>,
      (const void*)axis_pass_kernel<32, 16, Ld, St>,  (const void*)axis_pass_kernel<64, 16, Ld, St>,
      (const void*)axis_pass_kernel<128, 16, Ld, St>, (const void*)axis_pass_kernel<256, 16, Ld, St>,
      (const void*)axis_pass_kernel<512, 16, Ld, St>, (const void*)axis_pass_kernel<1024, 16, Ld, St>,
  };
  return (radix16 && log2L >= 4 && log2L <= 10) ? table[log2L - 4] : nullptr;
}
}  // namespace

const void* axis_kernel_dct2in(int log2L, int radix16) { return line_pass<LoadDCT2Line, StoreCplx>(log2L, radix16); }
const void* axis_kernel_dct2out(int log2L, int radix16) { return line_pass<LoadCplx, StoreDCT2Line>(log2L, radix16); }
const void* axis_kernel_dct3in(int log2L, int radix16) { return line_pass<LoadDCT3Line, StoreCplx>(log2L, radix16); }
const void* axis_kernel_dct3out(int log2L, int radix16) { return line_pass<LoadCplx, StoreDCT3Line>(log2L, radix16); }
const void* axis_kernel_c2rin(int log2L, int radix16) { return line_pass<LoadC2RLine, StoreCplx>(log2L, radix16); }
const void* axis_kernel_r2cout(int log2L, int radix16) { return line_pass<LoadCplx, StoreR2CLine>(log2L, radix16); }

}  // namespace mb
