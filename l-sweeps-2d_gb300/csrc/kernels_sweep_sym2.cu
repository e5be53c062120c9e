// The symmetric-tile sweep kernels on 2 CTAs per half chain (a translation unit
// per cluster size, so that they compile in parallel).
#include "sweep_sym.cuh"

namespace lsw {
SymKernel sym_kernel_2(bool split) { return split ? k_front_sym<2, true> : k_front_sym<2, false>; }
}  // namespace lsw
