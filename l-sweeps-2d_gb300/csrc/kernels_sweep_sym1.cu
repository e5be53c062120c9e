// The symmetric-tile sweep kernels on 1 CTA per half chain (a translation unit
// per cluster size, so that they compile in parallel).
#include "sweep_sym.cuh"

namespace lsw {
SymKernel sym_kernel_1(bool split) { return split ? k_front_sym<1, true> : k_front_sym<1, false>; }
}  // namespace lsw
