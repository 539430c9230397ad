// kernels_f64_const.cu -- the FP64 kernel of the single-pass classes, constant gap priors.
#include "kernel_table.cuh"

namespace rodv {
template KernelInfo rescue_info_for<kGapsConst>(int);
}  // namespace rodv
