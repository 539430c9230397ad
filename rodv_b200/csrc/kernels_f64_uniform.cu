// kernels_f64_uniform.cu -- the FP64 kernel of the single-pass classes, gap priors per read.
#include "kernel_table.cuh"

namespace rodv {
template KernelInfo rescue_info_for<kGapsUniform>(int);
}  // namespace rodv
