// kernels_f64_perrow.cu -- the FP64 kernel of the single-pass classes, per-row gap priors.
#include "kernel_table.cuh"

namespace rodv {
template KernelInfo rescue_info_for<kGapsPerRow>(int);
}  // namespace rodv
