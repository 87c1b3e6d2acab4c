// FP64 instantiation of the radiation column kernel.  Built with
// -fmad=false: products and sums round separately, in the reference's order.
#include "radiation_kernel.cuh"

namespace exotx {
exotx_status launch_radstep_fp64(const RadDev &D, int maxcols, bool list, cudaStream_t st) {
    return launch_radstep<double>(D, maxcols, list, st);
}
}  // namespace exotx
