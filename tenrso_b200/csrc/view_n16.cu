// The view kernel for 16-column tiles.
#include "view_kernel.cuh"

namespace tsr {
template int launch_view_bn<16>(tsr_ctx*, cudaStream_t, const ViewArgs&, int, dim3);
template int view_ctas_per_sm<16>(int);
}  // namespace tsr
