// The view kernel for 64-column tiles.
#include "view_kernel.cuh"

namespace tsr {
template int launch_view_bn<64>(tsr_ctx*, cudaStream_t, const ViewArgs&, int, dim3);
template int view_ctas_per_sm<64>(int);
}  // namespace tsr
