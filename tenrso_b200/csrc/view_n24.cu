// The view kernel for 24-column tiles.
#include "view_kernel.cuh"

namespace tsr {
template int launch_view_bn<24>(tsr_ctx*, cudaStream_t, const ViewArgs&, int, dim3);
template int view_ctas_per_sm<24>(int);
}  // namespace tsr
