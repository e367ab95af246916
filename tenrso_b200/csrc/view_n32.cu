// The view kernel for 32-column tiles.
#include "view_kernel.cuh"

namespace tsr {
template int launch_view_bn<32>(tsr_ctx*, cudaStream_t, const ViewArgs&, int, dim3);
template int view_ctas_per_sm<32>(int);
}  // namespace tsr
