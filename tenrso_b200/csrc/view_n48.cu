// The view kernel for 48-column tiles.
#include "view_kernel.cuh"

namespace tsr {
template int launch_view_bn<48>(tsr_ctx*, cudaStream_t, const ViewArgs&, int, dim3);
template int view_ctas_per_sm<48>(int);
}  // namespace tsr
