// moe_window_up_i.cu - the window kernel, gate/up, the codebook types (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_group<false, true, 1>(int, const WArgs&, cudaStream_t);
}
