// moe_window_down_i.cu - the window kernel, down, the codebook types (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_group<false, false, 1>(int, const WArgs&, cudaStream_t);
}
