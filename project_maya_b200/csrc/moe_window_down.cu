// moe_window_down.cu - the window kernel, down (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_type<false, false>(int, const WArgs&, cudaStream_t);
}
