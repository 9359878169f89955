// moe_window_up.cu - the window kernel, gate/up (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_type<false, true>(int, const WArgs&, cudaStream_t);
}
