// moe_window_down_sh.cu - the window kernel, down with a Q8_0 shared expert (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_type<true, false>(int, const WArgs&, cudaStream_t);
}
