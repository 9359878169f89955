// moe_window_up_sh.cu - the window kernel, gate/up with a Q8_0 shared expert (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_type<true, true>(int, const WArgs&, cudaStream_t);
}
