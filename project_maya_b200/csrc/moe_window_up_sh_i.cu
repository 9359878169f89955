// moe_window_up_sh_i.cu - the window kernel, gate/up with a Q8_0 shared expert, the codebook types (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_group<true, true, 1>(int, const WArgs&, cudaStream_t);
}
