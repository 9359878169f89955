// moe_window_down_sh_k.cu - the window kernel, down with a Q8_0 shared expert, Q8_0, the K-quants and IQ4_XS (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_group<true, false, 0>(int, const WArgs&, cudaStream_t);
}
