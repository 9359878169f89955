// moe_window_up_sh_k.cu - the window kernel, gate/up with a Q8_0 shared expert, Q8_0, the K-quants and IQ4_XS (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_group<true, true, 0>(int, const WArgs&, cudaStream_t);
}
