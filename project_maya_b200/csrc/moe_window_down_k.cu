// moe_window_down_k.cu - the window kernel, down, Q8_0, the K-quants and IQ4_XS (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_group<false, false, 0>(int, const WArgs&, cudaStream_t);
}
