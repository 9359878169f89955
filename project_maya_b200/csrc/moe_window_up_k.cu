// moe_window_up_k.cu - the window kernel, gate/up, Q8_0, the K-quants and IQ4_XS (see moe_window.cuh).
#include "moe_window.cuh"

namespace maya {
template int launch_window_group<false, true, 0>(int, const WArgs&, cudaStream_t);
}
