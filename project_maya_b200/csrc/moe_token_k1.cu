// moe_token_k1.cu - the token kernel for gate/up rows of Q8_0 and Q4_K (see moe_token.cuh).
#include "moe_token.cuh"

namespace maya {
template int token_by_type<MAYA_Q8_0>(const TokArgs&, cudaStream_t);
template int token_by_type<MAYA_Q4_K>(const TokArgs&, cudaStream_t);
}  // namespace maya
