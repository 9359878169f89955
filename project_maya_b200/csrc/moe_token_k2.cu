// moe_token_k2.cu - the token kernel for gate/up rows of Q5_K and Q6_K (see moe_token.cuh).
#include "moe_token.cuh"

namespace maya {
template int token_by_type<MAYA_Q5_K>(const TokArgs&, cudaStream_t);
template int token_by_type<MAYA_Q6_K>(const TokArgs&, cudaStream_t);
}  // namespace maya
