// moe_token_k3.cu - the token kernel for gate/up rows of IQ4_XS and IQ1_S (see moe_token.cuh).
#include "moe_token.cuh"

namespace maya {
template int token_by_type<MAYA_IQ4_XS>(const TokArgs&, cudaStream_t);
template int token_by_type<MAYA_IQ1_S>(const TokArgs&, cudaStream_t);
}  // namespace maya
