// moe_token_i1.cu - the token kernel for gate/up rows of IQ2_S and IQ3_S (see moe_token.cuh).
#include "moe_token.cuh"

namespace maya {
template int token_by_type<MAYA_IQ2_S>(const TokArgs&, cudaStream_t);
template int token_by_type<MAYA_IQ3_S>(const TokArgs&, cudaStream_t);
}  // namespace maya
