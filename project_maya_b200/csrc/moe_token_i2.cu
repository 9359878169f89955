// moe_token_i2.cu - the token kernel for gate/up rows of IQ3_XXS and IQ2_XXS (see moe_token.cuh).
#include "moe_token.cuh"

namespace maya {
template int token_by_type<MAYA_IQ3_XXS>(const TokArgs&, cudaStream_t);
template int token_by_type<MAYA_IQ2_XXS>(const TokArgs&, cudaStream_t);
}  // namespace maya
