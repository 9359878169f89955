// moe_token.cu - host side of the token kernel (moe_token.cuh): which layers it takes.
#include "maya_fused_args.cuh"
#include "maya_internal.cuh"

namespace maya {

template<int T> int token_by_type(const TokArgs& A, cudaStream_t s);

// kNotHere: not this kernel's, nothing launched.
int token_layer(const maya_moe_layer& L, const FusedArgs& F, unsigned* unit_count, unsigned polls, cudaStream_t s) {
    if (F.ar.nm >= 2) return kNotHere;                 // the cross-rank sum is moe_fused.cu's
    // bulk copies take aligned 16-byte windows around the rows: blobs have to start and end on 16-byte boundaries
    if ((((uintptr_t) F.experts) | F.expert_stride | (uintptr_t) F.shared) & 15u) return kNotHere;
    if (F.shared != nullptr && (L.sh_gu_type != MAYA_Q8_0 || L.sh_d_type != MAYA_Q8_0)) return kNotHere;
    TokArgs A{};
    (FusedArgs&) A = F;
    A.d_type = L.d_type;
    A.up_off = row_bytes(L.gu_type, L.n_embd) * (size_t) L.n_ff;
    A.down_off = 2 * A.up_off;
    A.unit_count = unit_count;
    A.polls = polls;
    switch (L.gu_type) {
        case MAYA_Q8_0: return token_by_type<MAYA_Q8_0>(A, s);
        case MAYA_Q4_K: return token_by_type<MAYA_Q4_K>(A, s);
        case MAYA_Q5_K: return token_by_type<MAYA_Q5_K>(A, s);
        case MAYA_Q6_K: return token_by_type<MAYA_Q6_K>(A, s);
        case MAYA_IQ4_XS: return token_by_type<MAYA_IQ4_XS>(A, s);
        case MAYA_IQ2_S: return token_by_type<MAYA_IQ2_S>(A, s);
        case MAYA_IQ3_S: return token_by_type<MAYA_IQ3_S>(A, s);
        case MAYA_IQ3_XXS: return token_by_type<MAYA_IQ3_XXS>(A, s);
        case MAYA_IQ2_XXS: return token_by_type<MAYA_IQ2_XXS>(A, s);
        case MAYA_IQ1_S: return token_by_type<MAYA_IQ1_S>(A, s);
        default: return kNotHere;
    }
}

}  // namespace maya
