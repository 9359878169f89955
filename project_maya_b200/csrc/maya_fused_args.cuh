// maya_fused_args.cuh - the argument blocks of the single-token layer kernels (moe_fused.cu, moe_token.cuh).
#pragma once

#include "maya_common.cuh"

namespace maya {

struct FusedArgs {
    const float* logits;       // [n_expert]
    int router;                // 0 softmax, 1 sigmoid (+ bias for the selection, weight scale, optional normalisation)
    const float* router_bias;
    float router_w_scale;
    int router_norm_w;
    const float* cpu_part;     // [n_embd] the host lane's contribution, added when *cpu_flag != 0 (NULL: none)
    const int* cpu_flag;
    const void* x;             // [n_embd] f32 or bf16
    int x_is_bf16;
    int n_embd, n_ff, n_expert, k;
    const uint8_t* experts;
    size_t expert_stride;
    int expert_lo, expert_hi;
    const uint8_t* shared;     // NULL: none (or not on this rank)
    int n_ff_sh;
    int sh_lo, sh_hi;          // this rank's slice of the shared expert's FFN width (multiples of 32): its gate/up rows
                               // and the same columns of every down row; the ranks' partial outputs add up
    float limit;
    int* ids;                  // [k] out
    float* weights;            // [k] out
    float* out;                // [n_embd] out
    float* h;                  // scratch [(k + 1)][max(n_ff, n_ff_sh)] f32
    maya_peer_ar ar;           // ar.nm >= 2: sum `out` over the ranks in the epilogue
    int ar_rank;
    unsigned ar_seq;
    maya_hc_post_args hc;      // hc.R_new != NULL: the hyper-connection write of `out` into the residual stack, last
    unsigned* sync;            // scratch: [0] arrivals, [1] epoch, [2] error, [4..15] block 0's phase time stamps (ns), [kTokMark] the mark
                               // of the last launch in which a block of the token kernel gave up
};

// moe_token.cuh: the rows' places in a blob, and the launch's carve-up of shared memory.
struct TokArgs : FusedArgs {
    int d_type;
    size_t up_off, down_off;   // byte offsets of the up and of the down rows in a routed blob
    unsigned* unit_count;      // scratch [(MAYA_MAX_K + 1) * blocks of h]: items done of units that two blocks share, modulo 16
    unsigned polls;            // looks at a row's copy before a warp gives up
    unsigned drain_polls;      // and, at the end, at the copies still in flight
    int stage, tab, cols;      // bytes of a ring stage, of the codebook, of the activation columns
    int units;                 // units of h a block may work on
};
constexpr int kTokWarps = 16;
constexpr int kTokMark = 32;    // a 128-byte line away from the arrivals, which every block is polling when the mark is read
constexpr size_t kTokMostSmem = 232448 - 8192;                  // dynamic shared memory, beside the static part
#define MAYA_TOK_TYPES(X) X(MAYA_IQ2_S) X(MAYA_IQ3_S) X(MAYA_IQ3_XXS) X(MAYA_IQ2_XXS) X(MAYA_IQ1_S)      // types with a codebook
__host__ __device__ inline int tok_col_bytes(int nblk) { return (nblk * 40 + 15) & ~15; }       // of an activation column
// The launch's carve-up, into A; what it takes of shared memory beside the static part, 0: more than there is.
size_t token_smem(int gu_type, TokArgs& A, int grid);

}  // namespace maya
