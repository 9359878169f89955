// maya_internal.cuh - host-side entry points shared between translation units of the library.
#pragma once

#include "maya_common.cuh"

namespace maya {

// How the group kernels find their work: group g = blob ptr[g] with entries [start[g], start[g+1]) (start NULL: the
// single entry g).  Entry e has an h / partial slot (ent_slot[e], NULL: e), an activation column (ent_tok[e]; NULL:
// slot >> 3 when tok_from_slot, else 0) and an output row for the down product (ent_out[e], NULL: its slot).
struct GroupArgs {
    const unsigned long long* ptr;
    const int* start;
    const int* n_groups;
    const int* ent_slot;
    const int* ent_tok;
    const int* ent_out;
    const int* skip;
    int tok_from_slot;
    int cap_entries;      // > 0: the kernels touch no entry at or beyond it
};

int gate_up_groups(int gu_type, const GroupArgs& A, int n_groups_grid, int n_embd, int n_ff, size_t up_off, float limit,
                   const void* xq, size_t xq_stride, void* hq, const void* sh_down, int sh_type, const void* sh_hq,
                   int n_ff_sh, float* sh_out, cudaStream_t s);
int down_groups(int d_type, const GroupArgs& A, int n_groups_grid, int n_embd, int n_ff, size_t down_off, const void* hq,
                float* part, cudaStream_t s);
int down_plan(int d_type, const maya_moe_plan& P, int k, int n_embd, int n_ff, size_t down_off, const void* hq,
              const float* sh_out, float* out, cudaStream_t s);
// The streamed forms (moe_window.cuh), for up to 128 groups.  kWindowTooWide: the shapes do not fit them, nothing launched.
// sh: a Q8_0 shared expert every one of n_tok tokens (whose columns are xq, xq_stride apart) uses, in the same launches: gate/up
// leaves its h in sh->hq [n_tok][n_ff / 32], down its output in sh->out [n_tok][n_embd].
constexpr int kWindowTooWide = 1;
struct SharedArgs {
    const uint8_t* blob;         // [gate rows | up rows | down rows]
    int n_ff, n_tok;
    void* hq;
    float* out;
};
// How often a warp looks at its rows' copies before it gives up, and who is told: `error` (optional, a sticky word) is set to 1 and
// *n_groups, the launch's group count, to -1.
struct WaitArgs {
    int* n_groups;
    unsigned* error;
    unsigned polls;
};
inline bool window_fits(int n_embd, int n_ff, int n_ff_sh) { return n_embd <= 8192 && n_ff <= 8192 && n_ff_sh <= 8192; }
int window_gate_up(int gu_type, const GroupArgs& A, int cap_groups, int n_embd, int n_ff, size_t up_off, float limit, const void* xq,
                   size_t xq_stride, void* hq, const SharedArgs* sh, const WaitArgs& wait, cudaStream_t s);
int window_down(int d_type, const GroupArgs& A, int cap_groups, int n_embd, int n_ff, size_t down_off, const void* hq, float* part,
                const SharedArgs* sh, const WaitArgs& wait, cudaStream_t s);
int win_combine(const unsigned long long* plan_ptr, const float* plan_w, int T, int k, int n_embd, const float* part,
                const float* cpu_part, const int* cpu_flag, const float* sh_out, float* out, size_t out_stride,
                cudaStream_t s);

int win_experts(int gu_type, int d_type, const maya_moe_win* w, bool grouped, const SharedArgs* sh, unsigned polls, unsigned* error,
                const maya_peer_ar* ar, int mi, unsigned seq, cudaStream_t s);

// One token through a layer in one launch: the token kernel (moe_token.cuh) or the fused kernel (moe_fused.cu).  kNotHere: neither
// takes the layer, nothing launched.
constexpr int kNotHere = 1;
struct FusedArgs;
bool fused_t1_supported(const maya_moe_layer& L);
int fused_t1(const maya_moe_layer& L, const float* logits, const void* x, int x_is_bf16, int* ids, float* weights,
             float* out, float* h_scratch, unsigned* unit_count, unsigned* sync, const maya_peer_ar* ar, int ar_rank, unsigned ar_seq,
             const maya_hc_post_args* hc, int kernel, unsigned polls, cudaStream_t s);
int token_layer(const maya_moe_layer& L, const FusedArgs& F, unsigned* unit_count, unsigned polls, cudaStream_t s);
bool token_takes(const maya_moe_layer& L, const FusedArgs& F, int sms);           // the token kernel's limits
bool token_better(int type, const FusedArgs& A, int sms);
// The kernel maya_moe_layer_decode runs one token with (enum maya_layer_kernel), with a sum over n_ranks ranks where that is 2 or more.
int layer_kernel(const maya_moe_layer& L, int n_ranks, int sms);

}  // namespace maya
