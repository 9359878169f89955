// moe_window.cu - host side of the streamed window kernels (moe_window.cuh): the groups' gate/up and down.
#include "moe_window_args.cuh"

namespace maya {
namespace {
WArgs common(const GroupArgs& A, int cap_groups, int n_embd, int n_ff, const SharedArgs* sh, const WaitArgs& wait) {
    WArgs W{};
    W.ptr = A.ptr; W.start = A.start; W.n_groups = wait.n_groups; W.error = wait.error; W.polls = wait.polls; W.ent_slot = A.ent_slot;
    W.cap = cap_groups; W.n_embd = n_embd; W.n_ff = n_ff;
    if (sh != nullptr) { W.n_ff_sh = sh->n_ff; W.n_tok = sh->n_tok; W.sh_hq = (uint8_t*) sh->hq; W.sh_out = sh->out; }
    return W;
}
template<bool SH, bool UP> int launch_window_type(int type, const WArgs& W, cudaStream_t s) {
    switch (type) {
        case MAYA_Q8_0: case MAYA_Q4_K: case MAYA_Q5_K: case MAYA_Q6_K: case MAYA_IQ4_XS: return launch_window_group<SH, UP, 0>(type, W, s);
        default: return launch_window_group<SH, UP, 1>(type, W, s);
    }
}
}  // namespace

int window_gate_up(int gu_type, const GroupArgs& A, int cap_groups, int n_embd, int n_ff, size_t up_off, float limit, const void* xq,
                   size_t xq_stride, void* hq, const SharedArgs* sh, const WaitArgs& wait, cudaStream_t s) {
    if (cap_groups > kWMaxGroups) return kWindowTooWide;
    WArgs W = common(A, cap_groups, n_embd, n_ff, sh, wait);
    W.up_off = up_off; W.limit = limit;
    W.xq = (const uint8_t*) xq; W.xq_stride = xq_stride; W.hq = (uint8_t*) hq;
    if (sh == nullptr) return launch_window_type<false, true>(gu_type, W, s);
    W.sh = sh->blob;
    return launch_window_type<true, true>(gu_type, W, s);
}
int window_down(int d_type, const GroupArgs& A, int cap_groups, int n_embd, int n_ff, size_t down_off, const void* hq, float* part,
                const SharedArgs* sh, const WaitArgs& wait, cudaStream_t s) {
    if (cap_groups > kWMaxGroups) return kWindowTooWide;
    WArgs W = common(A, cap_groups, n_embd, n_ff, sh, wait);
    W.row_off = down_off;
    W.xq = (const uint8_t*) hq; W.xq_stride = (size_t) (n_ff / 32) * kQ81Bytes; W.part = part;
    if (sh == nullptr) return launch_window_type<false, false>(d_type, W, s);
    W.sh = sh->blob + 2 * (size_t) sh->n_ff * row_bytes(MAYA_Q8_0, n_embd);
    return launch_window_type<true, false>(d_type, W, s);
}

}  // namespace maya
