// The attention step with one CTA a head, and the choice between that and several (attn_step.cuh).
#include "attn_step.cuh"

namespace fc {

// Other widths of a head, and contexts whose scores alone fill shared memory, keep the kernels that read the caches in place.
bool attn_step_covers(int hd, int ctx) { return (hd == 32 || hd == 64 || hd == 128) && (size_t)ctx * 4 <= kSmem; }

int launch_attn_step(const float* qkv, int n_q, int n_kv, int hd, int rope_dim, int neox, const float2* ftab, float inv_linear,
                     float* kc, float* vc, int ctx, int split, const StepState* state, float* out, cudaStream_t st) {
    if (!attn_step_covers(hd, ctx)) return fail(FC_E_SHAPE, "attention step: heads of %d, context %d", hd, ctx);
    const AttnStep a = {qkv, n_q, n_kv, rope_dim / 2, neox, ftab, inv_linear, kc, vc, ctx, split};
    if (split > 1) return launch_attn_step_split(hd, a, state, out, st);
    auto go = hd == 32 ? launch<32, false> : hd == 64 ? launch<64, false> : launch<128, false>;
    return go(a, state, out, st);
}

}  // namespace fc
