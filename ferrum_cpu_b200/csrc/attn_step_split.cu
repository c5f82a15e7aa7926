// The attention step with a cluster of CTAs a head (attn_step.cuh).
#include <climits>

#include "attn_step.cuh"

namespace fc {

namespace {

// CTAs that share a head: as many as its longest cache has parts for and as find room at the same time.
template <int HD>
int choose_split(int n_q, int ctx, int* split) {
    FC_TRY((prepare<HD, true>()));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(THREADS);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    for (*split = MAX_SPLIT; *split >= MIN_SPLIT; *split /= 2) {
        if ((*split - 1) * PART >= ctx) continue;
        int cap = 0, fit = 0;
        room<HD>(ctx, *split, &cap, &cfg.dynamicSmemBytes);
        cfg.gridDim = dim3(n_q * *split);
        attr[0].val.clusterDim.x = *split;
        FC_CUDA(cudaOccupancyMaxActiveClusters(&fit, attn_step_kernel<HD, true>, &cfg));
        if (fit >= n_q) return FC_OK;
    }
    *split = 1;
    return FC_OK;
}

}  // namespace

// Splitting a head pays once a part is long enough to outweigh the cluster's start and its meeting, which the layers behind
// it feel on every SM that holds a part. Us a token, one CTA a head against a shared head: 12 heads in 8 parts 217 against 229 at
// 32 positions, 231.5 against 231.4 at 128, 250 against 238 at 256, 477 against 257 at 900; 16 heads in 8 parts 476 against 478 at
// 128, 516 against 490 at 256, 1217 against 535 at 900; 32 heads in 4 parts 633 against 665 at 33, 672 against 686 at 256, 820
// against 702 at 512, 1208 against 730 at 1024. So: from 160 positions on with 8 parts, from 320 on with 4.
int attn_step_split(int n_q, int hd, int ctx, int* split, int* from) {
    *split = 1;
    *from = INT_MAX;
    if (!attn_step_covers(hd, ctx)) return FC_OK;
    FC_TRY(hd == 32 ? choose_split<32>(n_q, ctx, split) : hd == 64 ? choose_split<64>(n_q, ctx, split) : choose_split<128>(n_q, ctx, split));
    if (*split > 1) *from = 1280 / *split;
    return FC_OK;
}

int launch_attn_step_split(int hd, const AttnStep& a, const StepState* state, float* out, cudaStream_t st) {
    auto go = hd == 32 ? launch<32, true> : hd == 64 ? launch<64, true> : launch<128, true>;
    return go(a, state, out, st);
}

}  // namespace fc
