// The streaming kernel's instantiations as the launch code sees them.  The ones for 128-wide groups are built in
// linear_mma.cu, those for smaller groups in linear_mma_groups.cu.
#pragma once

#include "kernels.h"
#include "linear_mma_body.cuh"

namespace w4a16 {

struct Variant {
    const void* fn;
    const void* fn_exchange;   // the build with the tensor-parallel paths; null where it is not instantiated
    const void* fn_early;      // the build for early weights and no bias; null where it is not instantiated
    int red_bytes;     // shared memory for the cross-warp reduction
    int stage_bytes;   // shared memory of one pipeline stage
    int stages;
    int x_rows;        // batch rows stored per chunk of x (XB)
};

// nt: n8 tiles of the batch (1, 2 or 4); false when the shape is not built (one row tile per warp, k_warps 2 or 8).
bool pick_group_variant(int group, int nt, bool single_row, const w4a16_linear_config& c, Variant* v);

namespace {

// Hooks of the stand-alone kernel: programmatic dependent launch on the way in, nothing on the way out.
struct KernelHooks {
    // The successor is released with the very first instruction: its CTAs only take SM resources this grid does not
    // use, and the earlier they are resident the more of their prologue and weight prefetch hides under this grid.
    __device__ __forceinline__ void at_start() { pdl_release_downstream(); }
    __device__ __forceinline__ bool weights_wait(const MmaParams& p) const { return p.early_weights == 0; }
    __device__ __forceinline__ void before_activations() { pdl_wait_for_upstream(); }
    __device__ __forceinline__ void after_outputs() {}
};

template <int NT, int XB, int TILES, int KW, int U, int STAGES, int GROUP>
__global__ void __launch_bounds__(kThreads, min_ctas_per_sm<NT, TILES>())
linear_mma_kernel(const MmaParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    KernelHooks hooks;
    linear_mma_body<NT, XB, TILES, KW, U, STAGES, GROUP, 0>(p, smem, hooks);
}

// The same kernel with the tensor-parallel sender and reader paths compiled in (launches that carry a
// w4a16_peer_target or a w4a16_peer_source).
template <int NT, int XB, int TILES, int KW, int U, int STAGES>
__global__ void __launch_bounds__(kThreads, min_ctas_per_sm<NT, TILES>())
linear_mma_exchange_kernel(const MmaParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    KernelHooks hooks;
    linear_mma_body<NT, XB, TILES, KW, U, STAGES, kGroup, kFeatExchange>(p, smem, hooks);
}

// The same kernel for a single row whose weights are in place, without a bias.
template <int KW, int U, int STAGES>
__global__ void __launch_bounds__(kThreads, min_ctas_per_sm<1, 1>())
linear_mma_early_kernel(const MmaParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    KernelHooks hooks;
    linear_mma_body<1, 1, 1, KW, U, STAGES, kGroup, kFeatEarly>(p, smem, hooks);
}

template <int NT, int XB, int TILES, int KW, int U, int STAGES, int GROUP>
Variant variant_of() {
    constexpr int RW = kWarpsPerCta / KW;
    constexpr int red = KW > 1 ? 2 * KW * TILES * NT * 4 * 32 * RW * static_cast<int>(sizeof(float)) : 0;
    const void* exchange = nullptr;
    if constexpr (TILES == 1 && GROUP == kGroup) {   // sharded layers always run one 16-row tile per warp
        exchange = reinterpret_cast<const void*>(&linear_mma_exchange_kernel<NT, XB, TILES, KW, U, STAGES>);
    }
    const void* early = nullptr;
    if constexpr (XB == 1 && TILES == 1 && GROUP == kGroup) early = reinterpret_cast<const void*>(&linear_mma_early_kernel<KW, U, STAGES>);
    return {reinterpret_cast<const void*>(&linear_mma_kernel<NT, XB, TILES, KW, U, STAGES, GROUP>), exchange, early, red,
            stage_bytes<TILES, U, GROUP>(), STAGES, XB};
}

}  // namespace
}  // namespace w4a16
