// The streaming kernel for scale groups of 64 and 32 (linear_mma_body.cuh: GROUP).  One row tile per warp and two splits of
// a tile's K between warps only: these shapes cover the others within a few per cent, and each is built twice here.
//
// Replaces the byte-at-a-time generic kernel for these groups: 8192 -> 8192, 64-wide groups, back to back: M = 1 196 -> 10.8 us,
// M = 4 218 -> 13.7, M = 64 1502 -> 96 (128-wide groups: 10.3, 13.3 and, by the GEMM, 33).
#include "linear_mma_variants.cuh"

namespace w4a16 {
namespace {

template <int GROUP, int NT, int XB, int KW>
bool pick_pipeline(const w4a16_linear_config& c, Variant* v) {
    if (c.unroll == 1) {
        if (c.stages != 3) return false;
        *v = variant_of<NT, XB, 1, KW, 1, 3, GROUP>();
        return true;
    }
    if (c.unroll != 2) return false;
    if (c.stages == 3) { *v = variant_of<NT, XB, 1, KW, 2, 3, GROUP>(); return true; }
    if (c.stages == 4) { *v = variant_of<NT, XB, 1, KW, 2, 4, GROUP>(); return true; }
    return false;
}

template <int GROUP, int NT, int XB>
bool pick_kw(const w4a16_linear_config& c, Variant* v) {
    if (c.row_tiles != 1) return false;
    if (c.k_warps == 2) return pick_pipeline<GROUP, NT, XB, 2>(c, v);
    if (c.k_warps == 8) return pick_pipeline<GROUP, NT, XB, 8>(c, v);
    return false;
}

template <int GROUP>
bool pick_batch(int nt, bool single_row, const w4a16_linear_config& c, Variant* v) {
    switch (nt) {
        case 1: return single_row ? pick_kw<GROUP, 1, 1>(c, v) : pick_kw<GROUP, 1, 8>(c, v);
        case 2: return pick_kw<GROUP, 2, 16>(c, v);
        case 4: return pick_kw<GROUP, 4, 32>(c, v);
        default: return false;
    }
}

}  // namespace

bool pick_group_variant(int group, int nt, bool single_row, const w4a16_linear_config& c, Variant* v) {
    if (group == 64) return pick_batch<64>(nt, single_row, c, v);
    if (group == 32) return pick_batch<32>(nt, single_row, c, v);
    return false;
}

}  // namespace w4a16
