// rt_plane.cuh -- what the two bit-plane kernels share.
#pragma once

#include "rt_internal.h"

namespace rtb {

template <int FAM>
struct PlaneModel {
    static constexpr bool DOM = FAM != FAM_LOZENGE8;
    static constexpr int NC = DOM ? 2 : 3;  // colour arrays
    static constexpr int NP = DOM ? 4 : 6;  // bit planes per colour
    static constexpr int ROFF = DOM ? 1 : 0;
    static constexpr int COFF = DOM ? 1 : 0;
};

__device__ __forceinline__ uint32_t col_next(uint32_t cur, uint32_t nxt) { return __funnelshift_r(cur, nxt, 1); }
__device__ __forceinline__ uint32_t col_prev(uint32_t prv, uint32_t cur) { return __funnelshift_l(prv, cur, 1); }

// Bits [lo, hi) of the 32 columns starting at column 32 w.
__device__ __forceinline__ uint32_t col_mask(int w, int lo, int hi) {
    const int a = max(lo - 32 * w, 0), b = min(hi - 32 * w, 32);
    if (b <= a) return 0u;
    const uint32_t upper = b >= 32 ? 0xffffffffu : ((1u << b) - 1u);
    return upper & ~((1u << a) - 1u);
}

// Plans the walk with one word per thread (rt_planeband.cu); an error if the
// bands do not fit it.
rt_status plan_plane_band(int family, int device, int nlat, int rows, int width, int ctas_hint, int depth_hint,
                          WalkPlan* plan, std::string* err);

}  // namespace rtb
