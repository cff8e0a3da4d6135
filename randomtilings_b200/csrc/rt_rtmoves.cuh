// rt_rtmoves.cuh -- the rectangle-triangle moves as a table of whole-number tests.
//
// The flip rule (RectTriRule::flip) divides and multiplies floats, but which
// quarter a draw k falls into depends on k alone, and within a quarter the
// rescaled draw never falls as k grows: a move is kept for every k below one
// bound.  A CTA finds the bounds of its weights once, with the rule's own float
// operations, and a flip is one 16-byte load and two compares (a step of a
// 147-site lattice takes 0.40 us, 1.17 with the rule evaluated in place).
#pragma once

#include "rt_models.cuh"

namespace rtb {

// The first draw of quarter q; of q = 4, the first that proposes nothing.
// k 2^-23 is exact, as in single01().
constexpr uint32_t rt_quarter(int q) {
    uint32_t lo = 0, hi = 1u << 23;
    while (lo < hi) {
        const uint32_t k = lo + (hi - lo) / 2;
        const float rd = (float)k * (1.0f / 8388608.0f);
        if (q == 4 ? rd < 0.9f : rd / 0.9f < 0.25f * (float)q)
            lo = k + 1;
        else
            hi = k;
    }
    return lo;
}
constexpr uint32_t kRtQuarter1 = rt_quarter(1), kRtQuarter2 = rt_quarter(2), kRtQuarter3 = rt_quarter(3),
                   kRtDraws = rt_quarter(4);

constexpr int kRtStates = 17;  // states that move
struct RtStates {
    uint32_t v[kRtStates] = {0x122133, 0x331221, 0x8ebbe8, 0xfc99cf, 0xa7dd7a, 0x47d47a, 0xd22a33, 0xa74d74, 0x33a22d,
                             0x8eb558, 0x331eb1, 0x855be8, 0x1be133, 0x6699cf, 0xcf1221, 0xfc9966, 0x1221fc};
};
// Slot of a state: the top bits of a product, one state a slot.
__host__ __device__ constexpr uint32_t rt_slot(uint32_t v) { return (v * 0xc324c985u) >> 27; }
constexpr bool rt_slots_differ() {
    const RtStates states;
    uint32_t seen = 0;
    for (uint32_t v : states.v) {
        if (seen >> rt_slot(v) & 1u) return false;
        seen |= 1u << rt_slot(v);
    }
    return true;
}
static_assert(rt_slots_differ(), "two moving states share a slot");

// updateTiles (recttrianglekernel.cl:120-146): the colour after the one flipped,
// and the one after that, from neighbours of the flipped colour.
__device__ __forceinline__ int rt_next(int up, int east, int low) {
    return ((up & 0xff) << 16) | ((east >> 8) & 0xf00f) | ((low >> 8) & 0xff0);
}
__device__ __forceinline__ int rt_next2(int west, int upr, int down) {
    return ((west << 8) & 0xf00f00) | ((upr << 8) & 0xff000) | ((down >> 16) & 0xff);
}

struct RectTriMoves {
    uint4 move[32 * 4];  // [slot][quarter]: state, state proposed, bound of the draws that keep it

    __device__ void clear(int tid, int threads) {
        for (int e = tid; e < 32 * 4; e += threads) move[e] = make_uint4(0u, 0u, 0u, 0u);
    }
    // After clear() and a barrier; a barrier follows.
    template <class A>
    __device__ void fill(const A& a, int tid, int threads) {
        for (int e = tid; e < kRtStates * 4; e += threads) {
            const int q = e & 3;
            constexpr RtStates states;
            uint32_t v = states.v[0];
#pragma unroll
            for (int k = 1; k < kRtStates; ++k)
                if (e >> 2 == k) v = states.v[k];
            uint32_t lo = q == 0 ? 0u : q == 1 ? kRtQuarter1 : q == 2 ? kRtQuarter2 : kRtQuarter3;
            uint32_t hi = q == 0 ? kRtQuarter1 : q == 1 ? kRtQuarter2 : q == 2 ? kRtQuarter3 : kRtDraws;
            int nv = 0;
            const int kind = RectTriRule::propose((int)v, q, nv);
            const float ratio = __fdiv_rn(RectTriRule::weight(a, nv), RectTriRule::weight(a, (int)v));
            if (RectTriRule::kept(ratio, kind, q, hi - 1u)) {
                lo = hi;  // every draw (weights that do not fall)
            } else {
                while (lo < hi) {
                    const uint32_t k = lo + (hi - lo) / 2u;
                    if (RectTriRule::kept(ratio, kind, q, k))
                        lo = k + 1u;
                    else
                        hi = k;
                }
            }
            move[rt_slot(v) * 4 + q] = make_uint4(v, (uint32_t)nv, lo, 0u);
        }
    }
    // A draw with its quarter in the top bits; draws that propose nothing lie
    // above every bound.
    __device__ static uint32_t prepare(uint32_t k) {
        return k | ((uint32_t)(k >= kRtQuarter1) + (uint32_t)(k >= kRtQuarter2) + (uint32_t)(k >= kRtQuarter3)) << 23;
    }
    __device__ int flip(int v, uint32_t draw) const {
        const uint4 m = move[rt_slot((uint32_t)v) * 4 + (draw >> 23)];
        return (uint32_t)v == m.x && (draw & 0x7fffffu) < m.z ? (int)m.y : v;
    }
};

}  // namespace rtb
