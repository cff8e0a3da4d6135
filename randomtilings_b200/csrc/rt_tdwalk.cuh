// rt_tdwalk.cuh -- a band of a triangle-dimer chain as bit planes in shared
// memory, and one phase of the phase program on it: what the batched kernel
// (rt_batch.cu) and the single walk (rt_td.cu) share.
//
// A chain's rows are split over the CTAs of a cluster.  A CTA holds the planes
// (rt_tdplane.cuh) of its rows and of `halo` rows above and below, which it
// computes itself: a phase that reads neighbouring rows leaves one row less of
// the halo current, and when none is left the CTAs store their edge rows into
// each other's halos (distributed shared memory).  So most phases end with a
// block barrier, and the two cluster barriers of an exchange, with the fences
// they carry, come once in eight to ten phases.
#pragma once

#include <cooperative_groups.h>

#include "rt_device.cuh"
#include "rt_tdplane.cuh"
#include "rt_tridimer.cuh"

namespace cg = cooperative_groups;

namespace rtb {

// Halo rows of a band when `rows` rows are split over `ctas` CTAs (a lattice on
// one CTA has one empty row on either side): at most `cap`.  Halo rows cost
// words to compute and, with generators, decisions to make; an exchange costs
// about 3 us.  136 rows on 16 CTAs, us per step: Philox 3.86, 3.84, 3.89 at
// caps 8, 12, 16; TinyMT 5.66, 5.52, 5.69 at 4, 6, 8.
__host__ __device__ inline int td_halo(int rows, int ctas, int cap) {
    return ctas == 1 ? 1 : (rows / ctas < cap ? rows / ctas : cap);
}
__host__ __device__ constexpr int td_halo_cap(bool philox) { return philox ? 12 : 6; }
// First row of CTA `rank`: every band has floor or ceil(rows / ctas) rows.
__host__ __device__ inline int td_first_row(int rows, int ctas, int rank) {
    return (int)((int64_t)rank * rows / ctas);
}
// Words of shared memory a band takes: one zero word, then per plane its rows
// and halo rows of wb + 1 words (the last word of a row stays zero).
__host__ __device__ inline size_t td_band_words(int rows, int width, int ctas, int cap, int planes) {
    const int rpc = (rows + ctas - 1) / ctas;
    return 1 + (size_t)planes * (rpc + 2 * td_halo(rows, ctas, cap)) * (((width + 31) >> 5) + 1);
}

// Rows by which phase d's results depend on neighbouring rows.
__device__ __forceinline__ int td_reach(uint32_t d) {
    const uint32_t op = ph_op(d);
    return (op == TD_ROT_LOZ || op == TD_ROT_TRI || op == TD_ROT_BFLY || op == TD_LOZ_FROM_BFLY ||
            (op == TD_BFLY_SAME && ph_a(d) == 0))
               ? 0
               : 1;
}

// The view of a thread's words: all of one word column, whose lane masks the
// thread keeps.
template <class BITS>
struct TdView : tdp::ViewOf<BITS> {
    uint32_t inner, used;
    int c2;  // 2 c mod 3
    __device__ __forceinline__ uint32_t inner_cols(int) const { return inner; }
    __device__ __forceinline__ uint32_t used_cols(int) const { return used; }
    __device__ __forceinline__ uint32_t cols_mod3(int r) const {
        const int k = r - c2;  // 0x49249249 << k: the lanes l = k (mod 3)
        return 0x49249249u << (k < 0 ? k + 3 : k);
    }
};

template <class BITS>
struct TdBand {
    uint32_t* planes;  // plane 0, row 0 (array row row0), word 0
    int ps, rs, wb;    // plane and row strides in words, words per row
    int r0, r1;        // array rows of the band
    int row0, halo, depth;  // depth: halo rows that are current
    int rows, m, width, rank, ctas;
    // This thread's words: column c of rows g, g + stride, ... of a phase's rows
    // (idle: g beyond the threads that make up whole rows).
    int g, stride;
    bool idle;
    TdView<BITS> view;
    // Its words of an exchange: column xc of halo row xh, of every xstride-th
    // plane from xp on; arrays written since the last exchange.
    int xc, xh, xp, xstride;
    uint32_t written;

    // ctas: CTAs that hold rows; a CTA of rank >= ctas has none.
    __device__ __forceinline__ TdBand(uint32_t* smem, int rows_, int width_, int m_, int rank_, int cluster, int cap,
                                      int tid, int BLOCK) {
        rows = rows_, width = width_, m = m_, rank = rank_;
        ctas = min(cluster, rows);
        halo = depth = td_halo(rows, ctas, cap);
        planes = smem + 1;
        wb = (width + 31) >> 5;
        rs = wb + 1;
        ps = ((rows + ctas - 1) / ctas + 2 * halo) * rs;
        r0 = rank < ctas ? td_first_row(rows, ctas, rank) : rows;
        r1 = rank < ctas ? td_first_row(rows, ctas, rank + 1) : rows;
        row0 = r0 - halo;
        stride = BLOCK / wb;
        const int c = tid % wb;
        g = tid / wb;
        idle = g >= stride || r0 == r1;
        static_cast<tdp::ViewOf<BITS>&>(view) = tdp::ViewOf<BITS>{planes, ps, rs, row0, 0, c};
        view.inner = tdp::col_range(c, 1, m - 2);
        view.used = tdp::col_range(c, 0, width - 1);
        view.c2 = 2 * c % 3;
        const int per = halo * wb;  // words of a plane that a side exchanges
        xc = c;
        xh = tid / wb % halo;
        xp = tid / per;
        xstride = BLOCK / per;  // 0: fewer threads than words
        if (xp >= xstride) xp = BITS::planes;
        written = 0u;
    }

    // Stores this CTA's edge rows into the neighbours' halos.  All threads of the
    // cluster; ends with every halo current.
    __device__ __forceinline__ void exchange(cg::cluster_group& cluster) {
        cluster.sync();  // the neighbours are done with the halo rows they have
        if (r0 < r1) {
            uint32_t* up = rank > 0 ? cluster.map_shared_rank(planes, rank - 1) : nullptr;
            uint32_t* dn = rank + 1 < ctas ? cluster.map_shared_rank(planes, rank + 1) : nullptr;
            const int up_row = halo + r0 - (rank > 0 ? td_first_row(rows, ctas, rank - 1) : 0);  // below its rows
            auto word = [&](int p, int h, int c) {
                const uint32_t* mine = planes + p * ps + c;
                if (up) up[p * ps + (up_row + h) * rs + c] = mine[(halo + h) * rs];
                if (dn) dn[p * ps + h * rs + c] = mine[(r1 - r0 + h) * rs];
            };
            for (uint32_t w = written; w; w &= w - 1) {
                const int arr = __ffs((int)w) - 1, p0 = BITS::plane_of(arr), n = BITS::bits_of(arr);
                if (xstride > 0)
                    for (int k = xp; k < n; k += xstride) word(p0 + k, xh, xc);
                else if (!idle)
                    for (int k = 0; k < n; ++k)
                        for (int h = g; h < halo; h += stride) word(p0 + k, h, xc);
            }
        }
        cluster.sync();
        depth = halo;
        written = 0u;
    }
};

// Global int32 rows of the band and its halo -> planes (cleared before); one
// warp per 32 columns, with a ballot per bit.
template <class BITS>
__device__ __forceinline__ void td_load(const TdBand<BITS>& b, void* const* arr, int arows, int warp, int nwarps, int lane) {
    for (int it = warp; it < (b.r1 - b.r0 + 2 * b.halo) * 8 * b.wb; it += nwarps) {
        const int sr = it / (8 * b.wb), rem = it - sr * 8 * b.wb, a = rem / b.wb, c = rem - a * b.wb;
        const int rr = b.row0 + sr, j = 32 * c + lane;
        int32_t v = 0;
        if (rr >= 0 && rr < arows && j < b.width) v = static_cast<const int32_t*>(arr[a])[(size_t)rr * b.width + j];
        for (int k = 0; k < BITS::bits_of(a); ++k) {
            const uint32_t w = __ballot_sync(0xffffffffu, (v >> k) & 1);
            if (lane == 0) b.planes[(BITS::plane_of(a) + k) * b.ps + sr * b.rs + c] = w;
        }
    }
}
// planes -> global int32 rows r0 .. r1 - 1
template <class BITS>
__device__ __forceinline__ void td_store(const TdBand<BITS>& b, void* const* arr, int warp, int nwarps, int lane) {
    for (int it = warp; it < (b.r1 - b.r0) * 8 * b.wb; it += nwarps) {
        const int rr = it / (8 * b.wb), sr = b.halo + rr, rem = it - rr * 8 * b.wb, a = rem / b.wb, c = rem - a * b.wb;
        const int j = 32 * c + lane;
        int32_t v = 0;
        for (int k = 0; k < BITS::bits_of(a); ++k)
            v |= (int32_t)((b.planes[(BITS::plane_of(a) + k) * b.ps + sr * b.rs + c] >> lane) & 1u) << k;
        if (j < b.width) static_cast<int32_t*>(arr[a])[(size_t)(b.r0 + rr) * b.width + j] = v;
    }
}

// The fast mode's draws of the lanes F of array row r, word c: quad cq of the
// row is Philox4x32-10 of (r Gw + cq, step, chain), and a site flips when its
// output word is below 2^31 (k = word >> 9 below 2^22).  Few sites of a word
// can flip, so only the quads that hold one are drawn: 1 to 3 of 8.
struct TdPhilox {
    int Gw;
    int64_t step;
    uint32_t chain, key0, key1;
    __device__ __forceinline__ uint32_t operator()(int r, int c, uint32_t F) const {
        uint32_t out = 0u;
        while (F) {
            const int q = (__ffs((int)F) - 1) >> 2;
            const uint4 w = philox4((uint32_t)(r * Gw + 8 * c + q), (uint32_t)step, (uint32_t)((uint64_t)step >> 32), chain,
                                    key0, key1);
            out |= ((~w.x >> 31) | ((~w.y >> 31) << 1) | ((~w.z >> 31) << 2) | ((~w.w >> 31) << 3)) << (4 * q);
            F &= ~(15u << (4 * q));
        }
        return out;
    }
};

// Phase (OP, a, b) on rows lo .. hi - 1: only those TriDimerRule::live_rows
// admits, one 32-site word per work item.
template <uint32_t OP, int T, int B, class BITS, class Draw>
__device__ __forceinline__ void td_op(const TdBand<BITS>& d, int lo, int hi, uint32_t a, uint32_t b, const Draw& draw) {
    constexpr bool DRAWS = OP == TD_ROT_LOZ || OP == TD_ROT_TRI || OP == TD_ROT_BFLY;
    int S, o;
    TriDimerRule::live_rows<OP>(T >= 0 ? (uint32_t)T : a, b, &S, &o);
    TdView<BITS> v = d.view;
    for (v.i = lo + ((o - lo) % S + S) % S + S * d.g; v.i < hi; v.i += S * d.stride) {
        if (DRAWS) {
            uint32_t F = tdp::rot_mask<OP, T>(v, a, b, d.width);
            if (F) F &= draw(v.i, v.c, F);
            if (F) tdp::rot_flip<OP, T>(v, a, F);
        } else {
            tdp::word_op<OP, T, B>(v, a, b, d.m, d.width, 0u);
        }
    }
}

template <class BITS, class Draw>
__device__ __forceinline__ void td_phase(uint32_t d, TdBand<BITS>& band, const Draw& draw) {
    const uint32_t pa = ph_a(d), pb = ph_b(d);
    // the band's rows and the halo rows that can be kept current
    const int keep = band.ctas == 1 ? 0 : band.depth - td_reach(d);
    const int lo = max(0, band.r0 - keep), hi = min(band.rows, band.r1 + keep);
    if (band.ctas > 1) {
        band.depth = keep;
        band.written |= TriDimerRule::written(d);
    }
    if (band.idle) return;
    switch (ph_op(d)) {
#define RT_TD_PHASE(OP)                                               \
    case OP:                                                          \
        if (pa == 0)                                                  \
            td_op<OP, 0, -1>(band, lo, hi, pa, pb, draw);         \
        else if (pa == 1)                                             \
            td_op<OP, 1, -1>(band, lo, hi, pa, pb, draw);         \
        else                                                          \
            td_op<OP, 2, -1>(band, lo, hi, pa, pb, draw);         \
        break;
        RT_TD_PHASE(TD_ROT_LOZ)
        RT_TD_PHASE(TD_LOZ_FLIPPED)
        RT_TD_PHASE(TD_LOZ_OTHER)
        RT_TD_PHASE(TD_ROT_BFLY)
        RT_TD_PHASE(TD_BFLY_SAME)
        RT_TD_PHASE(TD_BFLY_21)
        RT_TD_PHASE(TD_BFLY_22)
        RT_TD_PHASE(TD_BFLY_23)
        RT_TD_PHASE(TD_LOZ_FROM_BFLY)
#undef RT_TD_PHASE
#define RT_TD_PHASE2(OP, B)                                           \
    case OP:                                                          \
        if (pa == 0)                                                  \
            td_op<OP, 0, B>(band, lo, hi, pa, pb, draw);          \
        else                                                          \
            td_op<OP, 1, B>(band, lo, hi, pa, pb, draw);          \
        break;
        RT_TD_PHASE2(TD_TRI_OTHER, 0)
        RT_TD_PHASE2(TD_ROT_TRI, -1)
        RT_TD_PHASE2(TD_TRI_FLIPPED, -1)
#undef RT_TD_PHASE2
        case TD_UP_FROM_LOZ: td_op<TD_UP_FROM_LOZ, 0, 0>(band, lo, hi, pa, pb, draw); break;
        case TD_LOZ_FROM_TRI: td_op<TD_LOZ_FROM_TRI, 0, 0>(band, lo, hi, pa, pb, draw); break;
        case TD_BFLY_FROM_LOZ:
            if (pa == 0 && pb == 1)
                td_op<TD_BFLY_FROM_LOZ, 0, 1>(band, lo, hi, pa, pb, draw);
            else if (pa == 0 && pb == 2)
                td_op<TD_BFLY_FROM_LOZ, 0, 2>(band, lo, hi, pa, pb, draw);
            else if (pa == 0 && pb == 4)
                td_op<TD_BFLY_FROM_LOZ, 0, 4>(band, lo, hi, pa, pb, draw);
            else
                td_op<TD_BFLY_FROM_LOZ, -1, -1>(band, lo, hi, pa, pb, draw);
            break;
        default: break;
    }
}

}  // namespace rtb
