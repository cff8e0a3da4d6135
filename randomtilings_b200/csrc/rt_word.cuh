// rt_word.cuh -- word-parallel site arithmetic of the int8 models
// (dominoes, uniform lozenges): four sites of a colour-array row per 32-bit
// word.  Used by the single-walk word kernel (rt_word.cu) and the batched
// kernels (rt_batch.cu).
#pragma once

#include "rt_internal.h"
#include "rt_models.cuh"

namespace rtb {

// 0xff in byte b iff (w[b] >> 9) < thr_b: the top byte of the difference of
// two numbers up to 2^23 is its sign.  n_b = -thr_b.
__device__ __forceinline__ uint32_t below4(const uint32_t (&w)[4], uint32_t n0, uint32_t n1, uint32_t n2, uint32_t n3) {
    const uint32_t lo = __byte_perm((w[0] >> 9) + n0, (w[1] >> 9) + n1, 0x0073);
    const uint32_t hi = __byte_perm((w[2] >> 9) + n2, (w[3] >> 9) + n3, 0x7300);
    return __byte_perm(lo, hi, 0x7610);
}
__device__ __forceinline__ uint32_t below4(const uint32_t (&w)[4], uint32_t n) { return below4(w, n, n, n, n); }

__device__ __forceinline__ uint32_t lds(const unsigned char* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ void sts(unsigned char* p, uint32_t v) { *reinterpret_cast<uint32_t*>(p) = v; }
// old where mask is clear, nw where it is set
__device__ __forceinline__ uint32_t merge(uint32_t old, uint32_t nw, uint32_t mask) { return (old & ~mask) | (nw & mask); }

// Fixed facts of one word of the band: its byte offset in a colour plane, its
// row's class (lozenges: i mod 3; dominoes: i mod 2), and two byte masks: `um`
// (0xff) marks the sites an Update refreshes (1 <= i <= N-2, 1 <= j <=
// width-2), `vm` (0x80) the sites that are Rotate positions.
struct WordInfo {
    int off;
    int cls;
    uint32_t um;
    uint32_t vm;
};

template <int FAM>
struct WordModel {
    static constexpr bool DOM = FAM != FAM_LOZENGE8;
    static constexpr int NC = DOM ? 2 : 3;
    static constexpr int ROFF = DOM ? 1 : 0;
    static constexpr int COFF = DOM ? 1 : 0;
    __device__ static uint32_t written(uint32_t d) {
        if (ph_op(d) != OP_STEP) return 0u;
        return 1u << (DOM ? 1 - (int)ph_a(d) : (int)ph_a(d));
    }
};

// Decoded phase descriptor.  dst: byte offset of the plane written (dominoes:
// the array flipped or, at the end, refreshed; lozenges: the colour flipped
// or, at the end, t+1); src: of the flipped colour t whose Update is pending;
// oth (lozenges): of the other colour that Update refreshes.  flags: the
// WP_* bits, the pending Update's colour t in bits 8..9.
enum : uint32_t { WP_STEP = 1u, WP_UPD = 2u, WP_NEXT = 4u /* dst is colour t+1 */ };
struct __align__(16) WordPhase {
    int dst, src, oth;
    uint32_t flags;
    __device__ __forceinline__ int t() const { return (int)(flags >> 8) & 3; }
};

// Phases take few values, so they are decoded once, into a table.
constexpr int kWordPhases = 32;
__device__ __forceinline__ int word_phase_index(uint32_t d) {
    return (int)(((d & OP_FINAL) << 3) | ((d >> 6) & 12u) | ((d >> 16) & 3u));
}
// Entry `idx` of the table for planes of `plane` bytes.
template <int FAM>
__device__ __forceinline__ WordPhase word_phase_entry(int idx, int plane) {
    const bool step = !(idx & 16);
    const int ca = (idx >> 2) & 3, cb = idx & 3;  // cb = 3: none
    const bool upd = step ? (cb != 3 && cb != ca) : true;
    const int t = step ? (upd ? cb : 0) : ca;
    WordPhase P;
    P.flags = (step ? WP_STEP : 0u) | (upd ? WP_UPD : 0u) | ((uint32_t)t << 8);
    if (FAM != FAM_LOZENGE8) {
        // Reference colour r flips array 1 - r, then refreshes array r from it.
        const int dst = step ? 1 - ca : ca;
        P.dst = dst * plane;
        P.src = (1 - dst) * plane;
        P.oth = 0;
    } else {
        const int t1 = t == 2 ? 0 : t + 1, t2 = t == 0 ? 2 : t - 1;
        const bool next = !step || ca == t1;
        P.dst = (step ? ca : t1) * plane;
        P.src = t * plane;
        P.oth = (next ? t2 : t1) * plane;
        if (next) P.flags |= WP_NEXT;
    }
    return P;
}

// Byte selectors of the lozenge column shifts for pending colour t and row
// class i mod 3 (index 3 t + class): the reads from the row above (x: words
// w, w+1), the row below (y: w-1, w), the left (z: w-1, w) and the right
// (w: w, w+1).  Exactly one of the three shifts applies in a row.
constexpr int kLozengeSel = 9;
__device__ __forceinline__ uint4 lozenge_sel_entry(int e) {
    const int t = e / 3, cls = e % 3;
    const bool sa = cls == (2 * t + 1) % 3, sw = cls == (2 * t + 2) % 3, se = cls == (2 * t) % 3;
    return make_uint4(sa ? 0x4321u : 0x3210u, sa ? 0x6543u : 0x7654u, sw ? 0x6543u : 0x7654u, se ? 0x4321u : 0x3210u);
}

// The words of the flipped colour in the rows next to a word's row, as its
// Update reads them: dominoes up[0] and dn[0] (same column); lozenges also
// up[1] (the next word of the row above) and dn[1] (the previous word of the
// row below).
struct WordNbr {
    uint32_t up[2], dn[2];
};

// One phase on one word of one lattice (planes at `lat`, a pending Update or
// none), in two parts: `begin` reads the word and its own row (sel_tab: the
// column shifts, null where no table is at hand), `finish` takes the rows next to
// it.  m0 / m1: byte masks (0xff) of the phase's draws -- dominoes: m0 where the
// site toggles (heat bath: becomes 12, else 3); lozenges: m0 where a cube is added,
// m1 where one is removed.
template <int FAM>
struct WordOp {
    static constexpr bool DOM = FAM != FAM_LOZENGE8;
    uint32_t v, o;    // the word written; lozenges: the other refreshed colour's
    uint32_t ta, tb;  // the own row's share of the refreshed bits (dominoes: ta)
    uint4 sel;

    __device__ __forceinline__ void begin(const unsigned char* lat, const WordPhase& P, const WordInfo& wi,
                                          const uint4* sel_tab) {
        v = lds(lat + P.dst + wi.off);
        if (!(P.flags & WP_UPD)) return;
        const unsigned char* f = lat + P.src + wi.off;
        const uint32_t l = lds(f - 4), c = lds(f), r = lds(f + 4);
        if (DOM) {
            // UpdateTiles (dominokernel.cl:22-31): edge bits 1 up, 2 down, 4 towards
            // j-1, 8 towards j+1; the neighbour towards j+1 shares the column in rows
            // with i + t odd, towards j-1 in the others.
            const uint32_t p = (uint32_t)((wi.cls ^ P.t()) & 1) * 0x1111u;
            const uint32_t west = __byte_perm(l, c, 0x6543u + p), east = __byte_perm(c, r, 0x3210u + p);
            ta = ((west >> 1) & 0x04040404u) | ((east << 1) & 0x08080808u);
        } else {
            // UpdateTiles (lozengekernel.cl:36-54): colour t+1 keeps all but bits
            // {2,4,32} and takes them from f[i-1][j+sa], f[i][j-sw], f[i+1][j]; colour
            // t+2 keeps all but {1,8,16} and takes them from f[i-1][j], f[i][j+se],
            // f[i+1][j-sa].  The bit fields never overlap: sums are ORs.
            sel = sel_tab ? sel_tab[3 * P.t() + wi.cls] : lozenge_sel_entry(3 * P.t() + wi.cls);
            o = lds(lat + P.oth + wi.off);
            ta = (__byte_perm(l, c, sel.z) >> 1) & 0x04040404u;
            tb = (__byte_perm(c, r, sel.w) << 1) & 0x08080808u;
        }
    }
    // Rows above and below from the band in shared memory (row stride W).
    __device__ __forceinline__ static void load_up(WordNbr& nb, const unsigned char* lat, const WordPhase& P,
                                                   const WordInfo& wi, int W) {
        const unsigned char* f = lat + P.src + wi.off - W;
        nb.up[0] = lds(f);
        nb.up[1] = DOM ? 0u : lds(f + 4);
    }
    __device__ __forceinline__ static void load_dn(WordNbr& nb, const unsigned char* lat, const WordPhase& P,
                                                   const WordInfo& wi, int W) {
        const unsigned char* f = lat + P.src + wi.off + W;
        nb.dn[0] = lds(f);
        nb.dn[1] = DOM ? 0u : lds(f - 4);
    }
    __device__ __forceinline__ void finish(const WordPhase& P, const WordInfo& wi, const WordNbr& nb, uint32_t m0,
                                           uint32_t m1) {
        if (P.flags & WP_UPD) {
            if (DOM) {
                const uint32_t x = ((nb.up[0] >> 1) & 0x01010101u) | ta;
                v = merge(v, ((nb.dn[0] << 1) & 0x02020202u) | x, wi.um);
            } else {
                const uint32_t fu = __byte_perm(nb.up[0], nb.up[1], sel.x), fd = __byte_perm(nb.dn[1], nb.dn[0], sel.y);
                const uint32_t na = ((nb.dn[0] << 5) & 0x20202020u) | (((fu >> 3) & 0x02020202u) | ta);
                const uint32_t nbv = ((fd << 3) & 0x10101010u) | (((nb.up[0] >> 5) & 0x01010101u) | tb);
                const uint32_t ma = wi.um & 0x26262626u, mb = wi.um & 0x19191919u;
                const bool next = (P.flags & WP_NEXT) != 0u;
                v = merge(v, next ? na : nbv, next ? ma : mb);
                o = merge(o, next ? nbv : na, next ? mb : ma);
            }
        }
        if (P.flags & WP_STEP) {
            // bit 7 of a byte of z is clear iff the byte equals the pattern (bytes < 0x80)
            uint32_t tog;
            if (DOM) {
                const uint32_t z3 = (v ^ 0x03030303u) + 0x7f7f7f7fu, z12 = (v ^ 0x0c0c0c0cu) + 0x7f7f7f7fu;
                if (FAM == FAM_DOMINO_HB)  // dominokernelCFTP.cl:19-28
                    tog = (~z3 & m0) | (~z12 & ~m0);
                else  // dominokernel.cl:11-17
                    tog = ~(z3 & z12) & m0;
            } else {  // lozengekernel.cl:19-31: a cube is added (25 -> 38) or removed (38 -> 25)
                const uint32_t z25 = (v ^ 0x19191919u) + 0x7f7f7f7fu, z38 = (v ^ 0x26262626u) + 0x7f7f7f7fu;
                tog = (~z25 & m0) | (~z38 & m1);
            }
            // 0x80 per toggled site -> 15 or 63 per byte: the high word of a product
            v ^= __umulhi(tog & wi.vm, (DOM ? 15u : 63u) << 25);
        }
    }
    __device__ __forceinline__ void store(unsigned char* lat, const WordPhase& P, const WordInfo& wi) const {
        sts(lat + P.dst + wi.off, v);
        if (!DOM && (P.flags & WP_UPD)) sts(lat + P.oth + wi.off, o);
    }
};

// 0x01 per byte of the bits set in mask, one bit per byte index.
__device__ __forceinline__ uint32_t lane_bytes(uint32_t bits) {
    return (bits & 1u) | ((bits & 2u) << 7) | ((bits & 4u) << 14) | ((bits & 8u) << 21);
}

// What the draws k of one step do to the word at array row i, columns c0 .. c0 + 3,
// as the byte masks of WordOp: combined into m0 / m1, which hold what the run's
// earlier steps did.  Within a run the sites' neighbours do not change, so a
// rotatable site stays rotatable: toggles add up modulo 2, and of the other
// rules' draws the last one that acts on a site decides.  nt0, nt1: the negated
// thresholds (WT: rt_word.cu).
template <int FAM, int WT>
__device__ __forceinline__ void word_combine(const WalkArgs& a, uint32_t d, int i, int c0, const uint32_t (&k)[4],
                                             uint32_t nt0, uint32_t nt1, uint32_t& m0, uint32_t& m1) {
    constexpr bool DOM = FAM != FAM_LOZENGE8;
    uint32_t lo;
    if (WT == 1) {
        // Periodic weights: a threshold per site from its vertex (i, j); array
        // column c of the rotated array A is vertex column 2 c + ((i + A) & 1)
        // (dominoes) or 3 c + (A + i) mod 3 (lozenges).
        const int step = DOM ? 2 : 3;
        const int j0 = step * c0 + (DOM ? (i + 1 - (int)ph_a(d)) & 1 : ((int)ph_a(d) + i) % 3);
        lo = below4(k, 0u - weight_thr(a, i, j0), 0u - weight_thr(a, i, j0 + step), 0u - weight_thr(a, i, j0 + 2 * step),
                    0u - weight_thr(a, i, j0 + 3 * step));
    } else {
        lo = below4(k, nt0);
    }
    if (FAM == FAM_DOMINO) {
        m0 ^= lo;
    } else if (FAM == FAM_DOMINO_HB) {
        m0 = lo;
    } else {
        const uint32_t rem = below4(k, nt1) & (WT == 2 ? ~below4(k, 0u - (1u << 22)) : ~lo);
        m0 = lo | (m0 & ~rem);
        m1 = rem | (m1 & ~lo);
    }
}

__device__ __forceinline__ uint32_t lozenge_shift_table(int t) {
    uint32_t tab = 0;
#pragma unroll
    for (int rr = 0; rr < 3; ++rr) {
        const uint32_t sa = rr == (2 * t + 1) % 3, sw = rr == (2 * t + 2) % 3, se = rr == (2 * t) % 3;
        tab |= (sa | (sw << 1) | (se << 2)) << (3 * rr);
    }
    return tab;
}

}  // namespace rtb
