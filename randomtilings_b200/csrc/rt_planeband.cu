// rt_planeband.cu -- the bit-plane walk (rt_plane.cu has the rules) with one
// word of 32 sites per thread.
//
// A thread owns the words of one place (row, column / 32) of every colour for
// the whole walk, halo rows included, and keeps them in registers; shared
// memory holds a copy for the neighbours.  The four threads of a quad share
// one Philox call per step, so they make the calls of four steps at once, one
// each, and exchange the words: a quarter of the calls.  Halo rows go from
// the registers of their owner to the registers of the thread that keeps them
// in the neighbouring CTA, with no index arithmetic.  Every walk on several CTAs
// makes an exchange (launch_walk): it orders a CTA's loads before its neighbours'
// stores.
//
// What bounds it: the latency of a phase (barrier, neighbours, rule: 0.25 us)
// and, on large lattices, instruction issue; the exchange every H phases adds
// 1.5 us.  A step of the Aztec diamond of order 1000 takes 0.72 us (2.47 in
// rt_plane.cu), of order 24 0.26 (2.27), of the hexagon of side 600 0.62 (1.92).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <type_traits>

#include "rt_exchange.cuh"
#include "rt_internal.h"
#include "rt_models.cuh"
#include "rt_plane.cuh"
#include "rt_word.cuh"

namespace rtb {

constexpr int kBandBlock = 512;  // threads of the largest block: 128 registers each

// Shared memory: planes [lattice][colour][plane][stored row][RS words], as in
// rt_plane.cu: stored row s is colour-array row a0 - H + s; word 0 and word
// WW + 1 of a row are zero padding for the funnel shifts.
// RPT: rows of a thread (one below the other).
template <int FAM, int NL, int RPT>
__global__ void __launch_bounds__(kBandBlock, 1) plane_band_kernel(const __grid_constant__ WalkArgs a) {
    using M = PlaneModel<FAM>;
    constexpr int NC = M::NC, NP = M::NP;
    extern __shared__ __align__(16) uint32_t psm[];
    const int BLOCK = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    const int cta = blockIdx.x, nct = gridDim.x;
    const int H = a.depth, WW = a.pwords, RS = WW + 2;
    const int QPR = (WW + 3) >> 2;  // Philox calls per row
    const int r0 = (int)((int64_t)cta * a.rows / nct), r1 = (int)((int64_t)(cta + 1) * a.rows / nct);
    const int nrows = r1 - r0;
    const int R = (a.rows_per_cta + 2 * H + RPT - 1) / RPT * RPT;
    const int PLANE = R * RS;
    const int a0 = r0 + M::ROFF;
    const bool has_top = cta > 0, has_bot = cta + 1 < nct;

    // This thread's words: stored rows s0 .. s0 + RPT - 1, word w (quads of words
    // are quads of lanes).  Rows that no position lies in have empty masks, so
    // computing them changes nothing.
    const int s0 = tid / (4 * QPR) * RPT, w = tid % (4 * QPR);
    const int i0 = a0 - H + s0;  // colour-array row
    const bool live = s0 < R && w < WW;
    const int o = min(s0, R - RPT) * RS + min(w, WW - 1) + 1;
    uint32_t um[RPT], vm[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int i = i0 + r;
        const bool in = live && i >= M::ROFF && i < M::ROFF + a.rows;
        um[r] = in && i >= 1 && i <= a.n - 2 ? col_mask(w, 1, a.width - 1) : 0u;
        vm[r] = in ? col_mask(w, M::COFF, M::COFF + a.cols) : 0u;
    }
    const int o_up = s0 > 0 ? -RS : 0, o_dn = s0 + RPT < R ? RPT * RS : (RPT - 1) * RS;  // the rows next to the thread's

    uint32_t x[NL][RPT][NC][NP];
    for (int e = tid; e < NL * NC * NP * PLANE; e += BLOCK) psm[e] = 0u;
    __syncthreads();
    // A warp turns one word after the other into planes: 32 bytes, a ballot a plane.
#pragma unroll
    for (int l = 0; l < NL; ++l)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int8_t* g = static_cast<const int8_t*>(a.arr[l][c]);
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int mine = live && s0 + r < nrows + 2 * H ? i0 + r : -1;
#pragma unroll
                for (int q = 0; q < NP; ++q) x[l][r][c][q] = 0u;
#pragma unroll 16
                for (int y = 0; y < 32; ++y) {
                    const int yi = __shfl_sync(0xffffffffu, mine, y), j = 32 * __shfl_sync(0xffffffffu, w, y) + lane;
                    uint32_t v = 0u;
                    if (yi >= 0 && yi < a.arows && j < a.width) v = (uint32_t)(uint8_t)__ldg(g + (size_t)yi * a.width + j);
                    if (v >> NP) atomicOr(a.err, ERR_BADOP);
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        const uint32_t bits = __ballot_sync(0xffffffffu, v >> q & 1u);
                        if (lane == y) x[l][r][c][q] = bits;
                    }
                }
                if (live)
#pragma unroll
                    for (int q = 0; q < NP; ++q) psm[((l * NC + c) * NP + q) * PLANE + r * RS + o] = x[l][r][c][q];
            }
        }
    // lozenge column shifts, three bits a row class (i mod 3) and pending colour
    uint32_t shifts[M::DOM ? 1 : 3] = {};
    if (!M::DOM)
        for (int t = 0; t < 3; ++t) shifts[M::DOM ? 0 : t] = lozenge_shift_table(t);
    const int cls0 = (i0 + 3 * H) % 3;

    int epoch = -1;
    int64_t next_epoch = a.nepochs > 0 ? a.epoch_start[0] : INT64_MAX;
    uint32_t key0 = 0, key1 = 0;
    int64_t dbase = 0;                    // step of the first draw in `bits`
    uint32_t bits[RPT][4];                // the words' draws of four steps
    int drawn = 4;                        // how many of them are used up

    // The draws of four steps from dbase on: lane x of the quad makes the call of
    // step dbase + x, and a 4 x 4 transpose hands each lane its own word.
    auto refill = [&]() {
        const int64_t st = dbase + (lane & 3);
#pragma unroll
        for (int y = 0; y < RPT; ++y) {
            const uint32_t quad = (uint32_t)((i0 + y - M::ROFF) * QPR + (w >> 2));
            uint4 r = philox4(quad, (uint32_t)st, (uint32_t)((uint64_t)st >> 32), a.chain, key0, key1);
            if (FAM == FAM_DOMINO) {
                const uint4 r2 =
                    philox4(quad | 0x80000000u, (uint32_t)st, (uint32_t)((uint64_t)st >> 32), a.chain, key0, key1);
                r = make_uint4(r.x | r2.x, r.y | r2.y, r.z | r2.z, r.w | r2.w);
            }
            const bool odd = lane & 1, high = lane & 2;
            const uint32_t t0 = __shfl_xor_sync(0xffffffffu, odd ? r.x : r.y, 1);
            const uint32_t t1 = __shfl_xor_sync(0xffffffffu, odd ? r.z : r.w, 1);
            (odd ? r.x : r.y) = t0;
            (odd ? r.z : r.w) = t1;
            const uint32_t t2 = __shfl_xor_sync(0xffffffffu, high ? r.x : r.z, 2);
            const uint32_t t3 = __shfl_xor_sync(0xffffffffu, high ? r.y : r.w, 2);
            bits[y][0] = high ? t2 : r.x;
            bits[y][1] = high ? t3 : r.y;
            bits[y][2] = high ? r.z : t2;
            bits[y][3] = high ? r.w : t3;
        }
    };

    // One phase of this thread's words; C: the colour flipped (dominoes: the
    // array), as a constant.
    auto phase = [&](auto cc, bool step, bool upd, bool next, const uint32_t (&b)[RPT]) {
        constexpr int C = decltype(cc)::value;
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            uint32_t* const L = psm + l * NC * NP * PLANE + o;
            if constexpr (M::DOM) {
                if (upd) {
                    // domino_refresh (dominokernel.cl:22-31): bit 1 <- up's bit 2,
                    // bit 2 <- down's bit 1, bit 4 <- west's bit 8, bit 8 <- east's bit 4;
                    // west / east share the column in rows of one parity.
                    const uint32_t* const F = L + (1 - C) * NP * PLANE;
                    const uint32_t top = F[PLANE + o_up], bottom = F[o_dn];
                    uint32_t side[RPT];
#pragma unroll
                    for (int r = 0; r < RPT; ++r)
                        side[r] = F[((i0 + r) ^ C) & 1 ? 2 * PLANE + r * RS + 1 : 3 * PLANE + r * RS - 1];
#pragma unroll
                    for (int r = 0; r < RPT; ++r) {
                        uint32_t(&D)[NP] = x[l][r][C];
                        const uint32_t(&S)[NP] = x[l][r][1 - C];
                        const bool p = ((i0 + r) ^ C) & 1;
                        const uint32_t up = r > 0 ? x[l][r > 0 ? r - 1 : 0][1 - C][1] : top;
                        const uint32_t dn = r + 1 < RPT ? x[l][r + 1 < RPT ? r + 1 : r][1 - C][0] : bottom;
                        const uint32_t west = p ? S[3] : col_prev(side[r], S[3]);
                        const uint32_t east = p ? col_next(S[2], side[r]) : S[2];
                        D[0] = (D[0] & ~um[r]) | (up & um[r]);
                        D[1] = (D[1] & ~um[r]) | (dn & um[r]);
                        D[2] = (D[2] & ~um[r]) | (west & um[r]);
                        D[3] = (D[3] & ~um[r]) | (east & um[r]);
                    }
                }
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    uint32_t(&D)[NP] = x[l][r][C];
                    if (step) {
                        const uint32_t rot = ((D[0] & D[1] & ~D[2] & ~D[3]) | (~D[0] & ~D[1] & D[2] & D[3])) & vm[r];
                        if (FAM == FAM_DOMINO_HB) {
                            // heat bath: 12 (planes 2, 3) where the bit is 1, else 3 (planes 0, 1)
                            D[0] = (D[0] & ~rot) | (~b[r] & rot);
                            D[1] = (D[1] & ~rot) | (~b[r] & rot);
                            D[2] = (D[2] & ~rot) | (b[r] & rot);
                            D[3] = (D[3] & ~rot) | (b[r] & rot);
                        } else {
#pragma unroll
                            for (int q = 0; q < NP; ++q) D[q] ^= rot & b[r];
                        }
                    }
#pragma unroll
                    for (int q = 0; q < NP; ++q) L[(C * NP + q) * PLANE + r * RS] = D[q];
                }
            } else {
                // lozenge_refresh (lozengekernel.cl:36-54): colour T + 1 takes bits
                // {2, 4, 32} from the flipped colour T at (i-1, j+sa), (i, j-sw),
                // (i+1, j); colour T + 2 takes {1, 8, 16} from (i-1, j), (i, j+se),
                // (i+1, j-sa).
                auto refresh = [&](auto tt) {
                    constexpr int T = decltype(tt)::value;
                    const uint32_t* const F = L + T * NP * PLANE;
                    const uint32_t top4 = F[4 * PLANE + o_up], top5 = F[5 * PLANE + o_up];
                    const uint32_t bottom0 = F[o_dn], bottom1 = F[PLANE + o_dn];
                    int cls = cls0;
#pragma unroll
                    for (int r = 0; r < RPT; ++r) {
                        const uint32_t sh = shifts[M::DOM ? 0 : T] >> (3 * cls);
                        cls = cls == 2 ? 0 : cls + 1;
                        const int up = r > 0 ? (r - 1) * RS : o_up, dn = r + 1 < RPT ? (r + 1) * RS : o_dn;
                        const uint32_t(&S)[NP] = x[l][r][T];
                        uint32_t(&A)[NP] = x[l][r][(T + 1) % 3];
                        uint32_t(&B)[NP] = x[l][r][(T + 2) % 3];
                        const uint32_t f4 = r > 0 ? x[l][r > 0 ? r - 1 : 0][T][4] : top4;
                        const uint32_t m0 = r > 0 ? x[l][r > 0 ? r - 1 : 0][T][5] : top5;
                        const uint32_t n5 = r + 1 < RPT ? x[l][r + 1 < RPT ? r + 1 : r][T][0] : bottom0;
                        const uint32_t f1 = r + 1 < RPT ? x[l][r + 1 < RPT ? r + 1 : r][T][1] : bottom1;
                        // exactly one of the three shifts applies in a row
                        const uint32_t n1 = (sh & 1u) ? col_next(f4, F[4 * PLANE + up + 1]) : f4;
                        const uint32_t m4 = (sh & 1u) ? col_prev(F[PLANE + dn - 1], f1) : f1;
                        const uint32_t n2 = (sh & 2u) ? col_prev(F[3 * PLANE + r * RS - 1], S[3]) : S[3];
                        const uint32_t m3 = (sh & 4u) ? col_next(S[2], F[2 * PLANE + r * RS + 1]) : S[2];
                        A[1] = (A[1] & ~um[r]) | (n1 & um[r]);
                        A[2] = (A[2] & ~um[r]) | (n2 & um[r]);
                        A[5] = (A[5] & ~um[r]) | (n5 & um[r]);
                        B[0] = (B[0] & ~um[r]) | (m0 & um[r]);
                        B[3] = (B[3] & ~um[r]) | (m3 & um[r]);
                        B[4] = (B[4] & ~um[r]) | (m4 & um[r]);
                    }
                };
                if (!step)
                    refresh(std::integral_constant<int, C>{});
                else if (upd && next)
                    refresh(std::integral_constant<int, (C + 2) % 3>{});
                else if (upd)
                    refresh(std::integral_constant<int, (C + 1) % 3>{});
                if (step) {
                    // heat bath: 25 (planes 0, 3, 4) -> 38 (planes 1, 2, 5) where the bit is 1, back where 0
#pragma unroll
                    for (int r = 0; r < RPT; ++r) {
                        uint32_t(&D)[NP] = x[l][r][C];
                        const uint32_t e25 = D[0] & ~D[1] & ~D[2] & D[3] & D[4] & ~D[5];
                        const uint32_t e38 = ~D[0] & D[1] & D[2] & ~D[3] & ~D[4] & D[5];
                        const uint32_t tog = ((e25 & b[r]) | (e38 & ~b[r])) & vm[r];
#pragma unroll
                        for (int q = 0; q < NP; ++q) {
                            D[q] ^= tog;
                            L[(C * NP + q) * PLANE + r * RS] = D[q];
                        }
                    }
                }
            }
        }
    };

    __syncthreads();
    uint32_t blk = 0;  // halo exchanges made (modulo 2^32, as the tags)
    int k = 0;         // phases since the last one
    const int s_top = has_top ? 1 : H, s_bot = H + nrows + (has_bot ? H - 1 : 0);
    // After phase k of a block the rows within H - k - 1 of the band are
    // current; rows beyond them may hold anything until the next exchange.
    auto computed = [&]() {
        return live && s0 + RPT - 1 >= s_top + (has_top ? k : 0) && s0 < s_bot - (has_bot ? k : 0);
    };
    auto draw = [&](bool active, uint32_t (&b)[RPT]) {
        if (__builtin_expect(drawn == 4, 0)) {
            dbase += 4;
            drawn = 0;
            // Rows that are not computed any more before the next exchange need no draws.
            if (__any_sync(0xffffffffu, active || (live && nct > 1 && k + 4 > H))) refill();
        }
        ++drawn;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            b[r] = bits[r][0];
            bits[r][0] = bits[r][1];
            bits[r][1] = bits[r][2];
            bits[r][2] = bits[r][3];
        }
    };
    // The band's first and last H rows of every colour go to the CTAs above
    // and below (tagged words, one tag a block), the H rows next to the band
    // come from them.  A slot is rewritten two blocks later, after the
    // neighbour's next rows were read, which it sent after reading this one.
    auto exchange = [&]() -> bool {
        const int par = (int)(blk & 1u);
        const uint32_t tag = blk + 1u;
        if (live && !(cta == 0 && blk == a.drop_phase)) {
            auto publish = [&](int side, int r, int j) {
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    unsigned long long* const to = slot(a, cta, side, par, l, 0) + j * WW + w;
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int q = 0; q < NP; ++q)
                            st_relaxed64(to + (c * NP + q) * H * WW, (unsigned long long)tag << 32 | x[l][r][c][q]);
                }
            };
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int s = s0 + r;
                if (has_top && s >= H && s < 2 * H) publish(0, r, s - H);
                if (has_bot && s >= nrows && s < H + nrows) publish(1, r, s - nrows);
            }
        }
        __syncthreads();  // the halo rows in shared memory are not read any more
        bool ok = true;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int s = s0 + r;
            const bool above = live && has_top && s < H, below = live && has_bot && s >= H + nrows && s < 2 * H + nrows;
            if (!(above || below)) continue;
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                const unsigned long long* const from =
                    (above ? slot(a, cta - 1, 1, par, l, 0) + s * WW : slot(a, cta + 1, 0, par, l, 0) + (s - H - nrows) * WW) + w;
                // all words in one round trip, again until the last one is there
                unsigned long long v[NC * NP];
                unsigned spins = 0;
                uint64_t t0 = 0;
                for (;;) {
                    bool here = true;
#pragma unroll
                    for (int q = 0; q < NC * NP; ++q) v[q] = ld_relaxed64(from + q * H * WW);
#pragma unroll
                    for (int q = 0; q < NC * NP; ++q) here = here && (uint32_t)(v[q] >> 32) == tag;
                    if (here || !ok) break;
                    if ((++spins & 63u) == 0u) ok = wait_more(a, t0);
                }
#pragma unroll
                for (int q = 0; q < NC * NP; ++q) {
                    x[l][r][q / NP][q % NP] = (uint32_t)v[q];
                    psm[(l * NC * NP + q) * PLANE + r * RS + o] = (uint32_t)v[q];
                }
            }
        }
        k = 0;
        ++blk;
        return !__syncthreads_or(!ok);
    };
    int64_t ph = 0;
    while (ph < a.nphases) {
        if (ph == next_epoch) {
            while (epoch + 1 < a.nepochs && a.epoch_start[epoch + 1] == ph) ++epoch;
            next_epoch = epoch + 1 < a.nepochs ? a.epoch_start[epoch + 1] : INT64_MAX;
            key0 = (uint32_t)a.epoch_seed[epoch];
            key1 = (uint32_t)(a.epoch_seed[epoch] >> 32);
            dbase = -4;
            drawn = 4;
        }
        const uint32_t d = __ldg(a.phases + ph);
        const bool step = ph_op(d) == OP_STEP;
        const int ca = (int)ph_a(d), cb = (int)ph_b(d);
        const bool upd = step ? (cb != (int)NO_COLOUR && cb != ca) : true;
        // reference colour r of the dominoes flips array 1 - r; at the end array r is refreshed
        const int col = M::DOM && step ? 1 - ca : ca;
        const bool next = !M::DOM && ca == (cb == 2 ? 0 : cb + 1);
        const bool active = computed();
        uint32_t b[RPT] = {};
        if (d & PH_DRAWS) draw(active, b);
        if (active) {
            if (col == 0)
                phase(std::integral_constant<int, 0>{}, step, upd, next, b);
            else if (col == 1)
                phase(std::integral_constant<int, 1>{}, step, upd, next, b);
            else
                phase(std::integral_constant<int, 2 % NC>{}, step, upd, next, b);
        }
        ++ph;
        ++k;
        __syncthreads();
        if (nct > 1 && k == H && ph < a.nphases && !exchange()) return;
        // The fast modes' colours go round within an epoch, so its phases after
        // the first are known: NC of them make one round of this loop, with
        // nothing to decode.
        if (!step || col != NC - 1) continue;
        int64_t rounds = (min(a.nphases - 1, next_epoch) - ph) / NC;
        if (rounds <= 0) continue;
        ph += rounds * NC;
        for (; rounds > 0; --rounds) {
            bool ok = true;
            auto regular = [&](auto cc) {
                const bool act = computed();
                uint32_t bb[RPT];
                draw(act, bb);
                if (act) phase(cc, true, true, true, bb);
                ++k;
                __syncthreads();
                if (nct > 1 && __builtin_expect(k == H, 0)) ok = ok && exchange();
            };
            regular(std::integral_constant<int, 0>{});
            regular(std::integral_constant<int, 1>{});
            if (NC == 3) regular(std::integral_constant<int, 2 % NC>{});
            if (!ok) return;
        }
    }

    // Band rows back to bytes: a warp writes one word after the other.
#pragma unroll
    for (int l = 0; l < NL; ++l)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            int8_t* g = static_cast<int8_t*>(a.arr[l][c]);
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int mine = live && s0 + r >= H && s0 + r < H + nrows ? i0 + r : -1;
#pragma unroll 4
                for (int y = 0; y < 32; ++y) {
                    const int yi = __shfl_sync(0xffffffffu, mine, y), j = 32 * __shfl_sync(0xffffffffu, w, y) + lane;
                    uint32_t v = 0u;
#pragma unroll
                    for (int q = 0; q < NP; ++q) v |= (__shfl_sync(0xffffffffu, x[l][r][c][q], y) >> lane & 1u) << q;
                    if (yi >= 0 && j < a.width) g[(size_t)yi * a.width + j] = (int8_t)v;
                }
            }
        }
}

using PlaneFn = void (*)(WalkArgs);

template <int FAM, int NL>
static PlaneFn band_fn_of(int rpt) {
    return rpt == 1 ? plane_band_kernel<FAM, NL, 1> : rpt == 2 ? plane_band_kernel<FAM, NL, 2> : plane_band_kernel<FAM, NL, 4>;
}

static PlaneFn band_fn(int family, int nlat, int rpt) {
    switch (family) {
        case FAM_DOMINO: return nlat == 1 ? band_fn_of<FAM_DOMINO, 1>(rpt) : nullptr;  // not monotone
        case FAM_DOMINO_HB: return nlat == 1 ? band_fn_of<FAM_DOMINO_HB, 1>(rpt) : band_fn_of<FAM_DOMINO_HB, 2>(rpt);
        case FAM_LOZENGE8: return nlat == 1 ? band_fn_of<FAM_LOZENGE8, 1>(rpt) : band_fn_of<FAM_LOZENGE8, 2>(rpt);
        default: return nullptr;
    }
}

rt_status plan_plane_band(int family, int device, int nlat, int rows, int width, int ctas_hint, int depth_hint,
                          WalkPlan* plan, std::string* err) {
    int sms = 0, smem_optin = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) {
        *err = "cudaDeviceGetAttribute failed";
        return RT_E_CUDA;
    }
    const int nc = family == FAM_LOZENGE8 ? 3 : 2, np = family == FAM_LOZENGE8 ? 6 : 4;
    const int ww = (width + 31) / 32, rs = ww + 2, wp = (ww + 3) / 4 * 4;
    // Microseconds per step (dominoes of order n / hexagons of side n; best depth):
    //   CTAs   24    60    100   250   500   700   1000 / 50    100   250   400   600
    //   1      0.26  0.36  -     -     -     -     -      0.50  -     -     -     -
    //   8      -     0.30  0.30  -     -     -     -      0.45  0.48  -     -     -
    //   24     -     -     0.31  0.37  -     -     -      -     0.44  0.54  -     -
    //   50     -     -     -     0.35  -     -     -      -     -     0.51  0.56  -
    //   100    -     -     -     -     0.42  -     -      -     -     -     0.56  0.65
    //   148    -     -     -     -     0.45  0.75  0.72   -     -     -     0.65  0.62
    // So: one CTA while ten warps hold the lattice; else bands of ten rows.  An
    // exchange takes 1.5 us or so and a phase 0.25 to 0.6, so blocks are as long
    // as the band has rows for the neighbours (up to 32) and the block has
    // threads for the halo.
    int ctas = ctas_hint;
    if (ctas <= 0) ctas = (int64_t)(rows + 2) * wp <= 320 ? 1 : std::min(sms, rows / 10);
    ctas = std::max(1, std::min(ctas, rows));
    const int rpc = (rows + ctas - 1) / ctas;
    const int depth_max = ctas == 1 ? 1 : std::max(1, std::min(depth_hint > 0 ? depth_hint : 32, std::min(32, rows / ctas)));
    int rpt = 1, depth = 0;
    auto stored = [&]() { return (rpc + 2 * depth + rpt - 1) / rpt * rpt; };
    // One row a thread, unless that leaves too few halo rows: dominoes 5 (order
    // 700: 0.75 with one row and 5, 0.74 with two rows and 9), lozenges 2 (their
    // 36 words do not fit the registers: side 1000, 0.99 with one row and 3, 1.59
    // with two rows and 8).
    for (;; rpt *= 2) {
        const int want = std::min(depth_max, rpt > 1 ? 1 : family == FAM_LOZENGE8 || nlat > 1 ? 2 : 5);
        for (depth = depth_max; depth >= want; --depth)
            if ((int64_t)(stored() / rpt) * wp <= kBandBlock &&
                (size_t)nlat * nc * np * stored() * rs * 4 <= (size_t)smem_optin)
                break;
        if (depth >= want) break;
        if (rpt == 4) {
            *err = "band too large for the words of one block";
            return RT_E_INVAL;
        }
    }
    const size_t smem = (size_t)nlat * nc * np * stored() * rs * 4;
    const int block = (stored() / rpt * wp + 31) / 32 * 32;
    PlaneFn fn = band_fn(family, nlat, rpt);
    if (!fn) {
        *err = "no such bit-plane walk";
        return RT_E_INVAL;
    }
    if (const rt_status s = allow_shared((const void*)fn, device, smem, err); s != RT_OK) return s;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)fn, block, smem) != cudaSuccess) {
        *err = "cudaOccupancyMaxActiveBlocksPerMultiprocessor failed";
        return RT_E_CUDA;
    }
    if (per_sm < 1 || ctas > per_sm * sms) {
        *err = "bit-plane grid cannot be co-resident";
        return RT_E_INVAL;
    }
    plan->items = 0;
    plan->block = block;
    plan->rows_per_cta = rpc;
    plan->ctas = ctas;
    plan->smem = smem;
    plan->wpad = rs;
    plan->xwords = nc * np * depth * ww;
    plan->xslots = 1;
    plan->depth = depth;
    plan->pwords = ww;
    plan->fn = (const void*)fn;
    return RT_OK;
}

}  // namespace rtb
