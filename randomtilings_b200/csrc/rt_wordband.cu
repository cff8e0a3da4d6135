// rt_wordband.cu -- the word-parallel walk on bands with halos.
//
// The rules and words of rt_word.cu, one word per thread.  A draw depends on the
// site and how often it drew, so a CTA can compute the rows next to its band
// itself: it keeps H rows of every colour above and below -- in bit-exact mode
// with their generators, which go on in step with their owners' -- and after
// phase k of a block of H phases the rows within H - k - 1 of the band are
// current.  Then each CTA's first and last H rows go to its neighbours through
// tagged words (rt_exchange.cuh), all words of a thread in one round trip.  H is
// less than the walk's phases (launch_walk), so that no CTA writes its band back
// before its neighbours have read it.
//
// What bounds it: the latency of a phase -- the draws, the word's update, the
// barrier, 0.2 us a step on one CTA -- and the exchange, 1.5 us or so every H
// phases; in bit-exact mode, from some 360 words a CTA on, the draws (118 issue
// cycles a warp's word and step), halo rows included.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "rt_exchange.cuh"
#include "rt_internal.h"
#include "rt_models.cuh"
#include "rt_word.cuh"

namespace rtb {

constexpr int kWbBlockMid = 640;  // 65,536 registers / 96, in whole warps

// Shared memory: 16 bytes of slack, for each lattice NC colour planes of (band
// rows + 2 H) x wpad bytes, 16 bytes of slack (rt_word.cu).
template <int FAM, int WT, int NL, bool PHILOX, int LB>
__global__ void __launch_bounds__(LB, 1) word_band_kernel(const __grid_constant__ WalkArgs a) {
    using M = WordModel<FAM>;
    constexpr int NC = M::NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* const lat = smem_raw + 16;
    const int BLOCK = blockDim.x, tid = threadIdx.x;
    const int cta = blockIdx.x, nct = gridDim.x, H = a.depth;
    const int r0 = (int)((int64_t)cta * a.rows / nct), r1 = (int)((int64_t)(cta + 1) * a.rows / nct);
    const int nrows = r1 - r0;
    const int a0 = r0 + M::ROFF;  // colour-array row of the band's first row
    const int W = a.wpad, Gw = W >> 2;
    const int plane = (a.rows_per_cta + 2 * H) * W;
    const bool has_top = cta > 0, has_bot = cta + 1 < nct;

    for (int l = 0; l < NL; ++l)
        for (int c = 0; c < NC; ++c) {
            const int8_t* g = static_cast<const int8_t*>(a.arr[l][c]);
            unsigned char* s = lat + (l * NC + c) * plane;
            for (int e = tid; e < plane; e += BLOCK) {
                const int i = a0 - H + e / W, j = e % W;
                s[e] = i >= 0 && i < a.arows && e < (nrows + 2 * H) * W && j < a.width ? (unsigned char)g[(size_t)i * a.width + j] : 0;
            }
        }
    __shared__ WordPhase s_phase[kWordPhases];
    __shared__ uint4 s_sel[kLozengeSel];
    if (tid < kWordPhases) s_phase[tid] = word_phase_entry<FAM>(tid, plane);
    if (tid < kLozengeSel) s_sel[tid] = lozenge_sel_entry(tid);
    const uint32_t nt0 = 0u - (WT == 2 ? a.thr[2] : a.thr[0]), nt1 = 0u - (WT == 2 ? a.thr[3] : a.thr[1]);

    // This thread's word: stored row s, word w.
    const int s = tid / Gw, w = tid - s * Gw;
    const bool live = s < nrows + 2 * H;
    const int i = a0 - H + s;
    WordInfo wi{0, 0, 0u, 0u};
    if (live) {
        wi.off = s * W + 4 * w;
        wi.cls = M::DOM ? i & 1 : (i + 3 * H) % 3;
        uint32_t ub = 0, vb = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int j = 4 * w + b;
            if (j >= 1 && j <= a.width - 2) ub |= 1u << b;
            if (j >= M::COFF && j < M::COFF + a.cols) vb |= 1u << b;
        }
        wi.um = i >= 1 && i <= a.n - 2 ? lane_bytes(ub) * 0xffu : 0u;
        wi.vm = lane_bytes(vb) << 7;
    }
    const uint32_t quad = (uint32_t)(i * Gw + w);
    const TinyParams tp{a.mat1, a.mat2, a.tmat};
    TinyState st[PHILOX ? 1 : 4];

    int epoch = -1;
    int64_t next_epoch = a.nepochs > 0 ? a.epoch_start[0] : INT64_MAX;
    uint32_t key0 = 0, key1 = 0;
    int64_t dstep = 0;
    // Draws restart at phase `ph` when an epoch begins there.
    auto begin_phase = [&](int64_t ph) {
        if (ph != next_epoch) return;
        while (epoch + 1 < a.nepochs && a.epoch_start[epoch + 1] == ph) ++epoch;
        next_epoch = epoch + 1 < a.nepochs ? a.epoch_start[epoch + 1] : INT64_MAX;
        key0 = (uint32_t)a.epoch_seed[epoch];
        key1 = (uint32_t)(a.epoch_seed[epoch] >> 32);
        dstep = 0;
        if (!PHILOX)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                // a site that is not a Rotate position has no stream; its draws are not used
                const uint32_t sid = (uint32_t)(4 * w + b - M::COFF) + (uint32_t)a.cols * (uint32_t)(i - M::ROFF);
                tiny_seed(st[PHILOX ? 0 : b], tp, key0 + sid);
            }
    };
    // The masks of this word for phase d (WordOp).  They depend on the draws
    // alone, so they are made a phase ahead, while the rows the phase needs are on
    // their way.  used: the word is computed in that phase (generators go on anyway).
    uint32_t m0 = 0u, m1 = 0u;
    auto draw_masks = [&](uint32_t d, bool used) {
        m0 = m1 = 0u;
        if (!(d & PH_DRAWS)) return;
        if (PHILOX) {
            if (used) {
                const uint4 r = philox4(quad, (uint32_t)dstep, (uint32_t)((uint64_t)dstep >> 32), a.chain, key0, key1);
                const uint32_t k[4] = {r.x, r.y, r.z, r.w};
                word_combine<FAM, WT>(a, d, i, 4 * w, k, nt0, nt1, m0, m1);
            }
            ++dstep;
        } else if (live) {
#pragma unroll 1
            for (uint32_t c = 0; c < ph_steps(d); ++c) {
                uint32_t k[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) k[b] = tiny_draw32(st[PHILOX ? 0 : b], tp);
                word_combine<FAM, WT>(a, d, i, 4 * w, k, nt0, nt1, m0, m1);
            }
        }
    };
    // Phases after `ph` until one before which an epoch begins, or the last.
    auto until_special = [&](int64_t ph) {
        return (int)min(min(a.nphases - 1, next_epoch - 1 >= ph ? next_epoch - 1 : INT64_MAX) - ph, (int64_t)1 << 30);
    };
    uint32_t d = a.nphases > 0 ? __ldg(a.phases) : 0u;
    const uint32_t* ahead = a.phases + 1;
    int until = 0;
    bool more = a.nphases > 0;
    int64_t blk = 0;  // halo exchanges made
    const int64_t drop_blk = a.drop_phase >= 0 ? a.drop_phase / H : -1;
    int lo = has_top ? 1 : H, hi = H + nrows + (has_bot ? H - 1 : 0);  // stored rows computed in this phase
    int k = 0;                                                        // phases since the last exchange
    if (more) {
        begin_phase(0);
        draw_masks(d, s >= lo && s < hi);
        until = until_special(0);
    }
    __syncthreads();
    WordPhase P = s_phase[word_phase_index(d)];
    while (more) {
        uint32_t d_next = 0u;
        int64_t begin = -1;  // the next phase, if its epoch may begin there
        if (__builtin_expect(until-- > 0, 1)) {
            d_next = __ldg(ahead);
        } else {
            const int64_t ph = ahead - a.phases - 1;
            more = ph + 1 < a.nphases;
            if (more) d_next = __ldg(ahead);
            if (more) begin = ph + 1;
        }
        ++ahead;
        if (s >= lo && s < hi) {
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                unsigned char* const L = lat + l * NC * plane;
                WordOp<FAM> op;
                WordNbr nb;
                op.load_up(nb, L, P, wi, W);
                op.load_dn(nb, L, P, wi, W);
                op.begin(L, P, wi, s_sel);
                op.finish(P, wi, nb, m0, m1);
                op.store(L, P, wi);
            }
        }
        d = d_next;
        P = s_phase[word_phase_index(d)];
        ++k;
        lo += has_top;
        hi -= has_bot;
        auto draw_ahead = [&]() {
            if (begin >= 0) {
                begin_phase(begin);
                until = until_special(begin);
            }
            draw_masks(d, s >= lo && s < hi);
        };
        if (__builtin_expect(nct == 1 || k < H || !more, 1)) {
            if (more) draw_ahead();
            __syncthreads();
            continue;
        }
        lo = has_top ? 1 : H;
        hi = H + nrows + (has_bot ? H - 1 : 0);
        // A slot is rewritten two blocks later, after the neighbour's next rows were
        // read, which it sent after reading this one.
        const int par = (int)(blk & 1);
        const uint32_t tag = (uint32_t)blk + 1u;
        if (live && !(cta == 0 && blk == drop_blk)) {
            auto publish = [&](int side, int j) {
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    unsigned long long* const to = slot(a, cta, side, par, l, 0) + j * Gw + w;
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        st_relaxed64(to + c * H * Gw, (unsigned long long)tag << 32 | lds(lat + (l * NC + c) * plane + wi.off));
                }
            };
            if (has_top && s >= H && s < 2 * H) publish(0, s - H);
            if (has_bot && s >= nrows && s < H + nrows) publish(1, s - nrows);
        }
        draw_ahead();
        __syncthreads();  // the halo rows are not read any more
        bool ok = true;
        const bool above = live && has_top && s < H, below = live && has_bot && s >= H + nrows;
        if (above || below) {
            const unsigned long long* const from =
                (above ? slot(a, cta - 1, 1, par, 0, 0) + s * Gw : slot(a, cta + 1, 0, par, 0, 0) + (s - H - nrows) * Gw) + w;
            unsigned long long v[NL * NC];
            unsigned spins = 0;
            uint64_t t0 = 0;
            for (;;) {
                bool here = true;
#pragma unroll
                for (int q = 0; q < NL * NC; ++q) v[q] = ld_relaxed64(from + (q / NC) * a.xwords + (q % NC) * H * Gw);
#pragma unroll
                for (int q = 0; q < NL * NC; ++q) here = here && (uint32_t)(v[q] >> 32) == tag;
                if (here || !ok) break;
                if ((++spins & 63u) == 0u) ok = wait_more(a, t0);
            }
#pragma unroll
            for (int q = 0; q < NL * NC; ++q) sts(lat + q * plane + wi.off, (uint32_t)v[q]);
        }
        if (__syncthreads_or(!ok)) return;
        k = 0;
        ++blk;
    }
    for (int l = 0; l < NL; ++l)
        for (int c = 0; c < NC; ++c) {
            int8_t* g = static_cast<int8_t*>(a.arr[l][c]);
            const unsigned char* src = lat + (l * NC + c) * plane + H * W;
            for (int e = tid; e < nrows * a.width; e += BLOCK) {
                const int rr = e / a.width, j = e % a.width;
                g[(size_t)(a0 + rr) * a.width + j] = (int8_t)src[rr * W + j];
            }
        }
}

using KernelFn = void (*)(WalkArgs);

template <int FAM, int WT, int NL, bool PHILOX>
static KernelFn wb_fn1(int block) {
    return block <= kWbBlockMid ? word_band_kernel<FAM, WT, NL, PHILOX, kWbBlockMid>
                                : word_band_kernel<FAM, WT, NL, PHILOX, 1024>;
}
template <int NL>
static KernelFn wb_kernel_for(int family, int block, bool philox, bool weighted) {
#define wb_fn_(F, WT, N) (philox ? wb_fn1<F, WT, N, true>(block) : wb_fn1<F, WT, N, false>(block))
    switch (family) {
        case FAM_DOMINO: return NL == 1 ? wb_fn_(FAM_DOMINO, 0, 1) : nullptr;  // not monotone: no coupled chains
        case FAM_DOMINO_HB: return weighted ? wb_fn_(FAM_DOMINO_HB, 1, NL) : wb_fn_(FAM_DOMINO_HB, 0, NL);
        case FAM_LOZENGE8: return weighted ? wb_fn_(FAM_LOZENGE8, 1, NL) : wb_fn_(FAM_LOZENGE8, 0, NL);
        case FAM_QLOZENGE8: return weighted ? nullptr : wb_fn_(FAM_LOZENGE8, 2, NL);
        default: return nullptr;
    }
#undef wb_fn_
}

rt_status plan_word_band(int family, int device, int nlat, int rows, int width, bool philox, int ctas_hint, bool weighted,
                         WalkPlan* plan, std::string* err) {
    int sms = 0, smem_optin = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) {
        *err = "cudaDeviceGetAttribute failed";
        return RT_E_CUDA;
    }
    const int nc = family == FAM_LOZENGE8 || family == FAM_QLOZENGE8 ? 3 : 2;
    const int wpad = (width + 3) & ~3, gw = wpad / 4;
    // Microseconds per step, this kernel / rt_word.cu.
    // Philox: Aztec diamonds of order 24 0.41 / 0.52, 50 0.48 / 0.65, 100 0.58 /
    // 0.75, 200 0.78 / 1.03, 300 (bands of 4 rows, H = 4) 0.99 / 1.00, 400 (6 rows,
    // H = 2) 1.44 / 1.10; hexagons of side 30 0.46 / 1.03, 100 0.62 / 0.80, 250 0.84 /
    // 1.38, 400 1.19 / 1.28, 450 (H = 3) 1.26 / 1.42, 500 (H = 2) 1.44 / 1.46; Aztec
    // diamond of order 350 (H = 3) 1.12 / 1.04; volume weight, 190 x 131 x 83 0.68 / 1.20.
    // TinyMT: Aztec diamonds of order 8 0.18 / 0.20, 24 0.28 / 0.35, 50 0.32 / 0.34,
    // 100 0.38 / 0.43, 200 0.48 / 0.56, 300 (H = 2) 0.54 / 0.55, 400 (803 words)
    // 0.94 / 0.64; hexagons of side 30 0.37 / 0.74, 60 0.40 / 0.51, 100 0.44 / 0.56,
    // 150 0.50 / 0.81, 250 0.64 / 0.92, 320 0.74 / 0.91, 500 (924 words) 1.21 / 1.00.
    // So: bands of four rows or more, until band and halo have some 200 to 270
    // words (order 24: 0.41 on 4 CTAs, 0.48 on 11; order 50: 0.58, 0.48, 0.52 on 8,
    // 16, 26); of two where TinyMT's draws would be the longer part (order 200: 0.47
    // on 148 CTAs with H = 2, 0.53 on 100, 0.62 there with H = 4).  Philox halos of
    // fewer than four rows (lozenges: three) and TinyMT bands beyond 640 words stay
    // on rt_word.cu.
    int ctas = ctas_hint;
    if (ctas <= 0) {
        const int band = std::max(!philox && gw > 40 ? 2 : 4, std::min(16, (philox ? 90 : 64) / gw));
        ctas = (int64_t)rows * gw <= (philox ? 192 : 100) ? 1 : std::min(sms, rows / band);
    }
    ctas = std::max(1, std::min(ctas, rows));
    const int rpc = (rows + ctas - 1) / ctas;
    const int most = philox ? 16 : 8, least = ctas == 1 ? 1 : !philox ? 2 : nc == 3 ? 3 : 4, room = philox ? 1024 : kWbBlockMid;
    int depth = ctas == 1 ? 1 : std::min(most, rows / ctas);
    while (depth > least && (int64_t)(rpc + 2 * depth) * gw > (philox ? room : 360)) --depth;
    const int64_t words = (int64_t)(rpc + 2 * depth) * gw;
    const size_t smem = 32 + (size_t)nlat * nc * (rpc + 2 * depth) * wpad;
    if (depth < least || words > room || smem > (size_t)smem_optin) {
        *err = "no room for a word per thread and a halo";
        return RT_E_INVAL;
    }
    const int block = (int)(words + 31) / 32 * 32;
    KernelFn fn = nlat == 1 ? wb_kernel_for<1>(family, block, philox, weighted) : wb_kernel_for<2>(family, block, philox, weighted);
    if (!fn) {
        *err = "no word kernel for this configuration";
        return RT_E_INVAL;
    }
    if (const rt_status s = allow_shared((const void*)fn, device, smem, err); s != RT_OK) return s;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)fn, block, smem) != cudaSuccess) {
        *err = "cudaOccupancyMaxActiveBlocksPerMultiprocessor failed";
        return RT_E_CUDA;
    }
    if (per_sm < 1 || ctas > per_sm * sms) {
        *err = "word-band grid cannot be co-resident";
        return RT_E_INVAL;
    }
    plan->items = 1;
    plan->block = block;
    plan->rows_per_cta = rpc;
    plan->ctas = ctas;
    plan->smem = smem;
    plan->wpad = wpad;
    plan->xwords = nc * depth * gw;
    plan->xslots = 1;
    plan->depth = depth;
    plan->merge_runs = !philox;
    plan->fn = (const void*)fn;
    return RT_OK;
}

}  // namespace rtb
