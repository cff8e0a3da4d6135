// rt_word.cu -- the word-parallel walk kernel of the int8 models.
//
// Dominoes (dominokernel.cl, dominokernelCFTP.cl) and lozenges
// (lozengekernel.cl, qlozengekernel.cl) store one byte per site.  This kernel
// treats a 32-bit word of four consecutive sites of a colour-array row as its
// unit of work: the Update of a colour is a handful of masks and byte shifts
// on words of the flipped colour (neighbours at j +- 1 are byte permutes of
// two adjacent words), the flip test is a per-byte compare, and each thread
// keeps the TinyMT states of the four positions of each of its words in
// registers for the whole walk (bit-exact mode) or draws them from one Philox
// call per word (fast mode).
//
// A phase is a run of steps that flip the same colour (the reference's random
// colour order repeats a colour with probability 1/2 or 1/3).  Within a run
// the sites' neighbours do not change, so its draws combine into two byte
// masks per word before the lattice is touched, and the lattice is refreshed,
// flipped and exchanged once per run instead of once per step.  The masks of
// the next phase are made while its rows are on their way.
//
// What bounds it: the integer work of the draws (about 100 instructions a
// word and step), the latency of one word's update, and the exchange.  On the
// a = b = c = 500 hexagon (148 CTAs) a step takes 0.98 us, 1.83 with a phase
// per step, a halo row copied through shared memory and a block-wide vote.
// Lattices whose bands have room for halo rows run on rt_wordband.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "rt_exchange.cuh"
#include "rt_internal.h"
#include "rt_models.cuh"
#include "rt_word.cuh"

namespace rtb {

constexpr int kWordBlockMax = 512;  // threads that keep 2 or 4 words' generator states each
constexpr int kWordBlockMid = 640;  // 65,536 registers / 96, in whole warps

// Shared memory: 16 bytes of slack, then for each lattice NC colour planes of
// (band rows + 2) x wpad bytes, then 16 bytes of slack (the funnel shifts read one
// word beyond a row; those bytes only reach sites outside the update / flip masks).
// MAXW: words per thread kept in registers (facts, draw masks and, in
// bit-exact mode, generator states); 0: words walked at run time (fast mode
// on large bands).
// WT: 0 the uniform rules; 1 periodic weights (a.wper > 0), a per-site
// threshold instead of thr[0]; 2 the lozenges' volume weight q
// (qlozengekernel.cl), add below thr[2], remove in [2^22, thr[3]).  Separate
// instantiations, so that the uniform kernel carries none of it.
// NL: lattices (2: coupled CFTP chains).
template <int FAM, int MAXW, bool PHILOX, int LB, int WT, int NL>
__global__ void __launch_bounds__(LB, 1) word_kernel(const __grid_constant__ WalkArgs a) {
    using M = WordModel<FAM>;
    constexpr int NC = M::NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* lat = smem_raw + 16;

    const int BLOCK = blockDim.x;
    const int cta = blockIdx.x, nct = gridDim.x, tid = threadIdx.x;
    const int r0 = cta * a.rows_per_cta;
    const int r1 = min(a.rows, r0 + a.rows_per_cta);
    const int nrows = r1 - r0;
    const int a0 = r0 + M::ROFF;
    const int W = a.wpad;
    const int plane = (nrows + 2) * W;
    const int Gw = W >> 2;  // words per row (the fast mode's counter stride too)
    const int nwords = nrows * Gw;
    const int N = a.n;
    const WordExchange<false> xch{a, nullptr, cta};
    for (int l = 0; l < NL; ++l)
        for (int c = 0; c < NC; ++c) {
            const int8_t* g = static_cast<const int8_t*>(a.arr[l][c]);
            unsigned char* s = lat + (l * NC + c) * plane;
            for (int e = tid; e < plane; e += BLOCK) {
                const int rr = a0 - 1 + e / W, j = e % W;
                int8_t v = 0;
                if (rr >= 0 && rr < a.arows && j < a.width) v = g[(size_t)rr * a.width + j];
                s[e] = (unsigned char)v;
            }
        }

    const bool has_top = cta > 0, has_bot = cta + 1 < nct;
    // Update mask of band row rr / word w: rows 1..N-2, columns 1..width-2;
    // Rotate positions: columns COFF..COFF+cols-1 (all band rows).
    auto info_at = [&](int rr, int w) {
        WordInfo wi;
        wi.off = (rr + 1) * W + 4 * w;
        const int i = a0 + rr;
        wi.cls = M::DOM ? (i & 1) : i % 3;
        const int j0 = 4 * w;
        uint32_t ub = 0, vb = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int j = j0 + b;
            if (j >= 1 && j <= a.width - 2) ub |= 1u << b;
            if (j >= M::COFF && j < M::COFF + a.cols) vb |= 1u << b;
        }
        if (!(i >= 1 && i <= N - 2)) ub = 0;
        wi.um = lane_bytes(ub) * 0xffu;
        wi.vm = lane_bytes(vb) << 7;
        return wi;
    };
    // Decoded phases: a table, or for the largest bands (MAXW = 0), where its 512
    // bytes would cost the last sides that fit, this phase's and the next one's.
    constexpr bool TABLE = MAXW > 0;
    __shared__ WordPhase s_phase[TABLE ? kWordPhases : 2];
    __shared__ uint4 s_sel[kLozengeSel];
    if (TABLE && tid < kWordPhases) s_phase[TABLE ? tid : 0] = word_phase_entry<FAM>(tid, plane);
    if (tid < kLozengeSel) s_sel[tid] = lozenge_sel_entry(tid);
    __shared__ int s_fail[2];
    if (tid < 2) s_fail[tid] = 0;
    const uint32_t nt0 = 0u - (WT == 2 ? a.thr[2] : a.thr[0]), nt1 = 0u - (WT == 2 ? a.thr[3] : a.thr[1]);

    // The words u = tid + m * BLOCK (m < MAXW) of this thread.
    constexpr int NW = MAXW > 0 ? MAXW : 1;
    WordInfo winfo[NW];
    int wcol[NW];  // word column
    TinyState st[PHILOX ? 1 : NW][4];
    uint32_t wflags = 0;  // per word, 4 bits: it exists, it is in the band's first row / last row next to another CTA
    if (MAXW > 0) {
#pragma unroll
        for (int m = 0; m < MAXW; ++m) {
            const int u = tid + m * BLOCK;
            if (u < nwords) {
                const int rr = u / Gw;
                wcol[m] = u - rr * Gw;
                winfo[m] = info_at(rr, wcol[m]);
                wflags |= (1u | (has_top && rr == 0 ? 2u : 0u) | (has_bot && rr == nrows - 1 ? 4u : 0u)) << (4 * m);
            } else {
                winfo[m] = WordInfo{0, 0, 0u, 0u};
                wcol[m] = 0;
            }
        }
    }
    const TinyParams tp{a.mat1, a.mat2, a.tmat};

    int epoch = -1;
    int64_t next_epoch = a.nepochs > 0 ? a.epoch_start[0] : INT64_MAX;
    uint32_t key0 = 0, key1 = 0;
    int64_t dstep = 0;
    // Draws restart at phase `ph` when an epoch begins there.
    auto begin_phase = [&](int64_t ph) {
        if (ph != next_epoch) return;
        while (epoch + 1 < a.nepochs && a.epoch_start[epoch + 1] == ph) ++epoch;
        next_epoch = epoch + 1 < a.nepochs ? a.epoch_start[epoch + 1] : INT64_MAX;
        const uint64_t eseed = a.epoch_seed[epoch];
        if (PHILOX) {
            key0 = (uint32_t)eseed;
            key1 = (uint32_t)(eseed >> 32);
            dstep = 0;
        } else {
            // A site that is not a Rotate position has no stream; what its
            // generator holds is never used.
#pragma unroll
            for (int m = 0; m < NW; ++m) {
                if (!(wflags >> (4 * m) & 1u)) continue;
                const int rpos = r0 + winfo[m].off / W - 1;  // position row
                const int jw = winfo[m].off % W;             // 4 * word
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint32_t sid = (uint32_t)(jw + b - M::COFF) + (uint32_t)a.cols * (uint32_t)rpos;
                    tiny_seed(st[PHILOX ? 0 : m][b], tp, (uint32_t)eseed + sid);
                }
            }
        }
    };
    auto combine = [&](uint32_t d, const WordInfo& wi, const uint32_t (&k)[4], uint32_t& m0, uint32_t& m1) {
        word_combine<FAM, WT>(a, d, a0 + wi.off / W - 1, wi.off % W, k, nt0, nt1, m0, m1);
    };
    auto philox_draws = [&](uint32_t d, int u, const WordInfo& wi, int64_t s, uint32_t& m0, uint32_t& m1) {
        m0 = m1 = 0u;
        if (!(d & PH_DRAWS)) return;
        // the fast mode's colours go round in turn: one step a phase
        const uint4 w4 =
            philox4((uint32_t)(a0 * Gw + u), (uint32_t)s, (uint32_t)((uint64_t)s >> 32), a.chain, key0, key1);
        const uint32_t k[4] = {w4.x, w4.y, w4.z, w4.w};
        combine(d, wi, k, m0, m1);
    };
    // The masks of this thread's words for phase descriptor d.  They depend on
    // the draws alone, so they are made a phase ahead, while the rows the
    // phase needs are on their way.
    uint32_t mk0[NW], mk1[NW];
    auto draw_masks = [&](uint32_t d) {
#pragma unroll
        for (int m = 0; m < NW; ++m) {
            mk0[m] = mk1[m] = 0u;
            if (!(wflags >> (4 * m) & 1u) || !(d & PH_DRAWS)) continue;
            if (PHILOX) {
                philox_draws(d, (winfo[m].off >> 2) - Gw, winfo[m], dstep, mk0[m], mk1[m]);
            } else {
#pragma unroll 1
                for (uint32_t c = 0; c < ph_steps(d); ++c) {
                    uint32_t k[4];
#pragma unroll
                    for (int b = 0; b < 4; ++b) k[b] = tiny_draw32(st[PHILOX ? 0 : m][b], tp);
                    combine(d, winfo[m], k, mk0[m], mk1[m]);
                }
            }
        }
        if (PHILOX && (d & PH_DRAWS)) ++dstep;
    };

    // Phases that need more than the plain loop body: those that begin an
    // epoch (a phase earlier where the draws are made ahead), the tests'
    // withheld one and the last two.  Returns how many phases after `ph` the
    // next one comes.
    auto until_special = [&](int64_t ph) {
        int64_t s = a.nphases - 2;
        const int64_t e = MAXW > 0 ? next_epoch - 1 : next_epoch;
        if (e >= ph) s = min(s, e);
        if (cta == 0 && a.drop_phase >= ph) s = min(s, a.drop_phase);
        return (int)min(max(s - ph, (int64_t)0), (int64_t)1 << 30);
    };
    uint32_t d = a.nphases > 0 ? __ldg(a.phases) : 0u;
    uint32_t d_next = a.nphases > 1 ? __ldg(a.phases + 1) : 0u;
    if (MAXW > 0 && a.nphases > 0) {
        begin_phase(0);
        draw_masks(d);
    }
    const uint32_t* ahead = a.phases + 2;  // the descriptor two phases on
    const int lat1 = NC * plane;           // second lattice (coupled CFTP chains)
    uint32_t p32 = 0;                      // phase number modulo 2^32
    int until = until_special(0);
    bool fail = false, more = a.nphases > 0;
    if (!TABLE && tid == 0) s_phase[0] = word_phase_entry<FAM>(word_phase_index(d), plane);
    __syncthreads();
    WordPhase P = s_phase[TABLE ? word_phase_index(d) : 0];
    while (more) {
        const int par = (int)(p32 & 1u);
        const bool failed = *(volatile int*)&s_fail[1 - par] != 0;
        if (!TABLE && tid == 0) s_phase[1 - par] = word_phase_entry<FAM>(word_phase_index(d_next), plane);
        const bool first = ahead == a.phases + 2;
        // Rows are exchanged after every phase but the last, whether or not the
        // next one has an Update pending: the waits keep the slots' order.
        bool pub = true;
        uint32_t d_after = 0u;
        if (until-- > 0) {
            d_after = __ldg(ahead);
        } else {
            const int64_t ph = ahead - a.phases - 2;
            if (ph + 2 < a.nphases) d_after = __ldg(ahead);
            more = ph + 1 < a.nphases;
            pub = more && !(cta == 0 && ph == a.drop_phase);
            if (MAXW == 0)
                begin_phase(ph);
            else if (more)
                begin_phase(ph + 1);
            until = until_special(ph + 1);
        }
        ++ahead;
        // One word: flags bit 1 (2) -- it needs the row above (below) the band
        // from the neighbour and publishes itself to it.
        auto do_word = [&](const WordInfo& wi, int w, uint32_t flags, uint32_t m0, uint32_t m1) {
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                unsigned char* const L = lat + l * lat1;
                WordOp<FAM> op;
                WordNbr nb;
                op.load_up(nb, L, P, wi, W);
                op.load_dn(nb, L, P, wi, W);
                if (flags && !first) {
                    bool ok = true;
                    if (flags & 2u) ok = xch.read(0, 1 - par, l, w, M::DOM ? w : min(w + 1, Gw - 1), p32, nb.up);
                    if (ok && (flags & 4u)) ok = xch.read(1, 1 - par, l, w, M::DOM ? w : max(w - 1, 0), p32, nb.dn);
                    if (!ok) {
                        fail = true;
                        return;
                    }
                }
                op.begin(L, P, wi, s_sel);
                op.finish(P, wi, nb, m0, m1);
                if (pub) {
                    if (flags & 2u) xch.write(0, par, l, w, p32 + 1u, op.v);
                    if (flags & 4u) xch.write(1, par, l, w, p32 + 1u, op.v);
                }
                op.store(L, P, wi);
            }
        };
        if (MAXW > 0) {
            // words away from the neighbours first
#pragma unroll
            for (int m = 0; m < NW; ++m)
                if ((wflags >> (4 * m) & 7u) == 1u) do_word(winfo[m], 0, 0u, mk0[m], mk1[m]);
#pragma unroll
            for (int m = 0; m < NW; ++m)
                if (wflags >> (4 * m) & 6u) do_word(winfo[m], wcol[m], wflags >> (4 * m) & 6u, mk0[m], mk1[m]);
            draw_masks(d_next);  // none after the last phase
        } else {
            // Words walked with an incremental (row, word) pair; the edge rows last.
            auto range = [&](int u_lo, int u_hi, uint32_t flags) {
                int u = u_lo + tid;
                if (u >= u_hi) return;
                int rr = u / Gw, w = u - rr * Gw;
                const int drr = BLOCK / Gw, dw = BLOCK - drr * Gw;
                for (; u < u_hi; u += BLOCK) {
                    const WordInfo wi = info_at(rr, w);
                    uint32_t m0, m1;
                    philox_draws(d, u, wi, dstep, m0, m1);
                    do_word(wi, w, flags, m0, m1);
                    rr += drr;
                    w += dw;
                    if (w >= Gw) {
                        w -= Gw;
                        ++rr;
                    }
                }
            };
            const bool one = has_top && has_bot && nrows == 1;
            range(has_top ? Gw : 0, nwords - (has_bot ? Gw : 0), 0u);
            if (has_top) range(0, Gw, one ? 6u : 2u);
            if (has_bot && !one) range(nwords - Gw, nwords, 4u);
            if (d & PH_DRAWS) ++dstep;
        }
        d = d_next;
        d_next = d_after;
        if (TABLE) P = s_phase[TABLE ? word_phase_index(d) : 0];
        // A wait that ran out is seen by every thread one phase later: the flag
        // of this phase is read after its barrier and acted on before the next
        // one, and not written again until then.
        if (fail) s_fail[par] = 1;
        if (failed) break;
        __syncthreads();
        if (!TABLE) P = s_phase[1 - par];
        ++p32;
    }
    __syncthreads();
    if (s_fail[0] | s_fail[1]) return;
    for (int l = 0; l < NL; ++l)
        for (int c = 0; c < NC; ++c) {
            int8_t* g = static_cast<int8_t*>(a.arr[l][c]);
            const unsigned char* s = lat + (l * NC + c) * plane;
            for (int e = tid; e < nrows * a.width; e += BLOCK) {
                const int rr = e / a.width, j = e % a.width;
                g[(size_t)(a0 + rr) * a.width + j] = (int8_t)s[(rr + 1) * W + j];
            }
        }
}

using KernelFn = void (*)(WalkArgs);

// One word per thread, up to `block` threads: blocks of at most kWordBlockMid
// threads have 96 registers a thread instead of 64.
template <int FAM, bool PHILOX, int WT, int NL>
static KernelFn word_fn1(int block) {
    return block <= kWordBlockMid ? word_kernel<FAM, 1, PHILOX, kWordBlockMid, WT, NL>
                                  : word_kernel<FAM, 1, PHILOX, 1024, WT, NL>;
}
template <int FAM, int WT, int NL>
static KernelFn word_fn(int maxw, int block, bool philox) {
    if (maxw == 1) return philox ? word_fn1<FAM, true, WT, NL>(block) : word_fn1<FAM, false, WT, NL>(block);
    if (philox) {
        switch (maxw) {
            case 0: return word_kernel<FAM, 0, true, 1024, WT, NL>;
            case 2: return word_kernel<FAM, 2, true, 1024, WT, NL>;
            case 4: return word_kernel<FAM, 4, true, 1024, WT, NL>;
            default: return nullptr;
        }
    }
    switch (maxw) {
        case 2: return word_kernel<FAM, 2, false, 512, WT, NL>;
        case 4: return word_kernel<FAM, 4, false, 512, WT, NL>;
        default: return nullptr;
    }
}

template <int NL>
static KernelFn word_kernel_for(int family, int maxw, int block, bool philox, bool weighted) {
    switch (family) {
        case FAM_DOMINO:  // not monotone: no coupled chains
            return NL == 1 ? word_fn<FAM_DOMINO, 0, 1>(maxw, block, philox) : nullptr;
        case FAM_DOMINO_HB:
            return weighted ? word_fn<FAM_DOMINO_HB, 1, NL>(maxw, block, philox)
                            : word_fn<FAM_DOMINO_HB, 0, NL>(maxw, block, philox);
        case FAM_LOZENGE8:
            return weighted ? word_fn<FAM_LOZENGE8, 1, NL>(maxw, block, philox)
                            : word_fn<FAM_LOZENGE8, 0, NL>(maxw, block, philox);
        case FAM_QLOZENGE8: return weighted ? nullptr : word_fn<FAM_LOZENGE8, 2, NL>(maxw, block, philox);
        default: return nullptr;
    }
}

bool word_family(int family) { return family == FAM_DOMINO || family == FAM_DOMINO_HB || family == FAM_LOZENGE8; }

// Plans the walk on (at most) `ctas` co-resident CTAs.
static rt_status plan_word_grid(int family, int device, int nlat, int rows, int width, bool philox, int ctas,
                                bool weighted, WalkPlan* plan, std::string* err) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        *err = "cudaDeviceGetAttribute failed";
        return RT_E_CUDA;
    }
    const int nc = family == FAM_LOZENGE8 || family == FAM_QLOZENGE8 ? 3 : 2;
    const int wpad = (width + 3) & ~3;
    const int gw = wpad / 4;
    const int rpc = (rows + ctas - 1) / ctas;
    ctas = (rows + rpc - 1) / rpc;
    const int words = rpc * gw;
    // One word per thread up to 1024 threads; bit-exact mode then keeps 2
    // or 4 words' generator states per thread in registers (512 threads).
    int maxw = 1, block = 0;
    if (philox) {
        // Fast mode keeps no generator state: up to 4 words' facts per thread
        // in registers, beyond that words are walked at run time.
        maxw = words <= 1024 ? 1 : words <= 2048 ? 2 : words <= 4096 ? 4 : 0;
        block = maxw == 0 ? 1024 : std::min(1024, ((words + maxw - 1) / maxw + 31) / 32 * 32);
    } else if (words <= 1024) {
        block = (words + 31) / 32 * 32;
    } else {
        for (maxw = 2; maxw <= 4; maxw *= 2)
            if ((words + maxw - 1) / maxw <= kWordBlockMax) break;
        if (maxw > 4) {
            *err = "band too wide for register-resident generator states";
            return RT_E_INVAL;
        }
        block = ((words + maxw - 1) / maxw + 31) / 32 * 32;
    }
    const size_t smem = 32 + (size_t)nlat * nc * (rpc + 2) * wpad;
    KernelFn fn = nlat == 1 ? word_kernel_for<1>(family, maxw, block, philox, weighted)
                            : word_kernel_for<2>(family, maxw, block, philox, weighted);
    if (!fn) {
        *err = "no word kernel for this configuration";
        return RT_E_INVAL;
    }
    if (const rt_status s = allow_shared((const void*)fn, device, smem, err); s != RT_OK) return s;
    plan->items = maxw;
    plan->block = block;
    plan->rows_per_cta = rpc;
    plan->ctas = ctas;
    plan->smem = smem;
    plan->wpad = wpad;
    plan->xwords = gw;
    plan->xslots = 1;
    plan->merge_runs = true;
    plan->fn = (const void*)fn;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)fn, block, smem) != cudaSuccess) {
        *err = "cudaOccupancyMaxActiveBlocksPerMultiprocessor failed";
        return RT_E_CUDA;
    }
    if (per_sm < 1 || ctas > per_sm * sms) {
        *err = "word-kernel grid cannot be co-resident";
        return RT_E_INVAL;
    }
    return RT_OK;
}

rt_status plan_word_walk(int family, int device, int nlat, int rows, int width, bool philox, int ctas_hint,
                         WalkPlan* plan, std::string* err, bool weighted) {
    if (!word_family(family) && family != FAM_QLOZENGE8) {
        *err = "no word kernel for this model";
        return RT_E_INVAL;
    }
    // Small and middle lattices run on bands with halos (ctas_hint < 0: not wanted).
    if (ctas_hint >= 0 &&
        plan_word_band(family, device, nlat, rows, width, philox, ctas_hint, weighted, plan, err) == RT_OK)
        return RT_OK;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        *err = "cudaDeviceGetAttribute failed";
        return RT_E_CUDA;
    }
    // What gets here is larger than the bands' words, or (the walk of a program
    // that owns the memory) has no scratch left for their slots.  Microseconds per
    // step (Aztec diamonds TinyMT / hexagons TinyMT / hexagons Philox; words =
    // 32-bit words of one colour array):
    //   CTAs     378-432 words     945-1326          9,156            13,366-13,872
    //   1        0.34 0.58 0.75    1.09 1.07 1.40    -                -
    //   74       0.63 1.12 1.63    0.75 1.33 1.96    -    0.89 1.37   0.55 0.90 1.34
    //   148      0.63 1.12 1.62    0.67 1.17 1.75    -    0.88 1.32   0.51 0.86 1.26
    // So: one CTA (no exchange) while three warps a scheduler hold the lattice;
    // else the whole GPU, with bands of three rows or more, whose first and last
    // rows are different warps' (258 rows: 0.71 at two rows a band, 0.54 at four).
    int ctas = ctas_hint;
    if (ctas_hint <= 0) ctas = (int64_t)rows * ((width + 3) / 4) <= 384 ? 1 : std::min(sms, rows / 3);
    ctas = std::max(1, std::min(ctas, rows));
    return plan_word_grid(family, device, nlat, rows, width, philox, ctas, weighted, plan, err);
}

}  // namespace rtb
