// rt_recttri.cu -- the rectangle-triangle walk, one site per thread.
//
// A site (six hex face digits, recttrianglekernel.cl) is refreshed by copying
// digits of three neighbours of the colour flipped last; nothing of its old
// value is kept.  So a phase refreshes only the colour that it flips -- the
// third colour is written anew before it is read -- and a run of steps that
// flip the same colour (the reference repeats a colour with probability 1/3)
// is one phase: its draws are made a phase ahead, and each site takes its
// moves one after the other in a register.
//
// What bounds it: the latency of one site's update and the exchange of the
// rows next to a band.  A step takes 0.60 us on a 135 x 135 tiling (6,075 sites
// a colour, one cluster of 16) and 0.40 us on a 21 x 21 one (one CTA); the
// generic kernel, with a phase per step on 135 CTAs of one row, took 2.9 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "rt_exchange.cuh"
#include "rt_internal.h"
#include "rt_models.cuh"
#include "rt_rtmoves.cuh"

namespace rtb {

constexpr int kRtClusterMax = 16;   // CTAs of the largest thread-block cluster (non-portable size)
constexpr int kRtBlockMid = 640;    // 65,536 registers / 96, in whole warps
constexpr int kRtAhead = 3;         // draws of a run made ahead (longer runs: 1 in 27, the rest in place)

// Shared memory: the inbox (CLUSTER), then three colour planes of (band rows
// + 2) x wpad sites.
template <bool PHILOX, bool CLUSTER, int LB>
__global__ void __launch_bounds__(LB, 1) recttri_kernel(const __grid_constant__ WalkArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_fail[2];
    __shared__ RectTriMoves s_moves;
    const int inbox_words = CLUSTER ? 4 * a.xwords : 0;
    int* const lat = reinterpret_cast<int*>(smem_raw + (size_t)inbox_words * 8);

    const int BLOCK = blockDim.x;
    const int cta = blockIdx.x, nct = gridDim.x, tid = threadIdx.x;
    const int r0 = cta * a.rows_per_cta;
    const int r1 = min(a.rows, r0 + a.rows_per_cta);
    const int W = a.wpad;
    const int plane = (r1 - r0 + 2) * W;
    const WordExchange<CLUSTER> xch{a, reinterpret_cast<unsigned long long*>(smem_raw), cta};

    if (CLUSTER) {
        for (int e = tid; e < inbox_words; e += BLOCK) xch.inbox[e] = 0ull;
        __syncthreads();
        cluster_sync_all();  // every inbox is clear before anyone writes into it
    }
    for (int c = 0; c < 3; ++c) {
        const int32_t* g = static_cast<const int32_t*>(a.arr[0][c]);
        for (int e = tid; e < plane; e += BLOCK) {
            const int rr = r0 - 1 + e / W, j = e % W;
            lat[c * plane + e] = rr >= 0 && rr < a.arows && j < a.width ? g[(size_t)rr * a.width + j] : 0;
        }
    }
    if (tid < 2) s_fail[tid] = 0;
    s_moves.clear(tid, BLOCK);
    __syncthreads();
    s_moves.fill(a, tid, BLOCK);

    // This thread's site (i, j).
    const bool live = tid < (r1 - r0) * a.cols;
    const int i = live ? r0 + tid / a.cols : r0, j = live ? tid % a.cols : 0;
    const int off = (i - r0 + 1) * W + j;
    const int cls = i % 3;
    const bool inner = live && i >= 1 && i <= a.n - 2 && j >= 1 && j <= a.width - 2;
    const bool top = live && cta > 0 && i == r0, bot = live && cta + 1 < nct && i == r1 - 1;
    const int j_up = min(j + 1, a.width - 1), j_dn = max(j - 1, 0);
    const uint32_t sid = (uint32_t)j + (uint32_t)a.cols * (uint32_t)i;
    TinyParams tp{a.mat1, a.mat2, a.tmat};
    if (!PHILOX && live && a.params) {
        const uint4 p = __ldg(a.params + sid);
        tp = TinyParams{p.x, p.y, p.z};
    }
    TinyState st{0u, 0u, 0u, 0u};
    const uint32_t quad = (uint32_t)i * (uint32_t)(W >> 2) + (uint32_t)(j >> 2);

    int epoch = -1;
    int64_t next_epoch = a.nepochs > 0 ? a.epoch_start[0] : INT64_MAX;
    uint32_t key0 = 0, key1 = 0;
    int64_t dstep = 0;
    auto begin_phase = [&](int64_t ph) {
        if (ph != next_epoch) return;
        while (epoch + 1 < a.nepochs && a.epoch_start[epoch + 1] == ph) ++epoch;
        next_epoch = epoch + 1 < a.nepochs ? a.epoch_start[epoch + 1] : INT64_MAX;
        const uint64_t eseed = a.epoch_seed[epoch];
        key0 = (uint32_t)eseed;
        key1 = (uint32_t)(eseed >> 32);
        dstep = 0;
        if (!PHILOX) tiny_seed(st, tp, key0 + sid);
    };
    auto draw = [&]() -> uint32_t {
        if (!PHILOX) return RectTriMoves::prepare(tiny_draw23(st, tp));
        const uint4 w = philox4(quad, (uint32_t)dstep, (uint32_t)((uint64_t)dstep >> 32), a.chain, key0, key1);
        ++dstep;
        return RectTriMoves::prepare(quad_word(w, j & 3) >> 9);
    };
    uint32_t kd[kRtAhead];
    auto draw_ahead = [&](uint32_t d) {
#pragma unroll
        for (int c = 0; c < kRtAhead; ++c)
            if ((d & PH_DRAWS) && c < (int)ph_steps(d)) kd[c] = draw();
    };

    uint32_t d = a.nphases > 0 ? __ldg(a.phases) : 0u;
    uint32_t d_next = a.nphases > 1 ? __ldg(a.phases + 1) : 0u;
    if (a.nphases > 0) {
        begin_phase(0);
        draw_ahead(d);
    }
    bool fail = false;
    __syncthreads();
    for (int64_t ph = 0; ph < a.nphases; ++ph) {
        const int par = (int)(ph & 1);
        const bool failed = *(volatile int*)&s_fail[1 - par] != 0;
        const uint32_t d_after = ph + 2 < a.nphases ? __ldg(a.phases + ph + 2) : 0u;
        const bool pub = ph + 1 < a.nphases && !(cta == 0 && ph == a.drop_phase);
        // STEP: apply the pending Update of colour t to the colour ca that is
        // flipped; FINAL: to both other colours.
        const bool step = ph_op(d) == OP_STEP;
        const int ca = (int)ph_a(d), cb = (int)ph_b(d);
        const bool upd = !step || (cb != (int)NO_COLOUR && cb != ca);
        const int t = step ? (upd ? cb : 0) : ca;
        const int t1 = t == 2 ? 0 : t + 1, t2 = t == 0 ? 2 : t - 1;
        const int s1 = cls == t, s2 = cls == t1, s3 = cls == t2;  // column shifts of the reads
        if (live) {
            const int* const f = lat + t * plane + off;
            int up = f[-W], upr = f[s2 - W], low = f[W - s2], down = f[W];
            const int east = f[s1], west = f[-s3];
            if ((top | bot) && ph > 0) {
                uint32_t x[2];
                bool ok = true;
                if (top && (ok = xch.read(0, 1 - par, 0, j, j_up, (uint32_t)ph, x))) {
                    up = (int)x[0];
                    upr = (int)x[s2];
                }
                if (bot && ok && (ok = xch.read(1, 1 - par, 0, j, j_dn, (uint32_t)ph, x))) {
                    down = (int)x[0];
                    low = (int)x[s2];
                }
                fail |= !ok;
            }
            const int na = rt_next(up, east, low), nb = rt_next2(west, upr, down);
            if (step) {
                int* const cur = lat + ca * plane + off;
                int v = upd && inner ? (ca == t1 ? na : nb) : *cur;
                if (d & PH_DRAWS) {
                    const int ns = (int)ph_steps(d);
#pragma unroll
                    for (int c = 0; c < kRtAhead; ++c)
                        if (c < ns) v = s_moves.flip(v, kd[c]);
                    for (int c = kRtAhead; c < ns; ++c) v = s_moves.flip(v, draw());
                }
                if (pub && !fail) {
                    if (top) xch.write(0, par, 0, j, (uint32_t)ph + 1u, (uint32_t)v);
                    if (bot) xch.write(1, par, 0, j, (uint32_t)ph + 1u, (uint32_t)v);
                }
                *cur = v;
            } else if (inner) {
                lat[t1 * plane + off] = na;
                lat[t2 * plane + off] = nb;
            }
        }
        if (ph + 1 < a.nphases) {
            begin_phase(ph + 1);
            draw_ahead(d_next);
        }
        d = d_next;
        d_next = d_after;
        // A wait that ran out is seen by every thread one phase later: the flag
        // of this phase is read after its barrier and acted on before the next.
        if (fail) s_fail[par] = 1;
        if (failed) break;
        __syncthreads();
    }
    __syncthreads();
    if (CLUSTER) cluster_sync_all();  // no CTA leaves while another may write into its inbox
    if (s_fail[0] | s_fail[1]) return;
    for (int c = 0; c < 3; ++c) {
        int32_t* g = static_cast<int32_t*>(a.arr[0][c]);
        for (int e = tid; e < (r1 - r0) * a.width; e += BLOCK) {
            const int rr = e / a.width, jj = e % a.width;
            g[(size_t)(r0 + rr) * a.width + jj] = lat[c * plane + (rr + 1) * W + jj];
        }
    }
}

using KernelFn = void (*)(WalkArgs);

static rt_status plan_recttri_grid(int device, int rows, int width, bool philox, int ctas, bool cluster,
                                   WalkPlan* plan, std::string* err) {
    int sms = 0, smem_optin = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) {
        *err = "cudaDeviceGetAttribute failed";
        return RT_E_CUDA;
    }
    const int rpc = (rows + ctas - 1) / ctas;
    ctas = (rows + rpc - 1) / rpc;
    cluster = cluster && ctas > 1;
    const int64_t sites = (int64_t)rpc * width;
    const int wpad = (width + 3) & ~3;
    const size_t smem = (size_t)3 * (rpc + 2) * wpad * 4 + (cluster ? (size_t)4 * wpad * 8 : (size_t)0);
    if (sites > 1024 || smem > (size_t)smem_optin) {
        *err = "rectangle-triangle band too large for one site per thread";
        return RT_E_INVAL;
    }
    const int block = std::max(32, (int)((sites + 31) / 32 * 32));
    KernelFn fn;
    if (block <= kRtBlockMid)
        fn = cluster ? (philox ? recttri_kernel<true, true, kRtBlockMid> : recttri_kernel<false, true, kRtBlockMid>)
                     : (philox ? recttri_kernel<true, false, kRtBlockMid> : recttri_kernel<false, false, kRtBlockMid>);
    else
        fn = cluster ? (philox ? recttri_kernel<true, true, 1024> : recttri_kernel<false, true, 1024>)
                     : (philox ? recttri_kernel<true, false, 1024> : recttri_kernel<false, false, 1024>);
    if (const rt_status s = allow_shared((const void*)fn, device, smem, err); s != RT_OK) return s;
    if (cluster && cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        *err = "cudaFuncSetAttribute failed";
        return RT_E_CUDA;
    }
    plan->items = 1;
    plan->block = block;
    plan->rows_per_cta = rpc;
    plan->ctas = ctas;
    plan->smem = smem;
    plan->wpad = wpad;
    plan->xwords = wpad;
    plan->xslots = 1;
    plan->cluster = cluster;
    plan->merge_runs = true;
    plan->fn = (const void*)fn;
    if (cluster) {
        int active = 0;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        walk_launch_config(*plan, &cfg, attr);
        if (cudaOccupancyMaxActiveClusters(&active, (const void*)fn, &cfg) != cudaSuccess || active < 1) {
            cudaGetLastError();
            *err = "rectangle-triangle cluster cannot be resident";
            return RT_E_INVAL;
        }
        return RT_OK;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)fn, block, smem) != cudaSuccess) {
        *err = "cudaOccupancyMaxActiveBlocksPerMultiprocessor failed";
        return RT_E_CUDA;
    }
    if (per_sm < 1 || ctas > per_sm * sms) {
        *err = "rectangle-triangle grid cannot be co-resident";
        return RT_E_INVAL;
    }
    return RT_OK;
}

rt_status plan_recttri_walk(int device, int rows, int width, bool philox, int ctas_hint, WalkPlan* plan,
                            std::string* err) {
    int sms = 0;
    if (rows < 1 || width < 1 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        *err = "cudaDeviceGetAttribute failed";
        return RT_E_CUDA;
    }
    // Microseconds per step, TinyMT (Philox adds 0.4 to 0.6), by sites of a colour:
    //   CTAs      147   363   507   768   1,323  6,075  11,907  31,827
    //   1         0.40  0.47  0.53  0.72  -      -      -       -
    //   16        0.62  0.61  0.61  0.50  0.51   0.60   0.71    -
    //   68 to 90  -     -     -     -     -      1.15   0.80    0.92
    //   136, 148  -     -     -     -     -      1.14   0.94    0.86
    // So: one CTA, which exchanges nothing, up to 512 sites; one cluster of 16
    // while its blocks hold the lattice; else the whole GPU.
    const int64_t sites = (int64_t)rows * width;
    bool cluster = ctas_hint > 0 && ctas_hint <= kRtClusterMax;
    int ctas = ctas_hint;
    if (ctas_hint <= 0) {
        cluster = sites <= (int64_t)kRtClusterMax * 1024;
        ctas = sites <= 512 ? 1 : cluster ? kRtClusterMax : std::min(sms, rows / 3);
    }
    ctas = std::max(1, std::min(ctas, rows));
    if (cluster && plan_recttri_grid(device, rows, width, philox, ctas, true, plan, err) == RT_OK) return RT_OK;
    if (ctas_hint <= 0) ctas = std::max(1, std::min(sms, rows / 3));
    return plan_recttri_grid(device, rows, width, philox, ctas, false, plan, err);
}

}  // namespace rtb
