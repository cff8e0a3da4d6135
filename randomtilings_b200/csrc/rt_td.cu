// rt_td.cu -- the single triangle-dimer walk on bit planes.
//
// The phase program (rt_tdschedule.h) runs on the chain's bit planes
// (rt_tdwalk.cuh) in the shared memory of one thread-block cluster, for the
// whole walk.  Bit-exact mode keeps the TinyMT states of the CTA's positions in
// shared memory, the 32 of a word side by side; a warp advances the 32
// generators of a word and their 32 "k < 2^22" decisions are one ballot.  Warps
// of their own make the decisions of the next drawing phase while the others
// run the phases; the two meet at drawing phases and exchanges.
//
// What bounds it: the latency of a phase -- one word's operation, about 1,000
// cycles, and the barrier -- since 18,496 sites are 680 words.  The int32 kernel
// took one CTA per array row and exchanged halo rows through global memory
// after each of the reference's 5.7 phases a move.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "rt_internal.h"
#include "rt_models.cuh"
#include "rt_tdwalk.cuh"

namespace rtb {

constexpr int kTdBlock = 512;
constexpr int kTdDeciders = 256;  // threads that make the decisions (bit-exact mode)

template <bool PHILOX>
__global__ void __launch_bounds__(kTdBlock, 1) td_walk_kernel(const __grid_constant__ WalkArgs a) {
    cg::cluster_group cluster = cg::this_cluster();
    const int CL = (int)gridDim.x, rank = (int)blockIdx.x;
    const int BLOCK = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    // threads that run the phases; the others decide
    const int RUN = BLOCK - (PHILOX ? 0 : kTdDeciders);
    extern __shared__ __align__(16) uint32_t td_smem[];
    const int ctas = min(CL, a.rows), halo = td_halo(a.rows, ctas, td_halo_cap(PHILOX));
    const int wb = (a.width + 31) >> 5, slots = ((a.rows + ctas - 1) / ctas + 2 * halo) * wb;
    // TinyMT: [s0 | s1 | s2 | s3][word][lane], then the decisions of two drawing
    // phases, for the band's rows and its halo's
    uint32_t* st = td_smem;
    uint32_t* draws = st + (PHILOX ? 0 : 4 * 32 * slots);
    uint32_t* sm = draws + (PHILOX ? 0 : 2 * slots);
    TdBand<tdp::AllBits> band(sm, a.rows, a.width, a.n / 2, rank, CL, td_halo_cap(PHILOX), min(tid, RUN - 1), RUN);
    const int first = max(0, band.row0), words = (min(a.rows, band.r1 + halo) - first) * wb;  // rows that draw

    for (int e = tid; e < (int)td_band_words(a.rows, a.width, ctas, td_halo_cap(PHILOX), tdp::kPlanes); e += BLOCK) sm[e] = 0u;
    __syncthreads();
    td_load(band, a.arr[0], a.arows, tid >> 5, BLOCK >> 5, lane);
    __syncthreads();

    int epoch = -1;
    int64_t next_epoch = a.nepochs > 0 ? a.epoch_start[0] : INT64_MAX;
    // Epochs that begin up to phase `ph`: true if one does, its seed in *seed.
    auto new_epoch = [&](int64_t ph, uint64_t* seed) {
        if (next_epoch > ph) return false;
        while (epoch + 1 < a.nepochs && a.epoch_start[epoch + 1] <= ph) ++epoch;
        next_epoch = epoch + 1 < a.nepochs ? a.epoch_start[epoch + 1] : INT64_MAX;
        *seed = a.epoch_seed[epoch];
        return true;
    };
    auto exchange_due = [&](uint32_t d) { return band.ctas > 1 && band.depth < td_reach(d); };

    if (tid < RUN) {
        TdPhilox philox{(a.width + 3) >> 2, 0, a.chain, 0u, 0u};
        int par = 0;
        uint32_t d = a.nphases > 0 ? __ldg(a.phases) : 0u;
        for (int64_t ph = 0; ph < a.nphases; ++ph) {
            const uint32_t d_next = ph + 1 < a.nphases ? __ldg(a.phases + ph + 1) : 0u;
            if (exchange_due(d)) band.exchange(cluster);
            if (PHILOX) {
                uint64_t seed;
                if (new_epoch(ph, &seed)) {
                    philox.key0 = (uint32_t)seed;
                    philox.key1 = (uint32_t)(seed >> 32);
                    philox.step = 0;
                }
                td_phase(d, band, philox);
                if (d & PH_DRAWS) ++philox.step;
                __syncthreads();
            } else {
                const uint32_t* mine = draws + par * slots;
                if (d & PH_DRAWS) {
                    __syncthreads();  // this phase's decisions are made; the other buffer is free
                    par ^= 1;
                }
                td_phase(d, band, [&](int r, int c, uint32_t) { return mine[(r - first) * wb + c]; });
                asm volatile("bar.sync 1, %0;" ::"r"(RUN) : "memory");
            }
            d = d_next;
        }
    } else {
        const int warp = (tid - RUN) >> 5, nwarps = (BLOCK - RUN) >> 5;  // a word's generators belong to one warp
        auto params_of = [&](uint32_t sid) {
            if (!a.params) return TinyParams{a.mat1, a.mat2, a.tmat};
            const uint4 p = __ldg(a.params + sid);
            return TinyParams{p.x, p.y, p.z};
        };
        auto stream_of = [&](int w) {  // of this lane's site of word w; a column past the array has none
            const int rr = w / wb, j = 32 * (w - rr * wb) + lane;
            return j < a.width ? (uint32_t)j + (uint32_t)band.m * (uint32_t)(first + rr) : 0u;
        };
        int64_t at = -1;  // the drawing phase whose decisions were made last
        int par = 0;
        auto decide_next = [&] {
            for (++at; at < a.nphases && !(__ldg(a.phases + at) & PH_DRAWS);) ++at;
            if (at >= a.nphases) return;
            uint64_t seed;
            const bool reseed = new_epoch(at, &seed);
            // four words at a time: their loads and chains overlap
            for (int w0 = warp; w0 < words; w0 += 4 * nwarps) {
                TinyState s[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t* p = st + 32 * min(w0 + q * nwarps, words - 1) + lane;
                    s[q] = TinyState{p[0], p[32 * slots], p[64 * slots], p[96 * slots]};
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int w = w0 + q * nwarps;
                    if (w >= words) break;
                    const uint32_t sid = a.params || reseed ? stream_of(w) : 0u;
                    const TinyParams tp = params_of(sid);
                    if (reseed) tiny_seed(s[q], tp, (uint32_t)seed + sid);
                    const uint32_t k = tiny_draw32(s[q], tp);
                    uint32_t* p = st + 32 * w + lane;
                    p[0] = s[q].s0;
                    p[32 * slots] = s[q].s1;
                    p[64 * slots] = s[q].s2;
                    p[96 * slots] = s[q].s3;
                    const uint32_t yes = __ballot_sync(0xffffffffu, (int32_t)k >= 0);  // k >> 9 < 2^22
                    if (lane == 0) draws[par * slots + w] = yes;
                }
            }
            par ^= 1;
        };
        decide_next();
        for (int64_t ph = 0; ph < a.nphases; ++ph) {
            const uint32_t d = __ldg(a.phases + ph);
            if (exchange_due(d)) {  // the cluster barriers of the exchange count every thread
                cluster.sync();
                cluster.sync();
                band.depth = band.halo;
            }
            if (band.ctas > 1) band.depth -= td_reach(d);
            if (d & PH_DRAWS) {
                __syncthreads();
                decide_next();
            }
        }
    }
    cluster.sync();  // no CTA leaves while another may write into its halo
    td_store(band, a.arr[0], tid >> 5, BLOCK >> 5, lane);
}

// One cluster; ctas_hint > 0 sets its size.
rt_status plan_td_walk(int device, int rows, int width, bool philox, int ctas_hint, WalkPlan* plan, std::string* err) {
    const void* fn = philox ? (const void*)td_walk_kernel<true> : (const void*)td_walk_kernel<false>;
    // us per step on 1 / 8 / 16 CTAs (words of one plane): Philox 2.4 / 3.6 / 4.3
    // (90), 3.0 / 3.6 / 4.0 (261), 4.7 / 3.9 / 3.8 (680); TinyMT 3.1 / 4.5 / 5.1,
    // 6.2 / 4.9 / 5.0, - / 6.2 / 5.5.
    const int words = rows * ((width + 31) / 32);
    int ctas = words <= (philox ? 300 : 150) ? 1 : words <= 400 ? 8 : 16;
    ctas = std::min(ctas_hint > 0 ? ctas_hint : ctas, std::min(rows, 16));
    const int rpc = (rows + ctas - 1) / ctas;
    const size_t slots = (size_t)(rpc + 2 * td_halo(rows, ctas, td_halo_cap(philox))) * ((width + 31) / 32);
    const size_t smem = 4 * (td_band_words(rows, width, ctas, td_halo_cap(philox), tdp::kPlanes) + (philox ? 0 : (4 * 32 + 2) * slots));
    if (const rt_status s = allow_shared(fn, device, smem, err); s != RT_OK) return s;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        *err = "cudaFuncSetAttribute failed";
        return RT_E_CUDA;
    }
    plan->items = 0;
    // a thread per word of a band and its halo, as far as there are threads
    const int most = kTdBlock - (philox ? 0 : kTdDeciders);
    plan->block = std::min(most, (int)(slots + 31) / 32 * 32) + (philox ? 0 : kTdDeciders);
    plan->rows_per_cta = rpc;
    plan->ctas = ctas;
    plan->smem = smem;
    plan->wpad = width;
    plan->xwords = 1;  // no exchange buffer
    plan->xslots = 1;
    plan->cluster = true;
    plan->merge_runs = false;
    plan->fn = fn;
    int active = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    walk_launch_config(*plan, &cfg, attr);
    if (cudaOccupancyMaxActiveClusters(&active, fn, &cfg) != cudaSuccess || active < 1) {
        cudaGetLastError();
        *err = "triangle-dimer cluster cannot be resident";
        return RT_E_INVAL;
    }
    return RT_OK;
}

}  // namespace rtb
