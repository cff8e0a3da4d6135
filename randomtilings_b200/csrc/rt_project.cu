// rt_project.cu -- exact integer Lipschitz projection of a height surface
// (include/rt_b200_project.h) on the GPU.
//
// Step 2 is a monotone min-plus relaxation: every pass lowers each interior
// vertex to min(h(w), h(v) + c(v -> w)) over its in-domain neighbours v,
// in place.  Values only decrease and never drop below the largest
// constraint-satisfying function under the start, so any order of updates
// (a racing read sees an old or a new value, both upper bounds) converges to
// that same unique function.  It runs over 32 x 64-vertex tiles, as the
// extremal flood does (rt_extremal.cu): a CTA relaxes its tile to a local
// fixpoint in shared memory and marks the neighbours that read a border value
// it lowered; a pass visits only marked tiles, and a pass that changes nothing
// ends the relaxation.
#include <cuda_runtime.h>

#include <climits>

#include "../../include/rt_b200_project.h"
#include "rt_domain.cuh"
#include "rt_internal.h"
#include "rt_guard.h"

using rtb::guarded;

namespace rtb {

namespace {

constexpr int PR = 32, PC = 64;      // tile rows x columns
constexpr int PT = 256;              // 64 columns x 4 groups of 8 rows
constexpr int kLocalCap = 4096;      // sweeps of one tile per pass (the tile is marked again if it is cut short)
constexpr int kGroup = 8;            // passes between two reads of the change counters
enum : int { C_BAD = kGroup, C_LOWERED, C_RAISED, C_COUNT };

// Step 1 for one vertex of kind `k`.
template <bool DOM>
__device__ __forceinline__ int32_t rounded(int k, int32_t lo, int32_t hi, float target) {
    if (k == 2) return lo;
    const double M = DOM ? 4.0 : 3.0;
    const double q = floor(((double)target - (double)lo) / M + 0.5);
    double g = (double)lo + M * q;
    g = g < (double)lo ? (double)lo : g > (double)hi ? (double)hi : g;
    return (int32_t)g;
}

// Vertex kinds and edges from the domain, step 1, and the check that hmin and
// hmax are a pair of height functions of this domain.
template <bool DOM>
__global__ void project_init(const int32_t* __restrict__ d, int m, const int32_t* __restrict__ hmin,
                             const int32_t* __restrict__ hmax, const float* __restrict__ target, uint8_t* kind,
                             uint8_t* edges, int32_t* h, unsigned* counts) {
    const int n = m + 1;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool bad = false;
    if (v < (int64_t)n * n) {
        const int i = (int)(v / n), j = (int)(v % n);
        const int k = vertex_kind<DOM>(d, m, i, j);
        kind[v] = (uint8_t)k;
        edges[v] = (uint8_t)(k == 1 ? edge_bits<DOM>(d, m, i, j) : 0u);  // only interior vertices move
        int32_t g = INT_MAX;
        if (k) {
            const int32_t lo = hmin[v], hi = hmax[v];
            bad = lo == INT_MAX || hi == INT_MAX || lo > hi || ((int64_t)hi - lo) % (DOM ? 4 : 3) != 0;
            g = rounded<DOM>(k, lo, hi, target[v]);
        }
        h[v] = g;
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicAdd(counts + C_BAD, 1u);
}

// One pass over the marked tiles.  h(w) - h(v) <= 1 along s(v -> w) = +1, i.e.
// s(w -> v) = -1, and <= M - 1 otherwise: dominoes, 1 along vertical and 3
// along horizontal edges into an even vertex (i + j even), the reverse into an
// odd one (DominoTiler.cpp:221-231); lozenges, 1 for directions 0, 2, 4 and 2
// for 1, 3, 5 (LozengeTiler.h:12-16).
template <bool DOM>
__global__ void __launch_bounds__(PT) project_relax(const uint8_t* __restrict__ edges, int32_t* h, int n, int tiles_x,
                                                    int tiles_y, uint8_t* dirty_in, uint8_t* dirty_out,
                                                    unsigned* changed_tiles) {
    const int tile = blockIdx.x;
    if (!dirty_in[tile]) return;  // the same answer for the whole block
    __shared__ int32_t sh[PR + 2][PC + 2];
    __shared__ unsigned s_mark;
    const int ty = tile / tiles_x, tx = tile % tiles_x;
    const int r0 = ty * PR, c0 = tx * PC;
    for (int e = threadIdx.x; e < (PR + 2) * (PC + 2); e += PT) {
        const int r = e / (PC + 2), c = e % (PC + 2);
        const int gi = r0 + r - 1, gj = c0 + c - 1;
        sh[r][c] = gi >= 0 && gj >= 0 && gi < n && gj < n ? *(volatile int32_t*)(h + (int64_t)gi * n + gj) : INT_MAX;
    }
    // Thread: column c, rows 8 grp .. 8 grp + 7 of the tile, kept in registers.
    // An iteration reads the other columns and the rows just outside its
    // segment, sweeps the segment down and then up, and publishes what changed.
    const int c = threadIdx.x & (PC - 1), grp = threadIdx.x / PC;
    const int cc = c + 1, rb = 8 * grp + 1, gj = c0 + c;
    const int p0 = (r0 + 8 * grp + gj) & 1;  // parity of the segment's first vertex (dominoes)
    uint32_t ed[8], any = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int gi = r0 + 8 * grp + k;
        ed[k] = gi < n && gj < n ? edges[(int64_t)gi * n + gj] : 0u;
        any |= ed[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        dirty_in[tile] = 0;  // nothing else writes dirty_in during this pass
        s_mark = 0;          // read after the barriers of the sweep loop
    }
    int32_t x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = sh[rb + k][cc];
    auto over = [](uint32_t e, int bit, int32_t hv, int cost) { return e >> bit & 1u ? hv + cost : INT_MAX; };
    uint32_t wrote = 0;  // bit k: x[k] lowered
    bool capped = true;
    for (int it = 0; it < kLocalCap; ++it) {
        uint32_t chg = 0;
        if (any) {
            int32_t a[8];  // from the other columns, fixed for this iteration
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int r = rb + k;
                if (DOM) {
                    const int side = ((p0 ^ k) & 1) == 0 ? 3 : 1;
                    a[k] = min(over(ed[k], 2, sh[r][cc + 1], side), over(ed[k], 3, sh[r][cc - 1], side));
                } else {
                    a[k] = min(min(over(ed[k], 0, sh[r][cc + 1], 1), over(ed[k], 1, sh[r - 1][cc + 1], 2)),
                               min(over(ed[k], 3, sh[r][cc - 1], 2), over(ed[k], 4, sh[r + 1][cc - 1], 1)));
                }
            }
            const int32_t xt = sh[rb - 1][cc], xb = sh[rb + 8][cc];
#pragma unroll
            for (int sweep = 0; sweep < 2; ++sweep) {
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    const int k = sweep == 0 ? kk : 7 - kk;
                    const int32_t up = k > 0 ? x[k - 1] : xt, dn = k < 7 ? x[k + 1] : xb;
                    const int cu = DOM ? (((p0 ^ k) & 1) == 0 ? 1 : 3) : 1, cd = DOM ? cu : 2;
                    const int32_t nx = min(a[k], min(over(ed[k], DOM ? 1 : 2, up, cu), over(ed[k], DOM ? 0 : 5, dn, cd)));
                    if (nx < x[k]) {
                        x[k] = nx;
                        chg |= 1u << k;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (chg >> k & 1u) sh[rb + k][cc] = x[k];
            wrote |= chg;
        }
        if (!__syncthreads_or(chg != 0)) {
            capped = false;
            break;
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (wrote >> k & 1u) h[(int64_t)(r0 + 8 * grp + k) * n + gj] = x[k];
    // Which neighbours read a lowered value (lozenges also across two corners).
    enum : unsigned { M_UP = 1, M_DOWN = 2, M_LEFT = 4, M_RIGHT = 8, M_UPRIGHT = 16, M_DOWNLEFT = 32, M_SELF = 64,
                      M_ANY = 128 };
    const bool top = grp == 0 && (wrote & 1u), bottom = grp == PR / 8 - 1 && (wrote >> 7 & 1u);
    unsigned mark = wrote ? M_ANY : 0u;
    if (top) mark |= M_UP;
    if (bottom) mark |= M_DOWN;
    if (c == 0 && wrote) mark |= M_LEFT;
    if (c == PC - 1 && wrote) mark |= M_RIGHT;
    if (!DOM && c == PC - 1 && top) mark |= M_UPRIGHT;
    if (!DOM && c == 0 && bottom) mark |= M_DOWNLEFT;
    if (capped && threadIdx.x == 0) mark |= M_SELF;
    if (mark) atomicOr(&s_mark, mark);
    __syncthreads();
    if (threadIdx.x == 0 && s_mark) {
        const unsigned m = s_mark;
        auto set = [&](int y, int x2) {
            if (y >= 0 && x2 >= 0 && y < tiles_y && x2 < tiles_x) dirty_out[y * tiles_x + x2] = 1;
        };
        if (m & M_UP) set(ty - 1, tx);
        if (m & M_DOWN) set(ty + 1, tx);
        if (m & M_LEFT) set(ty, tx - 1);
        if (m & M_RIGHT) set(ty, tx + 1);
        if (m & M_UPRIGHT) set(ty - 1, tx + 1);
        if (m & M_DOWNLEFT) set(ty + 1, tx - 1);
        if (m & M_SELF) set(ty, tx);
        if (m & M_ANY) atomicAdd(changed_tiles, 1u);
    }
}

// Step 3, and how many vertices steps 2 and 3 moved.
template <bool DOM>
__global__ void project_finish(const uint8_t* __restrict__ kind, const int32_t* __restrict__ hmin,
                               const int32_t* __restrict__ hmax, const float* __restrict__ target, int32_t* h, int64_t nn,
                               unsigned* counts) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = v < nn ? kind[v] : 0;
    bool lowered = false, raised = false;
    if (k) {
        const int32_t lo = hmin[v], x = h[v];
        lowered = x < rounded<DOM>(k, lo, hmax[v], target[v]);
        raised = x < lo;
        if (raised) h[v] = lo;
    }
    const int l = __syncthreads_count(lowered), r = __syncthreads_count(raised);
    if (threadIdx.x == 0) {
        if (l) atomicAdd(counts + C_LOWERED, (unsigned)l);
        if (r) atomicAdd(counts + C_RAISED, (unsigned)r);
    }
}

}  // namespace
}  // namespace rtb

using namespace rtb;

namespace {

// The call's device memory (one allocation), stream and events.
struct Workspace {
    char* p = nullptr;
    size_t used = 0;
    cudaStream_t s = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    // Offset of the next `bytes` bytes, 256-aligned.
    size_t take(size_t bytes) {
        const size_t at = used;
        used += (bytes + 255) & ~(size_t)255;
        return at;
    }
    ~Workspace() {
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (s) cudaStreamDestroy(s);
        if (p) cudaFree(p);
    }
};

template <bool DOM>
rt_status project(const int32_t* d, int64_t dlen, int m, const int32_t* hmin, const int32_t* hmax, const float* target,
                  int32_t* out, rt_project_stats* stats) {
    const int n = m + 1;
    const int64_t nn = (int64_t)n * n;
    const int tiles_x = (n + PC - 1) / PC, tiles_y = (n + PR - 1) / PR;
    const int64_t tiles = (int64_t)tiles_x * tiles_y;
    Workspace w;
    const size_t od = w.take((size_t)dlen * 4), olo = w.take((size_t)nn * 4), ohi = w.take((size_t)nn * 4),
                 ot = w.take((size_t)nn * 4), oh = w.take((size_t)nn * 4), ok = w.take((size_t)nn), oe = w.take((size_t)nn),
                 of = w.take((size_t)tiles * 2), oc = w.take(C_COUNT * sizeof(unsigned));
    if (cudaMalloc(&w.p, w.used) != cudaSuccess) {
        cudaGetLastError();
        return RT_E_NOMEM;
    }
    if (cudaStreamCreateWithFlags(&w.s, cudaStreamNonBlocking) != cudaSuccess || cudaEventCreate(&w.e0) != cudaSuccess ||
        cudaEventCreate(&w.e1) != cudaSuccess)
        return RT_E_CUDA;
    cudaStream_t s = w.s;
    auto *D = reinterpret_cast<int32_t*>(w.p + od), *LO = reinterpret_cast<int32_t*>(w.p + olo),
         *HI = reinterpret_cast<int32_t*>(w.p + ohi), *H = reinterpret_cast<int32_t*>(w.p + oh);
    auto* T = reinterpret_cast<float*>(w.p + ot);
    auto *K = reinterpret_cast<uint8_t*>(w.p + ok), *E = reinterpret_cast<uint8_t*>(w.p + oe),
         *F = reinterpret_cast<uint8_t*>(w.p + of);
    auto* C = reinterpret_cast<unsigned*>(w.p + oc);
    cudaMemsetAsync(F, 1, (size_t)tiles, s);
    cudaMemsetAsync(F + tiles, 0, (size_t)tiles, s);
    cudaMemsetAsync(C, 0, C_COUNT * sizeof(unsigned), s);
    cudaMemcpyAsync(D, d, (size_t)dlen * 4, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(LO, hmin, (size_t)nn * 4, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(HI, hmax, (size_t)nn * 4, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(T, target, (size_t)nn * 4, cudaMemcpyHostToDevice, s);
    const int threads = 256;
    const unsigned blocks = (unsigned)((nn + threads - 1) / threads);
    unsigned cnt[C_COUNT] = {};
    auto read_counts = [&] {
        cudaError_t e = cudaMemcpyAsync(cnt, C, sizeof cnt, cudaMemcpyDeviceToHost, s);
        return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    };
    cudaEventRecord(w.e0, s);
    project_init<DOM><<<blocks, threads, 0, s>>>(D, m, LO, HI, T, K, E, H, C);
    if (read_counts() != cudaSuccess) return RT_E_CUDA;
    if (cnt[C_BAD]) return RT_E_INVAL;  // not a pair of height functions of this domain
    // Passes in groups; the counters of a group are read once.  A pass that
    // changes nothing leaves no tile marked, so the relaxation has converged.
    int64_t passes = 0;
    const int64_t cap = nn + 32;  // Bellman-Ford bound: no more passes than vertices
    for (;;) {
        cudaMemsetAsync(C, 0, kGroup * sizeof(unsigned), s);
        for (int p = 0; p < kGroup; ++p)
            project_relax<DOM><<<(unsigned)tiles, PT, 0, s>>>(E, H, n, tiles_x, tiles_y, F + (p & 1) * tiles,
                                                              F + ((p & 1) ^ 1) * tiles, C + p);
        passes += kGroup;
        if (read_counts() != cudaSuccess) return RT_E_CUDA;
        if (cnt[kGroup - 1] == 0 || passes > cap) break;
    }
    project_finish<DOM><<<blocks, threads, 0, s>>>(K, LO, HI, T, H, nn, C);
    cudaEventRecord(w.e1, s);
    cudaMemcpyAsync(out, H, (size_t)nn * 4, cudaMemcpyDeviceToHost, s);
    if (read_counts() != cudaSuccess) return RT_E_CUDA;
    float ms = 0;
    cudaEventElapsedTime(&ms, w.e0, w.e1);
    if (stats) {
        stats->passes = passes;
        stats->lowered = cnt[C_LOWERED];
        stats->raised = cnt[C_RAISED];
        stats->device_ms = ms;
    }
    return RT_OK;
}

}  // namespace

extern "C" rt_status rt_project_heights(int32_t model, const int32_t* d, int64_t dlen, const int32_t* hmin,
                                        const int32_t* hmax, const float* target, int32_t* out, int64_t hlen,
                                        int32_t device, rt_project_stats* stats) {
    return guarded([&]() -> rt_status {
        if ((model != RT_DOMINO && model != RT_LOZENGE) || !d || !hmin || !hmax || !target || !out) return RT_E_INVAL;
        const int m = domain_side(model, dlen);
        if (m < 0 || (int64_t)(m + 1) * (m + 1) != hlen) return RT_E_INVAL;
        if (cudaSetDevice(device) != cudaSuccess) return RT_E_NODEVICE;
        return model == RT_DOMINO ? project<true>(d, dlen, m, hmin, hmax, target, out, stats)
                                  : project<false>(d, dlen, m, hmin, hmax, target, out, stats);
    });
}
