// rt_sixv.cu -- the six-vertex model (square ice) with domain-wall boundary
// conditions (include/rt_b200_sixv.h).
//
// The reference names the model (README.md:3) without code; this is the
// domino height machinery applied to it.  Heights live on the faces as int16.
// A colour step updates one of the four face classes (i mod 2, j mod 2); an
// epoch's steps run in one launch of the band kernel below when the bands
// fit shared memory, else one launch per step on the heights in HBM.  A
// thread owns four faces of its class in one row, (i, 8q + p + 2b) for
// b = 0..3, takes the four output words of one Philox4x32-10 call as their
// draws, and applies the heat bath: a face whose four edge neighbours share
// the height m becomes m+1 when its draw is below the threshold of its
// diagonal pattern, else m-1.  Faces of one class share no neighbour (edge
// or diagonal), so a launch is race-free and the result is independent of the
// order of the threads.  Coupled CFTP chains are two lattices of the same
// launch fed the same draws.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/rt_b200_sixv.h"
#include "rt_device.cuh"
#include "rt_exchange.cuh"
#include "rt_internal.h"
#include "rt_guard.h"

using rtb::guarded;

namespace rtb {

struct SixvArgs {
    int16_t* h[2];  // heights of each lattice, (n+1) x (n+1), row stride n+1
    int nlat;
    int n;
    int pi, pj;     // class: row parity, column parity
    int rows, Q;    // rows of the class, quads per row
    uint32_t s_lo, s_hi, chain, k0, k1;
    uint32_t thr[16];
};

__global__ void __launch_bounds__(256) sixv_step_kernel(const __grid_constant__ SixvArgs a) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= a.rows * a.Q) return;
    const int r = idx / a.Q, q = idx - r * a.Q;
    const int i = (a.pi == 0 ? 2 : 1) + 2 * r;
    const int S = a.n + 1;
    const uint4 w4 = philox4((uint32_t)(i * a.Q + q), a.s_lo, a.s_hi, a.chain, a.k0, a.k1);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int j = 8 * q + a.pj + 2 * b;
        if (j < 1 || j > a.n - 1) continue;
        const uint32_t k = quad_word(w4, b) >> 9;
        for (int l = 0; l < a.nlat; ++l) {
            int16_t* f = a.h[l] + (size_t)i * S + j;
            const int m = f[-S];
            if (f[S] != m || f[-1] != m || f[1] != m) continue;
            const int p = (f[-S - 1] > m) | ((f[-S + 1] > m) << 1) | ((f[S - 1] > m) << 2) | ((f[S + 1] > m) << 3);
            *f = (int16_t)(k < a.thr[p] ? m + 1 : m - 1);
        }
    }
}

// ---------------------------------------------------------------------------
// The heights on chip for a whole epoch.  CTA c owns face rows [r0, r1) of
// every lattice and keeps them, with H rows above and below, in shared memory
// as two planes: the even columns and the odd ones (4 Q halfwords a row each,
// column 2 x + parity at x).  The four faces of a work item, and the same
// columns of any row, are then one 64-bit access, and faces go two to a
// register: with m the height above a face, the others are compared by
// exclusive or, and the diagonals, which differ from m by one where it matters,
// by a subtraction whose borrow a set top bit keeps out of the other half.
//
// Steps 2t and 2t + 1 update rows of one parity from themselves and the rows
// next to them, so after a pair of steps one row less on each side of the band
// is current: H pairs run between two exchanges, the halo rows recomputed by
// both CTAs (the draws depend on the face and the step only).  Then the band's
// first and last H rows go to the neighbours through tagged 64-bit global slots
// (32 bits of heights and the exchange's number), double-buffered by its
// parity.  A CTA publishes exchange t + 1 only after it read exchange t, which
// each neighbour published after reading exchange t - 1 from it, so a slot is
// rewritten only after it was read, and no CTA writes its band back before its
// neighbours have read it.  Every wait is bounded: past timeout_ns the
// CTA sets ERR_TIMEOUT in *err and returns, and the others see it.  The launch
// is cooperative, so every CTA is resident.
//
// What bounds it: the arithmetic -- a Philox call a quad (73 issue cycles a warp),
// the logic of the rule at half rate -- and the latency of a step (0.26 us at n =
// 10).  n = 1000: 400 steps take 0.38 ms (0.9 us a step; 2.4 with int16 accesses
// one by one and an exchange every two steps).
// ---------------------------------------------------------------------------
struct SixvBandArgs {
    int16_t* h[2];
    int nlat, n, Q;
    uint32_t chain, k0, k1;
    uint32_t thr[16];
    int64_t steps;
    int rows_max, H, xwords;   // most rows of a CTA; halo rows; slot words of a side: H rows x 4 Q
    unsigned long long* xbuf;  // [cta][side][parity][lattice][xwords]
    int* err;
    uint64_t timeout_ns;
    int64_t drop_blk;  // an exchange whose rows CTA 0 withholds (bounded-wait tests); -1: none
};

__device__ __forceinline__ unsigned long long* sixv_slot(const SixvBandArgs& a, int cta, int side, int par, int l) {
    return a.xbuf + ((((size_t)cta * 2 + side) * 2 + par) * a.nlat + l) * a.xwords;
}

// ONE: the sixteen thresholds are equal, and neither 0 nor 2^23 (as with equal
// weights): the diagonals need not be looked at.
template <int NLAT, bool ONE>
__global__ void __launch_bounds__(1024, 1) sixv_band_kernel(const __grid_constant__ SixvBandArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_thr[16];
    int16_t* const sh = reinterpret_cast<int16_t*>(smem_raw);
    const int S = a.n + 1, Q = a.Q, ST = 4 * Q, H = a.H;
    const int cta = blockIdx.x, nct = gridDim.x, tid = threadIdx.x, BLOCK = blockDim.x;
    const int r0 = (int)((int64_t)cta * S / nct), r1 = (int)((int64_t)(cta + 1) * S / nct), nrows = r1 - r0;
    const int base = r0 - H;                         // face row of stored row 0
    const int plane = (a.rows_max + 2 * H) * ST;     // halfwords of one parity
    const bool has_top = cta > 0, has_bot = cta + 1 < nct;
    if (tid < 16) s_thr[tid] = a.thr[tid];
    for (int l = 0; l < NLAT; ++l)
        for (int e = tid; e < (nrows + 2 * H) * 2 * ST; e += BLOCK) {
            const int rr = e / (2 * ST), j = e - rr * 2 * ST, i = base + rr;
            sh[(2 * l + (j & 1)) * plane + rr * ST + (j >> 1)] =
                i >= 0 && i < S && j < S ? a.h[l][(size_t)i * S + j] : (int16_t)0;
        }

    // The launch has a multiple of Q threads: a thread keeps its column.
    const int q = tid % Q, rr0 = tid / Q, dr = BLOCK / Q;
    // the faces of the quad that move, two to a register, by column parity
    auto inside = [&](int j) { return (j >= 1 && j < a.n ? 0x2u : 0u) | (j + 2 < a.n ? 0x20000u : 0u); };
    const uint32_t in0[2] = {inside(8 * q), inside(8 * q + 1)}, in2[2] = {inside(8 * q + 4), inside(8 * q + 5)};
    auto draws = [&](int i, int64_t st) {
        return philox4((uint32_t)(i * Q + q), (uint32_t)st, (uint32_t)((uint64_t)st >> 32), a.chain, a.k0, a.k1);
    };

    const uint32_t one = a.thr[0] << 9;
    // The four faces (i, 8 q + PJ + 2 b) of every lattice.
    auto item = [&](auto pj, int i, const uint4& w4) {
        constexpr int PJ = decltype(pj)::value;
#pragma unroll
        for (int l = 0; l < NLAT; ++l) {
            int16_t* const P = sh + (2 * l + PJ) * plane + (i - base) * ST + 4 * q;
            const int16_t* const O = sh + (2 * l + 1 - PJ) * plane + (i - base) * ST + 4 * q;
            const uint2 up = *reinterpret_cast<const uint2*>(P - ST), dn = *reinterpret_cast<const uint2*>(P + ST);
            const uint2 old = *reinterpret_cast<const uint2*>(P);
            // the columns left and right of the faces, in the rows above, at and below
            uint32_t L01[3], L23[3], R01[3], R23[3];
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                if (ONE && y != 1) continue;
                const int16_t* const row = O + (y - 1) * ST;
                const uint2 v = *reinterpret_cast<const uint2*>(row);
                // beyond a row's ends this is another row's face, which only masked ones see
                const uint32_t ext = (uint16_t)row[PJ ? 4 : -1];
                const uint32_t mid = __byte_perm(v.x, v.y, 0x5432);
                L01[y] = PJ ? v.x : __byte_perm(ext, v.x, 0x5410);
                L23[y] = PJ ? v.y : mid;
                R01[y] = PJ ? mid : v.x;
                R23[y] = PJ ? __byte_perm(v.y, ext, 0x5432) : v.y;
            }
            // Neighbours of a face differ from one another by 0 or 2, and what
            // differs by 2 differs in bit 1: so one logic operation compares two
            // pairs of them.
            auto two = [&](uint32_t m, uint32_t below, const uint32_t(&L)[3], const uint32_t(&R)[3], uint32_t in,
                           uint32_t was, uint32_t wa, uint32_t wb) -> uint32_t {
                const uint32_t flat = ~((below ^ m) | (L[1] ^ m) | (R[1] ^ m)) & in;  // bit 1 of each half
                const uint32_t high = m + 0x00010001u;
                bool la, lb;  // the draw takes m - 1
                if (ONE) {
                    la = wa >= one;
                    lb = wb >= one;
                } else {
                    // a diagonal is m + 1 where its bit 1 is that of m + 1
                    const uint32_t d0 = ~(L[0] ^ high) & 0x00020002u, d1 = ~(R[0] ^ high) & 0x00020002u;
                    const uint32_t d2 = ~(L[2] ^ high) & 0x00020002u, d3 = ~(R[2] ^ high) & 0x00020002u;
                    const uint32_t p = d0 + 2u * d1 + 4u * d2 + 8u * d3;
                    la = wa >> 9 >= s_thr[p >> 1 & 15u];
                    lb = wb >> 9 >= s_thr[p >> 17];
                }
                // m >= 1 in every flat face: no borrow
                const uint32_t v = high - (((la ? 0x2u : 0u) | (lb ? 0x20000u : 0u)) & flat);
                const uint32_t mask = (flat >> 1) * 0xffffu;
                return (was & ~mask) | (v & mask);
            };
            uint2 out;
            out.x = two(up.x, dn.x, L01, R01, in0[PJ], old.x, w4.x, w4.y);
            out.y = two(up.y, dn.y, L23, R23, in2[PJ], old.y, w4.z, w4.w);
            *reinterpret_cast<uint2*>(P) = out;
        }
    };
    using C0 = std::integral_constant<int, 0>;
    using C1 = std::integral_constant<int, 1>;

    __syncthreads();
    int k = 0;          // pairs of steps since the last exchange
    uint32_t blk = 0;   // exchanges made
    for (int64_t s = 0; s < a.steps; s += 2) {
        // rows of the pair's parity that are computed: within the lattice, one
        // less on each side with every pair
        const int odd = (int)(s >> 1 & 1);  // the first pair takes the even rows
        const int lo = max(1, has_top ? base + 1 + k : r0), hi = min(a.n, has_bot ? r1 + H - 1 - k : r1);
        const int first = lo + ((lo & 1) != odd);
        const int nlive = first < hi ? (hi - first + 1) / 2 : 0;
        if (nlive <= dr) {
            // one item a thread: the draws of both steps are made together
            const int i = first + 2 * rr0;
            uint4 w0, w1;
            if (rr0 < nlive) {
                w0 = draws(i, s);
                w1 = draws(i, s + 1);
                item(C0{}, i, w0);
            }
            __syncthreads();
            if (rr0 < nlive) item(C1{}, i, w1);
        } else {
            for (int rr = rr0; rr < nlive; rr += dr) item(C0{}, first + 2 * rr, draws(first + 2 * rr, s));
            __syncthreads();
            for (int rr = rr0; rr < nlive; rr += dr) item(C1{}, first + 2 * rr, draws(first + 2 * rr, s + 1));
        }
        __syncthreads();
        ++k;
        if (nct == 1 || k < H || s + 2 >= a.steps) continue;

        // Row y of a side's H rows, quad q: slot words (4 y + z) Q + q, z = 0, 1 the
        // quad's even columns, 2, 3 its odd ones.
        const int par = (int)(blk & 1u);
        const uint32_t tag = blk + 1u;
#pragma unroll
        for (int l = 0; l < NLAT; ++l)
            for (int yy = rr0; yy < 2 * H; yy += dr) {
                const int side = yy >= H, y = yy - side * H;
                if ((side == 0 ? !has_top : !has_bot) || (cta == 0 && blk == a.drop_blk)) continue;
                const int16_t* const row = sh + 2 * l * plane + ((side == 0 ? H : nrows) + y) * ST + 4 * q;
                const uint2 ev = *reinterpret_cast<const uint2*>(row), od = *reinterpret_cast<const uint2*>(row + plane);
                unsigned long long* const to = sixv_slot(a, cta, side, par, l) + 4 * y * Q + q;
                const unsigned long long t = (unsigned long long)tag << 32;
                st_relaxed64(to, t | ev.x);
                st_relaxed64(to + Q, t | ev.y);
                st_relaxed64(to + 2 * Q, t | od.x);
                st_relaxed64(to + 3 * Q, t | od.y);
            }
        bool ok = true;
#pragma unroll
        for (int l = 0; l < NLAT; ++l)
            for (int yy = rr0; yy < 2 * H; yy += dr) {
                const int side = yy >= H, y = yy - side * H;
                if (side == 0 ? !has_top : !has_bot) continue;
                const unsigned long long* const from =
                    sixv_slot(a, side == 0 ? cta - 1 : cta + 1, 1 - side, par, l) + 4 * y * Q + q;
                // the four words in one round trip, again until the last one is there
                unsigned long long v[4];
                unsigned spins = 0;
                uint64_t t0 = 0;
                for (;;) {
                    bool here = true;
#pragma unroll
                    for (int z = 0; z < 4; ++z) v[z] = ld_relaxed64(from + z * Q);
#pragma unroll
                    for (int z = 0; z < 4; ++z) here = here && (uint32_t)(v[z] >> 32) == tag;
                    if (here || !ok) break;
                    if ((++spins & 63u) == 0u) ok = wait_more(a, t0);
                }
                int16_t* const row = sh + 2 * l * plane + ((side == 0 ? 0 : H + nrows) + y) * ST + 4 * q;
                *reinterpret_cast<uint2*>(row) = make_uint2((uint32_t)v[0], (uint32_t)v[1]);
                *reinterpret_cast<uint2*>(row + plane) = make_uint2((uint32_t)v[2], (uint32_t)v[3]);
            }
        if (__syncthreads_or(!ok)) return;
        k = 0;
        ++blk;
    }
    for (int l = 0; l < NLAT; ++l)
        for (int e = tid; e < nrows * S; e += BLOCK) {
            const int rr = e / S, j = e - rr * S;
            a.h[l][(size_t)(r0 + rr) * S + j] = sh[(2 * l + (j & 1)) * plane + (H + rr) * ST + (j >> 1)];
        }
}

// Vertex type of faces NW a, NE b, SW c, SE d (the header's numbering), -1 if none.
static int vertex_type(int a, int b, int c, int d) {
    if (b == a + 1 && c == a - 1 && d == a) return 0;
    if (b == a - 1 && c == a + 1 && d == a) return 1;
    if (b == a + 1 && c == a + 1) return d == a + 2 ? 2 : d == a ? 4 : -1;
    if (b == a - 1 && c == a - 1) return d == a - 2 ? 3 : d == a ? 5 : -1;
    return -1;
}

// Heat-bath thresholds of the 16 diagonal patterns (heights relative to m).
static void sixv_thresholds(const double w[6], uint32_t thr[16], bool* monotone) {
    for (int p = 0; p < 16; ++p) {
        const int d1 = (p & 1) ? 1 : -1, d2 = (p & 2) ? 1 : -1, d3 = (p & 4) ? 1 : -1, d4 = (p & 8) ? 1 : -1;
        double wt[2];
        for (int up = 0; up < 2; ++up) {
            const int h = up ? 1 : -1;
            wt[up] = w[vertex_type(d1, 0, 0, h)] * w[vertex_type(0, d2, h, 0)] * w[vertex_type(0, h, d3, 0)] *
                     w[vertex_type(h, 0, 0, d4)];
        }
        thr[p] = below_threshold(wt[1] / (wt[0] + wt[1]));
    }
    bool mono = true;
    for (int p = 0; p < 16; ++p)
        for (int b = 0; b < 4; ++b)
            if (!(p & (1 << b)) && thr[p | (1 << b)] < thr[p]) mono = false;
    *monotone = mono;
}

}  // namespace rtb

using namespace rtb;

// Heights cross to and from the device as int16 through two pinned chunks: the
// host narrows (and checks) or widens one while the other is on its way, half the
// bytes of int32 and no pageable copies (n = 1000, both ways: 0.51 ms, 1.1 before).
constexpr size_t kStageBytes = size_t(1) << 19;

struct rt_sixv {
    int device = 0;
    cudaStream_t stream = nullptr;
    double w[6] = {1, 1, 1, 1, 1, 1};
    uint32_t thr[16] = {};
    bool monotone = true;
    std::string err;
    void* d_h[2] = {nullptr, nullptr};  // int16 lattices
    size_t cap = 0;                     // bytes of each
    int16_t* stage[2] = {nullptr, nullptr};  // pinned chunks of whole rows, in turn
    cudaEvent_t staged[2] = {nullptr, nullptr};
    unsigned long long* d_count = nullptr;
    unsigned long long* d_xbuf = nullptr;  // band kernel: halo slots
    size_t xcap = 0;
    int* d_err = nullptr;                  // band kernel: error word
    uint64_t timeout_ns = 5000000000ull;   // band kernel: limit of one wait
    int64_t drop_blk = -1;                 // RT_TEST_DROP_PUBLISH

    rt_status fail(rt_status s, const std::string& m) {
        err = m;
        return s;
    }
    rt_status cuda_fail(cudaError_t e, const char* what) {
        return fail(RT_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    }
    bool reserve(int n) {
        const size_t bytes = (((size_t)(n + 1) * (n + 1) * 2) + 255) & ~(size_t)255;
        if (bytes > cap) {
            for (auto& p : d_h) {
                if (p) cudaFree(p);
                p = nullptr;
            }
            cap = 0;
            if (cudaMalloc(&d_h[0], bytes) != cudaSuccess || cudaMalloc(&d_h[1], bytes) != cudaSuccess) return false;
            cap = bytes;
        }
        for (int k = 0; k < 2; ++k) {
            if (!stage[k] && cudaMallocHost(&stage[k], kStageBytes) != cudaSuccess) return false;
            if (!staged[k] && cudaEventCreateWithFlags(&staged[k], cudaEventDisableTiming) != cudaSuccess) return false;
        }
        if (!d_count && cudaMalloc(&d_count, sizeof *d_count) != cudaSuccess) return false;
        return true;
    }
    ~rt_sixv() {
        for (auto& p : d_h)
            if (p) cudaFree(p);
        for (auto& p : stage)
            if (p) cudaFreeHost(p);
        for (auto& e : staged)
            if (e) cudaEventDestroy(e);
        if (d_count) cudaFree(d_count);
        if (d_xbuf) cudaFree(d_xbuf);
        if (d_err) cudaFree(d_err);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

int chunk_rows(int n) { return (int)std::max<size_t>(1, kStageBytes / ((size_t)(n + 1) * 2)); }

// Host heights -> int16 lattice l (its padding zeroed, so that lattices
// compare word by word).  check: RT_E_INVAL if they are no domain-wall height
// function, found on the way; nothing has run on them then.
rt_status upload(rt_sixv* h, const int32_t* heights, int n, int l, bool check) {
    const int S = n + 1, step = chunk_rows(n);
    cudaError_t e = cudaMemsetAsync(h->d_h[l], 0, h->cap, h->stream);
    bool bad = false;
    const int16_t* above = nullptr;  // the row above, in either chunk
    for (int i = 0, k = 0; i < S && e == cudaSuccess && !bad; i += step, k ^= 1) {
        const int rows = std::min(step, S - i);
        e = cudaEventSynchronize(h->staged[k]);  // the chunk's last copy
        if (e != cudaSuccess) break;
        for (int r = i; r < i + rows && !bad; ++r) {
            int16_t* const to = h->stage[k] + (size_t)(r - i) * S;
            sixv_narrow_row(heights + (size_t)r * S, S, to);
            bad = check && !sixv_row_ok(to, above, n, r);
            above = to;
        }
        if (bad) break;
        e = cudaMemcpyAsync(static_cast<int16_t*>(h->d_h[l]) + (size_t)i * S, h->stage[k], (size_t)rows * S * 2,
                            cudaMemcpyHostToDevice, h->stream);
        if (e == cudaSuccess) e = cudaEventRecord(h->staged[k], h->stream);
    }
    if (bad) return h->fail(RT_E_INVAL, "not a domain-wall height function of this size");
    return e == cudaSuccess ? RT_OK : h->cuda_fail(e, "upload");
}

rt_status download(rt_sixv* h, int32_t* heights, int n, int l) {
    const int S = n + 1, step = chunk_rows(n);
    cudaError_t e = cudaSuccess;
    auto fetch = [&](int i, int k) {
        if (i >= S || e != cudaSuccess) return;
        e = cudaMemcpyAsync(h->stage[k], static_cast<const int16_t*>(h->d_h[l]) + (size_t)i * S,
                            (size_t)std::min(step, S - i) * S * 2, cudaMemcpyDeviceToHost, h->stream);
        if (e == cudaSuccess) e = cudaEventRecord(h->staged[k], h->stream);
    };
    fetch(0, 0);
    fetch(step, 1);
    for (int i = 0, k = 0; i < S && e == cudaSuccess; i += step, k ^= 1) {
        e = cudaEventSynchronize(h->staged[k]);
        if (e != cudaSuccess) break;
        const size_t count = (size_t)std::min(step, S - i) * S;
        sixv_widen(h->stage[k], count, heights + (size_t)i * S);
        fetch(i + 2 * step, k);
    }
    return e == cudaSuccess ? RT_OK : h->cuda_fail(e, "download");
}

// Colour steps 0 .. 4 sweeps - 1 of one epoch on `nlat` lattices.
rt_status run_epoch(rt_sixv* h, int n, int nlat, int64_t sweeps, uint64_t key, uint32_t chain) {
    SixvArgs a;
    std::memset(&a, 0, sizeof a);
    a.h[0] = static_cast<int16_t*>(h->d_h[0]);
    a.h[1] = static_cast<int16_t*>(h->d_h[1]);
    a.nlat = nlat;
    a.n = n;
    a.Q = (n + 1 + 7) / 8;
    a.chain = chain;
    a.k0 = (uint32_t)key;
    a.k1 = (uint32_t)(key >> 32);
    std::memcpy(a.thr, h->thr, sizeof a.thr);
    if (sweeps <= 0) return RT_OK;
    {
        // The band kernel, when every CTA's rows (and halo) fit shared memory.
        int dev = 0, sms = 0, optin = 0;
        const int S = n + 1;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess && sms > 0) {
            // Microseconds per step: n = 30 0.28 on one CTA, 0.37 on four; n = 64
            // 0.44 on one, 0.39 on eight; n = 200 0.49 with bands of six rows, 0.45
            // of four; n = 400 0.66 and 0.52.  An exchange takes 1.5 us or so: n =
            // 1000 (bands of 7 rows) 0.97 with H = 1, 0.93 with 2, 0.91 with 3 or 4,
            // 1.0 with 6; n = 2000 (14 rows) 2.24 with 1, 1.99 with 2, 2.41 with 4;
            // n = 3500 5.2 with 1, 4.4 with 2.
            int ctas = (int64_t)S / 2 * a.Q <= 128 ? 1 : std::min(sms, std::max(1, S / 4));
            auto rows_max = [&]() { return (S + ctas - 1) / ctas; };
            int H = ctas == 1 ? 1 : std::min(rows_max() <= 8 ? 4 : 2, S / ctas);
            auto bytes = [&]() { return (size_t)nlat * (rows_max() + 2 * H) * 8 * a.Q * sizeof(int16_t); };
            while (H > 1 && bytes() + sizeof(uint32_t[16]) > (size_t)optin) --H;
            // Several CTAs make an exchange in every epoch, be it of one sweep (two
            // pairs): it orders a CTA's loads of its halo before its neighbours' stores.
            if (ctas > 1) H = (int)std::min<int64_t>(H, 2 * sweeps - 1);
            const size_t smem = bytes();
            const size_t xbytes = (size_t)ctas * 2 * 2 * nlat * (H * 4 * a.Q) * sizeof(unsigned long long);
            bool one = h->thr[0] > 0 && h->thr[0] < 1u << 23;
            for (int t = 1; t < 16; ++t) one = one && h->thr[t] == h->thr[0];
            const void* band_fn = nlat == 2 ? (one ? (const void*)sixv_band_kernel<2, true> : (const void*)sixv_band_kernel<2, false>)
                                            : (one ? (const void*)sixv_band_kernel<1, true> : (const void*)sixv_band_kernel<1, false>);
            const int block = std::max(1, 1024 / a.Q) * a.Q;
            bool ready = block <= 1024 && smem + sizeof(uint32_t[16]) <= (size_t)optin &&
                         // all there is: the limit is the function's, for every handle and thread
                         cudaFuncSetAttribute(band_fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              optin - (int)sizeof(uint32_t[16])) == cudaSuccess;
            if (ready && xbytes > h->xcap) {
                if (h->d_xbuf) cudaFree(h->d_xbuf);
                h->d_xbuf = nullptr;
                h->xcap = 0;
                ready = cudaMalloc(&h->d_xbuf, xbytes) == cudaSuccess;
                if (ready) h->xcap = xbytes;
            }
            if (ready && !h->d_err) ready = cudaMalloc(&h->d_err, sizeof(int)) == cudaSuccess;
            if (ready) {
                SixvBandArgs b;
                std::memset(&b, 0, sizeof b);
                b.h[0] = a.h[0];
                b.h[1] = a.h[1];
                b.nlat = nlat;
                b.n = n;
                b.Q = a.Q;
                b.chain = a.chain;
                b.k0 = a.k0;
                b.k1 = a.k1;
                std::memcpy(b.thr, a.thr, sizeof b.thr);
                b.steps = 4 * sweeps;
                b.rows_max = rows_max();
                b.H = H;
                b.xwords = H * 4 * a.Q;
                b.xbuf = h->d_xbuf;
                b.err = h->d_err;
                b.timeout_ns = h->timeout_ns;
                b.drop_blk = h->drop_blk;
                void* args[] = {&b};
                cudaError_t e = cudaMemsetAsync(h->d_xbuf, 0, xbytes, h->stream);
                if (e == cudaSuccess) e = cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream);
                if (e == cudaSuccess)
                    e = cudaLaunchCooperativeKernel(band_fn, dim3((unsigned)ctas), dim3((unsigned)block), args, smem,
                                                    h->stream);
                if (e == cudaSuccess) {
                    int flag = 0;
                    e = cudaMemcpyAsync(&flag, h->d_err, sizeof flag, cudaMemcpyDeviceToHost, h->stream);
                    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
                    if (e != cudaSuccess) return h->cuda_fail(e, "six-vertex band walk");
                    if (flag) return h->fail(RT_E_TIMEOUT, "six-vertex band walk: a halo wait timed out");
                    return RT_OK;
                }
                cudaGetLastError();  // not launched: one launch per colour step below
            }
        }
    }
    for (int64_t s = 0; s < 4 * sweeps; ++s) {
        a.pi = (int)((s & 3) >> 1);
        a.pj = (int)(s & 1);
        // rows i = 2, 4, .. or 1, 3, .. up to n - 1
        const int first = a.pi == 0 ? 2 : 1;
        a.rows = n - 1 >= first ? (n - 1 - first) / 2 + 1 : 0;
        if (a.rows <= 0) continue;
        a.s_lo = (uint32_t)s;
        a.s_hi = (uint32_t)((uint64_t)s >> 32);
        const int64_t threads = (int64_t)a.rows * a.Q;
        sixv_step_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, h->stream>>>(a);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? RT_OK : h->cuda_fail(e, "six-vertex step launch");
}

bool valid_n(int n) { return n >= 1 && n <= 32000; }

}  // namespace

extern "C" {

rt_status rt_sixv_create(int32_t device, rt_sixv** out) {
    return guarded([&]() -> rt_status {
        if (!out) return RT_E_INVAL;
        *out = nullptr;
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return RT_E_NODEVICE;
        cudaDeviceProp prop;
        if (cudaGetDeviceProperties(&prop, device) != cudaSuccess || prop.major != 10) return RT_E_NODEVICE;
        cudaSetDevice(device);
        rt_sixv* h = new rt_sixv();
        h->device = device;
        if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
            delete h;
            return RT_E_CUDA;
        }
        sixv_thresholds(h->w, h->thr, &h->monotone);
        if (const char* dp = std::getenv("RT_TEST_DROP_PUBLISH")) h->drop_blk = std::atoll(dp);
        if (const char* t = std::getenv("RT_WAIT_TIMEOUT_MS")) {
            const long ms = std::atol(t);
            if (ms > 0) h->timeout_ns = (uint64_t)ms * 1000000ull;
        }
        *out = h;
        return RT_OK;
    });
}

rt_status rt_sixv_destroy(rt_sixv* h) {
    return guarded([&]() -> rt_status {
        if (!h) return RT_E_INVAL;
        cudaSetDevice(h->device);
        cudaStreamSynchronize(h->stream);
        delete h;
        return RT_OK;
    });
}

const char* rt_sixv_last_error(rt_sixv* h) { return h ? h->err.c_str() : ""; }

rt_status rt_sixv_set_weights(rt_sixv* h, const double w[6]) {
    return guarded([&]() -> rt_status {
        if (!h || !w) return RT_E_INVAL;
        for (int t = 0; t < 6; ++t)
            if (!(w[t] > 0) || !std::isfinite(w[t])) return h->fail(RT_E_INVAL, "vertex weights must be finite and > 0");
        std::memcpy(h->w, w, sizeof h->w);
        sixv_thresholds(h->w, h->thr, &h->monotone);
        return RT_OK;
    });
}

rt_status rt_sixv_thresholds(rt_sixv* h, uint32_t thr[16], int32_t* monotone) {
    return guarded([&]() -> rt_status {
        if (!h) return RT_E_INVAL;
        if (thr) std::memcpy(thr, h->thr, sizeof h->thr);
        if (monotone) *monotone = h->monotone ? 1 : 0;
        return RT_OK;
    });
}

rt_status rt_sixv_dwbc_heights(int32_t n, int32_t* hmin, int32_t* hmax) {
    return guarded([&]() -> rt_status {
        if (!valid_n(n)) return RT_E_INVAL;
        for (int i = 0; i <= n; ++i)
            for (int j = 0; j <= n; ++j) {
                const size_t at = (size_t)i * (n + 1) + j;
                if (hmin) hmin[at] = std::abs(i - j);
                if (hmax) hmax[at] = std::min(i + j, 2 * n - i - j);
            }
        return RT_OK;
    });
}

rt_status rt_sixv_check(const int32_t* heights, int32_t n) {
    return guarded([&]() -> rt_status {
        if (!heights || !valid_n(n)) return RT_E_INVAL;
        const int S = n + 1;
        std::vector<int16_t> rows(2 * (size_t)S);
        for (int i = 0; i <= n; ++i) {
            int16_t* const row = rows.data() + (i & 1) * (size_t)S;
            sixv_narrow_row(heights + (size_t)i * S, S, row);
            if (!sixv_row_ok(row, i > 0 ? rows.data() + ((i - 1) & 1) * (size_t)S : nullptr, n, i)) return RT_E_INVAL;
        }
        return RT_OK;
    });
}

rt_status rt_sixv_to_asm(const int32_t* heights, int32_t n, int32_t* asm_out) {
    return guarded([&]() -> rt_status {
        if (!asm_out || rt_sixv_check(heights, n) != RT_OK) return RT_E_INVAL;
        const int S = n + 1;
        for (int i = 1; i <= n; ++i)
            for (int j = 1; j <= n; ++j) {
                const int a = heights[(size_t)(i - 1) * S + j - 1], b = heights[(size_t)(i - 1) * S + j];
                const int c = heights[(size_t)i * S + j - 1], d = heights[(size_t)i * S + j];
                asm_out[(size_t)(i - 1) * n + (j - 1)] = (b + c - a - d) / 2;
            }
        return RT_OK;
    });
}

rt_status rt_sixv_vertex_types(const int32_t* heights, int32_t n, int32_t* types) {
    return guarded([&]() -> rt_status {
        if (!types || rt_sixv_check(heights, n) != RT_OK) return RT_E_INVAL;
        const int S = n + 1;
        for (int i = 1; i <= n; ++i)
            for (int j = 1; j <= n; ++j)
                types[(size_t)(i - 1) * n + (j - 1)] =
                    vertex_type(heights[(size_t)(i - 1) * S + j - 1], heights[(size_t)(i - 1) * S + j],
                                heights[(size_t)i * S + j - 1], heights[(size_t)i * S + j]);
        return RT_OK;
    });
}

rt_status rt_sixv_walk(rt_sixv* h, int32_t* heights, int32_t n, int64_t sweeps, uint64_t key, uint32_t chain) {
    return guarded([&]() -> rt_status {
        if (!h) return RT_E_INVAL;
        if (!heights || !valid_n(n) || sweeps < 0) return h->fail(RT_E_INVAL, "bad arguments");
        if (sweeps > kMaxColourSteps / 4) return h->fail(RT_E_INVAL, "more than 2^38 sweeps in one call");
        cudaSetDevice(h->device);
        if (!h->reserve(n)) return h->fail(RT_E_NOMEM, "cudaMalloc six-vertex lattice");
        rt_status s = upload(h, heights, n, 0, true);
        if (s == RT_OK) s = run_epoch(h, n, 1, sweeps, key, chain);
        if (s == RT_OK) s = download(h, heights, n, 0);
        return s;
    });
}

rt_status rt_sixv_cftp(rt_sixv* h, int32_t n, int64_t first_sweeps, int64_t master_seed, int32_t max_trials,
                       int32_t* out_heights, rt_cftp_stats* stats) {
    return guarded([&]() -> rt_status {
        if (!h) return RT_E_INVAL;
        if (!valid_n(n) || first_sweeps <= 0 || max_trials <= 0) return h->fail(RT_E_INVAL, "bad CFTP arguments");
        if (first_sweeps > kMaxColourSteps / 4) return h->fail(RT_E_INVAL, "more than 2^38 sweeps in one call");
        if (!h->monotone) return h->fail(RT_E_INVAL, "these weights give a heat bath that is not monotone: no CFTP");
        cudaSetDevice(h->device);
        if (!h->reserve(n)) return h->fail(RT_E_NOMEM, "cudaMalloc six-vertex lattices");
        std::vector<int32_t> hmin((size_t)(n + 1) * (n + 1)), hmax(hmin.size());
        rt_sixv_dwbc_heights(n, hmin.data(), hmax.data());
        std::mt19937 mt((std::mt19937::result_type)master_seed);
        std::vector<int64_t> sweeps{first_sweeps};
        std::vector<uint64_t> keys{(uint64_t)mt()};
        rt_cftp_stats st{};
        cudaEvent_t e0, e1;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        rt_status s = RT_OK;
        double ms_total = 0;
        for (int trial = 0; trial < max_trials && s == RT_OK; ++trial) {
            s = upload(h, hmax.data(), n, 0, false);
            if (s == RT_OK) s = upload(h, hmin.data(), n, 1, false);
            if (s != RT_OK) break;
            cudaEventRecord(e0, h->stream);
            for (size_t e = 0; e < sweeps.size() && s == RT_OK; ++e) s = run_epoch(h, n, 2, sweeps[e], keys[e], 0);
            if (s != RT_OK) break;
            cudaEventRecord(e1, h->stream);
            s = launch_count_diff(h->d_h[0], h->d_h[1], h->cap, h->d_count, h->stream, &h->err);
            if (s != RT_OK) break;
            unsigned long long diff = 0;
            cudaError_t ce = cudaMemcpyAsync(&diff, h->d_count, sizeof diff, cudaMemcpyDeviceToHost, h->stream);
            if (ce == cudaSuccess) ce = cudaStreamSynchronize(h->stream);
            if (ce != cudaSuccess) {
                s = h->cuda_fail(ce, "coalescence readback");
                break;
            }
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            ms_total += ms;
            st.trials = trial + 1;
            int64_t total = 0;
            for (int64_t x : sweeps) total += x;
            st.total_steps = 4 * total;
            if (diff == 0) {
                st.coalesced = 1;
                break;
            }
            if (trial + 1 < max_trials && total > kMaxColourSteps / 8) {
                // the next trial would run 2 total sweeps
                s = h->fail(RT_E_INVAL, "CFTP schedule beyond 2^38 sweeps without coalescence");
                break;
            }
            sweeps.insert(sweeps.begin(), total);
            keys.insert(keys.begin(), (uint64_t)mt());
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        st.device_ms = ms_total;
        if (stats) *stats = st;
        if (s != RT_OK) return s;
        if (out_heights) return download(h, out_heights, n, 0);
        return RT_OK;
    });
}

}  // extern "C"
