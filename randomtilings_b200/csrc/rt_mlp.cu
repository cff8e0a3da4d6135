// rt_mlp.cu -- training and inference kernels of the coordinate MLP
// (include/rt_b200_mlp.h).
//
// One kernel takes tiles of 128 rows through the whole network: the rows are
// gathered into shared memory, layer 0 runs in FP32, layers 1 and 2 (128 x
// 128) on the fifth-generation tensor cores (tcgen05.mma, BF16 inputs, FP32
// accumulators in tensor memory), layer 3 in FP32; with gradients, the whole
// backward pass follows in the same CTA.  Activations live in shared memory
// as BF16 tiles that serve as the operands of every product they enter: the
// same 8 x 16-byte core matrices are read K-major (X W^T, dZ W) or MN-major
// (dZ^T X), so nothing is transposed or written to global memory.  GELU and
// its derivative share one tanh; the derivative waits in tensor memory or
// registers for the backward pass.
//
// Weight gradients of the 128 x 128 layers are sums over ranges of up to 256
// rows, each accumulated in tensor memory by a pair of CTAs in row order; a
// second kernel adds the ranges, sums the other gradients over the rows in a
// fixed order from the rows' FP32 values, and applies Adam.  No sum depends on
// timing, so training repeats bit for bit.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/rt_b200_mlp.h"
#include "rt_device.cuh"
#include "rt_guard.h"

using rtb::guarded;

namespace rtb {
namespace mlp {

constexpr int IN = RT_MLP_IN;
constexpr int H = RT_MLP_WIDTH;
// Offsets into the FP32 parameter vector.
constexpr int OW0 = 0, OB0 = OW0 + H * IN, OW1 = OB0 + H, OB1 = OW1 + H * H, OW2 = OB1 + H, OB2 = OW2 + H * H,
              OW3 = OB2 + H, OB3 = OW3 + H, NPARAM = OB3 + 1;
static_assert(NPARAM == RT_MLP_PARAMS, "parameter layout");

// GELU, tanh form: 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))).
__device__ __forceinline__ float gelu(float z) {
    const float u = 0.7978845608f * (z + 0.044715f * z * z * z);
    return 0.5f * z * (1.0f + tanhf(u));
}
// gelu(z), and its derivative in `grad`.
__device__ __forceinline__ float gelu_both(float z, float& grad) {
    const float u = 0.7978845608f * (z + 0.044715f * z * z * z);
    const float t = tanhf(u);
    grad = 0.5f * (1.0f + t) + 0.5f * z * (1.0f - t * t) * 0.7978845608f * (1.0f + 3.0f * 0.044715f * z * z);
    return 0.5f * z * (1.0f + t);
}

// ---------------------------------------------------------------------------
// Tiles.  An operand tile is 128 x 128 BF16 in shared memory, core matrices of
// 8 rows x 16 bytes (8 columns): element (r, c) at tile_off(r, c / 8) + 2 (c
// mod 8).  Read K-major (MN = rows, K = columns) the next core matrix along K
// is 128 bytes on (leading byte offset) and the next 8 rows 2 KB on (stride
// byte offset); read MN-major (MN = columns, K = rows) the next 8 columns are
// 128 bytes on (stride) and the next 8 rows 2 KB on (leading).
// ---------------------------------------------------------------------------
constexpr int TR = 128;                 // rows of a tile
constexpr int kTile = TR * H * 2;       // bytes of an operand tile
constexpr int kPart = 2 * H * H;        // floats of one CTA's partial dW1, dW2
// Instruction descriptor (PTX ISA, kind::f16): D = F32 (bits 4-5 = 1), A = B =
// BF16 (bits 7-9, 10-12 = 1), N >> 3 at bits 17-22, M >> 4 at bits 24-28; bits
// 15 / 16 mark A / B as MN-major.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(H >> 3) << 17) | ((uint32_t)(TR >> 4) << 24);
constexpr unsigned long long kWaitLimit = 1ull << 26;  // mbarrier polls before giving up

__device__ __forceinline__ uint32_t tile_off(int r, int c8) {
    return (uint32_t)(((r >> 3) * (H / 8) + c8) * 128 + (r & 7) * 16);
}
// Shared-memory matrix descriptor, no swizzle, version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, bool mn_major) {
    const uint32_t lead = mn_major ? 2048u : 128u, stride = mn_major ? 128u : 2048u;
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(lead >> 4) << 16) | ((uint64_t)(stride >> 4) << 32) | (1ull << 46);
}

// D (128 x 128) = or += A B over K = 128, eight MMAs of K = 16; one thread.
__device__ __forceinline__ void mma_tile(uint32_t d, uint32_t a, bool a_mn, uint32_t b, bool b_mn, bool accumulate) {
    const uint32_t idesc = kIdesc | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u);
#pragma unroll
    for (int k = 0; k < H / 16; ++k) {
        const uint64_t da = smem_desc(a + (a_mn ? 4096u : 256u) * k, a_mn), db = smem_desc(b + (b_mn ? 4096u : 256u) * k, b_mn);
        const uint32_t acc = (accumulate || k > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
            ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc)
            : "memory");
    }
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    for (unsigned long long it = 0; it < kWaitLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Eight columns of this warp's 32 tensor-memory lanes.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&f)[8]) {
    uint32_t v[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(v[i]);
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float (&f)[8]) {
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __float_as_uint(f[i]);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Columns 8 c8 .. 8 c8 + 7 of row r, rounded to BF16, into an operand tile; and back.
__device__ __forceinline__ void store8(unsigned char* tile, int r, int c8, const float (&f)[8]) {
    __nv_bfloat162 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        w[i].x = __float2bfloat16(f[2 * i]);
        w[i].y = __float2bfloat16(f[2 * i + 1]);
    }
    *reinterpret_cast<uint4*>(tile + tile_off(r, c8)) = *reinterpret_cast<uint4*>(w);
}
__device__ __forceinline__ void load8(const unsigned char* tile, int r, int c8, float (&f)[8]) {
    const uint4 q = *reinterpret_cast<const uint4*>(tile + tile_off(r, c8));
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

struct NetArgs {
    const float* P;                 // FP32 parameters
    const __nv_bfloat16 *w1, *w2;   // BF16 copies of W1, W2
    const float *x, *t;             // rows (IN features each) and, for gradients, targets
    int n;                          // rows of this call
    int range;                      // gradients: rows of a range (a pair of CTAs), 64 .. 256
    int chain;                      // gradients: every pair has one range (see net_kernel)
    int64_t pool;                   // > 0: row b is row floor(u pool) of x, t, with u from Philox (seed, step)
    uint64_t seed;
    int64_t step;
    float* y;      // forward: predictions
    float* part;   // gradients: partial dW1, dW2 (kPart floats) of each CTA
    float4* rows;  // gradients: dy h3, dz2, dz1, dz0 of every row (kRowArrays arrays, row_at)
    int64_t row_array;   // float4s of one of them
    float *dy, *xb, *err2;  // gradients, by tile: dy of the rows, their features ([IN][TR]), their shares of the loss
    int* err;      // set to 1 when a bounded wait gives up
};
constexpr int kRowArrays = 4;
// Columns 4 c4 .. 4 c4 + 3 of row r of a tile: a warp's rows side by side.
__host__ __device__ __forceinline__ int64_t row_at(int64_t tile, int c4, int r) { return (tile * (H / 4) + c4) * TR + r; }

// Shared memory: W1, W2 and one activation tile (forward) or h1, h2, dz2 and
// dz1 (gradients), then the FP32 parts.
struct NetSmall {
    float w0[H * IN], b0[H], b1[H], b2[H], w3[H];
    float x[TR * IN], t[TR];
    float y[8][TR];
    float w3h[32 * TR];  // gradients: a third of the products h3 W3
};
constexpr size_t net_smem(bool grad) {
    return (size_t)(grad ? 6 : 3) * kTile + sizeof(NetSmall) - (grad ? 0 : sizeof(NetSmall::w3h));
}

// Thread (warp w, lane l) owns row 32 (w mod 4) + l -- the tensor-memory lanes
// its warp can reach -- and, of every 128 x 128 array, the 8 NCH columns of
// column group w / 4, taken eight at a time in loops that are not unrolled
// across each other: with 32 columns at once in registers the kernel was
// three times as much code and waited for instructions.
//
// Gradients run as clusters of two CTAs, one per half of a range.  With one
// range per pair (chain; batches of up to 74 ranges), the second CTA starts
// its dW1, dW2 accumulators from the first one's results, so a range is one
// sum in row order.  With more ranges than pairs, each CTA adds its tiles'
// products to its own partial.
template <bool GRAD, int THREADS>
__global__ void __launch_bounds__(THREADS, GRAD ? 1 : 2) net_kernel(const __grid_constant__ NetArgs g) {
    constexpr int GROUPS = THREADS / TR, NCH = H / 8 / GROUPS;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *sW1 = smem, *sH1 = smem + 2 * kTile, *sH2 = GRAD ? sH1 + kTile : sH1, *sDz2 = sH1 + 2 * kTile,
                  *sDz1 = sH1 + 3 * kTile;
    NetSmall& S = *reinterpret_cast<NetSmall*>(smem + (GRAD ? 6 : 3) * kTile);
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cg = warp >> 2, r = 32 * (warp & 3) + lane, b0 = NCH * cg;  // columns 8 b0 .. 8 (b0 + NCH) - 1
    constexpr uint32_t kCols = GRAD ? 512 : 128;
    const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar);
    const uint32_t aW1 = (uint32_t)__cvta_generic_to_shared(sW1), aW2 = aW1 + kTile;
    const uint32_t aH1 = (uint32_t)__cvta_generic_to_shared(sH1), aH2 = (uint32_t)__cvta_generic_to_shared(sH2),
                   aDz2 = (uint32_t)__cvta_generic_to_shared(sDz2), aDz1 = (uint32_t)__cvta_generic_to_shared(sDz1);

    if (warp == 0) {
        const uint32_t slot = (uint32_t)__cvta_generic_to_shared(&tmem_slot);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    for (int e = tid; e < TR * (H / 8); e += THREADS) {
        const int o = e / (H / 8), k8 = e % (H / 8);
        cp_async16(aW1 + tile_off(o, k8), g.w1 + o * H + 8 * k8);
        cp_async16(aW2 + tile_off(o, k8), g.w2 + o * H + 8 * k8);
    }
    for (int e = tid; e < H * IN; e += THREADS) S.w0[e] = g.P[OW0 + e];
    for (int e = tid; e < H; e += THREADS) {
        S.b0[e] = g.P[OB0 + e];
        S.b1[e] = g.P[OB1 + e];
        S.b2[e] = g.P[OB2 + e];
        S.w3[e] = g.P[OW3 + e];
    }
    const float b3 = g.P[OB3];
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    // D1: z1, then gelu'(z1); D2: z2, then gelu'(z2), dz2 W2, dz1 W1; dW1, dW2.
    // gelu'(z0) waits where dW1 goes at the end of a tile.
    const uint32_t D1 = tmem, D2 = GRAD ? tmem + H : tmem, DW1 = tmem + 2 * H, DW2 = tmem + 3 * H;
    const uint32_t mine = ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(8 * b0);  // this warp's lanes and columns

    uint32_t parity = 0;
    // Operands written by everyone -> products issued by one thread (`issue`)
    // -> accumulators readable by everyone.  False when a wait gave up.
    auto products = [&](auto issue) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            issue();
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mb) : "memory");
        }
        if (!mbar_wait(mb, parity)) {
            s_fail = 1;  // racy but every writer writes 1
            atomicOr(g.err, 1);
        }
        parity ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return !__syncthreads_or(*(volatile int*)&s_fail);
    };
    // dW2 (+)= dz2^T h2, dW1 (+)= dz1^T h1 of the tile in shared memory
    auto weight_products = [&](bool acc) {
        return products([&] {
            mma_tile(DW2, aDz2, true, aH2, true, acc);
            mma_tile(DW1, aDz1, true, aH1, true, acc);
        });
    };
    // The accumulators dW1, dW2 and this CTA's partial, [k / 4][o][k mod 4], so
    // that a warp's accesses are contiguous.  `f` sees eight values and the two
    // float4s they belong to.
    auto each_part = [&](int cta, auto f) {
        float4* part = reinterpret_cast<float4*>(g.part + (int64_t)cta * kPart);
#pragma unroll 1
        for (int e = 0; e < 2 * NCH; ++e) {
            const int which = e >= NCH, ch = e - which * NCH;
            float4* at = part + which * (H * H / 4) + 2 * (b0 + ch) * H + r;
            f((which ? DW2 : DW1) + mine + 8 * ch, at, at + H);
        }
    };
    auto store_part = [&](bool add) {
        each_part((int)blockIdx.x, [&](uint32_t taddr, float4* lo, float4* hi) {
            float v[8];
            tmem_ld8(taddr, v);
            if (add) {
                const float4 a = __ldcg(lo), b = __ldcg(hi);
                v[0] += a.x, v[1] += a.y, v[2] += a.z, v[3] += a.w;
                v[4] += b.x, v[5] += b.y, v[6] += b.z, v[7] += b.w;
            }
            __stcg(lo, make_float4(v[0], v[1], v[2], v[3]));
            __stcg(hi, make_float4(v[4], v[5], v[6], v[7]));
        });
    };

    // Forward: tiles blockIdx.x, + gridDim.x, ...  Gradients: pair p takes the
    // ranges p, + pairs, ...; CTA 0 of it rows 0 .. 127 of the range, CTA 1 the rest.
    const int rank = GRAD ? (int)(blockIdx.x & 1) : 0, pair = GRAD ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int pairs = GRAD ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int span = GRAD ? g.range : TR, units = (g.n + span - 1) / span;
    for (int u = pair; u < units; u += pairs) {
        const int row0 = u * span + TR * rank, rows = max(0, min(min(span - TR * rank, TR), g.n - row0));
        const int tile = GRAD ? 2 * u + rank : u;
        const bool live = r < rows;
        if (tid < TR) {
            const int b = row0 + tid;
            float4 lo = make_float4(0, 0, 0, 0), hi = lo;
            float t = 0.0f;
            if (tid < rows) {
                int64_t src = b;
                if (GRAD && g.pool > 0) {
                    // batch rows drawn with replacement
                    const uint4 w = philox4((uint32_t)b, (uint32_t)g.step, (uint32_t)((uint64_t)g.step >> 32), 0x4d4c50u,
                                            (uint32_t)g.seed, (uint32_t)(g.seed >> 32));
                    src = (int64_t)((((uint64_t)w.x << 32) | w.y) % (uint64_t)g.pool);
                }
                lo = *reinterpret_cast<const float4*>(g.x + src * IN);
                hi = *reinterpret_cast<const float4*>(g.x + src * IN + 4);
                if (GRAD) t = g.t[src];
            }
            *reinterpret_cast<float4*>(S.x + tid * IN) = lo;
            *reinterpret_cast<float4*>(S.x + tid * IN + 4) = hi;
            S.t[tid] = t;
            if (GRAD) {
                float* xb = g.xb + (int64_t)tile * IN * TR + tid;
                xb[0] = lo.x, xb[TR] = lo.y, xb[2 * TR] = lo.z, xb[3 * TR] = lo.w;
                xb[4 * TR] = hi.x, xb[5 * TR] = hi.y, xb[6 * TR] = hi.z, xb[7 * TR] = hi.w;
            }
        }
        __syncthreads();
        float x[IN];
#pragma unroll
        for (int k = 0; k < IN; ++k) x[k] = S.x[r * IN + k];
        // The layers: z (layer 0 from x, the others from tensor memory), h =
        // gelu(z) rounded to BF16 into its tile, gelu'(z) into tensor memory.
        bool ok = true;
        float ysum = 0.0f;
#pragma unroll 1
        for (int layer = 0; layer < 3; ++layer) {
            const uint32_t src = (layer == 1 ? D1 : D2) + mine, dst = (layer == 0 ? DW1 : layer == 1 ? D1 : D2) + mine;
            const float* bias = layer == 0 ? S.b0 : layer == 1 ? S.b1 : S.b2;
            unsigned char* tile_h = layer == 0 ? sH1 : layer == 1 ? sH2 : sDz1;  // h3 waits where dz1 goes
#pragma unroll 1
            for (int ch = 0; ch < NCH; ++ch) {
                const int c = 8 * (b0 + ch);
                float z[8], h[8], d[GRAD ? 8 : 1];
                if (layer == 0) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 wa = *reinterpret_cast<const float4*>(S.w0 + (c + i) * IN);
                        const float4 wb = *reinterpret_cast<const float4*>(S.w0 + (c + i) * IN + 4);
                        z[i] = bias[c + i];
                        z[i] += wa.x * x[0], z[i] += wa.y * x[1], z[i] += wa.z * x[2], z[i] += wa.w * x[3];
                        z[i] += wb.x * x[4], z[i] += wb.y * x[5], z[i] += wb.z * x[6], z[i] += wb.w * x[7];
                    }
                } else {
                    tmem_ld8(src + 8 * ch, z);
#pragma unroll
                    for (int i = 0; i < 8; ++i) z[i] += bias[c + i];
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) h[i] = GRAD ? gelu_both(z[i], d[GRAD ? i : 0]) : gelu(z[i]);
                if (GRAD || layer < 2) {
                    store8(tile_h, r, b0 + ch, h);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) ysum += __bfloat162float(__float2bfloat16(h[i])) * S.w3[c + i];
                }
                if constexpr (GRAD) tmem_st8(dst + 8 * ch, d);
            }
            if (layer == 0) ok = products([&] { mma_tile(D1, aH1, false, aW1, false, false); });  // z1 = h1 W1^T
            if (layer == 1) ok = products([&] { mma_tile(D2, aH2, false, aW2, false, false); });  // z2 = h2 W2^T
            if (!ok) break;
        }
        if (!ok) break;
        if constexpr (!GRAD) {
            S.y[cg][r] = ysum;
            __syncthreads();
            if (cg == 0 && live) g.y[row0 + r] = ((S.y[0][r] + S.y[1][r]) + (S.y[2][r] + S.y[3][r])) + b3;
        } else {
            // y = h3 W3 + b3: the products of columns c, c + 32, c + 64 and c + 96 in
            // turn, then pairwise over c mod 32.  y - t cancels, so the order of this
            // sum shows in every gradient.  Columns 32 .. 127 pass through dz2's tile
            // and w3h as [c][row].
            float* const p1 = reinterpret_cast<float*>(sDz2);
#pragma unroll 1
            for (int ch = 0; ch < NCH; ++ch) {
                const int c = 8 * (b0 + ch);
                if (c < 32) continue;
                float h[8];
                load8(sDz1, r, b0 + ch, h);
                float* p = c < 96 ? p1 + (c - 32) * TR : S.w3h + (c - 96) * TR;
#pragma unroll
                for (int i = 0; i < 8; ++i) p[i * TR + r] = h[i] * S.w3[c + i];
            }
            __syncthreads();
            if (cg == 0) {
                float q[32];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float h[8];
                    load8(sDz1, r, k, h);
#pragma unroll
                    for (int i = 0; i < 8; ++i) q[8 * k + i] = h[i] * S.w3[8 * k + i];
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    q[i] = q[i] + p1[i * TR + r];
                    q[i] = q[i] + p1[(32 + i) * TR + r];
                    q[i] = q[i] + S.w3h[i * TR + r];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < o; ++i) q[i] += q[i + o];
                S.y[0][r] = q[0];
            }
            __syncthreads();
            const float e = S.y[0][r] + b3 - S.t[r];
            const float dy = live ? 2.0f * e / (float)g.n : 0.0f;
            if (cg == 0) {
                g.dy[(int64_t)tile * TR + r] = dy;
                g.err2[(int64_t)tile * TR + r] = live ? e * e / (float)g.n : 0.0f;
            }
            // Eight of this thread's values of row array `which`.
            auto put = [&](int which, int ch, const float (&f)[8]) {
                float4* dst = g.rows + which * g.row_array + row_at(tile, 2 * (b0 + ch), r);
                __stcg(dst, make_float4(f[0], f[1], f[2], f[3]));
                __stcg(dst + TR, make_float4(f[4], f[5], f[6], f[7]));
            };
#pragma unroll 1
            for (int ch = 0; ch < NCH; ++ch) {
                float v[8], d[8];
                load8(sDz1, r, b0 + ch, v);
                tmem_ld8(D2 + mine + 8 * ch, d);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[i] = dy * v[i];                              // dy h3
                    d[i] = dy * S.w3[8 * (b0 + ch) + i] * d[i];    // dz2
                }
                store8(sDz2, r, b0 + ch, d);
                put(0, ch, v);
                put(1, ch, d);
            }
            if (!products([&] { mma_tile(D2, aDz2, false, aW2, true, false); })) break;  // dz2 W2
#pragma unroll 1
            for (int ch = 0; ch < NCH; ++ch) {
                float v[8], d[8];
                tmem_ld8(D2 + mine + 8 * ch, v);
                tmem_ld8(D1 + mine + 8 * ch, d);
#pragma unroll
                for (int i = 0; i < 8; ++i) d[i] = v[i] * d[i];  // dz1
                store8(sDz1, r, b0 + ch, d);
                put(2, ch, d);
            }
            if (!products([&] { mma_tile(D2, aDz1, false, aW1, true, false); })) break;  // dz1 W1
#pragma unroll 1
            for (int ch = 0; ch < NCH; ++ch) {
                float v[8], d[8];
                tmem_ld8(D2 + mine + 8 * ch, v);
                tmem_ld8(DW1 + mine + 8 * ch, d);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = v[i] * d[i];  // dz0
                put(3, ch, v);
            }
            if (!(g.chain && rank == 1)) {
                if (!weight_products(false)) break;
                store_part(u != pair);
            }
        }
        __syncthreads();
    }

    if (GRAD && g.chain) {
        // both CTAs pass here, whatever happened to either
        __threadfence();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank == 1 && !s_fail) {
            each_part((int)blockIdx.x - 1, [&](uint32_t taddr, float4* lo, float4* hi) {
                const float4 a = __ldcg(lo), b = __ldcg(hi);
                const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                tmem_st8(taddr, v);
            });
            if (weight_products(true)) store_part(false);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        if (s_fail) {
            // the MMAs may still be running: wait for them (bounded) before freeing their accumulators
            mbar_wait(mb, parity ^ 1u);
        }
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
    }
}
constexpr int kFwdThreads = 512, kGradThreads = 512;

// BF16 copies of W1, W2 for the tensor-core products.
__global__ void to_bf16(const float* __restrict__ P, __nv_bfloat16* w1, __nv_bfloat16* w2) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= H * H) return;
    w1[e] = __float2bfloat16(P[OW1 + e]);
    w2[e] = __float2bfloat16(P[OW2 + e]);
}

// The second kernel of a gradient.  Blocks by role, 256 threads each, the
// longest first:
//   dW0, four rows and two inputs a block (128): lane p of warps 0 and 1 sums
//     the rows p, p + 32, ... of an input, staged through shared memory by the
//     block -- one chain of n / 32 additions a lane, and 384 KB of a batch of
//     16,384 through each block;
//   dW1, dW2 (128): the sum of the partials;
//   dW3, db2, db1, db0, four columns a block (128): thread s sums the rows
//     s, s + 256, ... of its columns, then the block the threads (within warps,
//     then warp by warp);
//   db3 and the loss (1).
// Rows that a tile does not have were written as zeros.  ADAM: the step, and
// the BF16 copies; else the gradient.  It reads 92 MB at batch 16,384, just
// written and still in L2: 18 us, 10 of them for the roles after the first.
struct SumArgs {
    const float* part;
    int parts, part_first, part_step;  // partials part_first, + part_step, ...
    const float4* rows;
    int64_t row_array;
    const float *dy, *xb, *err2;
    int n, range;
    float *P, *M1, *M2, *G, *loss;
    __nv_bfloat16 *w1, *w2;
    float lr, b1t, b2t;
};
constexpr int kW0Inputs = 2;  // dW0: inputs of a block
constexpr int kSumBlocks = 128 + 32 * kRowArrays + 32 * (IN / kW0Inputs) + 1;
constexpr int kStage = 8;  // dW0: tiles of a stage
constexpr int kBufs = 4;   // stages, three of them on their way
constexpr int kSumSmem = kBufs * kStage * TR * (16 + kW0Inputs * 4);

template <bool ADAM>
__device__ __forceinline__ void take_gradient(const SumArgs& a, int at, float grad) {
    if (!ADAM) {
        a.G[at] = grad;
        return;
    }
    const float m = 0.9f * a.M1[at] + 0.1f * grad;
    const float v = 0.999f * a.M2[at] + 0.001f * grad * grad;
    a.M1[at] = m;
    a.M2[at] = v;
    const float mh = m / (1.0f - a.b1t), vh = v / (1.0f - a.b2t);
    const float np = a.P[at] - a.lr * mh / (sqrtf(vh) + 1e-8f);
    a.P[at] = np;
    if (at >= OW1 && at < OB1) a.w1[at - OW1] = __float2bfloat16(np);
    if (at >= OW2 && at < OB2) a.w2[at - OW2] = __float2bfloat16(np);
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ float4 shfl_xor4(float4 a, int o) {
    return make_float4(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o),
                       __shfl_xor_sync(0xffffffffu, a.z, o), __shfl_xor_sync(0xffffffffu, a.w, o));
}

template <bool ADAM>
__global__ void __launch_bounds__(256) sum_kernel(const __grid_constant__ SumArgs a) {
    extern __shared__ __align__(16) unsigned char sum_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int role = blockIdx.x;
    // Place of row `row` among the tiles: tile * TR + row of the tile.
    auto place = [&](int row, int64_t* tile, int* r) {
        const int u = row / a.range, rem = row - u * a.range;
        *tile = 2 * (int64_t)u + (rem >= TR);
        *r = rem & (TR - 1);
    };
    const int ranges = (a.n + a.range - 1) / a.range;
    __shared__ float4 s_part[8];
    if (role < 32 * (IN / kW0Inputs)) {
        const int c4 = role & 31, k0 = kW0Inputs * (role >> 5);
        float4(*s_d)[kStage * TR] = reinterpret_cast<float4(*)[kStage * TR]>(sum_smem);
        float(*s_x)[kW0Inputs * kStage * TR] = reinterpret_cast<float(*)[kW0Inputs * kStage * TR]>(sum_smem + kBufs * kStage * TR * 16);
        const float4* src = a.rows + 3 * a.row_array;
        const int tiles = 2 * ranges, stages = (tiles + kStage - 1) / kStage;
        auto load = [&](int st) {
            if (st < stages) {
                const int buf = st % kBufs, n = min(kStage, tiles - st * kStage);
                for (int e = tid; e < n * TR; e += 256)
                    cp_async16((uint32_t)__cvta_generic_to_shared(&s_d[buf][e]),
                               src + row_at((int64_t)st * kStage + e / TR, c4, e % TR));
                constexpr int kQuads = kW0Inputs * TR / 4;  // the inputs of a tile are side by side
                for (int e = tid; e < n * kQuads; e += 256)
                    cp_async16((uint32_t)__cvta_generic_to_shared(&s_x[buf][4 * e]),
                               a.xb + (((int64_t)st * kStage + e / kQuads) * IN + k0) * TR + 4 * (e % kQuads));
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float4 s = make_float4(0, 0, 0, 0);
        for (int st = 0; st < kBufs - 1; ++st) load(st);
        for (int st = 0; st < stages; ++st) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kBufs - 2) : "memory");
            __syncthreads();  // the stage has arrived, and everyone is done with the one before
            load(st + kBufs - 1);
            if (warp >= kW0Inputs) continue;
            const int buf = st % kBufs, n = min(kStage, tiles - st * kStage);
            const float4* d = s_d[buf] + lane;
            const float* x = s_x[buf] + warp * TR + lane;
            auto product = [&](int e) {
                const float4 v = d[(e >> 2) * TR + 32 * (e & 3)];
                const float w = x[(e >> 2) * kW0Inputs * TR + 32 * (e & 3)];
                return make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
            };
            if (n == kStage) {
                float4 v[4 * kStage];
#pragma unroll
                for (int e = 0; e < 4 * kStage; ++e) v[e] = product(e);
#pragma unroll
                for (int e = 0; e < 4 * kStage; ++e) s = add4(s, v[e]);
            } else {
                for (int e = 0; e < 4 * n; ++e) s = add4(s, product(e));
            }
        }
        if (warp >= kW0Inputs) return;
        float4 t = make_float4(0, 0, 0, 0);
        for (int p = 0; p < 32; ++p)
            t = add4(t, make_float4(__shfl_sync(0xffffffffu, s.x, p), __shfl_sync(0xffffffffu, s.y, p),
                                    __shfl_sync(0xffffffffu, s.z, p), __shfl_sync(0xffffffffu, s.w, p)));
        if (lane < 4)
            take_gradient<ADAM>(a, OW0 + (4 * c4 + lane) * IN + k0 + warp,
                                lane == 0 ? t.x : lane == 1 ? t.y : lane == 2 ? t.z : t.w);
        return;
    }
    role -= 32 * (IN / kW0Inputs);
    if (role < 128) {
        // four lanes share four consecutive floats, each lane a quarter of the partials
        const int e4 = role * 64 + (tid >> 2), sub = tid & 3;
        const float4* p = reinterpret_cast<const float4*>(a.part) + e4;
        float4 s = make_float4(0, 0, 0, 0);
        p += (int64_t)a.part_first * (kPart / 4);
        const int64_t step = (int64_t)a.part_step * (kPart / 4);
        int b = sub;
        for (; b + 28 < a.parts; b += 32) {
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __ldcg(p + (b + 4 * k) * step);
#pragma unroll
            for (int k = 0; k < 8; ++k) s = add4(s, v[k]);
        }
        for (; b < a.parts; b += 4) s = add4(s, __ldcg(p + b * step));
        s = add4(s, shfl_xor4(s, 1));
        s = add4(s, shfl_xor4(s, 2));
        const float grad = sub == 0 ? s.x : sub == 1 ? s.y : sub == 2 ? s.z : s.w;
        const int which = e4 >= H * H / 4, e = e4 - which * (H * H / 4);  // e = (k / 4) H + o
        take_gradient<ADAM>(a, (which ? OW2 : OW1) + (e & (H - 1)) * H + (e / H) * 4 + sub, grad);
        return;
    }
    role -= 128;
    if (role < 32 * kRowArrays) {
        const int which = role >> 5, c4 = role & 31;
        const float4* src = a.rows + which * a.row_array;
        float4 s = make_float4(0, 0, 0, 0);
        if (a.range == 256) {
            const float4* q = src + row_at(tid >> 7, c4, tid & (TR - 1));
            int u = 0;
            for (; u + 16 <= ranges; u += 16) {
                float4 v[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) v[k] = __ldcg(q + (u + k) * row_at(2, 0, 0));
#pragma unroll
                for (int k = 0; k < 16; ++k) s = add4(s, v[k]);
            }
            for (; u < ranges; ++u) s = add4(s, __ldcg(q + u * row_at(2, 0, 0)));
        } else {
            for (int row = tid; row < a.n; row += 256) {
                int64_t tile;
                int r;
                place(row, &tile, &r);
                s = add4(s, __ldcg(src + row_at(tile, c4, r)));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = add4(s, shfl_xor4(s, o));
        if (lane == 0) s_part[warp] = s;
        __syncthreads();
        if (tid < 4) {
            float t = 0.0f;
            for (int w = 0; w < 8; ++w) t += reinterpret_cast<const float*>(s_part + w)[tid];
            take_gradient<ADAM>(a, (which == 0 ? OW3 : which == 1 ? OB2 : which == 2 ? OB1 : OB0) + 4 * c4 + tid, t);
        }
        return;
    }
    float s = 0.0f, loss = 0.0f;
    if (a.range == 256) {
        int u = 0;
        for (; u + 16 <= ranges; u += 16) {
            float v[16], w[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = __ldcg(a.dy + (u + k) * 256 + tid), w[k] = __ldcg(a.err2 + (u + k) * 256 + tid);
#pragma unroll
            for (int k = 0; k < 16; ++k) s += v[k], loss += w[k];
        }
        for (; u < ranges; ++u) {
            s += __ldcg(a.dy + u * 256 + tid);
            loss += __ldcg(a.err2 + u * 256 + tid);
        }
    } else {
        for (int row = tid; row < a.n; row += 256) {
            int64_t tile;
            int r;
            place(row, &tile, &r);
            s += __ldcg(a.dy + tile * TR + r);
            loss += __ldcg(a.err2 + tile * TR + r);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        loss += __shfl_xor_sync(0xffffffffu, loss, o);
    }
    if (lane == 0) s_part[warp] = make_float4(s, loss, 0.0f, 0.0f);
    __syncthreads();
    if (tid == 0) {
        float t = 0.0f, l = 0.0f;
        for (int w = 0; w < 8; ++w) t += s_part[w].x, l += s_part[w].y;
        take_gradient<ADAM>(a, OB3, t);
        *a.loss = l;
    }
}

}  // namespace mlp
}  // namespace rtb

using namespace rtb::mlp;

struct rt_mlp {
    int device = 0;
    cudaStream_t s = nullptr;
    float *P = nullptr, *G = nullptr, *M1 = nullptr, *M2 = nullptr;
    __nv_bfloat16 *w1 = nullptr, *w2 = nullptr;
    int64_t adam_t = 0;
    // workspace: up to `cap` rows from the host; gradients of up to `gtiles` tiles on `sms` CTAs
    int64_t cap = 0;
    float *x = nullptr, *t = nullptr, *y = nullptr, *loss = nullptr;
    float *part = nullptr, *dy = nullptr, *xb = nullptr, *err2 = nullptr;
    float4* rowvals = nullptr;
    int64_t gtiles = 0;
    int sms = 0;
    float *X = nullptr, *T = nullptr;
    int64_t rows = 0;
    int* err = nullptr;  // device: set when a bounded wait gave up
    size_t over = 0;     // RT_TEST_REFUSE_LAUNCH: bytes of shared memory asked for beyond what is allowed
};

namespace {

void free_ws(rt_mlp* m) {
    void* ps[] = {m->x, m->t, m->y};
    for (void* p : ps)
        if (p) cudaFree(p);
    m->x = m->t = m->y = nullptr;
    m->cap = 0;
}

bool reserve(rt_mlp* m, int64_t n) {
    if (n <= m->cap) return true;
    free_ws(m);
    bool ok = cudaMalloc(&m->x, (size_t)n * IN * 4) == cudaSuccess && cudaMalloc(&m->t, (size_t)n * 4) == cudaSuccess &&
              cudaMalloc(&m->y, (size_t)n * 4) == cudaSuccess;
    if (!ok) {
        free_ws(m);
        return false;
    }
    m->cap = n;
    return true;
}

NetArgs net_args(const rt_mlp* m, int n) {
    NetArgs g;
    std::memset(&g, 0, sizeof g);
    g.P = m->P;
    g.w1 = m->w1;
    g.w2 = m->w2;
    g.x = m->x;
    g.t = m->t;
    g.n = n;
    g.y = m->y;
    g.err = m->err;
    return g;
}

// `pair`: clusters of two CTAs.
template <class K, class A>
bool launch(rt_mlp* m, K kernel, int grid, int block, size_t smem, bool pair, const A& args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = m->s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pair ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kernel, args) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

// Predictions of the n rows in m->x into m->y: two CTAs a SM.
bool forward(rt_mlp* m, int n) {
    const int tiles = (n + TR - 1) / TR;
    return launch(m, net_kernel<false, kFwdThreads>, std::min(tiles, 2 * m->sms), kFwdThreads, net_smem(false) + m->over, false,
                  net_args(m, n));
}

// Rows of a range: 256, or less where that evens out the ranges (a multiple of 64).
int range_rows(int n) {
    const int ranges = (n + 255) / 256;
    return ((n + ranges - 1) / ranges + 63) / 64 * 64;
}

void free_gradient_ws(rt_mlp* m) {
    void* ps[] = {m->part, m->dy, m->xb, m->err2, m->rowvals};
    for (void* p : ps)
        if (p) cudaFree(p);
    m->part = m->dy = m->xb = m->err2 = nullptr;
    m->rowvals = nullptr;
    m->gtiles = 0;
}

bool reserve_gradient(rt_mlp* m, int n) {
    const int range = range_rows(n);
    const int64_t tiles = 2 * (((int64_t)n + range - 1) / range);
    if (tiles <= m->gtiles) return true;
    free_gradient_ws(m);
    const size_t rows = (size_t)tiles * TR;
    const bool ok = cudaMalloc(&m->part, (size_t)m->sms * kPart * 4) == cudaSuccess &&
                    cudaMalloc(&m->dy, rows * 4) == cudaSuccess && cudaMalloc(&m->err2, rows * 4) == cudaSuccess &&
                    cudaMalloc(&m->xb, rows * IN * 4) == cudaSuccess &&
                    cudaMalloc(&m->rowvals, rows * kRowArrays * H * 4) == cudaSuccess;
    if (!ok) {
        free_gradient_ws(m);
        cudaGetLastError();
        return false;
    }
    m->gtiles = tiles;
    return true;
}

// Loss and gradient of g's rows: into m->G and m->loss, or an Adam step.  False
// if a kernel did not start; the second one then does not either.
bool gradient(rt_mlp* m, NetArgs g, bool adam, float lr, float b1t, float b2t) {
    g.range = range_rows(g.n);
    const int ranges = (g.n + g.range - 1) / g.range, pairs = std::min(ranges, m->sms / 2);
    g.chain = ranges == pairs;
    g.part = m->part;
    g.rows = m->rowvals;
    g.row_array = m->gtiles * TR * (H / 4);
    g.dy = m->dy;
    g.xb = m->xb;
    g.err2 = m->err2;
    if (!launch(m, net_kernel<true, kGradThreads>, 2 * pairs, kGradThreads, net_smem(true) + m->over, true, g)) return false;
    SumArgs a;
    std::memset(&a, 0, sizeof a);
    a.part = m->part;
    a.parts = g.chain ? pairs : 2 * pairs;  // a chain's sum is its second CTA's
    a.part_first = g.chain ? 1 : 0;
    a.part_step = g.chain ? 2 : 1;
    a.rows = g.rows;
    a.row_array = g.row_array;
    a.dy = g.dy;
    a.xb = g.xb;
    a.err2 = g.err2;
    a.n = g.n;
    a.range = g.range;
    a.P = m->P;
    a.M1 = m->M1;
    a.M2 = m->M2;
    a.G = m->G;
    a.loss = m->loss;
    a.w1 = m->w1;
    a.w2 = m->w2;
    a.lr = lr;
    a.b1t = b1t;
    a.b2t = b2t;
    return adam ? launch(m, sum_kernel<true>, kSumBlocks, 256, kSumSmem, false, a)
                : launch(m, sum_kernel<false>, kSumBlocks, 256, kSumSmem, false, a);
}

rt_status sync(rt_mlp* m) {
    if (cudaStreamSynchronize(m->s) != cudaSuccess) return RT_E_CUDA;
    int e = 0;
    if (cudaMemcpy(&e, m->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return RT_E_CUDA;
    return e ? RT_E_TIMEOUT : RT_OK;
}

}  // namespace

extern "C" {

rt_status rt_mlp_create(int32_t device, uint64_t seed, rt_mlp** out) {
    return guarded([&]() -> rt_status {
        if (!out) return RT_E_INVAL;
        *out = nullptr;
        if (cudaSetDevice(device) != cudaSuccess) return RT_E_NODEVICE;
        rt_mlp* m = new rt_mlp();
        m->device = device;
        if (std::getenv("RT_TEST_REFUSE_LAUNCH")) m->over = 1024;
        bool ok = cudaStreamCreateWithFlags(&m->s, cudaStreamNonBlocking) == cudaSuccess &&
                  cudaMalloc(&m->P, NPARAM * 4) == cudaSuccess && cudaMalloc(&m->G, NPARAM * 4) == cudaSuccess &&
                  cudaMalloc(&m->M1, NPARAM * 4) == cudaSuccess && cudaMalloc(&m->M2, NPARAM * 4) == cudaSuccess &&
                  cudaMalloc(&m->w1, H * H * 2) == cudaSuccess && cudaMalloc(&m->w2, H * H * 2) == cudaSuccess &&
                  cudaMalloc(&m->loss, 4) == cudaSuccess && cudaMalloc(&m->err, sizeof(int)) == cudaSuccess &&
                  cudaMemset(m->err, 0, sizeof(int)) == cudaSuccess &&
                  cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
                  cudaFuncSetAttribute((const void*)net_kernel<false, kFwdThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)net_smem(false)) == cudaSuccess &&
                  cudaFuncSetAttribute((const void*)net_kernel<true, kGradThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)net_smem(true)) == cudaSuccess &&
                  cudaFuncSetAttribute((const void*)sum_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSumSmem) == cudaSuccess &&
                  cudaFuncSetAttribute((const void*)sum_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSumSmem) == cudaSuccess;
        if (!ok) {
            rt_mlp_destroy(m);
            return RT_E_NOMEM;
        }
        // Initialisation: weights uniform in +-1/sqrt(fan_in) from Philox(seed), biases 0.
        std::vector<float> p(NPARAM, 0.0f);
        auto fill = [&](int off, int count, int fan_in) {
            const float a = 1.0f / std::sqrt((float)fan_in);
            for (int i = 0; i < count; ++i) {
                const uint4 w = rtb::philox4((uint32_t)(off + i), 0x494e4954u, 0, 0, (uint32_t)seed, (uint32_t)(seed >> 32));
                p[off + i] = a * (2.0f * ((float)(w.x >> 8) * (1.0f / 16777216.0f)) - 1.0f);
            }
        };
        fill(OW0, H * IN, IN);
        fill(OW1, H * H, H);
        fill(OW2, H * H, H);
        fill(OW3, H, H);
        *out = m;
        return rt_mlp_set_params(m, p.data());
    });
}

rt_status rt_mlp_destroy(rt_mlp* m) {
    return guarded([&]() -> rt_status {
        if (!m) return RT_E_INVAL;
        cudaSetDevice(m->device);
        if (m->s) cudaStreamSynchronize(m->s);
        free_ws(m);
        free_gradient_ws(m);
        void* ps[] = {m->P, m->G, m->M1, m->M2, m->w1, m->w2, m->loss, m->X, m->T, m->err};
        for (void* p : ps)
            if (p) cudaFree(p);
        if (m->s) cudaStreamDestroy(m->s);
        delete m;
        return RT_OK;
    });
}

rt_status rt_mlp_get_params(rt_mlp* m, float* params) {
    return guarded([&]() -> rt_status {
        if (!m || !params) return RT_E_INVAL;
        cudaSetDevice(m->device);
        if (cudaMemcpyAsync(params, m->P, NPARAM * 4, cudaMemcpyDeviceToHost, m->s) != cudaSuccess) return RT_E_CUDA;
        return sync(m);
    });
}

rt_status rt_mlp_set_params(rt_mlp* m, const float* params) {
    return guarded([&]() -> rt_status {
        if (!m || !params) return RT_E_INVAL;
        cudaSetDevice(m->device);
        cudaMemcpyAsync(m->P, params, NPARAM * 4, cudaMemcpyHostToDevice, m->s);
        cudaMemsetAsync(m->M1, 0, NPARAM * 4, m->s);
        cudaMemsetAsync(m->M2, 0, NPARAM * 4, m->s);
        m->adam_t = 0;
        to_bf16<<<(H * H + 255) / 256, 256, 0, m->s>>>(m->P, m->w1, m->w2);
        return sync(m);
    });
}

rt_status rt_mlp_predict(rt_mlp* m, const float* x, int64_t n, float* y) {
    return guarded([&]() -> rt_status {
        if (!m || !x || !y || n < 0) return RT_E_INVAL;
        cudaSetDevice(m->device);
        const int64_t chunk = 1 << 18;
        for (int64_t r0 = 0; r0 < n; r0 += chunk) {
            const int rn = (int)std::min<int64_t>(chunk, n - r0);
            if (!reserve(m, rn)) return RT_E_NOMEM;
            cudaMemcpyAsync(m->x, x + r0 * IN, (size_t)rn * IN * 4, cudaMemcpyHostToDevice, m->s);
            if (!forward(m, rn)) return RT_E_CUDA;
            cudaMemcpyAsync(y + r0, m->y, (size_t)rn * 4, cudaMemcpyDeviceToHost, m->s);
            rt_status st = sync(m);
            if (st != RT_OK) return st;
        }
        return RT_OK;
    });
}

rt_status rt_mlp_loss_grad(rt_mlp* m, const float* x, const float* target, int64_t n, float* loss, float* grad) {
    return guarded([&]() -> rt_status {
        if (!m || !x || !target || n <= 0 || n > (1 << 22)) return RT_E_INVAL;
        cudaSetDevice(m->device);
        if (!reserve(m, n) || !reserve_gradient(m, (int)n)) return RT_E_NOMEM;
        cudaMemcpyAsync(m->x, x, (size_t)n * IN * 4, cudaMemcpyHostToDevice, m->s);
        cudaMemcpyAsync(m->t, target, (size_t)n * 4, cudaMemcpyHostToDevice, m->s);
        if (!gradient(m, net_args(m, (int)n), false, 0.0f, 0.0f, 0.0f)) return RT_E_CUDA;
        if (loss) cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, m->s);
        if (grad) cudaMemcpyAsync(grad, m->G, NPARAM * 4, cudaMemcpyDeviceToHost, m->s);
        return sync(m);
    });
}

rt_status rt_mlp_set_data(rt_mlp* m, const float* x, const float* target, int64_t n) {
    return guarded([&]() -> rt_status {
        // At most 2^40 rows, so that no byte count below can wrap.
        if (!m || !x || !target || n <= 0 || n > ((int64_t)1 << 40)) return RT_E_INVAL;
        cudaSetDevice(m->device);
        if (m->X) cudaFree(m->X);
        if (m->T) cudaFree(m->T);
        m->X = m->T = nullptr;
        m->rows = 0;
        // Both buffers or neither: training checks for both.
        float *X = nullptr, *T = nullptr;
        const bool okx = cudaMalloc(&X, (size_t)n * IN * 4) == cudaSuccess;
        const bool okt = okx && cudaMalloc(&T, (size_t)n * 4) == cudaSuccess;
        if (!okt) {
            if (okx) cudaFree(X);
            cudaGetLastError();
            return RT_E_NOMEM;
        }
        m->X = X;
        m->T = T;
        cudaMemcpyAsync(m->X, x, (size_t)n * IN * 4, cudaMemcpyHostToDevice, m->s);
        cudaMemcpyAsync(m->T, target, (size_t)n * 4, cudaMemcpyHostToDevice, m->s);
        m->rows = n;
        return sync(m);
    });
}

rt_status rt_mlp_train(rt_mlp* m, int64_t steps, int32_t batch, float lr, uint64_t seed, float* loss) {
    return guarded([&]() -> rt_status {
        if (!m || steps < 0 || batch <= 0 || batch > (1 << 22) || !m->X || !m->T || m->rows <= 0) return RT_E_INVAL;
        cudaSetDevice(m->device);
        if (!reserve_gradient(m, batch)) return RT_E_NOMEM;
        NetArgs g = net_args(m, batch);
        g.x = m->X;
        g.t = m->T;
        g.pool = m->rows;
        g.seed = seed;
        for (int64_t k = 0; k < steps; ++k) {
            g.step = m->adam_t++;
            const float b1t = std::pow(0.9f, (float)m->adam_t), b2t = std::pow(0.999f, (float)m->adam_t);
            if (!gradient(m, g, true, lr, b1t, b2t)) {
                --m->adam_t;
                return RT_E_CUDA;
            }
        }
        if (loss) cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, m->s);
        return sync(m);
    });
}

}  // extern "C"
