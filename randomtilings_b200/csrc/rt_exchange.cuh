// rt_exchange.cuh -- halo-row exchange between the CTAs of one walk.
#pragma once

#include "rt_models.cuh"

namespace rtb {

// ---------------------------------------------------------------------------
// Halo exchange.  After each flip phase a CTA publishes the first and last
// row of its band (of the colour it just flipped) into a slot of global
// memory; every 64-bit slot word carries 32 bits of lattice data and the
// phase tag (phase + 1), so a neighbour knows the row is complete by polling
// the words themselves -- no separate flag, no memory fence on the critical
// path.  Slots are double-buffered by phase parity; a CTA enters phase p only
// after both neighbours finished phase p-1, so a slot is never overwritten
// before it was read.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long* slot(const WalkArgs& a, int cta, int side, int parity, int lat,
                                                   int k) {
    return a.xbuf + (((((size_t)cta * 2 + side) * 2 + parity) * a.nlat + lat) * a.xslots + k) * a.xwords;
}

// Index of the k-th set bit of mask (k < popc(mask)).
__device__ __forceinline__ int nth_bit(uint32_t mask, int k) {
    for (int i = 0; i < k; ++i) mask &= mask - 1;
    return __ffs(mask) - 1;
}

template <class T>
__device__ __forceinline__ uint32_t pack_word(const T* row, int w) {
    if (sizeof(T) == 1) return reinterpret_cast<const uint32_t*>(row)[w];
    return (uint32_t)row[w];
}
template <class T>
__device__ __forceinline__ void unpack_word(T* row, int w, uint32_t v) {
    if (sizeof(T) == 1)
        reinterpret_cast<uint32_t*>(row)[w] = v;
    else
        row[w] = (T)v;
}

// Whether a wait goes on: false on timeout (a.timeout_ns from the first check
// of this wait's clock t0, 0 before it) or when another CTA already reported an
// error.  The clock starts at this wait, so a walk may run for any length of
// time; only a single wait is bounded.
template <class A>  // the kernel's arguments: err, timeout_ns
__device__ __forceinline__ bool wait_more(const A& a, uint64_t& t0) {
    if (*(volatile int*)a.err) return false;
    const uint64_t now = global_ns();
    if (t0 == 0) {
        t0 = now;
    } else if (now - t0 > a.timeout_ns) {
        atomicOr(a.err, ERR_TIMEOUT);
        return false;
    }
    return true;
}

// Waits for one tagged word; returns false where wait_more does.
__device__ __forceinline__ bool wait_word(const WalkArgs& a, const unsigned long long* p, uint32_t tag,
                                          uint32_t* out) {
    unsigned spins = 0;
    uint64_t t0 = 0;
    for (;;) {
        const unsigned long long x = ld_relaxed64(p);
        if ((uint32_t)(x >> 32) == tag) {
            *out = (uint32_t)x;
            return true;
        }
        if ((++spins & 63u) == 0u && !wait_more(a, t0)) return false;
    }
}

// ---------------------------------------------------------------------------
// Exchange of the rows next to a band.  A row of the colour flipped in phase
// p is published as tagged 64-bit words (32 bits of lattice, p + 1), double
// buffered by the parity of p; its reader is the thread that owns the word
// next to it, which polls the words it needs in phase p + 1 (never a copy of
// the row in shared memory), so a wait costs its own warp and no barrier.  A
// CTA publishes phase p + 2 only after it read its neighbour's phase p + 1,
// which the neighbour published after reading phase p: a slot is rewritten
// only after it was read.
//   CLUSTER = false: slots in global memory (any number of co-resident CTAs).
//   CLUSTER = true: the CTAs are one thread-block cluster and a row is written
//   straight into its reader's shared memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_addr(uint32_t saddr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}

template <bool CLUSTER>
struct WordExchange {
    const WalkArgs& a;
    unsigned long long* inbox;  // CLUSTER: [side][parity][lattice][word] in this CTA's shared memory
    int cta;

    __device__ __forceinline__ int at(int side, int par, int l, int w) const {
        return ((side * 2 + par) * a.nlat + l) * a.xwords + w;
    }
    __device__ __forceinline__ unsigned long long poll(const unsigned long long* p) const {
        if (!CLUSTER) return ld_relaxed64(p);
        unsigned long long x;
        asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];"
                     : "=l"(x)
                     : "r"((uint32_t)__cvta_generic_to_shared(p))
                     : "memory");
        return x;
    }
    // Words w and w2 (both polled in one round trip; w2 = w: one word) of the
    // row above (side 0) or below (side 1) the band, tagged `tag`.
    __device__ __forceinline__ bool read(int side, int par, int l, int w, int w2, uint32_t tag,
                                         uint32_t (&out)[2]) const {
        const unsigned long long* row =
            CLUSTER ? inbox + at(side, par, l, 0) : slot(a, side == 0 ? cta - 1 : cta + 1, 1 - side, par, l, 0);
        unsigned spins = 0;
        uint64_t t0 = 0;
        for (;;) {
            const unsigned long long x = poll(row + w), y = w2 == w ? x : poll(row + w2);
            if ((uint32_t)(x >> 32) == tag && (uint32_t)(y >> 32) == tag) {
                out[0] = (uint32_t)x;
                out[1] = (uint32_t)y;
                return true;
            }
            if ((++spins & (CLUSTER ? 1023u : 63u)) == 0u && !wait_more(a, t0)) return false;
        }
    }
    // Word w of the band's first (side 0) or last (side 1) row for the CTA above / below.
    __device__ __forceinline__ void write(int side, int par, int l, int w, uint32_t tag, uint32_t v) const {
        const unsigned long long x = (unsigned long long)tag << 32 | v;
        if (CLUSTER) {
            // the upper CTA receives it as its row below, the lower one as its row above
            const uint32_t mine = (uint32_t)__cvta_generic_to_shared(inbox + at(1 - side, par, l, w));
            const uint32_t theirs = cluster_addr(mine, side == 0 ? cta - 1 : cta + 1);
            asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(theirs), "l"(x) : "memory");
        } else {
            st_relaxed64(slot(a, cta, side, par, l, 0) + w, x);
        }
    }
};

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

}  // namespace rtb
