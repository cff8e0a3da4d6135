// rt_domain.cuh -- vertices and edges of a domino or lozenge domain on the
// device, as the host builders define them (rt_host.cpp).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace rtb {

__device__ __forceinline__ int dface(const int32_t* __restrict__ d, int m, int i, int j) {
    return (i >= 0 && j >= 0 && i < m && j < m) ? d[(int64_t)i * m + j] : 0;
}
__device__ __forceinline__ int lface(const int32_t* __restrict__ d, int m, int r, int c) {
    return (r >= 0 && c >= 0 && r < m && c < 2 * m) ? d[(int64_t)r * 2 * m + c] : 0;
}

// Vertex kind (DomainToVertices, DominoTiler.cpp:479-506,
// LozengeTiler.cpp:405-430): 0 outside, 1 interior, 2 boundary.  Dominoes: m x
// m faces; lozenges: m rows of 2m triangles; vertices (m + 1) x (m + 1).
template <bool DOM>
__device__ __forceinline__ int vertex_kind(const int32_t* __restrict__ d, int m, int i, int j) {
    if (DOM) {
        if (i == 0 || j == 0 || i == m || j == m) {
            const int i0 = i - (i == m), i1 = i - 1 + (i == 0), j0 = j - (j == m), j1 = j - 1 + (j == 0);
            return (dface(d, m, i0, j0) || dface(d, m, i1, j0) || dface(d, m, i0, j1) || dface(d, m, i1, j1)) ? 2 : 0;
        }
        const int s = (dface(d, m, i - 1, j - 1) != 0) + (dface(d, m, i - 1, j) != 0) + (dface(d, m, i, j - 1) != 0) +
                      (dface(d, m, i, j) != 0);
        return s == 4 ? 1 : s > 0 ? 2 : 0;
    }
    if (i < 1 || j < 1 || i >= m || j >= m) return 0;
    const int s = (lface(d, m, i, 2 * j) != 0) + (lface(d, m, i, 2 * j - 1) != 0) + (lface(d, m, i, 2 * j - 2) != 0) +
                  (lface(d, m, i - 1, 2 * j) != 0) + (lface(d, m, i - 1, 2 * j + 1) != 0) +
                  (lface(d, m, i - 1, 2 * j - 1) != 0);
    return s == 6 ? 1 : s > 0 ? 2 : 0;
}

// Bit nb: the edge of vertex (i, j) in direction nb touches a face of the
// domain and ends at a vertex of it.  Directions: dominoes (+1,0), (-1,0),
// (0,+1), (0,-1); lozenges (0,+1), (-1,+1), (-1,0), (0,-1), (+1,-1), (+1,0).
template <bool DOM>
__device__ __forceinline__ uint32_t edge_bits(const int32_t* __restrict__ d, int m, int i, int j) {
    if (DOM) {
        // the four faces around the vertex; an edge lies between two of them
        const bool nw = dface(d, m, i - 1, j - 1), ne = dface(d, m, i - 1, j), sw = dface(d, m, i, j - 1), se = dface(d, m, i, j);
        return (sw || se ? 1u : 0u) | (nw || ne ? 2u : 0u) | (ne || se ? 4u : 0u) | (nw || sw ? 8u : 0u);
    }
    // the six triangles around the vertex in turn, from the one below (0,+1)'s edge
    const bool t0 = lface(d, m, i, 2 * j), t1 = lface(d, m, i - 1, 2 * j + 1), t2 = lface(d, m, i - 1, 2 * j),
               t3 = lface(d, m, i - 1, 2 * j - 1), t4 = lface(d, m, i, 2 * j - 2), t5 = lface(d, m, i, 2 * j - 1);
    uint32_t e = (t0 || t1 ? 1u : 0u) | (t1 || t2 ? 2u : 0u) | (t2 || t3 ? 4u : 0u) | (t3 || t4 ? 8u : 0u) |
                 (t4 || t5 ? 16u : 0u) | (t5 || t0 ? 32u : 0u);
    // the outermost vertices are outside every domain
    if (j + 1 >= m) e &= ~3u;
    if (i - 1 < 1) e &= ~6u;
    if (j - 1 < 1) e &= ~24u;
    if (i + 1 >= m) e &= ~48u;
    return e;
}

}  // namespace rtb
