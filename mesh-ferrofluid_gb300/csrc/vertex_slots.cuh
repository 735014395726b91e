// vertex_slots.cuh -- per-thread sums over a block's test faces by their distinct vertices, for
// matrices packed by vertex ([V, V] from face pairs).
//
// A packed entry [row vertex, column vertex] receives a term from every pair of faces around the
// two.  A reduction in global memory per term is bound by L2 (0.87 ms for 5120 x 5120 pairs of nine),
// rows of the matrix in shared memory by the compare-and-swap loop of a shared FP32 addition.  Here a
// block has kPairRows consecutive test faces and each thread one source face: the terms are added
// to the thread's own words of shared memory, one per distinct vertex of the test faces and corner of
// its source face, and leave by one global reduction per word.  Consecutive faces of a mesh share
// vertices: 16 faces of the sphere have 15 to 17 distinct ones of 48 corners.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace mb {

// Measured for the packed Laplace operators at 5120 faces (three operators, us): 16 faces and 20 vertices 1448
// (5 blocks per SM), 32 and 40 1695 (3 blocks), 24 and 32 1757, 8 and 12 1585.
constexpr int kPairRows = 16;
constexpr int kPairVerts = 20;  // distinct vertices with a place; terms of the rest are reduced directly
constexpr int kPairThreads = 128;
constexpr int kPairSumBytes = 3 * kPairVerts * kPairThreads * (int)sizeof(float);

// Test faces per block (host) for `rows` test faces and gx blocks of source faces.  An SM's time is that of its share
// of the blocks, each worth its faces and about 0.6 more for its start; fewer than five blocks an SM leave it waiting
// (676 faces: 8 a block 35 us, 5 27.5, 2 28.7).  Among those within 1 % the most faces: fewer reductions.
inline int pair_rows(int64_t rows, int64_t gx) {
    int best = 1;
    double cost = 0.0;
    for (int per = 1; per <= kPairRows; ++per) {
        const int64_t blocks = (rows + per - 1) / per * gx;
        if (per > 1 && blocks < 5 * kSms) break;
        const double c = (double)((blocks + kSms - 1) / kSms) * (per + 0.6);
        if (per == 1 || c <= 1.01 * cost) {
            best = per;
            cost = per == 1 || c < cost ? c : cost;
        }
    }
    return best;
}

struct VertexSlots {
    int id[3 * kPairRows];        // vertex of each corner
    int first[3 * kPairRows];     // 1 at a vertex's first corner
    uint8_t slot[4 * kPairRows];  // the corners' slots, 4 bytes per face
    int vert[kPairVerts], n;
};

// Fills s.slot, s.vert and s.n from s.id (np faces); all threads of the block call it, with s.id written
// before.  At most 48 corners: the searches are short.
__device__ __forceinline__ void find_slots(VertexSlots& s, int np) {
    const int t = threadIdx.x, n = 3 * np;
    if (np == 1) {  // nothing to share: its terms are reduced directly
        if (t < 3) s.slot[t] = 255;
        if (t == 0) s.n = 0;
        __syncthreads();
        return;
    }
    __syncthreads();
    int first = 0;
    if (t < n) {
        while (s.id[first] != s.id[t]) ++first;
        s.first[t] = first == t;
    }
    __syncthreads();
    if (t < n) {
        int rank = 0;
        for (int j = 0; j < first; ++j) rank += s.first[j];
        s.slot[4 * (t / 3) + t % 3] = (uint8_t)rank;
        if (rank < kPairVerts) s.vert[rank] = s.id[t];
    }
    if (t == 0) {
        int c = 0;
        for (int j = 0; j < n; ++j) c += s.first[j];
        s.n = c < kPairVerts ? c : kPairVerts;
    }
    __syncthreads();
}

// The thread's words: [slot][corner b][thread]
__device__ __forceinline__ void clear_sums(float* sums, int n) {
    for (int u = 0; u < 3 * n; ++u) sums[u * kPairThreads + threadIdx.x] = 0.f;
}

// acc[3 a + b] of test face i and the thread's source face with vertices col
__device__ __forceinline__ void add_entries(const VertexSlots& s, int i, const float acc[9], const int32_t* col, int64_t nv,
                                            float* sums, float* __restrict__ packed) {
    const uint32_t slots = *reinterpret_cast<const uint32_t*>(s.slot + 4 * i);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int u = (slots >> (8 * a)) & 255;
        if (u < kPairVerts) {
            float* t = sums + 3 * u * kPairThreads + threadIdx.x;
#pragma unroll
            for (int b = 0; b < 3; ++b) t[b * kPairThreads] += acc[3 * a + b];
        } else {
            float* dst = packed + (int64_t)s.id[3 * i + a] * nv;
#pragma unroll
            for (int b = 0; b < 3; ++b) atomicAdd(dst + col[b], acc[3 * a + b]);
        }
    }
}

__device__ __forceinline__ void flush_sums(const VertexSlots& s, const int32_t* col, int64_t nv, const float* sums,
                                           float* __restrict__ packed) {
    for (int u = 0; u < s.n; ++u) {
        float* dst = packed + (int64_t)s.vert[u] * nv;
#pragma unroll
        for (int b = 0; b < 3; ++b) atomicAdd(dst + col[b], sums[(3 * u + b) * kPairThreads + threadIdx.x]);
    }
}

}  // namespace mb
