// face_order.cuh -- whether consecutive faces of a mesh share their vertices (or edges).
//
// Kernels that sum a block's terms by its faces' distinct vertices or edges (vertex_slots.cuh, sym_pairs_kernel) gain from
// faces listed neighbour by neighbour, as subdivision, strips and most files give them, and lose without: 16
// faces in any order have 48 vertices, and every term is a reduction of its own. The order is
// the caller's, so it is looked at before the kernel is chosen: on the device, from 16 samples spread over the list, by one
// small block (3 us; by every block of the packing instead it cost 18 % of its time).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mb {

constexpr int kOrderSamples = 16;

// How many different values a warp's lanes hold
__device__ __forceinline__ int distinct_lanes(int v) {
    const unsigned same = __match_any_sync(0xffffffffu, v);
    return __popc(__ballot_sync(0xffffffffu, (int)(threadIdx.x & 31) == __ffs(same) - 1));
}

struct FaceOrder {
    int ids;      // different ids of ten consecutive faces' 30, mean of the samples: 12 to 14 vertices along a strip, 14 on a
                  // subdivided sphere, 30 in any order; 21 to 23 edges, 30 in any order
    int sectors;  // of 32 consecutive faces, groups of eight ids (32 bytes of a float row) among the first corners, plus
                  // the second, plus the third: 12 along a strip of neighbouring ids, 19 to 37 on a subdivided sphere, 53 on strips
                  // across the ids, 90 in any order
};

// (all threads of a block of whole warps; ids: 3 per face)
__device__ __forceinline__ FaceOrder face_order(const int32_t* __restrict__ ids, int64_t nf) {
    __shared__ int s_ids, s_sectors;
    if (threadIdx.x == 0) s_ids = s_sectors = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    int a = 0, b = 0;
    for (int s = threadIdx.x >> 5; s < kOrderSamples; s += blockDim.x >> 5) {
        const int64_t f10 = (nf > 10 ? nf - 10 : 0) * s / (kOrderSamples - 1);
        const int64_t f32 = (nf > 32 ? nf - 32 : 0) * s / (kOrderSamples - 1);
        const int64_t f = min(f32 + lane, nf - 1);
        a += distinct_lanes(__ldg(ids + min(3 * f10 + min(lane, 29), 3 * nf - 1)));
        for (int c = 0; c < 3; ++c) b += distinct_lanes(__ldg(ids + 3 * f + c) >> 3);
    }
    if (lane == 0) {
        atomicAdd(&s_ids, a);
        atomicAdd(&s_sectors, b);
    }
    __syncthreads();
    return FaceOrder{s_ids / kOrderSamples, s_sectors / kOrderSamples};
}

}  // namespace mb
