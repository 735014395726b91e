// mesh_args.cu -- what every assembly needs of its mesh arguments: face areas and normals, and the check that
// indices are in range.
//
// Bound: launches and waits, not bytes.  As tensor operations the areas and normals of a mesh of a few hundred
// faces take 18 launches (two gathers of three vertices, two cross products, norms, divisions) and the range of
// one index array four launches and two waits; here one launch each and one wait.  A CFIE assembly with
// one excitation on 80 faces: 610 -> 171 us.
#include "common.cuh"
#include "face_order.cuh"

namespace mb {

namespace {

// areas [F] = |e0 x e1| / 2, normals [F, 3] = e0 x e1 / max(|e0 x e1|, 1e-12), e0 = v1 - v0, e1 = v2 - v1.  A face
// with an index outside the vertices gets zeros (the range check refuses it before anything is used).
template <typename T>
__global__ void __launch_bounds__(256) face_geometry_kernel(const T* __restrict__ verts, int64_t nv,
                                                            const int32_t* __restrict__ faces, int64_t nf,
                                                            T* __restrict__ areas, T* __restrict__ normals) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const int32_t i0 = faces[3 * f], i1 = faces[3 * f + 1], i2 = faces[3 * f + 2];
    V3<T> n = v3<T>(0, 0, 0);
    if (i0 >= 0 && i0 < nv && i1 >= 0 && i1 < nv && i2 >= 0 && i2 < nv) {
        const V3<T> v0 = load3(verts, i0), v1 = load3(verts, i1), v2 = load3(verts, i2);
        n = cross(v1 - v0, v2 - v1);
    }
    const T len = sqrt_t(dot(n, n));
    areas[f] = T(0.5) * len;
    if (!normals) return;
    const T den = len > T(1e-12) || len != len ? len : T(1e-12);
    normals[3 * f] = n.x / den;
    normals[3 * f + 1] = n.y / den;
    normals[3 * f + 2] = n.z / den;
}

__global__ void __launch_bounds__(256) index_range_kernel(const int32_t* __restrict__ idx, int64_t count,
                                                          int64_t limit, int32_t* __restrict__ outside) {
    bool bad = false;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = idx[i];
        bad |= v < 0 || v >= limit;
    }
    if (bad) *outside = 1;  // all writers store the same value
}

__global__ void __launch_bounds__(32 * kOrderSamples) face_order_kernel(const int32_t* __restrict__ ids, int64_t nf,
                                                                       FaceOrder* __restrict__ out) {
    const FaceOrder o = face_order(ids, nf);
    if (threadIdx.x == 0) *out = o;
}

}  // namespace

template <typename T>
int launch_face_geometry(const T* verts, int64_t nv, const int32_t* faces, int64_t nf, T* areas, T* normals,
                         cudaStream_t s) {
    if (nf <= 0) return MB_OK;
    face_geometry_kernel<T><<<(unsigned)((nf + 255) / 256), 256, 0, s>>>(verts, nv, faces, nf, areas, normals);
    return check_launch("face_geometry");
}
template int launch_face_geometry<float>(const float*, int64_t, const int32_t*, int64_t, float*, float*, cudaStream_t);
template int launch_face_geometry<double>(const double*, int64_t, const int32_t*, int64_t, double*, double*,
                                          cudaStream_t);

// *outside: 1 if an index is not in [0, limit), else 0 (waits for the stream).  work: 4 bytes on the device.  With order
// (count = 3 per face; work: 12 bytes) the order of the faces, too, by the same wait.
int index_range(const int32_t* idx, int64_t count, int64_t limit, int32_t* work, int32_t* outside, FaceOrder* order,
                cudaStream_t s) {
    *outside = 0;
    if (order) *order = FaceOrder{0, 0};
    if (count <= 0) return MB_OK;
    int32_t got[3] = {0, 0, 0};
    cudaError_t e = cudaMemsetAsync(work, 0, sizeof(int32_t), s);
    if (e == cudaSuccess) {
        // four indices a thread; at most two blocks an SM
        const int64_t blocks = (count + 1023) / 1024;
        index_range_kernel<<<(unsigned)(blocks < 2 * kSms ? blocks : 2 * kSms), 256, 0, s>>>(idx, count, limit, work);
        if (order)
            face_order_kernel<<<1, 32 * kOrderSamples, 0, s>>>(idx, count / 3, reinterpret_cast<FaceOrder*>(work + 1));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(got, work, sizeof(int32_t) * (order ? 3 : 1), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return set_error(MB_ERR_CUDA, "index range: %s", cudaGetErrorString(e));
    *outside = got[0];
    if (order) *order = FaceOrder{got[1], got[2]};
    return MB_OK;
}

}  // namespace mb
