// laplace_sym.cu -- 3D Laplace boundary operators with the symmetric 7-point rule and
// closed-form singular integrals: an accurate mode next to the reference's quadrature
// (laplace.cu), needed by the Neumann / mixed problems whose hypersingular operator the
// reference never implemented, and by the single-layer collocation system.
//
// Galerkin (P0 / P1), for every ordered face pair (fy, fx) -- fy the "y" face whose normal
// the double layer uses, as in the reference (integrations_3d.py:367, 412-415):
//     out[fy, fx, a, b] = int_{fy} int_{fx} phi_a(y) phi_b(x) k(x, y) dS_x dS_y
//     k = 1/(4 pi R)  (single layer)   or   n_y.(x - y)/(4 pi R^3)  (double layer).
// Separated pairs (no shared vertex): 7 x 7 points, FP32 or FP64 as the output type, the
// pair's coordinates moved to the first vertex of fy.  Pairs sharing a vertex (self, edge-
// and vertex-adjacent): 7 points on fx and the inner integral over fy in closed form, in
// FP64 (closed_form.cuh).  P1 inner integrals use that a hat function is affine:
//     phi_a(y) = phi_a~(x) + grad phi_a . (y - x),   grad phi_a = n x (P_{a+2} - P_{a+1}) / (2A),
// so int phi_a / R = phi_a~(x) I0 + grad phi_a . I1 and, with d = n.(x - P0),
//     int phi_a n.(x - y)/R^3 = -phi_a~(x) Omega + d grad phi_a . J.
//
// Collocation (P0 single layer): A[i, j] = int_{T_j} 1/(4 pi |c_i - y|) dS_y at the
// centroid c_i of face i, 7 points (FP32 / FP64) or closed form (FP64) when i and j share
// a vertex.  Each thread keeps one source triangle and sweeps 16 collocation rows.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "closed_form.cuh"
#include "common.cuh"
#include "face_order.cuh"
#include "packed.cuh"
#include "vertex_slots.cuh"

namespace mb {

constexpr int kSymThreads = 128;

__device__ __forceinline__ float rcp_sqrt(float x) { return rsqrtf(x); }
// FP64 1/sqrt(x): the FP32 estimate refined by two Newton steps r <- r (3 - x r^2) / 2
// (quadratic convergence: ~2^-23 -> 2^-46 -> below double rounding).
__device__ __forceinline__ double rcp_sqrt(double x) {
    double r = (double)rsqrtf((float)x);
    r = r * (1.5 - 0.5 * x * r * r);
    r = r * (1.5 - 0.5 * x * r * r);
    return r;
}


__device__ __forceinline__ bool share_vertex(const int32_t* f, int64_t p, int64_t q) {
    const int32_t a0 = __ldg(f + 3 * p), a1 = __ldg(f + 3 * p + 1), a2 = __ldg(f + 3 * p + 2);
    const int32_t b0 = __ldg(f + 3 * q), b1 = __ldg(f + 3 * q + 1), b2 = __ldg(f + 3 * q + 2);
    return (a0 == b0) | (a0 == b1) | (a0 == b2) | (a1 == b0) | (a1 == b1) | (a1 == b2) | (a2 == b0) |
           (a2 == b1) | (a2 == b2);
}

// The 7 x 7-point integral of a separated pair: fy's rule points (shifted to fy's first
// vertex) and weights w_j A_y in s_y, the barycentric rule in s_rule, fx's corners X0..X2 in
// the same shifted frame; acc[3 a + b] (P1) or acc[0] (P0), without the 1 / (4 pi).
template <typename T, int LAYER, int NPHI>
__device__ __forceinline__ void sym_far_pair(const T (*s_rule)[4], const T (*s_y)[4], const V3<T>& ny,
                                             const V3<T>& X0, const V3<T>& X1, const V3<T>& X2, T acc[9]) {
    const V3<T> nx = cross(X1 - X0, X2 - X1);
    const T ax = T(0.5) * sqrt_t(dot(nx, nx));
#pragma unroll 1
    for (int i = 0; i < 7; ++i) {
        const V3<T> x = s_rule[i][0] * X0 + s_rule[i][1] * X1 + s_rule[i][2] * X2;
        T s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            const V3<T> d = x - v3<T>(s_y[j][0], s_y[j][1], s_y[j][2]);
            const T ri = rcp_sqrt(dot(d, d));
            T g = ri * s_y[j][3];
            if constexpr (LAYER == 2) g *= ri * ri;
            if constexpr (NPHI == 3) {
                s0 += g * s_rule[j][0];
                s1 += g * s_rule[j][1];
                s2 += g * s_rule[j][2];
            } else {
                s0 += g;
            }
        }
        if constexpr (LAYER == 2) {
            const T dn = dot(x, ny);  // n_y.(x - y_j): the shifted y_j lie in the plane through 0
            s0 *= dn;
            s1 *= dn;
            s2 *= dn;
        }
        const T wx = s_rule[i][3] * ax;
        if constexpr (NPHI == 3) {
            const T sa[3] = {s0, s1, s2};
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) acc[3 * a + b] += sa[a] * (wx * s_rule[i][b]);
        } else {
            acc[0] += s0 * wx;
        }
    }
}

// Two separated pairs (fy, fxa) and (fy, fxb) at once in packed f32x2 arithmetic (lane .x
// the first source face, .y the second): the same sums as sym_far_pair with half the FP32
// instructions.  X0..X2 hold both faces' shifted corners per coordinate; acc as in
// sym_far_pair, packed.
template <int LAYER, int NPHI>
__device__ __forceinline__ void sym_far_pair2(const float4 (*s_r4)[2], const float4 (*s_y4)[2], const float3& ny,
                                              const float2 X0[3], const float2 X1[3], const float2 X2[3],
                                              float2 acc[9]) {
    // s_r4[j] = {(r0, r0, r1, r1), (r2, r2, w, w)}, s_y4[j] = {(y.x, y.x, y.y, y.y),
    // (y.z, y.z, wA, wA)}: every value already duplicated, so one 16-byte shared load yields two
    // packed operands and no register moves are needed to broadcast them
    float2 e1[3], e2[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        e1[c] = sub2(X1[c], X0[c]);
        e2[c] = sub2(X2[c], X1[c]);
    }
    const float2 nx0 = fma2(e1[1], e2[2], mul2(bc(-1.f), mul2(e1[2], e2[1])));
    const float2 nx1 = fma2(e1[2], e2[0], mul2(bc(-1.f), mul2(e1[0], e2[2])));
    const float2 nx2 = fma2(e1[0], e2[1], mul2(bc(-1.f), mul2(e1[1], e2[0])));
    const float2 n2 = fma2(nx0, nx0, fma2(nx1, nx1, mul2(nx2, nx2)));
    const float2 ax = make_float2(0.5f * sqrtf(n2.x), 0.5f * sqrtf(n2.y));
#pragma unroll 1
    for (int i = 0; i < 7; ++i) {
        // re-read the tables every outer point instead of holding all 28 of them in registers
        asm volatile("" ::: "memory");
        const float4 ra = s_r4[i][0], rb = s_r4[i][1];
        const float2 r0 = make_float2(ra.x, ra.y), r1 = make_float2(ra.z, ra.w), r2 = make_float2(rb.x, rb.y);
        float2 x[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c] = fma2(r0, X0[c], fma2(r1, X1[c], mul2(r2, X2[c])));
        float2 s0 = bc(0.f), s1 = bc(0.f), s2 = bc(0.f);
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            const float4 ya = s_y4[j][0], yb = s_y4[j][1];
            const float2 dx = sub2(x[0], make_float2(ya.x, ya.y));
            const float2 dy = sub2(x[1], make_float2(ya.z, ya.w));
            const float2 dz = sub2(x[2], make_float2(yb.x, yb.y));
            const float2 d2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
            const float2 ri = make_float2(rsqrtf(d2.x), rsqrtf(d2.y));
            float2 g = mul2(ri, make_float2(yb.z, yb.w));
            if constexpr (LAYER == 2) g = mul2(g, mul2(ri, ri));
            if constexpr (NPHI == 3) {
                const float4 qa = s_r4[j][0], qb = s_r4[j][1];
                s0 = fma2(g, make_float2(qa.x, qa.y), s0);
                s1 = fma2(g, make_float2(qa.z, qa.w), s1);
                s2 = fma2(g, make_float2(qb.x, qb.y), s2);
            } else {
                s0 = add2(s0, g);
            }
        }
        if constexpr (LAYER == 2) {
            const float2 dn = fma2(x[0], bc(ny.x), fma2(x[1], bc(ny.y), mul2(x[2], bc(ny.z))));
            s0 = mul2(s0, dn);
            s1 = mul2(s1, dn);
            s2 = mul2(s2, dn);
        }
        const float2 wx = mul2(make_float2(rb.z, rb.w), ax);
        if constexpr (NPHI == 3) {
            const float2 sa[3] = {s0, s1, s2};
            const float2 rr[3] = {r0, r1, r2};
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const float2 wb = mul2(wx, rr[b]);
#pragma unroll
                for (int a = 0; a < 3; ++a) acc[3 * a + b] = fma2(sa[a], wb, acc[3 * a + b]);
            }
        } else {
            acc[0] = fma2(s0, wx, acc[0]);
        }
    }
}

// Block set-up shared by the panel and packed kernels: the 7-point rule, fy's shifted rule
// points with weights, and fy's unit normal.
template <typename T>
__device__ __forceinline__ void sym_source_setup(const V3<T>& Y1, const V3<T>& Y2, T (*s_rule)[4], T (*s_y)[4],
                                                 T* s_n) {
    if (threadIdx.x < 7) {
        const int j = threadIdx.x;
        s_rule[j][0] = (T)c_d7[j][0];
        s_rule[j][1] = (T)c_d7[j][1];
        s_rule[j][2] = (T)c_d7[j][2];
        s_rule[j][3] = (T)c_d7[j][3];
        const V3<T> nr = cross(Y1, Y2 - Y1);
        const T ay = T(0.5) * sqrt_t(dot(nr, nr));
        const V3<T> y = (T)c_d7[j][1] * Y1 + (T)c_d7[j][2] * Y2;
        s_y[j][0] = y.x;
        s_y[j][1] = y.y;
        s_y[j][2] = y.z;
        s_y[j][3] = (T)c_d7[j][3] * ay;
        if (j == 0) {
            const T inv = rsqrt_t(dot(nr, nr));
            s_n[0] = nr.x * inv;
            s_n[1] = nr.y * inv;
            s_n[2] = nr.z * inv;
        }
    }
}

template <typename T, int LAYER, int NPHI>
__global__ void __launch_bounds__(kSymThreads)
    lap_sym_far_kernel(const T* __restrict__ verts, const int32_t* __restrict__ faces, int64_t nf,
                       int64_t row_begin, int64_t col_blocks, T* __restrict__ out) {
    __shared__ T s_rule[7][4];   // barycentric coordinates and weight of the 7-point rule
    __shared__ T s_y[7][4];      // source points (shifted) and weights w_j A_y
    __shared__ T s_n[3];
    __shared__ __align__(16) T s_out[kSymThreads * 9];
    const int64_t row_local = (int64_t)blockIdx.x / col_blocks;
    const int64_t fy = row_begin + row_local;
    const int64_t col0 = ((int64_t)blockIdx.x % col_blocks) * kSymThreads;
    const int64_t fx = col0 + threadIdx.x;
    const V3<T> o = load3(verts, __ldg(faces + 3 * fy));
    const V3<T> Y1 = load3(verts, __ldg(faces + 3 * fy + 1)) - o;
    const V3<T> Y2 = load3(verts, __ldg(faces + 3 * fy + 2)) - o;
    sym_source_setup(Y1, Y2, s_rule, s_y, s_n);
    __syncthreads();
    constexpr int nn = NPHI * NPHI;
    T acc[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) acc[c] = 0;
    if (fx < nf && !share_vertex(faces, fy, fx)) {
        const V3<T> X0 = load3(verts, __ldg(faces + 3 * fx)) - o;
        const V3<T> X1 = load3(verts, __ldg(faces + 3 * fx + 1)) - o;
        const V3<T> X2 = load3(verts, __ldg(faces + 3 * fx + 2)) - o;
        sym_far_pair<T, LAYER, NPHI>(s_rule, s_y, v3<T>(s_n[0], s_n[1], s_n[2]), X0, X1, X2, acc);
#pragma unroll
        for (int c = 0; c < 9; ++c) acc[c] *= T(kInv4Pi);
    }
#pragma unroll
    for (int c = 0; c < nn; ++c) s_out[threadIdx.x * nn + c] = acc[c];
    __syncthreads();
    const int64_t valid = (nf - col0) < kSymThreads ? (nf - col0) : kSymThreads;
    const int64_t base = (row_local * nf + col0) * nn;
    const int64_t n_out = valid * nn;
    for (int64_t c = threadIdx.x; c < n_out; c += kSymThreads) out[base + c] = s_out[c];
}

// Surface curls (p_{a+1} - p_{a+2}) / (2 A) of the P1 hat functions of a triangle
// (translation invariant, so any common shift of the corners gives the same curls).
template <typename T>
__device__ __forceinline__ void tri_curls(const V3<T>& p0, const V3<T>& p1, const V3<T>& p2, V3<T> c[3]) {
    const V3<T> nr = cross(p1 - p0, p2 - p1);
    const T inv2a = T(1) / sqrt_t(dot(nr, nr));
    c[0] = inv2a * (p1 - p2);
    c[1] = inv2a * (p2 - p0);
    c[2] = inv2a * (p0 - p1);
}

// Ten consecutive faces with more vertices than this (face_order.cuh) are not listed neighbour by neighbour.  5120
// faces, us, operators 1, 2, 3, a block per face / groups of faces: 14 vertices 1026 / 494, 1064 / 573, 801 / 429; 17: 1030 / 650,
// 1068 / 675, 806 / 626; 23: 1036 / 893, 1076 / 902, 818 / 877; 30: 1036 / 1171, 1074 / 1173, 815 / 1158.
constexpr int kOrderIds = 20;

__global__ void __launch_bounds__(32 * kOrderSamples) lap_face_order_kernel(const int32_t* __restrict__ faces, int64_t nf,
                                                                           FaceOrder* __restrict__ out) {
    const FaceOrder o = face_order(faces, nf);
    if (threadIdx.x == 0) *out = o;
}

// Packed operators [V, V] without the [F, F, 3, 3] panels: OP 1 single layer, 2 double layer
// (P1 x P1), 3 hypersingular (Maue: curl phi_a(fy) . curl phi_b(fx) times the P0 single
// layer).  One block per test face fy sweeps every source face fx, accumulates the three
// packed rows faces[fy, a] in shared memory (3 V values) and adds them to `packed` at the
// end.  Pairs sharing a vertex are skipped here and added by lap_sym_near_kernel.  FP64, and FP32 meshes of a few
// hundred faces (launch_sym_pairs).
template <typename T, int OP>
__global__ void __launch_bounds__(kSymThreads, sizeof(T) == 4 ? (OP == 3 ? 6 : 4) : 1)
    lap_sym_tight_kernel(const T* __restrict__ verts, const int32_t* __restrict__ faces, int64_t nf, int64_t nv,
                         int64_t row_begin, const FaceOrder* __restrict__ order, T* __restrict__ packed) {
    if constexpr (sizeof(T) == 4)
        if (order && order->ids <= kOrderIds) return;  // lap_sym_pairs_kernel's
    constexpr int LAYER = OP == 2 ? 2 : 1;
    constexpr int NPHI = OP == 3 ? 1 : 3;
    __shared__ T s_rule[7][4];
    __shared__ T s_y[7][4];
    __shared__ T s_n[3];
    __shared__ float4 s_r4[7][2];  // the same tables with every value duplicated (float path)
    __shared__ float4 s_y4[7][2];
    extern __shared__ __align__(16) unsigned char tight_smem[];
    T* rows = reinterpret_cast<T*>(tight_smem);
    const int64_t fy = row_begin + blockIdx.x;
    const V3<T> o = load3(verts, __ldg(faces + 3 * fy));
    const V3<T> Y1 = load3(verts, __ldg(faces + 3 * fy + 1)) - o;
    const V3<T> Y2 = load3(verts, __ldg(faces + 3 * fy + 2)) - o;
    sym_source_setup(Y1, Y2, s_rule, s_y, s_n);
    for (int64_t j = threadIdx.x; j < 3 * nv; j += blockDim.x) rows[j] = T(0);
    V3<T> cy[3];
    if constexpr (OP == 3) tri_curls(v3<T>(0, 0, 0), Y1, Y2, cy);
    __syncthreads();
    if (threadIdx.x < 7) {
        const int j = threadIdx.x;
        const float r0 = (float)s_rule[j][0], r1 = (float)s_rule[j][1], r2 = (float)s_rule[j][2];
        const float rw = (float)s_rule[j][3];
        s_r4[j][0] = make_float4(r0, r0, r1, r1);
        s_r4[j][1] = make_float4(r2, r2, rw, rw);
        const float y0 = (float)s_y[j][0], y1 = (float)s_y[j][1], y2 = (float)s_y[j][2], yw = (float)s_y[j][3];
        s_y4[j][0] = make_float4(y0, y0, y1, y1);
        s_y4[j][1] = make_float4(y2, y2, yw, yw);
    }
    __syncthreads();
    const V3<T> ny = v3<T>(s_n[0], s_n[1], s_n[2]);
    // each thread sweeps its own strip of consecutive source faces: neighbouring faces share
    // vertices, and lanes of a warp working on neighbours would collide in the shared-memory
    // accumulators (same-address atomics serialise)
    const int64_t strip = (nf + blockDim.x - 1) / blockDim.x;
    const int64_t strip0 = (int64_t)threadIdx.x * strip;
    const int64_t strip1 = strip0 + strip < nf ? strip0 + strip : nf;
    if constexpr (sizeof(T) == 4 && OP != 3) {
        // two source faces per thread and iteration (fxa, fxa + 1), packed arithmetic
        // (the P0 sums of OP 3 are light enough that occupancy matters more)
        const float3 nyf = make_float3(ny.x, ny.y, ny.z);
#pragma unroll 1
        for (int64_t k = 0; k < strip; k += 2) {
            const int64_t fxa = strip0 + k;
            if (fxa >= strip1) break;
            const int64_t fxb_raw = fxa + 1;
            const bool has_b = fxb_raw < strip1;
            const int64_t fxb = has_b ? fxb_raw : fxa;
            const bool use_a = !share_vertex(faces, fy, fxa);
            const bool use_b = has_b && !share_vertex(faces, fy, fxb);
            if (!use_a && !use_b) continue;
            const int32_t va[3] = {__ldg(faces + 3 * fxa), __ldg(faces + 3 * fxa + 1), __ldg(faces + 3 * fxa + 2)};
            const int32_t vb[3] = {__ldg(faces + 3 * fxb), __ldg(faces + 3 * fxb + 1), __ldg(faces + 3 * fxb + 2)};
            float2 X[3][3];  // corner, coordinate
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                const V3<T> pa = load3(verts, va[v]) - o;
                const V3<T> pb = load3(verts, vb[v]) - o;
                X[v][0] = make_float2(pa.x, pb.x);
                X[v][1] = make_float2(pa.y, pb.y);
                X[v][2] = make_float2(pa.z, pb.z);
            }
            float2 acc[9];
#pragma unroll
            for (int c = 0; c < 9; ++c) acc[c] = bc(0.f);
            sym_far_pair2<LAYER, NPHI>(s_r4, s_y4, nyf, X[0], X[1], X[2], acc);
            {
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        if (use_a) atomicAdd(rows + a * nv + va[b], acc[3 * a + b].x * T(kInv4Pi));
                        if (use_b) atomicAdd(rows + a * nv + vb[b], acc[3 * a + b].y * T(kInv4Pi));
                    }
            }
        }
    } else {
#pragma unroll 1
        for (int64_t fx = strip0; fx < strip1; ++fx) {
            if (share_vertex(faces, fy, fx)) continue;
            const int32_t vx[3] = {__ldg(faces + 3 * fx), __ldg(faces + 3 * fx + 1), __ldg(faces + 3 * fx + 2)};
            const V3<T> X0 = load3(verts, vx[0]) - o;
            const V3<T> X1 = load3(verts, vx[1]) - o;
            const V3<T> X2 = load3(verts, vx[2]) - o;
            T acc[9];
#pragma unroll
            for (int c = 0; c < 9; ++c) acc[c] = 0;
            sym_far_pair<T, LAYER, NPHI>(s_rule, s_y, ny, X0, X1, X2, acc);
            if constexpr (OP == 3) {
                V3<T> cx[3];
                tri_curls(X0, X1, X2, cx);
                const T w = acc[0] * T(kInv4Pi);
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) atomicAdd(rows + a * nv + vx[b], dot(cy[a], cx[b]) * w);
            } else {
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) atomicAdd(rows + a * nv + vx[b], acc[3 * a + b] * T(kInv4Pi));
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        T* dst = packed + (int64_t)__ldg(faces + 3 * fy + a) * nv;
        for (int64_t j = threadIdx.x; j < nv; j += blockDim.x) atomicAdd(dst + j, rows[a * nv + j]);
    }
}

// FP32 (which meshes: launch_sym_pairs): a thread keeps one source face fx and meets the block's test faces.  The 7-point rule is its
// centroid and two orbits s A_a of the corners A_a relative to the centroid (s = 1 - 3 q), so with
// D the difference of the centroids
//     R^2 = |D|^2 + 2 s D.A_a - 2 s' D.B_b + s^2 |A_a|^2 + s'^2 |B_b|^2 - 2 s s' A_a.B_b
// comes from 15 dot products of the pair at three operations per evaluation instead of six, and the
// hat functions at the points are (1 - s)/3 + s [corner], so two sums per evaluation (over all
// corners of fy, and corner by corner) hold all nine entries.  n_y.(x - y) depends on x alone.
// Lanes of a packed register are the two orbits of fx.  The sums are over k(R) - k(R_c): the
// constant's integrals are known, and the rounding is that of the differences.  Entries are added by
// vertex_slots.cuh.  Bound: SFU (49 reciprocal roots per pair, 0.28 ms at 5120 faces) and issue
// slots.  Measured (GB300, 5120 faces of a subdivided sphere, the pairs sharing a vertex included): single / double /
// hypersingular 1028 / 1065 / 805 -> 512 / 586 / 442 us.
// Pairs whose centroids are closer than twice the sum of the corner distances, where the
// expansion of R^2 would cancel, are listed and evaluated from coordinate differences.
constexpr int kRowRec = 28;  // floats per staged test face

struct FaceLocal {
    V3<float> v0, off, A[3];  // first corner; centroid - v0; corners - centroid
    float area, rho;
    int32_t id[3];
};

__device__ __forceinline__ FaceLocal face_local(const float* __restrict__ verts, const int32_t* __restrict__ faces,
                                                int64_t f) {
    FaceLocal o;
#pragma unroll
    for (int a = 0; a < 3; ++a) o.id[a] = __ldg(faces + 3 * f + a);
    o.v0 = load3(verts, o.id[0]);
    const V3<float> e1 = load3(verts, o.id[1]) - o.v0, e2 = load3(verts, o.id[2]) - o.v0;
    o.off = (1.f / 3.f) * (e1 + e2);
    o.A[0] = -1.f * o.off;
    o.A[1] = e1 - o.off;
    o.A[2] = e2 - o.off;
    const V3<float> n = cross(e1, e2);
    o.area = 0.5f * sqrtf(dot(n, n));
    o.rho = sqrtf(fmaxf(dot(o.A[0], o.A[0]), fmaxf(dot(o.A[1], o.A[1]), dot(o.A[2], o.A[2]))));
    return o;
}

// a close separated pair: coordinate differences, as lap_sym_far_kernel
template <int OP>
__device__ void close_pair_entries(const float* __restrict__ verts, const int32_t* __restrict__ faces, int64_t fy,
                                   int64_t fx, int64_t nv, float* __restrict__ packed) {
    constexpr int LAYER = OP == 2 ? 2 : 1, NPHI = OP == 3 ? 1 : 3;
    const int32_t row[3] = {faces[3 * fy], faces[3 * fy + 1], faces[3 * fy + 2]};
    const int32_t col[3] = {faces[3 * fx], faces[3 * fx + 1], faces[3 * fx + 2]};
    const V3<float> o = load3(verts, row[0]);
    const V3<float> Y1 = load3(verts, row[1]) - o, Y2 = load3(verts, row[2]) - o;
    const V3<float> X0 = load3(verts, col[0]) - o, X1 = load3(verts, col[1]) - o, X2 = load3(verts, col[2]) - o;
    float rule[7][4], y[7][4];
    const V3<float> n = cross(Y1, Y2 - Y1);
    const float l = sqrtf(dot(n, n));
#pragma unroll
    for (int j = 0; j < 7; ++j) {
#pragma unroll
        for (int c = 0; c < 4; ++c) rule[j][c] = (float)c_d7[j][c];
        const V3<float> p = rule[j][1] * Y1 + rule[j][2] * Y2;
        y[j][0] = p.x;
        y[j][1] = p.y;
        y[j][2] = p.z;
        y[j][3] = rule[j][3] * 0.5f * l;
    }
    float acc[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    sym_far_pair<float, LAYER, NPHI>(rule, y, (1.f / l) * n, X0, X1, X2, acc);
    if constexpr (OP == 3) {
        V3<float> cy[3], cx[3];
        tri_curls(v3<float>(0.f, 0.f, 0.f), Y1, Y2, cy);
        tri_curls(X0, X1, X2, cx);
        const float w = acc[0];
#pragma unroll
        for (int c = 0; c < 9; ++c) acc[c] = dot(cy[c / 3], cx[c % 3]) * w;
    }
#pragma unroll
    for (int c = 0; c < 9; ++c) atomicAdd(packed + (int64_t)row[c / 3] * nv + col[c % 3], acc[c] * float(kInv4Pi));
}

template <int OP>
__global__ void __launch_bounds__(kPairThreads, 5)
    lap_sym_pairs_kernel(const float* __restrict__ verts, const int32_t* __restrict__ faces, int64_t nf, int64_t nv,
                         int64_t row_begin, int64_t row_end, int rows_per_block, const FaceOrder* __restrict__ order,
                         float* __restrict__ packed) {
    if (order && order->ids > kOrderIds) return;  // lap_sym_tight_kernel's
    constexpr float s1 = (float)(1.0 - 3.0 * 0.10128650732345634), s2 = (float)(1.0 - 3.0 * 0.47014206410511509);
    constexpr float w0 = 0.225f, w1 = 0.12593918054482715f, w2 = 0.13239415278850619f;
    constexpr float a1 = (1.f - s1) / 3.f, a2 = (1.f - s2) / 3.f;
    __shared__ __align__(16) float s_rec[kPairRows][kRowRec];
    __shared__ VertexSlots s_slots;
    __shared__ uint16_t s_close[kPairRows * kPairThreads];
    __shared__ int s_n;
    extern __shared__ float s_sum[];
    const int64_t p0 = row_begin + (int64_t)blockIdx.y * rows_per_block;
    const int64_t q = (int64_t)blockIdx.x * kPairThreads + threadIdx.x;
    const int np = (int)min((int64_t)rows_per_block, row_end - p0);
    if (threadIdx.x == 0) s_n = 0;
    if (threadIdx.x < np) {
        const FaceLocal f = face_local(verts, faces, p0 + threadIdx.x);
        float* r = s_rec[threadIdx.x];
        const V3<float> n = cross(f.A[1] - f.A[0], f.A[2] - f.A[1]);
        const float inv = 1.f / sqrtf(dot(n, n));
        const float v[kRowRec] = {f.v0.x, f.v0.y, f.v0.z, f.rho, f.off.x, f.off.y, f.off.z, f.area,
                                  f.A[0].x, f.A[0].y, f.A[0].z, 0.f, f.A[1].x, f.A[1].y, f.A[1].z, 0.f,
                                  f.A[2].x, f.A[2].y, f.A[2].z, 0.f, n.x * inv, n.y * inv, n.z * inv, 0.f,
                                  dot(f.A[0], f.A[0]), dot(f.A[1], f.A[1]), dot(f.A[2], f.A[2]), 0.f};
#pragma unroll
        for (int c = 0; c < kRowRec; ++c) r[c] = v[c];
#pragma unroll
        for (int a = 0; a < 3; ++a) s_slots.id[3 * threadIdx.x + a] = f.id[a];
    }
    find_slots(s_slots, np);
    clear_sums(s_sum, s_slots.n);
    if (q < nf) {
        const FaceLocal x = face_local(verts, faces, q);
        float BB[3];
#pragma unroll
        for (int b = 0; b < 3; ++b) BB[b] = dot(x.A[b], x.A[b]);
#pragma unroll 1
        for (int i = 0; i < np; ++i) {
            const float4* r = reinterpret_cast<const float4*>(s_rec[i]);
            const float4 c0 = r[0], c1 = r[1], r2v = r[2], r3v = r[3], r4v = r[4], nv4 = r[5], aav = r[6];
            const float dx = (c0.x - x.v0.x) + (c1.x - x.off.x), dy = (c0.y - x.v0.y) + (c1.y - x.off.y),
                        dz = (c0.z - x.v0.z) + (c1.z - x.off.z);
            const float Rc2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx)), lim = 2.f * (c0.w + x.rho);
            if (!(Rc2 >= lim * lim)) {  // faces sharing a vertex are here, too: closed forms
                int shared = 0;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int id = s_slots.id[3 * i + a];
                    shared |= (id == x.id[0]) | (id == x.id[1]) | (id == x.id[2]);
                }
                if (!shared) s_close[atomicAdd(&s_n, 1)] = (uint16_t)(i * kPairThreads + threadIdx.x);
                continue;
            }
            const float A[3][3] = {{r2v.x, r2v.y, r2v.z}, {r3v.x, r3v.y, r3v.z}, {r4v.x, r4v.y, r4v.z}};
            const float AA[3] = {aav.x, aav.y, aav.z};
            float m[3][3], DA[3];
            float2 V[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const float DB = fmaf(dz, x.A[b].z, fmaf(dy, x.A[b].y, dx * x.A[b].x));
                V[b] = make_float2(s1 * (2.f * DB - s1 * BB[b]), s2 * (2.f * DB - s2 * BB[b]));
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                DA[a] = fmaf(dz, A[a][2], fmaf(dy, A[a][1], dx * A[a][0]));
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    m[a][b] = fmaf(A[a][2], x.A[b].z, fmaf(A[a][1], x.A[b].y, A[a][0] * x.A[b].x));
            }
            // sums over fy's points, lanes fx's orbits: S[a][b] with w s (corner a), S0[b] with
            // w (1 - s)/3 (OP 3: w); c[a], cc the same at fx's centroid; fy's centroid first
            float2 S[3][3], S0[3];
            float c[3] = {0.f, 0.f, 0.f}, cc = 0.f;
            const float ri = rsqrtf(Rc2), kc = OP == 2 ? ri * ri * ri : ri;
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const float2 d2 = sub2(bc(Rc2), V[b]);
                float2 h = make_float2(rsqrtf(d2.x), rsqrtf(d2.y));
                if constexpr (OP == 2) h = mul2(h, mul2(h, h));
                S0[b] = mul2(bc(OP == 3 ? w0 : w0 / 3.f), sub2(h, bc(kc)));
#pragma unroll
                for (int a = 0; a < 3; ++a) S[a][b] = bc(0.f);
            }
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const float s = o ? s2 : s1, w = o ? w2 : w1, al = o ? a2 : a1;
                const float2 K = make_float2(2.f * s * s1, 2.f * s * s2);
                const float2 W0 = bc(OP == 3 ? w : w * al), WS = bc(w * s);
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float u = fmaf(s * s, AA[a], 2.f * s * DA[a]);
                    {
                        float g = rsqrtf(Rc2 + u);
                        if constexpr (OP == 2) g = g * g * g;
                        g -= kc;
                        cc = fmaf(OP == 3 ? w : w * al, g, cc);
                        c[a] = fmaf(w * s, g, c[a]);
                    }
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const float2 d2 = sub2(bc(Rc2 + u), fma2(bc(m[a][b]), K, V[b]));
                        float2 h = make_float2(rsqrtf(d2.x), rsqrtf(d2.y));
                        if constexpr (OP == 2) h = mul2(h, mul2(h, h));
                        h = sub2(h, bc(kc));
                        S0[b] = fma2(W0, h, S0[b]);
                        if constexpr (OP != 3) S[a][b] = fma2(WS, h, S[a][b]);
                    }
                }
            }
            float acc[9];
            if constexpr (OP == 3) {
                const float2 t = add2(add2(S0[0], S0[1]), S0[2]);
                // curl_a . curl_b = (A_{a+1} - A_{a+2}).(B_{b+1} - B_{b+2}) / (4 area area)
                const float v0 = (kc + fmaf(w1, t.x, fmaf(w2, t.y, w0 * cc))) * (0.25f * float(kInv4Pi));
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const int p = (a + 1) % 3, e = (a + 2) % 3, u = (b + 1) % 3, v = (b + 2) % 3;
                        acc[3 * a + b] = ((m[p][u] - m[p][v]) - (m[e][u] - m[e][v])) * v0;
                    }
            } else {
                const float sc = c1.w * x.area * float(kInv4Pi);
                float k0[3] = {kc / 9.f, kc / 9.f, kc / 9.f};  // the constant's share of column b
                if constexpr (OP == 2) {                       // n_y.(x - y) at fx's points
                    const float nD = fmaf(nv4.z, dz, fmaf(nv4.y, dy, nv4.x * dx));
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const float nB = fmaf(nv4.z, x.A[b].z, fmaf(nv4.y, x.A[b].y, nv4.x * x.A[b].x));
                        const float2 dn = make_float2(fmaf(s1, nB, -nD), fmaf(s2, nB, -nD));
                        S0[b] = mul2(S0[b], dn);
                        k0[b] = (kc / 3.f) * fmaf(w1 * s1 * s1 + w2 * s2 * s2, nB, -nD / 3.f);
#pragma unroll
                        for (int a = 0; a < 3; ++a) S[a][b] = mul2(S[a][b], dn);
                    }
                    cc *= -nD;
#pragma unroll
                    for (int a = 0; a < 3; ++a) c[a] *= -nD;
                }
                // fx's weights: w' s' at corner b, w' (1 - s')/3 over all points
                const float2 t0 = add2(add2(S0[0], S0[1]), S0[2]);
                const float C0 = fmaf(w1 * a1, t0.x, fmaf(w2 * a2, t0.y, (w0 / 3.f) * cc));
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float2 t = add2(add2(S[a][0], S[a][1]), S[a][2]);
                    const float Ca = fmaf(w1 * a1, t.x, fmaf(w2 * a2, t.y, fmaf(w0 / 3.f, c[a], C0)));
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const float2 v = add2(S[a][b], S0[b]);
                        acc[3 * a + b] = sc * (k0[b] + fmaf(w1 * s1, v.x, fmaf(w2 * s2, v.y, Ca)));
                    }
                }
            }
            add_entries(s_slots, i, acc, x.id, nv, s_sum, packed);
        }
        flush_sums(s_slots, x.id, nv, s_sum, packed);
    }
    __syncthreads();
    const int n = s_n;
    for (int i = threadIdx.x; i < n; i += kPairThreads) {
        const int e = s_close[i];
        close_pair_entries<OP>(verts, faces, p0 + e / kPairThreads, (int64_t)blockIdx.x * kPairThreads + e % kPairThreads,
                               nv, packed);
    }
}

__device__ __forceinline__ V3<double> load3d(const float* p, int64_t i) {
    return v3<double>(p[3 * i], p[3 * i + 1], p[3 * i + 2]);
}
__device__ __forceinline__ V3<double> load3d(const double* p, int64_t i) {
    return v3<double>(p[3 * i], p[3 * i + 1], p[3 * i + 2]);
}

// Pairs sharing a vertex; overwrites the entry.  The closed forms run in the output's
// arithmetic T (float outputs: float logs and arctangents, ~1e-7 of each integral, below
// the rounding of the stored value; GB300's FP64 rate is 1/64 of its FP32 rate), on
// coordinates moved to fy's first vertex in FP64 first.  Eight lanes per listed pair
// (fy, fx): lane i < 7 integrates over fy at the i-th point of fx, lane 7 idles, and the
// eight partial blocks are summed by shuffles within the group.  With `packed` set the
// pair's block is added to the packed matrix [nv, nv] instead (op 1 / 2: single / double
// layer P1; op 3: hypersingular from the P0 single layer and the faces' curls).
constexpr int kNearLanes = 8;

template <typename T>
__global__ void __launch_bounds__(128)
    lap_sym_near_kernel(const T* __restrict__ verts, const int32_t* __restrict__ faces, int64_t nf,
                        const int32_t* __restrict__ pairs, int64_t n_pairs, int layer, int nphi,
                        int64_t row_begin, int64_t row_end, T* __restrict__ out, int op, int64_t nv,
                        T* __restrict__ packed) {
    const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t t = gt / kNearLanes;
    const int i = (int)(gt % kNearLanes);
    // every lane of a group sees the same t, so a group leaves (or stays) as a whole
    if (t >= n_pairs) return;
    const int64_t fy = pairs[2 * t], fx = pairs[2 * t + 1];
    if (fy < row_begin || fy >= row_end) return;
    const unsigned gmask = 0xFFu << (threadIdx.x & 24);
    const V3<double> o = load3d(verts, faces[3 * fy]);
    V3<T> P[3], Q[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        const V3<double> p = load3d(verts, faces[3 * fy + v]) - o;
        const V3<double> q = load3d(verts, faces[3 * fx + v]) - o;
        P[v] = v3<T>((T)p.x, (T)p.y, (T)p.z);
        Q[v] = v3<T>((T)q.x, (T)q.y, (T)q.z);
    }
    T acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (i < 7) {
        const V3<T> ny2 = cross(P[1] - P[0], P[2] - P[1]);
        const T two_ay = sqrt_t(dot(ny2, ny2));
        const V3<T> ny = (T(1) / two_ay) * ny2;
        const V3<T> nx2 = cross(Q[1] - Q[0], Q[2] - Q[1]);
        const T ax = T(0.5) * sqrt_t(dot(nx2, nx2));
        const V3<T> x = (T)c_d7[i][0] * Q[0] + (T)c_d7[i][1] * Q[1] + (T)c_d7[i][2] * Q[2];
        const T wx = (T)c_d7[i][3] * ax;
        T sa[3] = {0, 0, 0};
        V3<T> grad[3];
        V3<T> cy = v3<T>(0, 0, 0);
        if (nphi == 3) {
#pragma unroll
            for (int a = 0; a < 3; ++a) grad[a] = (T(1) / two_ay) * cross(ny, P[(a + 2) % 3] - P[(a + 1) % 3]);
            cy = T(1.0 / 3.0) * (P[0] + P[1] + P[2]);
        }
        if (layer == 1) {
            T I0;
            V3<T> I1;
            potential_integrals(x, P, &I0, &I1);
            if (nphi == 3) {
#pragma unroll
                for (int a = 0; a < 3; ++a) sa[a] = (T(1.0 / 3.0) + dot(grad[a], x - cy)) * I0 + dot(grad[a], I1);
            } else {
                sa[0] = I0;
            }
        } else {
            T hmax = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const V3<T> e = P[(a + 1) % 3] - P[a];
                hmax = fmax(hmax, sqrt_t(dot(e, e)));
            }
            // in-plane test: 1e-10 of the edge in FP64, 1e-5 in FP32 (its coordinate noise is ~1e-7)
            const T dtol = (sizeof(T) == 4 ? T(1e-5) : T(1e-10)) * hmax;
            T om, d;
            V3<T> J;
            dl_integrals(x, P, dtol, &om, &J, &d);
            if (nphi == 3) {
#pragma unroll
                for (int a = 0; a < 3; ++a) sa[a] = -(T(1.0 / 3.0) + dot(grad[a], x - cy)) * om + d * dot(grad[a], J);
            } else {
                sa[0] = -om;
            }
        }
        if (nphi == 3) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) acc[3 * a + b] = sa[a] * wx * (T)c_d7[i][b];
        } else {
            acc[0] = sa[0] * wx;
        }
    }
    const int nn = nphi * nphi;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        if (c < nn) {
            acc[c] += __shfl_xor_sync(gmask, acc[c], 1);
            acc[c] += __shfl_xor_sync(gmask, acc[c], 2);
            acc[c] += __shfl_xor_sync(gmask, acc[c], 4);
        }
    }
    T mine = acc[0];
#pragma unroll
    for (int c = 1; c < 8; ++c)
        if (i == c) mine = acc[c];
    if (packed == nullptr) {
        T* dst = out + ((fy - row_begin) * nf + fx) * nn;
        if (i < nn) dst[i] = mine * T(kInv4Pi);
        if (i == 0 && nn == 9) dst[8] = acc[8] * T(kInv4Pi);
        return;
    }
    // packed: lane i adds entry (a, b) = (i / 3, i % 3); lane 0 also (2, 2)
    V3<T> cy[3], cx[3];
    if (op == 3) {
        tri_curls(P[0], P[1], P[2], cy);
        tri_curls(Q[0], Q[1], Q[2], cx);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int c = k == 0 ? i : 8;
        if (k == 1 && i != 0) break;
        const int a = c / 3, b = c % 3;
        const T v = op == 3 ? dot(cy[a], cx[b]) * acc[0] * T(kInv4Pi) : (k == 0 ? mine : acc[8]) * T(kInv4Pi);
        atomicAdd(packed + (int64_t)faces[3 * fy + a] * nv + faces[3 * fx + b], v);
    }
}

// P0 single-layer collocation at face centroids with the 7-point rule.  A block covers
// kSymThreads source faces j (one per thread) and kColRows consecutive collocation rows i:
// each thread builds its source triangle's 7 points once and evaluates them against the
// kColRows centroids held in shared memory, writing out[(i - row_begin) * nf + j]
// (coalesced per row).  Pairs sharing a vertex are then rewritten by lap_colloc_near_kernel.
constexpr int kColRows = 64;

template <typename T>
__global__ void __launch_bounds__(kSymThreads)
    lap_colloc_sl_kernel(const T* __restrict__ verts, const int32_t* __restrict__ faces, int64_t nf,
                         int64_t row_begin, int64_t row_end, T* __restrict__ out) {
    __shared__ T s_c[kColRows][3];
    const int64_t i0 = row_begin + (int64_t)blockIdx.y * kColRows;
    const int64_t j = (int64_t)blockIdx.x * kSymThreads + threadIdx.x;
    for (int t = threadIdx.x; t < kColRows; t += blockDim.x) {
        const int64_t i = i0 + t;
        if (i < row_end) {
            const int32_t a0 = faces[3 * i], a1 = faces[3 * i + 1], a2 = faces[3 * i + 2];
            const V3<T> c = T(1.0 / 3.0) * (load3(verts, a0) + load3(verts, a1) + load3(verts, a2));
            s_c[t][0] = c.x;
            s_c[t][1] = c.y;
            s_c[t][2] = c.z;
        }
    }
    __syncthreads();
    if (j >= nf) return;
    const V3<T> B0 = load3(verts, __ldg(faces + 3 * j));
    const V3<T> E1 = load3(verts, __ldg(faces + 3 * j + 1)) - B0, E2 = load3(verts, __ldg(faces + 3 * j + 2)) - B0;
    const V3<T> nr = cross(E1, E2);
    const T scale = T(0.5) * sqrt_t(dot(nr, nr)) * T(kInv4Pi);
    V3<T> y[7];
    T w[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        y[k] = B0 + ((T)c_d7[k][1] * E1 + (T)c_d7[k][2] * E2);
        w[k] = (T)c_d7[k][3] * scale;
    }
    // Pairs sharing a vertex are evaluated here too (the value is discarded: the near-pair
    // kernel, launched next on the same stream, overwrites them); the only coincident point,
    // the centroid of a face against its own rule, gives +inf, never a fault.
    const int64_t rows = row_end - i0;
    if constexpr (sizeof(T) == 4) {
        if (rows >= kColRows) {
            // two collocation rows per packed f32x2 instruction (the source points broadcast)
            float2 yx[7], yy[7], yz[7], wk[7];
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                yx[k] = bc(y[k].x);
                yy[k] = bc(y[k].y);
                yz[k] = bc(y[k].z);
                wk[k] = bc(w[k]);
            }
#pragma unroll 2
            for (int r = 0; r < kColRows; r += 2) {
                const float2 cx = make_float2(s_c[r][0], s_c[r + 1][0]);
                const float2 cy = make_float2(s_c[r][1], s_c[r + 1][1]);
                const float2 cz = make_float2(s_c[r][2], s_c[r + 1][2]);
                float2 acc = bc(0.f);
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    const float2 dx = sub2(yx[k], cx), dy = sub2(yy[k], cy), dz = sub2(yz[k], cz);
                    const float2 r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
                    float2 ri;
                    ri.x = rsqrtf(r2.x);
                    ri.y = rsqrtf(r2.y);
                    acc = fma2(wk[k], ri, acc);
                }
                out[(i0 - row_begin + r) * nf + j] = acc.x;
                out[(i0 - row_begin + r + 1) * nf + j] = acc.y;
            }
            return;
        }
    }
    if (rows >= kColRows) {
#pragma unroll 4
        for (int r = 0; r < kColRows; ++r) {
            const V3<T> c = v3<T>(s_c[r][0], s_c[r][1], s_c[r][2]);
            T acc = 0;
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const V3<T> d = y[k] - c;
                acc += w[k] * rcp_sqrt(dot(d, d));
            }
            out[(i0 - row_begin + r) * nf + j] = acc;
        }
    } else {
        for (int r = 0; r < (int)rows; ++r) {
            const V3<T> c = v3<T>(s_c[r][0], s_c[r][1], s_c[r][2]);
            T acc = 0;
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const V3<T> d = y[k] - c;
                acc += w[k] * rcp_sqrt(dot(d, d));
            }
            out[(i0 - row_begin + r) * nf + j] = acc;
        }
    }
}

// Collocation pairs sharing a vertex (listed as (i, j)): closed form in FP64.
template <typename T>
__global__ void lap_colloc_near_kernel(const T* __restrict__ verts, const int32_t* __restrict__ faces, int64_t nf,
                                       const int32_t* __restrict__ pairs, int64_t n_pairs, int64_t row_begin,
                                       int64_t row_end, T* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_pairs) return;
    const int64_t i = pairs[2 * t], j = pairs[2 * t + 1];
    if (i < row_begin || i >= row_end) return;
    V3<double> P[3];
    V3<double> c = v3<double>(0, 0, 0);
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        P[v] = load3d(verts, faces[3 * j + v]);
        c = c + (1.0 / 3.0) * load3d(verts, faces[3 * i + v]);
    }
    double I0;
    V3<double> I1;
    potential_integrals(c, P, &I0, &I1);
    out[(i - row_begin) * nf + j] = (T)(I0 * kInv4Pi);
}

template <typename T>
int launch_laplace_sym(const T* verts, const int32_t* faces, int64_t nf, int layer, int order,
                       const int32_t* pairs, int64_t n_pairs, int64_t row_begin, int64_t row_end, T* out,
                       cudaStream_t s) {
    if (nf <= 0 || row_end <= row_begin) return MB_OK;
    if (layer != 1 && layer != 2) return set_error(MB_ERR_ARG, "layer must be 1 (single) or 2 (double)");
    if (order != 0 && order != 1) return set_error(MB_ERR_ARG, "order must be 0 or 1");
    const int nphi = order == 1 ? 3 : 1;
    const int64_t col_blocks = (nf + kSymThreads - 1) / kSymThreads;
    const int64_t blocks = (row_end - row_begin) * col_blocks;
    if (blocks > 0x7fffffffLL) return set_error(MB_ERR_SIZE, "mesh too large for one launch");
#define MB_FAR(LY, NP)                                                                                   \
    lap_sym_far_kernel<T, LY, NP><<<(unsigned)blocks, kSymThreads, 0, s>>>(verts, faces, nf, row_begin, \
                                                                            col_blocks, out)
    if (layer == 1 && nphi == 1) MB_FAR(1, 1);
    else if (layer == 1) MB_FAR(1, 3);
    else if (nphi == 1) MB_FAR(2, 1);
    else MB_FAR(2, 3);
#undef MB_FAR
    if (n_pairs > 0) {
        const int64_t near_blocks = (n_pairs * kNearLanes + 127) / 128;
        if (near_blocks > 0x7fffffffLL) return set_error(MB_ERR_SIZE, "near-pair list too long for one launch");
        lap_sym_near_kernel<T><<<(unsigned)near_blocks, 128, 0, s>>>(verts, faces, nf, pairs, n_pairs, layer, nphi,
                                                                     row_begin, row_end, out, 0, 0, nullptr);
    }
    return check_launch("laplace_sym");
}
// Packed operators (op 1 single layer, 2 double layer, 3 hypersingular) for test rows
// [row_begin, row_end), added to packed [nv, nv].  order: 8 bytes of device memory for the FP32 kernels' choice, or null
// (many rows of a large mesh then go by a block per face).
constexpr int64_t kTightSmemMax = 160 * 1024;

template <typename T>
static int launch_sym_rows(const T* verts, const int32_t* faces, int64_t nf, int64_t nv, int op, int64_t row_begin,
                           int64_t row_end, const FaceOrder* order, T* packed, cudaStream_t s) {
    if (row_end - row_begin > 0x7fffffffLL) return set_error(MB_ERR_SIZE, "mesh too large for one launch");
    auto go = [&](auto kernel) -> int {
        const size_t smem = (size_t)(3 * nv) * sizeof(T);
        if (smem > 48 * 1024) {
            // the same limit for every mesh: it is the process's, and another thread may be between these two calls
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTightSmemMax);
            if (e != cudaSuccess) return set_error(MB_ERR_CUDA, "%s", cudaGetErrorString(e));
        }
        kernel<<<(unsigned)(row_end - row_begin), kSymThreads, smem, s>>>(verts, faces, nf, nv,
                                                                                               row_begin, order, packed);
        return MB_OK;
    };
    return op == 1 ? go(lap_sym_tight_kernel<T, 1>) : op == 2 ? go(lap_sym_tight_kernel<T, 2>) : go(lap_sym_tight_kernel<T, 3>);
}

static int launch_sym_pairs(const double* verts, const int32_t* faces, int64_t nf, int64_t nv, int op, int64_t row_begin,
                            int64_t row_end, FaceOrder*, double* packed, cudaStream_t s) {
    return launch_sym_rows(verts, faces, nf, nv, op, row_begin, row_end, nullptr, packed, s);
}

// Whether a block per test face is the faster form for FP32: small meshes, where lap_sym_pairs_kernel's blocks are
// few and its set-up and its close pairs, one after the other, are most of their time.  Measured (GB300, us, rows form /
// pairs form, operators 1, 2, 3, without the pairs sharing a vertex where the rows are a window):
//   416 faces 25 / 35, 27 / 36, 25 / 34; 680 39 / 46, 41 / 49, 31 / 44; 1300 90 / 94, 98 / 102, 68 / 90;
//   1740 139 / 122, 150 / 131, 107 / 116; 2112 192 / 154, 207 / 166, 141 / 148; 2960 383 / 254, 397 / 267, 264 / 241;
//   300 rows of 680 faces 18 / 28, 19 / 30, 17 / 27, of 2112 39 / 42, 41 / 45, 37 / 41, of 2960 52 / 52, 54 / 54, 49 / 50, of
//   4048 80 / 56, 82 / 59, 68 / 53; 100 rows of 874 17 / 19, 19 / 20, 17 / 19; 30 rows of 680 14 / 10, 15 / 10, 16 / 10, of
//   126 8 / 8, 8 / 10, 8 / 8.
// Where many rows may go by pairs, the look at the faces' order and the other form's empty launch cost 10 to 18 us more,
// which a mesh in any order pays for nothing: 2.5 % of a call at these lines (5120 faces 1041 -> 1060 us), 5 % at 2600.
static bool rows_form(int64_t nf, int64_t rows, int op) {
    if (nf < 150) return true;
    return rows >= 64 && nf < (op == 3 ? 4800 : 3600);
}

static int launch_sym_pairs(const float* verts, const int32_t* faces, int64_t nf, int64_t nv, int op, int64_t row_begin,
                            int64_t row_end, FaceOrder* order, float* packed, cudaStream_t s) {
    const int64_t gx = (nf + kPairThreads - 1) / kPairThreads, rows = row_end - row_begin;
    // few rows: groups of faces in any order (each row form's block would sweep the mesh for one row)
    if (nf >= 150 && rows < 64) order = nullptr;
    else if (rows_form(nf, rows, op) || !order) return launch_sym_rows(verts, faces, nf, nv, op, row_begin, row_end, nullptr, packed, s);
    const int per = pair_rows(rows, gx);
    const int64_t gy = (rows + per - 1) / per;
    if (gx > 0x7fffffffLL || gy > 65535) return set_error(MB_ERR_SIZE, "mesh too large for one launch");
    if (order) {
        lap_face_order_kernel<<<1, 32 * kOrderSamples, 0, s>>>(faces, nf, order);
        if (int rc = launch_sym_rows(verts, faces, nf, nv, op, row_begin, row_end, order, packed, s)) return rc;
    }
    auto go = [&](auto kernel) -> int {
        kernel<<<dim3((unsigned)gx, (unsigned)gy), kPairThreads, kPairSumBytes, s>>>(verts, faces, nf, nv, row_begin,
                                                                                     row_end, per, order, packed);
        return MB_OK;
    };
    return op == 1 ? go(lap_sym_pairs_kernel<1>) : op == 2 ? go(lap_sym_pairs_kernel<2>) : go(lap_sym_pairs_kernel<3>);
}

template <typename T>
int launch_laplace_sym_tight(const T* verts, const int32_t* faces, int64_t nf, int64_t nv, int op,
                             const int32_t* pairs, int64_t n_pairs, int64_t row_begin, int64_t row_end,
                             FaceOrder* order, T* packed, cudaStream_t s) {
    if (nf <= 0 || row_end <= row_begin) return MB_OK;
    if (op < 1 || op > 3) return set_error(MB_ERR_ARG, "op must be 1 (single), 2 (double) or 3 (hypersingular)");
    if (3 * nv * (int64_t)sizeof(T) > kTightSmemMax) return set_error(MB_ERR_SIZE, "too many vertices for the packed assembly");
    if (int rc = launch_sym_pairs(verts, faces, nf, nv, op, row_begin, row_end, order, packed, s)) return rc;
    if (n_pairs > 0) {
        const int64_t near_blocks = (n_pairs * kNearLanes + 127) / 128;
        if (near_blocks > 0x7fffffffLL) return set_error(MB_ERR_SIZE, "near-pair list too long for one launch");
        lap_sym_near_kernel<T><<<(unsigned)near_blocks, 128, 0, s>>>(
            verts, faces, nf, pairs, n_pairs, op == 2 ? 2 : 1, op == 3 ? 1 : 3, row_begin, row_end, nullptr, op, nv,
            packed);
    }
    return check_launch("laplace_sym_tight");
}
template int launch_laplace_sym_tight<float>(const float*, const int32_t*, int64_t, int64_t, int, const int32_t*,
                                             int64_t, int64_t, int64_t, FaceOrder*, float*, cudaStream_t);
template int launch_laplace_sym_tight<double>(const double*, const int32_t*, int64_t, int64_t, int, const int32_t*,
                                              int64_t, int64_t, int64_t, FaceOrder*, double*, cudaStream_t);

template int launch_laplace_sym<float>(const float*, const int32_t*, int64_t, int, int, const int32_t*, int64_t,
                                       int64_t, int64_t, float*, cudaStream_t);
template int launch_laplace_sym<double>(const double*, const int32_t*, int64_t, int, int, const int32_t*,
                                        int64_t, int64_t, int64_t, double*, cudaStream_t);

template <typename T>
int launch_laplace_colloc_sl(const T* verts, const int32_t* faces, int64_t nf, const int32_t* pairs,
                             int64_t n_pairs, int64_t row_begin, int64_t row_end, T* out, cudaStream_t s) {
    if (nf <= 0 || row_end <= row_begin) return MB_OK;
    const int64_t gx = (nf + kSymThreads - 1) / kSymThreads;
    const int64_t gy = (row_end - row_begin + kColRows - 1) / kColRows;
    if (gx > 0x7fffffffLL || gy > 65535) return set_error(MB_ERR_SIZE, "mesh too large for one launch");
    lap_colloc_sl_kernel<T><<<dim3((unsigned)gx, (unsigned)gy), kSymThreads, 0, s>>>(verts, faces, nf, row_begin,
                                                                                      row_end, out);
    if (n_pairs > 0)
        lap_colloc_near_kernel<T><<<(unsigned)((n_pairs + 127) / 128), 128, 0, s>>>(verts, faces, nf, pairs, n_pairs,
                                                                                   row_begin, row_end, out);
    return check_launch("laplace_colloc_sl");
}
template int launch_laplace_colloc_sl<float>(const float*, const int32_t*, int64_t, const int32_t*, int64_t,
                                             int64_t, int64_t, float*, cudaStream_t);
template int launch_laplace_colloc_sl<double>(const double*, const int32_t*, int64_t, const int32_t*, int64_t,
                                              int64_t, int64_t, double*, cudaStream_t);

}  // namespace mb
