// mom_tiers.cu -- the reference-rule CFIE matrix in FP32 with each face pair's quadrature
// sized by its separation.
//
// The reference anchors its collapsed Gauss rule at every local edge's free vertex, so the
// nine entries of a face pair use nine point sets: 1296 kernel evaluations at gaussQR 4.
// What makes those sets differ is only what the rules do not integrate exactly: anchored
// at any vertex, the n x n collapsed rule is exact for polynomials of total degree 2n - 2.
// On a pair that is far apart, compared with its triangles, and small, compared with the
// wavelength, the integrand is such a polynomial up to less than the rounding of its FP32
// evaluation, and any rule of that degree -- one set of points for all nine entries -- gives
// the same entry.  With rho the larger distance of a corner from its centroid of the two
// faces and R the centroid distance, measured on spheres of 0.15 <= kh <= 1.5 in 64 bits
// (rms over entries, relative to them; FP32 evaluation of the 1296 points is off by
// 1e-5 .. 6e-5 at kh = 0.38, by 1.4e-6 .. 6e-6 at kh = 1.5, the four face pairs of an entry
// cancelling to (kh)^2 of their size):
//   tier 1   6-point degree-4 rule on both faces        36 evaluations
//            off by 2.7e-4 (k rho)^4 + 3.2e-2 (rho/R)^4, taken up to 2e-6
//   tier 2   7-point degree-5 rule on the test face, the anchored source rule   189
//            off by 1.2e-5 (k rho)^6 + 0.4 (rho/R)^6, taken up to 5e-7
//   tier 3   12-point degree-6 rule on the test face, the anchored source rule  324
//            off by 1.5e-6 (k rho)^8 + 0.73 (rho/R)^8, taken up to 6e-7 where k rho <= 0.8 (above, the SFU's
//            error in the phases relative to the centroids' exceeds that of the 1296 points' mean)
//   tier 4   the reference's points (mom_entry_fast)                           1296
// (counts at gaussQR 4).  gaussQR 3: its source rule has degree 2, so no tier 1; its test rule
// degree 4, so tier 2 up to the first bound.  gaussQR 5: all tiers.  A rule that is not
// Gauss-Legendre, a normal that is not perpendicular to its face and coordinates that are
// not finite put every pair concerned into tier 4.
//
// Measured on GB300 (2070 MHz), whole call: 20480 faces, k 10, unit sphere 500.0 -> 34.8 ms (far pairs 26.2, close
// pairs 4.0 + 3.6); 5120 faces, k 6, ellipsoid 32.2 -> 4.6 ms; all pairs in tier 4: 1280 faces, k 10, gaussQR 4 2.13 -> 2.10
// ms, gaussQR 5 5.12 -> 5.15, 5120 faces, k 30, 31.3 -> 31.3 and 78.8 -> 79.1.
// Error of the entries against 64 bits by distance, of the 1296 points' FP32 error: 1.0 .. 1.1 below 4 h, 0.5 .. 0.95
// beyond (kh 0.15 .. 0.9).  The four adds of an entry are atomic, so its last bit depends on their order.
//
// Rules: O. C. Zienkiewicz / D. A. Dunavant, Int. J. Numer. Meth. Eng. 21 (1985), degrees 4 to 6.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "face_order.cuh"
#include "face_record.cuh"
#include "mom_entry.cuh"
#include "packed.cuh"

namespace mb {

namespace {

// ---------------------------------------------------------------------------------------
// face records: 32 floats per face
// ---------------------------------------------------------------------------------------
// sin x = x (1 + SA x^2 + SB x^4) and cos x = 1 + CA x^2 + CB x^4 + CC x^6, least squares on |x| <= 0.43 (off by
// 5e-8 of x and 3e-10)
constexpr float SA = -0.16666371f, SB = 0.00828212f;
constexpr float CA = -0.49999997f, CB = 0.04166572f, CC = -0.00138007f;

// degree-4 rule: corners (1 - 2 q, q, q) of two orbits lie at s A_a from the centroid
constexpr float kS1 = (float)(1.0 - 3.0 * 0.445948490915965), kW1 = 0.223381589678011f;
constexpr float kS2 = (float)(1.0 - 3.0 * 0.091576213509771), kW2 = 0.109951743655322f;

// test rules of tiers 2 and 3: barycentric coordinates and weights (sum 1)
__constant__ float c_test[19][4] = {
    {0.33333333333f, 0.33333333333f, 0.33333333333f, 0.225f},
    {0.101286507323456f, 0.101286507323456f, 0.797426985353087f, 0.125939180544827f},
    {0.101286507323456f, 0.797426985353087f, 0.101286507323456f, 0.125939180544827f},
    {0.797426985353087f, 0.101286507323456f, 0.101286507323456f, 0.125939180544827f},
    {0.470142064105115f, 0.470142064105115f, 0.059715871789770f, 0.132394152788506f},
    {0.470142064105115f, 0.059715871789770f, 0.470142064105115f, 0.132394152788506f},
    {0.059715871789770f, 0.470142064105115f, 0.470142064105115f, 0.132394152788506f},
    {0.249286745170910f, 0.249286745170910f, 0.501426509658179f, 0.116786275726379f},
    {0.249286745170910f, 0.501426509658179f, 0.249286745170910f, 0.116786275726379f},
    {0.501426509658179f, 0.249286745170910f, 0.249286745170910f, 0.116786275726379f},
    {0.063089014491502f, 0.063089014491502f, 0.873821971016996f, 0.050844906370207f},
    {0.063089014491502f, 0.873821971016996f, 0.063089014491502f, 0.050844906370207f},
    {0.873821971016996f, 0.063089014491502f, 0.063089014491502f, 0.050844906370207f},
    {0.053145049844817f, 0.310352451033784f, 0.636502499121399f, 0.082851075618374f},
    {0.310352451033784f, 0.053145049844817f, 0.636502499121399f, 0.082851075618374f},
    {0.053145049844817f, 0.636502499121399f, 0.310352451033784f, 0.082851075618374f},
    {0.310352451033784f, 0.636502499121399f, 0.053145049844817f, 0.082851075618374f},
    {0.636502499121399f, 0.053145049844817f, 0.310352451033784f, 0.082851075618374f},
    {0.636502499121399f, 0.310352451033784f, 0.053145049844817f, 0.082851075618374f},
};

// Gauss-Legendre nodes and weights on [0, 1], n = 2 .. 5 (the second half mirrors the first)
__constant__ float c_gl[4][3][2] = {
    {{0.2113248654f, 0.5f}, {0.f, 0.f}, {0.f, 0.f}},
    {{0.1127016654f, 0.2777777778f}, {0.5f, 0.4444444444f}, {0.f, 0.f}},
    {{0.0694318442f, 0.1739274226f}, {0.3300094782f, 0.3260725774f}, {0.f, 0.f}},
    {{0.0469100770f, 0.1184634425f}, {0.2307653449f, 0.2393143352f}, {0.5f, 0.2844444444f}},
};

__device__ bool is_gauss(const float* p, const float* w, int n) {
    for (int i = 0; i < n; ++i) {
        const int j = i < (n + 1) / 2 ? i : n - 1 - i;
        const float x = j == i ? c_gl[n - 2][j][0] : 1.f - c_gl[n - 2][j][0];
        if (!(fabsf(p[i] - x) <= 1e-6f) || !(fabsf(w[i] - c_gl[n - 2][j][1]) <= 1e-6f)) return false;
    }
    return true;
}

__global__ void face_record_kernel(const float* __restrict__ verts, const int32_t* __restrict__ faces,
                                   const float* __restrict__ normals, const int32_t* __restrict__ fei, int64_t nf,
                                   const float* __restrict__ gpx, const float* __restrict__ gwx, int nx,
                                   const float* __restrict__ gpy, const float* __restrict__ gwy, int ny,
                                   float* __restrict__ rec) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    double v[3][3];
    int32_t id[3];
    float n[3];
    for (int a = 0; a < 3; ++a) {
        id[a] = faces[3 * f + a];
        n[a] = normals ? normals[3 * f + a] : 0.f;
        for (int d = 0; d < 3; ++d) v[a][d] = (double)verts[3 * (int64_t)id[a] + d];
    }
    float r[kRec];
    float A[3][3];
    for (int d = 0; d < 3; ++d) {
        const double c = (v[0][d] + v[1][d] + v[2][d]) * (1.0 / 3.0);
        r[kC + d] = (float)c;
        r[kCl + d] = (float)(c - (double)(float)c);
        for (int a = 0; a < 3; ++a) A[a][d] = (float)(v[a][d] - c);
        r[kN + d] = n[d];
    }
    float rho2 = 0.f;
    bool ok = !gpx || (is_gauss(gpx, gwx, nx) && is_gauss(gpy, gwy, ny));
    const float nn = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3, c = (a + 2) % 3;
        r[kAA + a] = A[a][0] * A[a][0] + A[a][1] * A[a][1] + A[a][2] * A[a][2];
        r[kAB + a] = A[a][0] * A[b][0] + A[a][1] * A[b][1] + A[a][2] * A[b][2];
        rho2 = fmaxf(rho2, r[kAA + a]);
        const double ex = v[c][0] - v[b][0], ey = v[c][1] - v[b][1], ez = v[c][2] - v[b][2];
        const float half = (float)(0.5 * sqrt(ex * ex + ey * ey + ez * ez));
        r[kHalf + 4 * a] = id[b] < id[c] ? half : -half;
        r[kEdge + 4 * a] = __int_as_float(fei[3 * f + a]);
        for (int d = 0; d < 3; ++d) r[kA + 4 * a + d] = A[a][d];
        const float na = n[0] * A[a][0] + n[1] * A[a][1] + n[2] * A[a][2];
        ok = ok && na * na <= 1e-10f * nn * r[kAA + a];
    }
    r[kRho2] = ok ? rho2 : __int_as_float(0x7fc00000);
    r[31] = 0.f;
    float4* out = reinterpret_cast<float4*>(rec) + (kRec / 4) * f;
    for (int q = 0; q < kRec / 4; ++q) out[q] = make_float4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
}

// ---------------------------------------------------------------------------------------
// the rule of a pair.  Both kernels below evaluate it and take disjoint sets of pairs, so its
// arithmetic is spelled out with rounding intrinsics (no contraction that differs by context).
// ---------------------------------------------------------------------------------------
template <int NX>
__device__ __forceinline__ int pair_tier(float r2, float rho2p, float rho2q, float k2) {
    // fmaxf drops a NaN operand; the sum does not
    const float rho2 = __fadd_rn(fmaxf(rho2p, rho2q), __fmul_rn(0.f, __fadd_rn(rho2p, rho2q)));
    const float u = __fmul_rn(rho2, __frcp_rn(r2)), q = __fmul_rn(k2, rho2);
    const float u2 = __fmul_rn(u, u), q2 = __fmul_rn(q, q);
    const bool t1 = __fmaf_rn(2.7e-4f, q2, __fmul_rn(3.2e-2f, u2)) <= 2e-6f;
    if (NX == 3) return t1 ? 2 : 4;
    if (t1) return 1;
    if (__fmaf_rn(1.2e-5f, __fmul_rn(q2, q), __fmul_rn(0.4f, __fmul_rn(u2, u))) <= 5e-7f) return 2;
    const bool t3 = __fmaf_rn(1.5e-6f, __fmul_rn(q2, q2), __fmul_rn(0.73f, __fmul_rn(u2, u2))) <= 6e-7f;
    return t3 && q <= 0.64f ? 3 : 4;
}

// The centroid distance of a pair in two floats -- the subtraction's error (TwoSum), the centroids'
// low parts, the squares' errors and the square root's -- and e^{-jkR_c} = c - j s from it, the
// wavenumber in turns as kth + ktl.  d = fl(c_p - c_q).
struct Centre {
    float r2, r, ri, ril, c, s;  // R^2, R, 1/R (ri + ril), cos and sin of k R
    // -e^{-jkR} j q / R in two floats (hi + lo): the entry's charge term at the centroids, common
    // to its nine entries and cancelling between an entry's four face pairs to (kh)^2 of itself
    float br, brl, bi, bil;
};
__device__ __forceinline__ Centre pair_centre(const float4& p, const float4& pl, const float4& q, const float4& ql,
                                              float dx, float dy, float dz, float kth, float ktl, float q4) {
    Centre o;
    const float bx = dx - p.x, by = dy - p.y, bz = dz - p.z;
    const float ex = ((p.x - (dx - bx)) - (q.x + bx)) + (pl.x - ql.x);
    const float ey = ((p.y - (dy - by)) - (q.y + by)) + (pl.y - ql.y);
    const float ez = ((p.z - (dz - bz)) - (q.z + bz)) + (pl.z - ql.z);
    // (rounding intrinsics: a contraction of these sums would void their error terms)
    const float sx = __fmul_rn(dx, dx), sy = __fmul_rn(dy, dy), sz = __fmul_rn(dz, dz);
    const float s1 = __fadd_rn(sx, sy), b1 = __fsub_rn(s1, sx);
    o.r2 = __fadd_rn(s1, sz);
    const float b2 = __fsub_rn(o.r2, s1);
    float lo = (fmaf(dx, dx, -sx) + fmaf(dy, dy, -sy)) + fmaf(dz, dz, -sz);
    lo += ((sx - (s1 - b1)) + (sy - b1)) + ((s1 - (o.r2 - b2)) + (sz - b2));
    lo = fmaf(2.f, fmaf(dx, ex, fmaf(dy, ey, dz * ez)), lo);
    o.ri = rsqrtf(o.r2);
    o.r = __fmul_rn(o.r2, o.ri);
    const float rl = (fmaf(-o.r, o.r, o.r2) + lo) * (0.5f * o.ri);
    o.ril = o.ri * fmaf(-o.r, o.ri, 1.f) - o.ri * o.ri * rl;
    const float t = __fmul_rn(kth, o.r), te = fmaf(kth, rl, fmaf(ktl, o.r, fmaf(kth, o.r, -t)));
    const float f0 = t - rintf(t), f = __fadd_rn(f0, te);
    sincospif(2.f * f, &o.s, &o.c);
    const float fl = 6.2831853f * (te - __fsub_rn(f, f0)), g = __fmul_rn(q4, o.ri), gl = fmaf(q4, o.ri, -g) + q4 * o.ril;
    const float pr = __fmul_rn(g, o.s), pi = __fmul_rn(g, o.c);
    o.br = -pr;
    o.bi = -pi;
    o.brl = -(fmaf(g, o.s, -pr) + fmaf(gl, o.s, g * o.c * fl));
    o.bil = -(fmaf(g, o.c, -pi) + fmaf(gl, o.c, -g * o.s * fl));
    return o;
}

// A squared centroid distance from which every pair of faces with rho^2 <= rho2 is in tier 1 (for gaussQR 3,
// in tier 2): pair_tier is monotone in both, and the factor covers its rounding.  Infinite where
// there is none, NaN for a NaN.
__device__ __forceinline__ float far_limit(float rho2, float k2) {
    const float q = k2 * rho2, rest = 2e-6f - 2.7e-4f * q * q;
    return rest > 2e-8f ? 1.001f * rho2 * sqrtf(3.2e-2f / rest) : rho2 == rho2 ? __int_as_float(0x7f800000) : rho2;
}

// One mesh of a launch: all meshes of a batch share the arrays, desc as in the batched kernels
// (n_mesh 0: one mesh, its values as arguments).
struct TierArgs {
    const float* verts;
    const int32_t* faces;
    const float* areas;
    const float* normals;
    const float* rec;
    const float *gpx, *gwx, *gpy, *gwy;
    const int64_t* desc;   // batch: [n_mesh, 6]
    const int64_t* boff;   // batch: first block of each mesh
    const double* ks;      // batch: wavenumbers
    int n_mesh;
    int64_t nf, n_edges;   // single mesh
    double k;
    float* z;
};

struct MeshRef {
    int64_t f0, nf, pitch, block;
    double k;
    float* z;
};

__device__ __forceinline__ MeshRef find_mesh(const TierArgs& a) {
    MeshRef m;
    if (a.n_mesh == 0) {
        m.f0 = 0;
        m.nf = a.nf;
        m.pitch = a.n_edges;
        m.block = blockIdx.x;
        m.k = a.k;
        m.z = a.z;
        return m;
    }
    int lo = 0, hi = a.n_mesh - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(a.boff + mid) <= (int64_t)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const int64_t* d = a.desc + 6 * lo;
    const int64_t ne = __ldg(d + 2);
    m.f0 = __ldg(d);
    m.nf = __ldg(d + 1);
    m.pitch = ne + (ne & 1);
    m.block = (int64_t)blockIdx.x - __ldg(a.boff + lo);
    m.k = __ldg(a.ks + lo);
    m.z = a.z + 2 * __ldg(d + 3);
    return m;
}

// ---------------------------------------------------------------------------------------
// tier 1.  A thread keeps one source face q and meets the block's test faces.  With centroids
// c_p, c_q, D = c_p - c_q, corners A_a, B_b relative to them, the rule points are s A_a and
// s' B_b, and everything the entry needs is built from the scalars m_ab = A_a.B_b, D.A_a,
// D.B_b, A_a.A_a', n.B_b, n.D (n the test normal) and from sums of w w' G and w w' h over the
// 36 points, h = G (1 + jkR) / R^2, weighted by powers of s, s':
//   sum G f_m.f_n    = T - sum_b m_mb M0b - sum_a m_an Ma0 + m_mn M00
//   MFIE part        = R_m - (n.B_n) S_m + (n.B_n - n.D)(U - U_m) + sum_a m_an Z_a - m_mn Z
// (h (x - A_m) . [r (n.rho) - rho (n.r)] with r = x - y, rho = y - B_n, summed term by term).
// The distance comes as R^2 = R_c^2 + sigma with sigma from the scalars (two operations), and
// R - R_c = (sigma - (R - R_c)^2) / (2 R_c), whose rounding is that of the small difference: the
// phase of an evaluation is k (R - R_c) relative to the pair's e^{-jkR_c}, which is computed
// once in two-float arithmetic.  An FP32 kR instead costs 1e-7 kR of phase per face pair,
// which the cancellation between an entry's four face pairs raises to 1e-5 .. 6e-5 of it.
//
// Lanes of a packed register are the two orbits of the source rule; they are weighted and
// added after the loop.  Bound: FMA pipe, 468 packed and ~600 scalar operations per pair.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float lanes(float2 v, float wx, float wy) { return fmaf(v.x, wx, v.y * wy); }

template <int NX>
__global__ void __launch_bounds__(128, 2) far_pairs_kernel(const TierArgs args, int rows_per_block) {
    __shared__ float4 s_rec[32 * (kRec / 4)];
    const MeshRef m = find_mesh(args);
    const int64_t col_tiles = (m.nf + 127) / 128;
    const int64_t p0 = (m.block / col_tiles) * rows_per_block;
    const int64_t q = (m.block % col_tiles) * 128 + threadIdx.x;
    const int np = (int)min((int64_t)rows_per_block, m.nf - p0);
    const float4* rec = reinterpret_cast<const float4*>(args.rec) + (kRec / 4) * m.f0;
    for (int i = threadIdx.x; i < np * (kRec / 4); i += 128) s_rec[i] = __ldg(rec + (kRec / 4) * p0 + i);
    __syncthreads();
    if (q >= m.nf) return;
    const float4* rq = rec + (kRec / 4) * q;
    const float k = (float)m.k, k2 = k * k;
    const float4 q0 = __ldg(rq);
    if (!(k2 * q0.w <= 0.09f)) return;  // tier 1 needs (k rho)^2 <= (2e-6 / 2.7e-4)^(1/2) = 0.086
    const float4 q1 = __ldg(rq + 1), q2 = __ldg(rq + 2), q3 = __ldg(rq + 3), q4 = __ldg(rq + 4),
                 q5 = __ldg(rq + 5), q6 = __ldg(rq + 6);
    const float B[3][3] = {{q2.x, q2.y, q2.z}, {q3.x, q3.y, q3.z}, {q4.x, q4.y, q4.z}};
    const float BB[3] = {q6.x, q6.y, q6.z}, hq[3] = {q4.w, q5.w, q6.w};
    const int col[3] = {__float_as_int(q1.w), __float_as_int(q2.w), __float_as_int(q3.w)};
    const double kt = m.k * kInv2Pi;
    const float kth = (float)kt, ktl = (float)(kt - (double)kth), four_k = 4.f / k;
    const float wqx = kW1, wqy = kW2, wsx = kW1 * kS1, wsy = kW2 * kS2;
#pragma unroll 1
    for (int i = 0; i < np; ++i) {
        const float4* rp = s_rec + (kRec / 4) * i;
        const float4 p0v = rp[0];
        const float dx = p0v.x - q0.x, dy = p0v.y - q0.y, dz = p0v.z - q0.z;
        if (pair_tier<NX>(centre_dist2(dx, dy, dz), p0v.w, q0.w, k2) != 1) continue;
        const float4 p1v = rp[1], p2v = rp[2], p3v = rp[3], p4v = rp[4], p5v = rp[5], p6v = rp[6], p7v = rp[7];
        const float A[3][3] = {{p2v.x, p2v.y, p2v.z}, {p3v.x, p3v.y, p3v.z}, {p4v.x, p4v.y, p4v.z}};
        const float AA[3] = {p6v.x, p6v.y, p6v.z};
        const Centre ce = pair_centre(p0v, p1v, q0, q1, dx, dy, dz, kth, ktl, four_k);
        const float Rc2 = ce.r2, R0 = ce.r, kp = k * (0.5f * ce.ri), C = ce.c, S = ce.s;
        const float2 G0 = bc(ce.ri);
        float mm[3][3], DA[3], nB[3];
        float2 V[3];  // -(sigma's source part) per b, lanes the two orbits
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            DA[a] = fmaf(dz, A[a][2], fmaf(dy, A[a][1], dx * A[a][0]));
            nB[a] = fmaf(p5v.z, B[a][2], fmaf(p5v.y, B[a][1], p5v.x * B[a][0]));
            const float DB = fmaf(dz, B[a][2], fmaf(dy, B[a][1], dx * B[a][0]));
            V[a] = make_float2(kS1 * (2.f * DB - kS1 * BB[a]), kS2 * (2.f * DB - kS2 * BB[a]));
#pragma unroll
            for (int b = 0; b < 3; ++b)
                mm[a][b] = fmaf(A[a][2], B[b][2], fmaf(A[a][1], B[b][1], A[a][0] * B[b][0]));
        }
        const float nD = fmaf(p5v.z, dz, fmaf(p5v.y, dy, p5v.x * dx));

        float2 Mr[3][3], Mi[3][3], M0r[3], M0i[3], Xr[3][3], Xi[3][3], X0r[3], X0i[3], Xgr[3], Xgi[3];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            M0r[b] = M0i[b] = X0r[b] = X0i[b] = Xgr[b] = Xgi[b] = bc(0.f);
#pragma unroll
            for (int a = 0; a < 3; ++a) Mr[a][b] = Mi[a][b] = Xr[a][b] = Xi[a][b] = bc(0.f);
        }
#pragma unroll 1
        for (int o = 0; o < 2; ++o) {
            const float s = o ? kS2 : kS1, w = o ? kW2 : kW1;
            const float2 W = bc(w), WS = bc(w * s), K2 = make_float2(2.f * s * kS1, 2.f * s * kS2);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float sd = s * DA[a], gam = fmaf(s * s, AA[a], sd);
                const float2 U = bc(-(gam + sd)), WG = bc(w * gam);
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const float2 ns = fma2(bc(mm[a][b]), K2, add2(U, V[b]));  // -sigma
                    const float2 r2 = sub2(bc(Rc2), ns);
                    float2 rinv;
                    rinv.x = rsqrtf(r2.x);
                    rinv.y = rsqrtf(r2.y);
                    const float2 R = mul2(r2, rinv), d0 = sub2(R, bc(R0));
                    const float2 th = mul2(fma2(d0, d0, ns), bc(kp));  // -k (R - R_c)
                    // |th| <= 0.43 by the rule of tier 1: polynomials; the SFU's error, 4e-7 and alike over a pair,
                    // would not average out
                    const float2 t = mul2(th, th);
                    const float2 sn = mul2(th, fma2(t, fma2(t, bc(SB), bc(SA)), bc(1.f)));
                    const float2 cs = fma2(t, fma2(t, fma2(t, bc(CC), bc(CB)), bc(CA)), bc(1.f));
                    const float2 gr = mul2(rinv, cs), gi = mul2(rinv, sn), ri2 = mul2(rinv, rinv), kR = mul2(bc(k), R);
                    const float2 hr = mul2(sub2(gr, mul2(gi, kR)), ri2), hi = mul2(fma2(gr, kR, gi), ri2);
                    // sums of G - 1/R_c: the constant drops out of the first moments (the corners' sums
                    // vanish) and is carried through M00 in two floats (ce.b)
                    const float2 gd = sub2(gr, G0);
                    Mr[a][b] = fma2(WS, gd, Mr[a][b]);
                    Mi[a][b] = fma2(WS, gi, Mi[a][b]);
                    M0r[b] = fma2(W, gd, M0r[b]);
                    M0i[b] = fma2(W, gi, M0i[b]);
                    Xr[a][b] = fma2(WS, hr, Xr[a][b]);
                    Xi[a][b] = fma2(WS, hi, Xi[a][b]);
                    X0r[b] = fma2(W, hr, X0r[b]);
                    X0i[b] = fma2(W, hi, X0i[b]);
                    Xgr[b] = fma2(WG, hr, Xgr[b]);
                    Xgi[b] = fma2(WG, hi, Xgi[b]);
                }
            }
        }
        // sums over the source orbits; re and im in the lanes of the complex values below
        float2 E[3][3], H[3][3];
        {
            float2 Tr = bc(0.f), Ti = bc(0.f), Ma[3], Mb[3], M00;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                Mb[a] = make_float2(lanes(M0r[a], wsx, wsy), lanes(M0i[a], wsx, wsy));
                const float2 sr = add2(add2(Mr[a][0], Mr[a][1]), Mr[a][2]), si = add2(add2(Mi[a][0], Mi[a][1]), Mi[a][2]);
                Ma[a] = make_float2(lanes(sr, wqx, wqy), lanes(si, wqx, wqy));
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    Tr = fma2(bc(mm[a][b]), Mr[a][b], Tr);
                    Ti = fma2(bc(mm[a][b]), Mi[a][b], Ti);
                }
            }
            const float2 s0r = add2(add2(M0r[0], M0r[1]), M0r[2]), s0i = add2(add2(M0i[0], M0i[1]), M0i[2]);
            M00 = make_float2(lanes(s0r, wqx, wqy), lanes(s0i, wqx, wqy));
            const float2 M0f = add2(M00, make_float2(ce.ri, 0.f));
            const float2 T = fma2(bc(-4.f / k2), M00, make_float2(lanes(Tr, wsx, wsy), lanes(Ti, wsx, wsy)));
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float2 u = fma2(bc(mm[a][2]), Mb[2], fma2(bc(mm[a][1]), Mb[1], mul2(bc(mm[a][0]), Mb[0])));
                const float2 Tu = sub2(T, u);
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const float2 v = fma2(bc(mm[2][b]), Ma[2], fma2(bc(mm[1][b]), Ma[1], mul2(bc(mm[0][b]), Ma[0])));
                    E[a][b] = fma2(bc(mm[a][b]), M0f, sub2(Tu, v));
                }
            }
        }
        {
            float2 Usr = bc(0.f), Usi = bc(0.f), Pa[3], Qa[3], X0[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                X0[a] = make_float2(lanes(X0r[a], wsx, wsy), lanes(X0i[a], wsx, wsy));
                const float2 sr = add2(add2(Xr[a][0], Xr[a][1]), Xr[a][2]), si = add2(add2(Xi[a][0], Xi[a][1]), Xi[a][2]);
                Qa[a] = make_float2(lanes(sr, wqx, wqy), lanes(si, wqx, wqy));
                float2 pr = mul2(bc(nB[0]), Xr[a][0]), pi = mul2(bc(nB[0]), Xi[a][0]);
                pr = fma2(bc(nB[2]), Xr[a][2], fma2(bc(nB[1]), Xr[a][1], pr));
                pi = fma2(bc(nB[2]), Xi[a][2], fma2(bc(nB[1]), Xi[a][1], pi));
                Pa[a] = make_float2(lanes(pr, wsx, wsy), lanes(pi, wsx, wsy));
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    Usr = fma2(bc(mm[a][b]), Xr[a][b], Usr);
                    Usi = fma2(bc(mm[a][b]), Xi[a][b], Usi);
                }
            }
            const float2 Us = make_float2(lanes(Usr, wsx, wsy), lanes(Usi, wsx, wsy));
            const float2 q0r = add2(add2(X0r[0], X0r[1]), X0r[2]), q0i = add2(add2(X0i[0], X0i[1]), X0i[2]);
            const float2 Q = make_float2(lanes(q0r, wqx, wqy), lanes(q0i, wqx, wqy));
            const float2 gr = add2(add2(Xgr[0], Xgr[1]), Xgr[2]), gi = add2(add2(Xgi[0], Xgi[1]), Xgi[2]);
            const float2 Qg = make_float2(lanes(gr, wqx, wqy), lanes(gi, wqx, wqy));
            const float2 pgr = fma2(bc(nB[2]), Xgr[2], fma2(bc(nB[1]), Xgr[1], mul2(bc(nB[0]), Xgr[0])));
            const float2 pgi = fma2(bc(nB[2]), Xgi[2], fma2(bc(nB[1]), Xgi[1], mul2(bc(nB[0]), Xgi[0])));
            const float2 Pg = make_float2(lanes(pgr, wsx, wsy), lanes(pgi, wsx, wsy));
            const float2 P = fma2(bc(nB[2]), X0[2], fma2(bc(nB[1]), X0[1], mul2(bc(nB[0]), X0[0])));
            const float2 Z = sub2(mul2(bc(nD), Q), P);
            float2 Za[3], Y[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) Za[a] = sub2(mul2(bc(nD), Qa[a]), Pa[a]);
#pragma unroll
            for (int b = 0; b < 3; ++b)
                Y[b] = fma2(bc(mm[2][b]), Za[2], fma2(bc(mm[1][b]), Za[1], mul2(bc(mm[0][b]), Za[0])));
            const float G[3][3] = {{AA[0], p7v.x, p7v.z}, {p7v.x, AA[1], p7v.y}, {p7v.z, p7v.y, AA[2]}};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float2 nDA = bc(-DA[a]);
                float2 R = fma2(nDA, P, Pg), Sm = fma2(nDA, Q, Qg);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    R = fma2(bc(-G[a][c]), Pa[c], R);
                    Sm = fma2(bc(-G[a][c]), Qa[c], Sm);
                }
                const float2 um = fma2(bc(mm[a][2]), X0[2], fma2(bc(mm[a][1]), X0[1], mul2(bc(mm[a][0]), X0[0])));
                const float2 du = sub2(Us, um);
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const float2 t = fma2(bc(nB[b] - nD), du, fma2(bc(-nB[b]), Sm, R));
                    H[a][b] = add2(t, fma2(bc(-mm[a][b]), Z, Y[b]));
                }
            }
        }
        const float hp[3] = {p4v.w, p5v.w, p6v.w};
        const int row[3] = {__float_as_int(p1v.w), __float_as_int(p2v.w), __float_as_int(p3v.w)};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float2* zr = reinterpret_cast<float2*>(m.z) + (int64_t)row[a] * m.pitch;
            const float ha = hp[a] * float(kInv4Pi);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                // jk E + H, times e^{-jkR_c}, and the charge term at the centroids
                const float re = fmaf(-k, E[a][b].y, H[a][b].x), im = fmaf(k, E[a][b].x, H[a][b].y), c = ha * hq[b];
                atomicAdd(zr + col[b], make_float2(fmaf(c, ce.br, c * fmaf(im, S, fmaf(re, C, ce.brl))),
                                                   fmaf(c, ce.bi, c * fmaf(-re, S, fmaf(im, C, ce.bil)))));
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// tiers 2 and 3: the three entries (m, e2), m = 0 .. 2, of one face pair -- nt shared test points,
// the NY x NY source points anchored at local edge e2.  Distances and phases as in tier 1, in
// units of 1/k: with y = B + r1 E1 + r2 E2 from the centroid, sigma takes three operations per
// evaluation.  Per test point the sums over the source points are S0 = sum G, and of G y and h y
// by the source's two barycentric coordinates; with the origin at the anchor,
// P = sum G y, H = sum h y the entry is
//   sum_i w_i [ (x_i - A_m) . (jk P_i - n x (H_i x x_i)) - (4j/k) S0_i ],
// whose vector is e1 E1 + e2 E2 + e3 x_i.  Bound: FMA pipe, 26 packed operations per two evaluations.
// ---------------------------------------------------------------------------------------
template <int NY>
__device__ __forceinline__ void shared_test_entries(const float* __restrict__ rp, const float* __restrict__ rq, int e2,
                                                    const float (*s_b)[4], int nt, const float4* s_s, float k,
                                                    float kth, float ktl, float wsum, int64_t pitch,
                                                    float* __restrict__ z) {
    constexpr int NS = NY * NY, NP = (NS + 1) / 2;  // an odd count is padded with a zero weight
    const float4* r4p = reinterpret_cast<const float4*>(rp);
    const float4* r4q = reinterpret_cast<const float4*>(rq);
    const float4 cp = r4p[0], cq = r4q[0];
    const float dx = cp.x - cq.x, dy = cp.y - cq.y, dz = cp.z - cq.z;
    // charge term at the centroids: 4/k / R, the sums below being over G / k
    const Centre ce = pair_centre(cp, r4p[1], cq, r4q[1], dx, dy, dz, kth, ktl, 4.f * wsum / (k * k));
    const float k2 = k * k, Rc2 = k2 * ce.r2, R0 = k * ce.r, hc = 0.5f * ce.ri / k;
    const float2 G0 = bc(-ce.ri / k);
    const int b1 = e2 == 2 ? 0 : e2 + 1, b2 = e2 == 0 ? 2 : e2 - 1;
    const V3<float> b0 = v3<float>(rq[kA + 4 * e2], rq[kA + 4 * e2 + 1], rq[kA + 4 * e2 + 2]);
    const V3<float> E1 = v3<float>(rq[kA + 4 * b1], rq[kA + 4 * b1 + 1], rq[kA + 4 * b1 + 2]) - b0;
    const V3<float> E2 = v3<float>(rq[kA + 4 * b2], rq[kA + 4 * b2 + 1], rq[kA + 4 * b2 + 2]) - b0;
    const V3<float> D = v3<float>(dx, dy, dz), o = D - b0;  // x' + o: the test point from the anchor
    const V3<float> n = v3<float>(rp[kN], rp[kN + 1], rp[kN + 2]);
    float2 wn[NP];  // -k^2 (|y|^2 - 2 D.y)
#pragma unroll
    for (int j = 0; j < 2 * NP; ++j) {
        const float4 r = s_s[j];
        const V3<float> y = b0 + r.x * E1 + r.y * E2;
        (reinterpret_cast<float*>(&wn[j / 2]) + (j & 1))[0] = k2 * (2.f * dot(D, y) - dot(y, y));
    }
    const float nB1 = dot(n, E1), nB2 = dot(n, E2);
    V3<float> er = v3<float>(0.f, 0.f, 0.f), ei = v3<float>(0.f, 0.f, 0.f);  // sum w e3 x
    float f1r = 0.f, f1i = 0.f, f2r = 0.f, f2i = 0.f;                         // sum w e1, w e2
    float t0r = 0.f, t0i = 0.f;                                               // sum w x.E - (4j/k) w S0
#pragma unroll 1
    for (int i = 0; i < nt; ++i) {
        V3<float> xc = v3<float>(0.f, 0.f, 0.f);
#pragma unroll
        for (int a = 0; a < 3; ++a) xc = xc + s_b[i][a] * v3<float>(rp[kA + 4 * a], rp[kA + 4 * a + 1], rp[kA + 4 * a + 2]);
        const V3<float> x = xc + o;
        const float2 U = bc(k2 * (2.f * dot(xc, b0 - D) - dot(xc, xc))), X1 = bc(2.f * k2 * dot(xc, E1)),
                     X2 = bc(2.f * k2 * dot(xc, E2));
        float2 s0r = bc(0.f), s0i = bc(0.f), p1r = bc(0.f), p1i = bc(0.f), p2r = bc(0.f), p2i = bc(0.f), h1r = bc(0.f),
               h1i = bc(0.f), h2r = bc(0.f), h2i = bc(0.f);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const float4 ra = s_s[2 * j], rb = s_s[2 * j + 1];  // (r1, r2, weight)
            const float2 c1 = make_float2(ra.x, rb.x), c2 = make_float2(ra.y, rb.y), w = make_float2(ra.z, rb.z);
            const float2 ns = fma2(c1, X1, fma2(c2, X2, add2(wn[j], U)));  // -k^2 sigma
            const float2 r2 = sub2(bc(Rc2), ns);
            float2 rinv;
            rinv.x = rsqrtf(r2.x);
            rinv.y = rsqrtf(r2.y);
            const float2 kR = mul2(r2, rinv), d0 = sub2(kR, bc(R0));
            const float2 th = mul2(fma2(d0, d0, ns), bc(hc));  // -k (R - R_c)
            float2 sn, cs;
            __sincosf(th.x, &sn.x, &cs.x);
            __sincosf(th.y, &sn.y, &cs.y);
            const float2 g = mul2(w, rinv), gr = mul2(g, cs), gi = mul2(g, sn), ri2 = mul2(rinv, rinv);
            const float2 hr = mul2(sub2(gr, mul2(gi, kR)), ri2), hi = mul2(fma2(gr, kR, gi), ri2);
            s0r = add2(s0r, fma2(w, G0, gr));  // of G - 1/R_c, as in tier 1
            s0i = add2(s0i, gi);
            p1r = fma2(c1, gr, p1r);
            p1i = fma2(c1, gi, p1i);
            p2r = fma2(c2, gr, p2r);
            p2i = fma2(c2, gi, p2i);
            h1r = fma2(c1, hr, h1r);
            h1i = fma2(c1, hi, h1i);
            h2r = fma2(c2, hr, h2r);
            h2i = fma2(c2, hi, h2i);
        }
        const float w = s_b[i][3], wk = w * k, wk2 = w * k2, nx = dot(n, x), xx = dot(x, x), x1 = dot(x, E1), x2 = dot(x, E2);
        const float u1r = h1r.x + h1r.y, u1i = h1i.x + h1i.y, u2r = h2r.x + h2r.y, u2i = h2i.x + h2i.y;
        // E = e1 E1 + e2 E2 + e3 x:  e1 = jk p1 - k^2 h1 (n.x),  e3 = k^2 (h1 n.E1 + h2 n.E2)
        const float e1r = -fmaf(wk2 * nx, u1r, wk * (p1i.x + p1i.y)), e1i = fmaf(-wk2 * nx, u1i, wk * (p1r.x + p1r.y));
        const float e2r = -fmaf(wk2 * nx, u2r, wk * (p2i.x + p2i.y)), e2i = fmaf(-wk2 * nx, u2i, wk * (p2r.x + p2r.y));
        const float e3r = wk2 * fmaf(nB1, u1r, nB2 * u2r), e3i = wk2 * fmaf(nB1, u1i, nB2 * u2i);
        f1r += e1r;
        f1i += e1i;
        f2r += e2r;
        f2i += e2i;
        er = er + e3r * x;
        ei = ei + e3i * x;
        const float q = 4.f * w / k;
        t0r += fmaf(x1, e1r, fmaf(x2, e2r, fmaf(xx, e3r, q * (s0i.x + s0i.y))));
        t0i += fmaf(x1, e1i, fmaf(x2, e2i, fmaf(xx, e3i, -q * (s0r.x + s0r.y))));
    }
    er = er + f1r * E1 + f2r * E2;
    ei = ei + f1i * E1 + f2i * E2;
    const float sc = 2.f * k * rq[kHalf + 4 * e2];  // the sums lack a factor k (1/R -> 1/(kR))
    const int64_t col = __float_as_int(rq[kEdge + 4 * e2]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float c = sc * rp[kHalf + 4 * a];
        const V3<float> A = v3<float>(rp[kA + 4 * a], rp[kA + 4 * a + 1], rp[kA + 4 * a + 2]) + o;
        const float re = t0r - dot(A, er), im = t0i - dot(A, ei);
        const int64_t row = __float_as_int(rp[kEdge + 4 * a]);
        atomicAdd(reinterpret_cast<float2*>(z) + row * pitch + col,
                  make_float2(fmaf(c, ce.br, c * fmaf(im, ce.s, fmaf(re, ce.c, ce.brl))),
                              fmaf(c, ce.bi, c * fmaf(-re, ce.s, fmaf(im, ce.c, ce.bil)))));
    }
}

// The pairs outside tier 1 of a block's tile of tp test x tq source faces (at most kTilePairs): sorted
// into lists in shared memory, then worked off by all threads -- CLOSE: tier 4, one (pair, e1, e2)
// entry per thread; else tiers 2 and 3, (pair, e2) items -- so that the few close pairs of a tile
// leave no lanes idle.  A tile without such pairs ends after the tests.  Two launches: in one
// kernel the two bodies spilled at 128 registers.
constexpr int kTilePairs = 1024;

template <int NX, int NY, bool CLOSE>
__global__ void __launch_bounds__(128, NX <= 4 ? 4 : CLOSE ? 2 : 3) close_pairs_kernel(const TierArgs args, int tp, int tq) {
    __shared__ float4 s_t[NX * NX], s_s[NY * NY], s_src[(NY * NY + 1) / 2 * 2];
    __shared__ float s_b[19][4];
    __shared__ float4 s_p[256], s_q[256];
    __shared__ uint16_t s_list[CLOSE ? 1 : 2][kTilePairs];
    __shared__ int s_n[2], s_rho;
    const MeshRef m = find_mesh(args);
    const int64_t col_tiles = (m.nf + tq - 1) / tq;
    const int64_t p0 = (m.block / col_tiles) * tp, q0 = (m.block % col_tiles) * tq;
    const int np = (int)min((int64_t)tp, m.nf - p0), nq = (int)min((int64_t)tq, m.nf - q0);
    const float4* rec4 = reinterpret_cast<const float4*>(args.rec) + (kRec / 4) * m.f0;
    if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
    // the tile's largest rho^2 (a NaN wins: as bits it is above every finite value)
    if (threadIdx.x == 0) s_rho = 0;
    __syncthreads();
    int top = 0;
    for (int i = threadIdx.x; i < np + nq; i += 128) {
        const float4 r = __ldg(rec4 + (kRec / 4) * (i < np ? p0 + i : q0 + (i - np)));
        (i < np ? s_p[i] : s_q[i - np]) = r;
        top = max(top, __float_as_int(r.w));
    }
    atomicMax(&s_rho, top);
    const float k = (float)m.k, k2 = k * k;
    __syncthreads();
    // tq is a power of two up to 128: a thread keeps one source face and steps through the test faces
    const float limit = CLOSE || NX > 3 ? far_limit(__int_as_float(s_rho), k2) : __int_as_float(0x7f800000);
    const int b = threadIdx.x & (tq - 1);
    // (tier 3 ends at k rho = 0.8: a larger face has nothing for the launch of tiers 2 and 3)
    if (b < nq && (CLOSE || k2 * s_q[b].w <= 0.65f)) {
        const float4 q = s_q[b];
        for (int a = threadIdx.x / tq; a < np; a += 128 / tq) {
            const float4 p = s_p[a];
            const float r2 = centre_dist2(p.x - q.x, p.y - q.y, p.z - q.z);
            if (r2 >= limit) continue;
            const int t = pair_tier<NX>(r2, p.w, q.w, k2);
            if (CLOSE ? t == 4 : (t == 2 || t == 3)) {
                const int l = CLOSE ? 0 : t - 2;
                s_list[l][atomicAdd(&s_n[l], 1)] = (uint16_t)(a * tq + b);
            }
        }
    }
    __syncthreads();
    const int n0 = s_n[0], n1 = s_n[1];
    if (n0 + n1 == 0) return;
    stage_rules<NX, NY>(args.gpx, args.gwx, args.gpy, args.gwy, s_t, s_s);
    if constexpr (!CLOSE)
        if (threadIdx.x < 76) (&s_b[0][0])[threadIdx.x] = (&c_test[0][0])[threadIdx.x];
    __syncthreads();
    const float* rec = args.rec + kRec * m.f0;
    if constexpr (CLOSE) {
        // e1 slowest: neighbouring threads have the same test corner and the corners of one source face
        const int per = 3 * n0;
        if constexpr (NX == 3) {
            // short entries: where the list gives every thread enough, all three by one thread, whose source points
            // serve them all (5120 faces, k 10: 10.65 -> 10.44 ms; gaussQR 4 and 5: no gain)
            const int span = n0 >= 512 ? 3 : 1;
            for (int i = threadIdx.x; i < (span == 3 ? per : 3 * per); i += 128) {
                const int first = (i >= per) + (i >= 2 * per), r = i - first * per, c = s_list[0][r / 3], e2 = r % 3;
                const int64_t p = p0 + c / tq, q = q0 + (c & (tq - 1));
                const int64_t col = __float_as_int(rec[kRec * q + kEdge + 4 * e2]);
#pragma unroll 1
                for (int e1 = first; e1 < first + span; ++e1) {
                    float re, im;
                    mom_entry_fast<NX, NY>(args.verts, args.faces, args.areas, args.normals, s_t, s_s, k, m.f0 + p, e1,
                                           m.f0 + q, e2, &re, &im);
                    const int64_t row = __float_as_int(rec[kRec * p + kEdge + 4 * e1]);
                    atomicAdd(reinterpret_cast<float2*>(m.z) + row * m.pitch + col, make_float2(re, im));
                }
            }
        } else {
            for (int i = threadIdx.x; i < 3 * per; i += 128) {
                const int e1 = (i >= per) + (i >= 2 * per), r = i - e1 * per, c = s_list[0][r / 3], e2 = r % 3;
                const int64_t p = p0 + c / tq, q = q0 + (c & (tq - 1));
                float re, im;
                mom_entry_fast<NX, NY>(args.verts, args.faces, args.areas, args.normals, s_t, s_s, k, m.f0 + p, e1,
                                       m.f0 + q, e2, &re, &im);
                const int64_t row = __float_as_int(rec[kRec * p + kEdge + 4 * e1]);
                const int64_t col = __float_as_int(rec[kRec * q + kEdge + 4 * e2]);
                atomicAdd(reinterpret_cast<float2*>(m.z) + row * m.pitch + col, make_float2(re, im));
            }
        }
    } else {
        if (threadIdx.x < (NY * NY + 1) / 2 * 2) {  // barycentric form of the source rule: (r3 - r4, r4, weight)
            const float4 r = threadIdx.x < NY * NY ? s_s[threadIdx.x] : make_float4(0.5f, 0.25f, 0.f, 0.f);
            s_src[threadIdx.x] = make_float4(r.x - r.y, r.y, r.z, 0.f);
        }
        __syncthreads();
        float wsum = 0.f;
        for (int j = 0; j < NY * NY; ++j) wsum += s_s[j].z;
        const double kt = m.k * kInv2Pi;
        const float kth = (float)kt, ktl = (float)(kt - (double)kth);
#pragma unroll 1
        for (int t = 1; t >= 0; --t) {
            const int n = 3 * (t ? n1 : n0);
            for (int i = threadIdx.x; i < n; i += 128) {
                const int c = s_list[t][i / 3];
                shared_test_entries<NY>(rec + kRec * (p0 + c / tq), rec + kRec * (q0 + (c & (tq - 1))), i % 3,
                                        t ? s_b + 7 : s_b, t ? 12 : 7, s_src, k, kth, ktl, wsum, m.pitch, m.z);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// the 7-point-rule EFIE (mom_sym.cu) on separated pairs, in the same arithmetic: the rule's points
// are the centroid and two orbits s A_a, so all 49 evaluations come from the pair's scalar products.
// The operator is symmetric and both faces carry the same rule: a pair is evaluated once, p < q, and
// its entries belong at (m, n) and (n, m).  The terms of kEdgeRows test faces are summed per thread in
// shared memory by distinct test edge (8 faces of the sphere have 16 to 18 of 24), so that about 2 edges
// x 3 of a face remain of 9 reductions per ordered pair: a reduction costs a cycle of its SM, which
// with 9 bounds the whole at 13 ms for 20480 faces.  Into a matrix of its own (not one that is added
// to) the kernel sums above the diagonal only, half the reductions, and mirror_kernel copies.
// Measured (GB300), 20480 faces: 22.35 (every ordered pair, row by row) -> 10.05 ms + 1.08 ms for
// the mirror, 0.49 instead of 0.96 for the zeros, 0.5 ms for the pairs left; on both sides 13.66.  (rows, slots, blocks per
// SM), both sides: 8/16/4 best of 4/8/5 15.4, 8/16/3 14.1, 12/22/3 14.1, 16/28/2 14.8 ms.  Bound: FMA pipe.  Entry errors
// against 64 bits 0.45 .. 0.65 of the row kernel's beyond 4 edges.
// Pairs with |D| >= 2 (rho_p + rho_q) and k (rho_p + rho_q) <= 0.6 (the phases' polynomials); the
// others are left to mom_sym_regular_rows_kernel, which applies the same test.  It takes all of them (sym_form_kernel):
//   * below 2400 faces, whose grid leaves the chip half empty: rows / pairs 121 / 166 us at 1280, 294 / 299 .. 310 at
//     2112, 538 / 428 .. 457 at 2960;
//   * where consecutive faces do not share edges, every term then a reduction: faces in any order 1.51 / 1.57 ms at 5120, 23.5 /
//     33.3 at 20480; in runs of two 23.5 / 23.1, of four 23.4 / 14.6; on both sides, where a transposed term's reductions
//     go down a column, also where neighbouring faces' edges are not numbered alike (groups of eight ids, face_order.cuh):
//     subdivided sphere (33) 23.3 / 11.9, in runs of eight (48) 23.3 / 19.2, of four (57) 23.4 / 25.3, strips across the ids
//     of 12798 faces (61) 8.8 / 11.8;
//   * where most faces are too large for the phases: k 10, 5120 faces, 1.50 / 1.75 ms.
// ---------------------------------------------------------------------------------------
constexpr int kEdgeRows = 8, kEdgeSlots = 16;
constexpr int kEdgeSumBytes = 3 * kEdgeSlots * 128 * (int)sizeof(float2);

struct EdgeSlots {
    int id[3 * kEdgeRows], first[3 * kEdgeRows], edge[kEdgeSlots], n;
    uint8_t slot[4 * kEdgeRows];
};

// e at (m, n) and (n, m); UPPER: at the one of them above the diagonal, for mirror_kernel to copy
template <bool UPPER>
__device__ __forceinline__ void add_both(float2* __restrict__ z, int64_t m, int64_t n, int64_t n_edges, float2 e) {
    atomicAdd(z + (UPPER ? min(m, n) : m) * n_edges + (UPPER ? max(m, n) : n), e);
    if (!UPPER || m == n) atomicAdd(z + n * n_edges + m, e);
}

// *form = 1 where sym_pairs_kernel pays (see above), from samples of the edge ids (face_order.cuh) and of the records.
constexpr int kFormThreads = 512;
__global__ void __launch_bounds__(kFormThreads) sym_form_kernel(const float* __restrict__ rec, const int32_t* __restrict__ fei,
                                                                int64_t nf, float k, int max_sectors,
                                                                int* __restrict__ form) {
    const FaceOrder o = face_order(fei, nf);  // 30 edges of ten faces in any order, 21 to 24 neighbour by neighbour
    const float rho2 = __ldg(rec + kRec * (nf * threadIdx.x / kFormThreads) + kRho2);
    const int small = __syncthreads_count(2.f * k * sqrtf(rho2) <= 0.6f);
    if (threadIdx.x == 0) *form = o.ids <= 25 && o.sectors <= max_sectors && 2 * small >= kFormThreads;
}

constexpr int kMirror = 32;  // tile of mirror_kernel

// Zeros from the diagonal's tiles to the right, a row per block.
__global__ void __launch_bounds__(256) zero_upper_kernel(float2* __restrict__ z, int64_t n) {
    float2* row = z + (int64_t)blockIdx.x * n;
    for (int64_t c = (int64_t)blockIdx.x / kMirror * kMirror + threadIdx.x; c < n; c += 256) row[c] = make_float2(0.f, 0.f);
}

// z[n, m] = z[m, n] for m < n (zero where sym_pairs_kernel summed nothing), a tile above the diagonal per block.  Tile rows y and t - 1 - y together
// have t + 1 tiles: the grid is (t + 1) x ceil(t / 2).
// Bound: HBM.  A thread's four loads are in flight together: 30720 edges (7.5 GB) 1.08 ms, 6.99 TB/s, against 1.47 one
// after the other; tiles of 64 1.27.
__global__ void __launch_bounds__(256) mirror_kernel(float2* __restrict__ z, int64_t n, int t, const int* __restrict__ form) {
    __shared__ float2 s[kMirror][kMirror + 1];
    const int x = blockIdx.x, y = blockIdx.y;
    if (x <= y && 2 * y == t - 1) return;  // the middle row pairs with itself
    const int64_t i0 = kMirror * (int64_t)(x > y ? y : t - 1 - y), j0 = kMirror * (int64_t)(x > y ? x - 1 : t - 1 - x);
    constexpr int kRows = 256 / kMirror;
    const int c = threadIdx.x % kMirror, r0 = threadIdx.x / kMirror;
    const bool sums = *form != 0;
#pragma unroll
    for (int q = 0; q < kMirror / kRows; ++q) {
        const int r = r0 + kRows * q;
        if (i0 + r < n && j0 + c < n) s[r][c] = sums ? z[(i0 + r) * n + j0 + c] : make_float2(0.f, 0.f);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kMirror / kRows; ++q) {
        const int r = r0 + kRows * q;
        if (j0 + r < n && i0 + c < n && j0 + r > i0 + c) z[(j0 + r) * n + i0 + c] = s[c][r];
    }
}

template <bool UPPER>
__global__ void __launch_bounds__(128, 4)
    sym_pairs_kernel(const float* __restrict__ rec, int64_t nf, int64_t n_edges, double kd, const int* __restrict__ form,
                     float* __restrict__ z) {
    if (!*form) return;
    constexpr float s1 = (float)(1.0 - 3.0 * 0.10128650732345634), s2 = (float)(1.0 - 3.0 * 0.47014206410511509);
    constexpr float w0 = 0.225f, w1 = 0.12593918054482715f, w2 = 0.13239415278850619f;
    __shared__ float4 s_rec[kEdgeRows * (kRec / 4)];
    __shared__ EdgeSlots s_e;
    extern __shared__ float2 s_sum[];  // [kEdgeSlots][3][128]
    const int64_t p0 = (int64_t)blockIdx.x * kEdgeRows, q0i = (int64_t)blockIdx.y * 128, q = q0i + threadIdx.x;
    if (q0i + 127 <= p0) return;  // no pair p < q in the tile
    const int np = (int)min((int64_t)kEdgeRows, nf - p0), t = threadIdx.x;
    const float4* rec4 = reinterpret_cast<const float4*>(rec);
    for (int i = t; i < np * (kRec / 4); i += 128) s_rec[i] = __ldg(rec4 + (kRec / 4) * p0 + i);
    if (t < 3 * np) s_e.id[t] = __float_as_int(__ldg(rec + kRec * (p0 + t / 3) + kEdge + 4 * (t % 3)));
    __syncthreads();
    int first = 0;
    if (t < 3 * np) {
        while (s_e.id[first] != s_e.id[t]) ++first;
        s_e.first[t] = first == t;
    }
    __syncthreads();
    if (t < 3 * np) {
        int rank = 0;
        for (int j = 0; j < first; ++j) rank += s_e.first[j];
        s_e.slot[4 * (t / 3) + t % 3] = (uint8_t)rank;
        if (rank < kEdgeSlots) s_e.edge[rank] = s_e.id[t];
    }
    if (t == 0) {
        int n = 0;
        for (int j = 0; j < 3 * np; ++j) n += s_e.first[j];
        s_e.n = min(n, kEdgeSlots);
    }
    __syncthreads();
    const int nslot = s_e.n;
    float2* mine = s_sum + t;
    for (int u = 0; u < 3 * nslot; ++u) mine[u * 128] = bc(0.f);
    if (q >= nf) return;
    const float4* rq = rec4 + (kRec / 4) * q;
    const float4 q0 = __ldg(rq), q1 = __ldg(rq + 1), q2 = __ldg(rq + 2), q3 = __ldg(rq + 3), q4 = __ldg(rq + 4),
                 q5 = __ldg(rq + 5), q6 = __ldg(rq + 6);
    const float B[3][3] = {{q2.x, q2.y, q2.z}, {q3.x, q3.y, q3.z}, {q4.x, q4.y, q4.z}};
    const float BB[3] = {q6.x, q6.y, q6.z}, hq[3] = {q4.w, q5.w, q6.w};
    const int col[3] = {__float_as_int(q1.w), __float_as_int(q2.w), __float_as_int(q3.w)};
    const float k = (float)kd, four_k = 4.f / k;
    const double kt = kd * kInv2Pi;
    const float kth = (float)kt, ktl = (float)(kt - (double)kth);
    float2* z2 = reinterpret_cast<float2*>(z);
#pragma unroll 1
    for (int i = 0; i < np && p0 + i < q; ++i) {
        const float4* rp = s_rec + (kRec / 4) * i;
        const float4 p0v = rp[0];
        const float dx = p0v.x - q0.x, dy = p0v.y - q0.y, dz = p0v.z - q0.z;
        if (!sym_pair_far(centre_dist2(dx, dy, dz), p0v.w, q0.w, k)) continue;
        const float4 p1v = rp[1], p2v = rp[2], p3v = rp[3], p4v = rp[4], p5v = rp[5], p6v = rp[6];
        const float A[3][3] = {{p2v.x, p2v.y, p2v.z}, {p3v.x, p3v.y, p3v.z}, {p4v.x, p4v.y, p4v.z}};
        const float AA[3] = {p6v.x, p6v.y, p6v.z};
        const Centre ce = pair_centre(p0v, p1v, q0, q1, dx, dy, dz, kth, ktl, four_k);
        const float Rc2 = ce.r2, R0 = ce.r, kp = k * (0.5f * ce.ri);
        float mm[3][3], DA[3];
        float2 V[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            DA[a] = fmaf(dz, A[a][2], fmaf(dy, A[a][1], dx * A[a][0]));
            const float DB = fmaf(dz, B[a][2], fmaf(dy, B[a][1], dx * B[a][0]));
            V[a] = make_float2(s1 * (2.f * DB - s1 * BB[a]), s2 * (2.f * DB - s2 * BB[a]));
#pragma unroll
            for (int b = 0; b < 3; ++b)
                mm[a][b] = fmaf(A[a][2], B[b][2], fmaf(A[a][1], B[b][1], A[a][0] * B[b][0]));
        }
        // (G - 1/R_c) e^{jkR_c} at squared distance Rc2 - ns
        auto green = [&](float2 ns, float2& gr, float2& gi) {
            const float2 r2 = sub2(bc(Rc2), ns);
            float2 rinv;
            rinv.x = rsqrtf(r2.x);
            rinv.y = rsqrtf(r2.y);
            const float2 d0 = sub2(mul2(r2, rinv), bc(R0));
            const float2 th = mul2(fma2(d0, d0, ns), bc(kp)), x2 = mul2(th, th);
            const float2 sn = mul2(th, fma2(x2, fma2(x2, bc(SB), bc(SA)), bc(1.f)));
            const float2 cs = fma2(x2, fma2(x2, fma2(x2, bc(CC), bc(CB)), bc(CA)), bc(1.f));
            gr = sub2(mul2(rinv, cs), bc(ce.ri));
            gi = mul2(rinv, sn);
        };
        float2 M0r[3], M0i[3], Ma[3], Mb[3], M00;
        float2 Tr = bc(0.f), Ti = bc(0.f);
#pragma unroll
        for (int b = 0; b < 3; ++b) {  // p's centroid
            float2 gr, gi;
            green(V[b], gr, gi);
            M0r[b] = mul2(bc(w0), gr);
            M0i[b] = mul2(bc(w0), gi);
        }
        float c0r = 0.f, c0i = 0.f;
        // corner by corner of p, its sums folded at once (fewer registers)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float2 Mr[3], Mi[3];
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const float s = o ? s2 : s1, w = o ? w2 : w1;
                const float2 W = bc(w), WS = bc(w * s), K2 = make_float2(2.f * s * s1, 2.f * s * s2);
                const float2 U = bc(-s * fmaf(s, AA[a], 2.f * DA[a]));
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    float2 gr, gi;
                    green(fma2(bc(mm[a][b]), K2, add2(U, V[b])), gr, gi);
                    Mr[b] = o ? fma2(WS, gr, Mr[b]) : mul2(WS, gr);
                    Mi[b] = o ? fma2(WS, gi, Mi[b]) : mul2(WS, gi);
                    M0r[b] = fma2(W, gr, M0r[b]);
                    M0i[b] = fma2(W, gi, M0i[b]);
                }
            }
            // q's centroid: lanes p's two orbits
            float2 cr, ci;
            green(make_float2(-s1 * (2.f * DA[a] + s1 * AA[a]), -s2 * (2.f * DA[a] + s2 * AA[a])), cr, ci);
            c0r += lanes(cr, w1, w2);
            c0i += lanes(ci, w1, w2);
            const float2 sr = add2(add2(Mr[0], Mr[1]), Mr[2]), si = add2(add2(Mi[0], Mi[1]), Mi[2]);
            Ma[a] = make_float2(fmaf(w0, lanes(cr, w1 * s1, w2 * s2), lanes(sr, w1, w2)),
                                fmaf(w0, lanes(ci, w1 * s1, w2 * s2), lanes(si, w1, w2)));
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                Tr = fma2(bc(mm[a][b]), Mr[b], Tr);
                Ti = fma2(bc(mm[a][b]), Mi[b], Ti);
            }
        }
        {
            const float2 s0r = add2(add2(M0r[0], M0r[1]), M0r[2]), s0i = add2(add2(M0i[0], M0i[1]), M0i[2]);
            M00 = make_float2(fmaf(w0, c0r, lanes(s0r, w1, w2)), fmaf(w0, c0i, lanes(s0i, w1, w2)));
        }
#pragma unroll
        for (int b = 0; b < 3; ++b)
            Mb[b] = make_float2(lanes(M0r[b], w1 * s1, w2 * s2), lanes(M0i[b], w1 * s1, w2 * s2));
        const float2 M0f = add2(M00, make_float2(ce.ri, 0.f));
        const float2 T = fma2(bc(-four_k / k), M00,
                              make_float2(lanes(Tr, w1 * s1, w2 * s2), lanes(Ti, w1 * s1, w2 * s2)));
        float2 v[3];
#pragma unroll
        for (int b = 0; b < 3; ++b)
            v[b] = fma2(bc(mm[2][b]), Ma[2], fma2(bc(mm[1][b]), Ma[1], mul2(bc(mm[0][b]), Ma[0])));
        const float hp[3] = {p4v.w, p5v.w, p6v.w};
        const uint32_t slots = *reinterpret_cast<const uint32_t*>(s_e.slot + 4 * i);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float2 u = fma2(bc(mm[a][2]), Mb[2], fma2(bc(mm[a][1]), Mb[1], mul2(bc(mm[a][0]), Mb[0])));
            const float2 Tu = sub2(T, u);
            const float ha = hp[a] * float(kInv4Pi);
            const int slot = (slots >> (8 * a)) & 255;
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const float2 E = fma2(bc(mm[a][b]), M0f, sub2(Tu, v[b]));
                const float re = -k * E.y, im = k * E.x, c = ha * hq[b];
                const float2 e = make_float2(fmaf(c, ce.br, c * fmaf(im, ce.s, fmaf(re, ce.c, ce.brl))),
                                             fmaf(c, ce.bi, c * fmaf(-re, ce.s, fmaf(im, ce.c, ce.bil))));
                if (slot < kEdgeSlots) {
                    float2* d = mine + (3 * slot + b) * 128;
                    *d = add2(*d, e);
                } else {
                    add_both<UPPER>(z2, s_e.id[3 * i + a], col[b], n_edges, e);
                }
            }
        }
    }
    for (int u = 0; u < nslot; ++u) {
        const int64_t m = s_e.edge[u];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const float2 e = mine[(3 * u + b) * 128];
            if (e.x != 0.f || e.y != 0.f) add_both<UPPER>(z2, m, col[b], n_edges, e);
        }
    }
}

}  // namespace

// Tile sizes for that many (test face, source face) pairs in a launch, over all its meshes.  Tier 1's test faces per
// block (its per-thread source set-up is amortised over them) matter little: 4 to 32 of them within 2 % of the call at 1280
// faces (the fewer the better), 8 / 16 / 32 3.40 / 3.35 / 3.36 ms at 5120, 35.0 / 34.4 / 34.3 at 20480.  The close pairs' tiles hold
// 1024 pairs on large meshes, fewer on small ones, so that the last wave is a small part of the time; 14 x 16 pairs are 2016
// entries, 15.75 rounds of 128 threads.  Measured, us, gaussQR 4, tp x tq 16x64 / 8x64 / 14x16 / 4x32 / 4x16 / 7x2:
// 3 meshes of 80 faces 314 / 172 / - / 82 / 57 / 59; one of 320, k 1, 370 / 268 / 192 / 176 / 151 / 200; 64 of 80 838 /
// 698 / - / 586 / 571 / 690; one of 1280, k 30, 2115 / 2090 / 2008 / 2025 / 2089 / 2351; 50 of 320 3788 / 3695 / - / 3981 /
// 4415 / 8230; one of 5120, k 10, gaussQR 3, 10.36 / 10.43 ms, 8x32 11.02.
void mom_tier_tiles(int64_t pairs, int* rows, int* tp, int* tq) {
    *rows = pairs >= 5000 * 5000 ? 32 : 8;
    const double per_block = (double)pairs / (kSms * 4 * 8);  // were there 8 times the resident blocks (4 an SM)
    *tp = per_block >= 4096 ? 16 : per_block >= 1024 ? 8 : per_block >= 200 ? 14 : per_block >= 3 ? 4 : 7;
    *tq = per_block >= 1024 ? 64 : per_block >= 200 ? 16 : per_block >= 40 ? 32 : per_block >= 3 ? 16 : 2;
}

int64_t mom_tier_blocks(int64_t nf, int64_t tp, int64_t tq) { return ((nf + tp - 1) / tp) * ((nf + tq - 1) / tq); }

template <int NX, int NY>
static int launch_tiers(TierArgs a, int64_t far_blocks, int64_t close_blocks, int rows, int tp, int tq,
                        const int64_t* far_off, const int64_t* close_off, cudaStream_t s) {
    if (far_blocks > 0x7fffffffLL || close_blocks > 0x7fffffffLL)
        return set_error(MB_ERR_SIZE, "mesh too large for one launch");
    a.boff = close_off;
    close_pairs_kernel<NX, NY, true><<<(unsigned)close_blocks, 128, 0, s>>>(a, tp, tq);
    close_pairs_kernel<NX, NY, false><<<(unsigned)close_blocks, 128, 0, s>>>(a, tp, tq);
    if (NX > 3) {
        a.boff = far_off;
        far_pairs_kernel<NX><<<(unsigned)far_blocks, 128, 0, s>>>(a, rows);
    }
    return check_launch("mom tiers");
}

static int tier_records(const float* verts, const int32_t* faces, const float* normals, const int32_t* fei, int64_t nf,
                        const float* gpx, const float* gwx, int nx, const float* gpy, const float* gwy, int ny,
                        float* rec, cudaStream_t s) {
    face_record_kernel<<<(unsigned)((nf + 127) / 128), 128, 0, s>>>(verts, faces, normals, fei, nf, gpx, gwx, nx, gpy,
                                                                    gwy, ny, rec);
    return check_launch("face records");
}

bool mom_tier_rule(int nx, int ny) { return nx >= 3 && nx <= 5 && ny == nx - 1; }

#define MB_TIERS(...)                                                    \
    (nx == 4 ? launch_tiers<4, 3>(__VA_ARGS__) : nx == 3 ? launch_tiers<3, 2>(__VA_ARGS__) : launch_tiers<5, 4>(__VA_ARGS__))

int launch_mom_tiers(const float* verts, const int32_t* faces, int64_t nf, const float* areas, const float* normals,
                     const int32_t* fei, int64_t n_edges, const float* gpx, const float* gwx, int nx, const float* gpy,
                     const float* gwy, int ny, double k, float* rec, float* z, cudaStream_t s) {
    if (nf <= 0) return MB_OK;
    if (int rc = tier_records(verts, faces, normals, fei, nf, gpx, gwx, nx, gpy, gwy, ny, rec, s)) return rc;
    int rows, tp, tq;
    mom_tier_tiles(nf * nf, &rows, &tp, &tq);
    const TierArgs a{verts, faces, areas, normals, rec, gpx, gwx, gpy, gwy, nullptr, nullptr, nullptr, 0, nf, n_edges, k, z};
    return MB_TIERS(a, mom_tier_blocks(nf, rows, 128), mom_tier_blocks(nf, tp, tq), rows, tp, tq, nullptr, nullptr, s);
}

int launch_mom_tiers_batched(const float* verts, const int32_t* faces, int64_t total_faces, const float* areas,
                             const float* normals, const int32_t* fei, const int64_t* desc, const int64_t* far_off,
                             int64_t far_blocks, const int64_t* close_off, int64_t close_blocks, int rows, int tp, int tq,
                             const double* ks, int n_mesh, const float* gpx, const float* gwx, int nx, const float* gpy,
                             const float* gwy, int ny, float* rec, float* z, cudaStream_t s) {
    if (total_faces <= 0) return MB_OK;
    if (int rc = tier_records(verts, faces, normals, fei, total_faces, gpx, gwx, nx, gpy, gwy, ny, rec, s)) return rc;
    const TierArgs a{verts, faces, areas, normals, rec, gpx, gwx, gpy, gwy, desc, nullptr, ks, n_mesh, 0, 0, 0.0, z};
    return MB_TIERS(a, far_blocks, close_blocks, rows, tp, tq, far_off, close_off, s);
}

// The separated pairs of the 7-point-rule EFIE over the whole mesh: records, sym_pairs_kernel, then the
// pairs it leaves (mom_sym.cu).  Added to z, or, with overwrite, the whole of z.
int launch_mom_sym_rest(const float* verts, const int32_t* faces, const int32_t* fei, int64_t n_edges, double k, int64_t nf,
                        const float* rec, const int* form, float* z, cudaStream_t s);
template <typename T>
int launch_mom_sym_regular(const T* verts, const int32_t* faces, const int32_t* fei, int64_t n_edges, double k, int64_t nf,
                           int64_t p_begin, int64_t p_end, T* z, cudaStream_t s);

int launch_mom_sym_pairs(const float* verts, const int32_t* faces, const int32_t* fei, int64_t nf, int64_t n_edges, double k,
                         bool overwrite, float* rec, float* z, cudaStream_t s) {
    if (nf <= 0) return MB_OK;
    if (nf < 2400) {
        if (overwrite) {
            const cudaError_t e = cudaMemsetAsync(z, 0, sizeof(float2) * (size_t)n_edges * n_edges, s);
            if (e != cudaSuccess) return set_error(MB_ERR_CUDA, "%s", cudaGetErrorString(e));
        }
        return launch_mom_sym_regular<float>(verts, faces, fei, n_edges, k, nf, 0, nf, z, s);
    }
    const int64_t gx = (nf + kEdgeRows - 1) / kEdgeRows, gy = (nf + 127) / 128;
    if (gx > 0x7fffffffLL || gy > 65535) return set_error(MB_ERR_SIZE, "mesh too large for one launch");
    // a matrix that is not added to is summed above the diagonal only, half the reductions, and mirrored
    const auto kernel = overwrite ? sym_pairs_kernel<true> : sym_pairs_kernel<false>;
    const bool mirror = overwrite && n_edges > 0;
    const int64_t tiles = (n_edges + kMirror - 1) / kMirror;
    if (mirror && (n_edges > 0x7fffffffLL || (tiles + 1) / 2 > 65535))
        return set_error(MB_ERR_SIZE, "matrix too large for one launch");
    if (int rc = tier_records(verts, faces, nullptr, fei, nf, nullptr, nullptr, 0, nullptr, nullptr, 0, rec, s)) return rc;
    int* form = reinterpret_cast<int*>(rec + kRec * nf);
    sym_form_kernel<<<1, kFormThreads, 0, s>>>(rec, fei, nf, (float)k, overwrite ? 96 : 53, form);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kEdgeSumBytes);
    if (e != cudaSuccess) return set_error(MB_ERR_CUDA, "%s", cudaGetErrorString(e));
    float2* z2 = reinterpret_cast<float2*>(z);
    if (mirror) zero_upper_kernel<<<(unsigned)n_edges, 256, 0, s>>>(z2, n_edges);
    // test groups fastest: blocks in flight share the rows of one source tile for the transposed terms
    kernel<<<dim3((unsigned)gx, (unsigned)gy), 128, kEdgeSumBytes, s>>>(rec, nf, n_edges, k, form, z);
    if (mirror)
        mirror_kernel<<<dim3((unsigned)(tiles + 1), (unsigned)((tiles + 1) / 2)), 256, 0, s>>>(z2, n_edges, (int)tiles, form);
    if (int rc = check_launch("mom sym pairs")) return rc;
    return launch_mom_sym_rest(verts, faces, fei, n_edges, k, nf, rec, form, z, s);
}

}  // namespace mb
