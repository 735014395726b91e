// mom_entry.cuh -- one face-edge entry of the reference-rule CFIE in FP32 (used by the
// kernels of mom_ref.cu and mom_tiers.cu).
#pragma once
#include "common.cuh"
#include "packed.cuh"

namespace mb {

// ---------------------------------------------------------------------------------------
// float fast path: compile-time rule sizes, projected moments, packed f32x2 arithmetic.
//
// Per test point x_i the entry needs only three complex sums over the source points:
//   S0 = sum G,   P = sum G (y.a),   Q = sum G (1 + jkR) R^-2 (y.u)
// with a = x - A0 and u = x x (a x n1) = a (x.n1) - n1 (x.a), because the old vector
// moments were only ever used as a.S1 and u.H1.  y.a = r1 (y.e1) + r2 (y.e2) with the test
// edge vectors e1 = A1 - A0, e2 = A2 - A1, so per source point the kernel keeps (y, w,
// y.e1, y.e2, y.n1) in registers and an evaluation costs ~26 FP32 ops.  Two source points
// ride in one packed f32x2 instruction (Blackwell `fma/mul/add/sub.rn.f32x2`); the SFU does
// rsqrt, sin and cos.  The entry is then
//   c1 c2 sum_i w_i [ -Q + jk P - (4j/k) S0 ]  (+ self term), identical to mom_entry.
// ---------------------------------------------------------------------------------------


// Rule tables staged in shared memory: test (r1, r2, w_a w_b r1), source
// (r3, r4, w_a w_b r3 / (4 pi)); index b*n + a as in the reference loops (:410-415).
template <int NX, int NY>
__device__ __forceinline__ void stage_rules(const float* gpx, const float* gwx, const float* gpy,
                                            const float* gwy, float4* s_t, float4* s_s) {
    const int t = threadIdx.x;
    if (t < NX * NX) {
        const float r1 = gpx[t / NX];
        s_t[t] = make_float4(r1, gpx[t % NX] * r1, gwx[t / NX] * gwx[t % NX] * r1, 0.f);
    } else if (t < NX * NX + NY * NY) {
        const int j = t - NX * NX;
        const float r3 = gpy[j / NY];
        s_s[j] = make_float4(r3, gpy[j % NY] * r3, gwy[j / NY] * gwy[j % NY] * r3 * float(kInv4Pi), 0.f);
    }
}

template <int NX, int NY>
__device__ __forceinline__ void mom_entry_fast(const float* __restrict__ verts,
                                               const int32_t* __restrict__ faces,
                                               const float* __restrict__ areas,
                                               const float* __restrict__ normals, const float4* s_t,
                                               const float4* s_s, float k, int64_t f1, int e1, int64_t f2,
                                               int e2, float* out_re, float* out_im) {
    // NP full pairs of source points in packed f32x2 registers; an odd count leaves one
    // source point (TAIL) that is evaluated with scalar instructions.
    constexpr int NT = NX * NX, NS = NY * NY, NP = NS / 2, TAIL = NS & 1;
    const int32_t a0 = __ldg(faces + 3 * f1 + e1);
    const int32_t a1 = __ldg(faces + 3 * f1 + (e1 + 1) % 3);
    const int32_t a2 = __ldg(faces + 3 * f1 + (e1 + 2) % 3);
    const int32_t b0 = __ldg(faces + 3 * f2 + e2);
    const int32_t b1 = __ldg(faces + 3 * f2 + (e2 + 1) % 3);
    const int32_t b2 = __ldg(faces + 3 * f2 + (e2 + 2) % 3);
    const V3<float> o = load3(verts, b0);
    const V3<float> A0 = load3(verts, a0) - o;
    const V3<float> A1 = load3(verts, a1) - o;
    const V3<float> A2 = load3(verts, a2) - o;
    const V3<float> B1 = load3(verts, b1) - o;
    const V3<float> B2 = load3(verts, b2) - o;
    const V3<float> n1 = load3(normals, f1);
    const float area1 = __ldg(areas + f1), area2 = __ldg(areas + f2);
    const V3<float> ev1 = A1 - A0, ev2 = A2 - A1;
    const V3<float> d2 = B2 - B1;
    const float c1 = (a1 < a2 ? 1.f : -1.f) * sqrtf(dot(ev2, ev2)) / (2.f * area1);
    const float c2 = (b1 < b2 ? 1.f : -1.f) * sqrtf(dot(d2, d2)) / (2.f * area2);

    // Source points (origin B0) packed two per register pair: coordinates scaled by k (only
    // distances use them: |k x - k y| = kR), the weight k w (so g = w / R = (k w) / (kR)), and
    // the projections k (y.e1), k (y.e2) on the test edge vectors and y.n1 on the normal.
    float2 yx[NP > 0 ? NP : 1], yy[NP > 0 ? NP : 1], yz[NP > 0 ? NP : 1], yw[NP > 0 ? NP : 1],
        ye1[NP > 0 ? NP : 1], ye2[NP > 0 ? NP : 1], yn[NP > 0 ? NP : 1];
    float tx = 0.f, ty = 0.f, tz = 0.f, tw = 0.f, te1 = 0.f, te2 = 0.f, tn = 0.f;  // the tail point
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        const float4 r = s_s[j];
        const V3<float> y = (r.x - r.y) * B1 + r.y * B2;
        const float w = r.z * (2.f * area2) * k;
        if (j < 2 * NP) {
            (reinterpret_cast<float*>(&yx[j / 2]) + (j & 1))[0] = k * y.x;
            (reinterpret_cast<float*>(&yy[j / 2]) + (j & 1))[0] = k * y.y;
            (reinterpret_cast<float*>(&yz[j / 2]) + (j & 1))[0] = k * y.z;
            (reinterpret_cast<float*>(&yw[j / 2]) + (j & 1))[0] = w;
            (reinterpret_cast<float*>(&ye1[j / 2]) + (j & 1))[0] = k * dot(y, ev1);
            (reinterpret_cast<float*>(&ye2[j / 2]) + (j & 1))[0] = k * dot(y, ev2);
            (reinterpret_cast<float*>(&yn[j / 2]) + (j & 1))[0] = dot(y, n1);
        } else {
            tx = k * y.x;
            ty = k * y.y;
            tz = k * y.z;
            tw = w;
            te1 = k * dot(y, ev1);
            te2 = k * dot(y, ev2);
            tn = dot(y, n1);
        }
    }
    // Per evaluation, with c = k (y.a) - 4/k, yu = (y.a)(x.n1) - (y.n1)(x.a), m = -R^-2 yu and
    // G = gr - j gs:  t_re += gs c + m Re[G(1 + jkR)],  t_im += gr c + m Im[G(1 + jkR)]
    // (Re = gr + gs kR, Im = gr kR - gs), i.e. the per-test-point combination
    // -Q + jk P - (4j/k) S0 of the three sums, summed directly.  yu = c (x.n1)/k + (4 (x.n1)/k^2 - (y.n1)(x.a)) and R^-2 = k^2 (kR)^-2, so
    // -R^-2 yu = (kR)^-2 [c (-k (x.n1)) + (y.n1) k^2 (x.a) - 4 (x.n1)].
    const float2 M4K = bc(-4.f / k);
    float2 acc_re = bc(0.f), acc_im = bc(0.f);
    float self_acc = 0.f;
    const bool same = (f1 == f2);
    // The test-point loop stays rolled: its body (the unrolled source loop) is ~2 KB of
    // code, and unrolling it 16 times overflows the instruction cache.
#pragma unroll 1
    for (int i = 0; i < NT; ++i) {
        const float4 t = s_t[i];
        const float w1 = t.z * (2.f * area1);
        const V3<float> a = t.x * ev1 + t.y * ev2;
        const V3<float> x = A0 + a;
        const float xn = dot(x, n1), xa = dot(x, a);
        const float2 X = bc(k * x.x), Y = bc(k * x.y), Z = bc(k * x.z), R1 = bc(t.x), R2 = bc(t.y),
                     CN = bc(-k * xn), CA = bc(k * k * xa), C4 = bc(-4.f * xn);
        float2 tr = bc(0.f), ti = bc(0.f);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const float2 dx = sub2(X, yx[p]);
            const float2 dy = sub2(Y, yy[p]);
            const float2 dz = sub2(Z, yz[p]);
            const float2 r2d = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));  // (kR)^2
            float2 rinv;                                                 // (kR)^-1
            rinv.x = rsqrtf(r2d.x);
            rinv.y = rsqrtf(r2d.y);
            const float2 kR = mul2(r2d, rinv);
            float2 sn, cs;
            __sincosf(kR.x, &sn.x, &cs.x);
            __sincosf(kR.y, &sn.y, &cs.y);
            const float2 g = mul2(yw[p], rinv);
            const float2 gr = mul2(g, cs), gs = mul2(g, sn);  // G = gr - j gs
            const float2 c = fma2(R1, ye1[p], fma2(R2, ye2[p], M4K));
            const float2 nyu = fma2(c, CN, fma2(yn[p], CA, C4));  // -k^2 yu
            const float2 m = mul2(mul2(rinv, rinv), nyu);         // -R^-2 yu
            // m G(1 + jkR) + c G in the conjugate form (gr + j gs)(u + j m), u = m kR + c
            const float2 u = fma2(m, kR, c);
            tr = fma2(gs, u, fma2(m, gr, tr));
            ti = sub2(fma2(gr, u, ti), mul2(m, gs));
        }
        if constexpr (TAIL) {
            // the odd source point, scalar: same algebra as one lane of the packed loop
            const float dx = k * x.x - tx, dy = k * x.y - ty, dz = k * x.z - tz;
            const float r2d = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            const float rinv = rsqrtf(r2d);
            const float kR = r2d * rinv;
            float sn, cs;
            __sincosf(kR, &sn, &cs);
            const float g = tw * rinv;
            const float gr = g * cs, gs = g * sn;
            const float c = fmaf(t.x, te1, fmaf(t.y, te2, -4.f / k));
            const float nyu = fmaf(c, -k * xn, fmaf(tn, k * k * xa, -4.f * xn));
            const float m = rinv * rinv * nyu;
            const float u = fmaf(m, kR, c);
            tr.x = fmaf(gs, u, fmaf(m, gr, tr.x));
            ti.x = fmaf(gr, u, fmaf(-m, gs, ti.x));
        }
        const float2 W1 = bc(w1);
        acc_re = fma2(W1, tr, acc_re);
        acc_im = fma2(W1, ti, acc_im);
        if (same) self_acc += w1 * xa;  // (x - A0) . (x - B0), B0 = 0
    }
    const float cc = c1 * c2;
    *out_re = cc * (acc_re.x + acc_re.y + 0.5f * self_acc);
    *out_im = cc * (acc_im.x + acc_im.y);
}

}  // namespace mb
