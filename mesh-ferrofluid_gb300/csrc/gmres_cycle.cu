// gmres_cycle.cu -- one restart cycle of mb_gmres_* as one cooperative kernel.
//
// A step of the launch-per-operation form (gmres.cu) is a matrix-vector product, four
// Gram-Schmidt kernels and three host round trips: at 1998 unknowns 0.15 ms of which the
// product is 0.01 ms, the Gram-Schmidt kernels running as 8 blocks over serial loops.  Here the
// grid stays resident for the cycle.  Each worker block owns a range of rows: it computes its
// part of the product and keeps its rows of the whole complex128 basis in shared memory, so
// Gram-Schmidt reads no global memory beyond the sums.  Per step the blocks meet three times:
// for the two passes' sums V^H w (FP64 atomics, as in gmres.cu) and for the new basis vector, and once
// more where its norm has to be summed again.  One more block applies the Givens rotations of a step while the workers are
// in the next step's product; when it finds the estimate below the target the workers drop
// that step and add V y to x.  Precisions are those of gmres.cu: products in FP32 (or FP64 for a
// float64 matrix) with FP64 lane sums, everything else FP64.
//
// Measured (GB300, complex64): 1998 unknowns, 186 steps in 5 cycles: 30.0 -> 4.9 ms; per step with its share
// of the residuals 120 unknowns 103 -> 28 us, 7680 264 -> 173 us, 15000 651 -> 653 us, 30720 2278 -> 2319 us: the product's
// reads dominate from there on, and one block per SM streams them a little slower, so above
// kMaxUnknowns the launch-per-operation form runs.
// Waits are on a counter that every block of the cooperative grid increments; each is bounded and a
// run-out ends the kernel with an error code.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "gmres_cycle.cuh"

namespace mb {

namespace {

constexpr int kThreads = 1024, kWarps = 32;
constexpr int64_t kMaxUnknowns = 12288;
constexpr int kStaticShared = 1024;  // bytes of shared memory left to the kernel's own variables
constexpr long long kPollLimit = 1ll << 22;  // about 2 s of polls

struct CycleArgs {
    const void* a;
    const double2* b;
    double2* x;
    const double2* r;
    float2* v32;     // the current basis vector, rounded (kinds 0, 1)
    double2* v64;    // the current basis vector (kind 2)
    GmresSync* sync;
    GmresState* st;
    double2* hsum;   // [2 steps][2 passes][m + 1]
    double2 *H, *y;  // [m][m + 1], [m]
    int64_t n;
    int m, rows, rows_pad;
    double tol;
    long long max_iters;
};

// Every block arrives; false when the wait ran out.
__device__ bool grid_wait(GmresSync* s, unsigned target, bool* s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&s->count, 1u);
        long long it = 0;
        unsigned v;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&s->count) : "memory");
        } while (v < target && ++it < kPollLimit);
        if (v < target) atomicExch(&s->error, 1);
        *s_ok = v >= target;
        __threadfence();
    }
    __syncthreads();
    return *s_ok;
}

// (re, im) summed over the warp's lanes in FP64: lanes 0-15 take re, 16-31 im after one exchange; the
// sums end in lanes 0 and 16
__device__ __forceinline__ double warp_sum_pair(float re, float im) {
    const bool hi = threadIdx.x & 16;
    double v = (double)(hi ? im : re);
    v += (double)__shfl_xor_sync(0xffffffffu, hi ? re : im, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_sum_pair(double re, double im) {
    const bool hi = threadIdx.x & 16;
    double v = hi ? im : re;
    v += __shfl_xor_sync(0xffffffffu, hi ? re : im, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// v at index i: the staged copy in shared memory, or L2 (the vector changes within the kernel, so no
// read-only or L1 path)
template <bool STAGED, typename T>
__device__ __forceinline__ T vget(const T* v, int64_t i) {
    if constexpr (STAGED) return v[i];
    else return __ldcg(v + i);
}

// Part [lane + 32 part, ...) of rows row .. row + NR - 1 of A times v.
template <int KIND, bool STAGED, int NR>
__device__ __forceinline__ void row_dots(const void* a, int64_t n, int64_t row, const float2* v32, const double2* v64,
                                         int64_t first, int64_t step, float (&re)[NR], float (&im)[NR],
                                         double (&dre)[NR], double (&dim)[NR]) {
    if constexpr (KIND == 0) {
        const float2* z = static_cast<const float2*>(a) + row * n;
        if (((n & 1) | (reinterpret_cast<uintptr_t>(a) & 15)) == 0) {
            const float4* v4 = reinterpret_cast<const float4*>(v32);
            const int64_t np = n >> 1;
            int64_t p = first;
            for (; p + 3 * step < np; p += 4 * step) {
                float4 q[NR][4];
#pragma unroll
                for (int i = 0; i < NR; ++i)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        q[i][u] = __ldcs(reinterpret_cast<const float4*>(z + i * n) + p + u * step);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 w = vget<STAGED>(v4, p + u * step);
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        const float4 c = q[i][u];
                        re[i] = fmaf(c.x, w.x, fmaf(-c.y, w.y, re[i]));
                        im[i] = fmaf(c.x, w.y, fmaf(c.y, w.x, im[i]));
                        re[i] = fmaf(c.z, w.z, fmaf(-c.w, w.w, re[i]));
                        im[i] = fmaf(c.z, w.w, fmaf(c.w, w.z, im[i]));
                    }
                }
            }
            for (; p < np; p += step) {
                const float4 w = vget<STAGED>(v4, p);
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const float4 c = __ldcs(reinterpret_cast<const float4*>(z + i * n) + p);
                    re[i] = fmaf(c.x, w.x, fmaf(-c.y, w.y, re[i]));
                    im[i] = fmaf(c.x, w.y, fmaf(c.y, w.x, im[i]));
                    re[i] = fmaf(c.z, w.z, fmaf(-c.w, w.w, re[i]));
                    im[i] = fmaf(c.z, w.w, fmaf(c.w, w.z, im[i]));
                }
            }
        } else {
            for (int64_t p = first; p < n; p += step) {
                const float2 w = vget<STAGED>(v32, p);
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const float2 c = __ldcs(z + i * n + p);
                    re[i] = fmaf(c.x, w.x, fmaf(-c.y, w.y, re[i]));
                    im[i] = fmaf(c.x, w.y, fmaf(c.y, w.x, im[i]));
                }
            }
        }
    } else if constexpr (KIND == 1) {
        const float* z = static_cast<const float*>(a) + row * n;
        int64_t done = 0;
        if (((n & 3) | (reinterpret_cast<uintptr_t>(a) & 15)) == 0) {
            const float4* v4 = reinterpret_cast<const float4*>(v32);
            done = n;
            for (int64_t p = first; p < (n >> 2); p += step) {
                const float4 w0 = vget<STAGED>(v4, 2 * p), w1 = vget<STAGED>(v4, 2 * p + 1);
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const float4 c = __ldcs(reinterpret_cast<const float4*>(z + i * n) + p);
                    re[i] = fmaf(c.x, w0.x, fmaf(c.y, w0.z, fmaf(c.z, w1.x, fmaf(c.w, w1.z, re[i]))));
                    im[i] = fmaf(c.x, w0.y, fmaf(c.y, w0.w, fmaf(c.z, w1.y, fmaf(c.w, w1.w, im[i]))));
                }
            }
        }
        for (int64_t p = done + first; p < n; p += step) {
            const float2 w = vget<STAGED>(v32, p);
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const float c = __ldcs(z + i * n + p);
                re[i] = fmaf(c, w.x, re[i]);
                im[i] = fmaf(c, w.y, im[i]);
            }
        }
    } else {
        const double* z = static_cast<const double*>(a) + row * n;
        for (int64_t p = first; p < n; p += step) {
            const double2 w = vget<STAGED>(v64, p);
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const double c = __ldcs(z + i * n + p);
                dre[i] = fma(c, w.x, dre[i]);
                dim[i] = fma(c, w.y, dim[i]);
            }
        }
    }
}

// w_s[row] = (A v)[r0 + row] for the block's nr rows.  Few rows: several warps share one (split), their
// partial sums meeting in s_part; many: a warp takes two rows at once, reading v once for both.
template <int KIND, bool STAGED>
__device__ void block_product(const CycleArgs& g, int64_t r0, int nr, const float2* v32, const double2* v64, double2* w_s,
                              double2* s_part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (nr >= kWarps) {
        for (int row = 2 * warp; row < nr; row += 2 * kWarps) {
            float re[2] = {0.f, 0.f}, im[2] = {0.f, 0.f};
            double dre[2] = {0.0, 0.0}, dim[2] = {0.0, 0.0};
            const int two = row + 1 < nr;
            if (two) {
                row_dots<KIND, STAGED, 2>(g.a, g.n, r0 + row, v32, v64, lane, 32, re, im, dre, dim);
            } else {
                float r1[1] = {0.f}, i1[1] = {0.f};
                double dr1[1] = {0.0}, di1[1] = {0.0};
                row_dots<KIND, STAGED, 1>(g.a, g.n, r0 + row, v32, v64, lane, 32, r1, i1, dr1, di1);
                re[0] = r1[0];
                im[0] = i1[0];
                dre[0] = dr1[0];
                dim[0] = di1[0];
            }
            for (int i = 0; i <= two; ++i) {
                const double v = KIND == 2 ? warp_sum_pair(dre[i], dim[i]) : warp_sum_pair(re[i], im[i]);
                if (lane == 0) w_s[row + i].x = v;
                if (lane == 16) w_s[row + i].y = v;
            }
        }
    } else if (nr > 0) {
        int split = 1;
        while (2 * split * nr <= kWarps) split *= 2;
        const int row = warp / split, part = warp % split;
        if (row < nr) {
            float re[1] = {0.f}, im[1] = {0.f};
            double dre[1] = {0.0}, dim[1] = {0.0};
            row_dots<KIND, STAGED, 1>(g.a, g.n, r0 + row, v32, v64, lane + 32 * part, 32 * split, re, im, dre, dim);
            const double v = KIND == 2 ? warp_sum_pair(dre[0], dim[0]) : warp_sum_pair(re[0], im[0]);
            if (lane == 0) s_part[warp].x = v;
            if (lane == 16) s_part[warp].y = v;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nr; i += kThreads) {
            double2 s = make_double2(0.0, 0.0);
            for (int q = 0; q < split; ++q) {
                s.x += s_part[i * split + q].x;
                s.y += s_part[i * split + q].y;
            }
            w_s[i] = s;
        }
    }
    __syncthreads();
}

// hsum[i] += sum over the block's rows of conj(V_i) w, i < nb: four threads per i
__device__ void block_dots(const double2* V, int ld, const double2* w_s, int nr, int nb, double2* hsum) {
    const int i = threadIdx.x >> 2, sub = threadIdx.x & 3;
    if (i < ((nb + 7) & ~7)) {  // whole warps
        double re = 0.0, im = 0.0;
        if (i < nb) {
            const double2* vi = V + (int64_t)i * ld;
            for (int k = sub; k < nr; k += 4) {
                const double2 v = vi[k], w = w_s[k];
                re = fma(v.x, w.x, fma(v.y, w.y, re));
                im = fma(v.x, w.y, fma(-v.y, w.x, im));
            }
        }
        // lanes 0, 1 of a quad end with re, 2, 3 with im
        double t = (sub & 2) ? im : re;
        t += __shfl_xor_sync(0xffffffffu, (sub & 2) ? re : im, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        if (i < nb && nr > 0) {
            if (sub == 0) atomicAdd(&hsum[i].x, t);
            if (sub == 2) atomicAdd(&hsum[i].y, t);
        }
    }
}

// sum of |w|^2 over the block's rows, in thread 0
__device__ double block_norm2(const double2* w_s, int nr) {
    double a = 0.0;
    if (threadIdx.x < 32) {
        for (int k = threadIdx.x; k < nr; k += 32) a = fma(w_s[k].x, w_s[k].x, fma(w_s[k].y, w_s[k].y, a));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    }
    return a;
}

// w -= sum_{i < nb} V_i h_i: eight threads per row over strided i
__device__ void block_subtract(const double2* V, int ld, const double2* h, double2* w_s, int nr, int nb) {
    const int sub = threadIdx.x & 7;
    for (int row = threadIdx.x >> 3; row < ((nr + 3) & ~3); row += kThreads / 8) {  // whole warps
        double re = 0.0, im = 0.0;
        if (row < nr) {
            for (int i = sub; i < nb; i += 8) {
                const double2 v = V[(int64_t)i * ld + row], c = h[i];
                re = fma(v.x, c.x, fma(-v.y, c.y, re));
                im = fma(v.x, c.y, fma(v.y, c.x, im));
            }
        }
        // lanes 0-3 of the eight end with re, 4-7 with im
        double t = (sub & 4) ? im : re;
        t += __shfl_xor_sync(0xffffffffu, (sub & 4) ? re : im, 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        if (row < nr && sub == 0) w_s[row].x -= t;
        if (row < nr && sub == 4) w_s[row].y -= t;
    }
    __syncthreads();
}

// The manager's Hessenberg column j: previous rotations, the new one, the residual estimate.  A rotation
// takes (a, b) to (conj(c) a + s b, c b - s a) with s real, so what it hands to the next is one FMA:
// the products c b are formed by all threads, two lanes run the recurrence (an FP64 instruction holds
// the pipe for 16 cycles however few its lanes), all threads form the column.  Sets the stop flag.
__device__ void givens_column(const CycleArgs& g, int j, const double2* h1, const double2* h2, double hn, double bnorm,
                              long long iters, double2* col, double2* chain, double2* cs, double* sn, double2* gv) {
    for (int i = threadIdx.x; i <= j; i += kThreads) {
        const double2 a = __ldcg(h1 + i), b = __ldcg(h2 + i);
        const double2 h = make_double2(a.x + b.x, a.y + b.y);
        col[i] = h;
        if (i == 0) {
            chain[0] = h;
        } else {
            const double2 c = cs[i - 1];
            chain[i] = make_double2(fma(c.x, h.x, -c.y * h.y), fma(c.x, h.y, c.y * h.x));
        }
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double* t = reinterpret_cast<double*>(chain) + threadIdx.x;
        double a = t[0];
        for (int i = 0; i < j; ++i) {
            a = fma(-sn[i], a, t[2 * (i + 1)]);
            t[2 * (i + 1)] = a;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < j; i += kThreads) {
        const double2 a = chain[i], b = col[i + 1], c = cs[i];
        const double s = sn[i];
        g.H[(int64_t)j * (g.m + 1) + i] =
            make_double2(fma(c.x, a.x, fma(c.y, a.y, s * b.x)), fma(c.x, a.y, fma(-c.y, a.x, s * b.y)));
    }
    if (threadIdx.x == 0) {
        const double2 a = chain[j];
        // a matrix of entries about 1e+-150: the squares leave the range, the values do not
        const double r2 = fma(a.x, a.x, fma(a.y, a.y, hn * hn));
        const double rr = r2 > 1e-280 && r2 < 1e280 ? sqrt(r2) : hypot(hypot(a.x, a.y), hn), ir = rr == 0.0 ? 0.0 : 1.0 / rr;
        const double2 c = rr == 0.0 ? make_double2(1.0, 0.0) : make_double2(a.x * ir, a.y * ir);
        const double s = hn * ir;
        cs[j] = c;
        sn[j] = s;
        g.H[(int64_t)j * (g.m + 1) + j] = make_double2(rr, 0.0);
        const double2 t = gv[j];
        const double2 nx = make_double2(-s * t.x, -s * t.y);
        gv[j + 1] = nx;
        gv[j] = make_double2(c.x * t.x + c.y * t.y, c.x * t.y - c.y * t.x);
        const double stop = 0.5 * g.tol * bnorm;
        if (fma(nx.x, nx.x, nx.y * nx.y) <= stop * stop || hn <= 1e-300 || iters + j + 1 >= g.max_iters ||
            j + 1 == g.m) {
            g.st->jdone = j + 1;
            __threadfence();
            atomicExch(&g.sync->stop, 1);
        }
    }
    __syncthreads();
}

template <int KIND, bool STAGED>
__global__ void __launch_bounds__(kThreads, 1) gmres_cycle_kernel(const CycleArgs g) {
    extern __shared__ double2 sm[];
    __shared__ bool s_ok;
    __shared__ double s_num[4];
    __shared__ int s_stop, s_again;
    const int nblk = gridDim.x, m = g.m, ld = g.rows_pad;
    const bool manager = blockIdx.x == nblk - 1;
    const int64_t r0 = (int64_t)blockIdx.x * g.rows;
    const int nr = manager ? 0 : (int)max((int64_t)0, min((int64_t)g.rows, g.n - r0));
    double2* V = sm;                       // workers: [m + 1][ld], ld >= 12; the manager: col, chain, cs, g, sn
    double2* w_s = V + (int64_t)(m + 1) * ld;
    double2* h_s = w_s + g.rows;
    double2* part = h_s + (m + 1);         // [32]
    double2* stage = part + kWarps;
    double2 *col = sm, *chain = col + (m + 1), *cs = chain + (m + 1), *gv = cs + m;
    double* sn = reinterpret_cast<double*>(gv + (m + 1));
    const long long iters = g.st->iters;  // written by the manager at the very end only
    unsigned target = 0;
#define MB_WAIT()                                     \
    do {                                              \
        target += (unsigned)nblk;                     \
        if (!grid_wait(g.sync, target, &s_ok)) return; \
    } while (0)

    // |r|, |b|
    for (int k = threadIdx.x; k < nr; k += kThreads) w_s[k] = g.r[r0 + k];
    __syncthreads();
    {
        const double rr = block_norm2(w_s, nr);
        double bb = 0.0;
        if (threadIdx.x < 32) {
            for (int k = threadIdx.x; k < nr; k += 32) {
                const double2 v = g.b[r0 + k];
                bb = fma(v.x, v.x, fma(v.y, v.y, bb));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) bb += __shfl_xor_sync(0xffffffffu, bb, o);
        }
        if (threadIdx.x == 0 && nr > 0) {
            atomicAdd(&g.sync->acc[0], rr);
            atomicAdd(&g.sync->acc[1], bb);
        }
    }
    MB_WAIT();
    // (FP64 square roots and divisions by one thread: by all 32 warps they take 13 us)
    if (threadIdx.x == 0) {
        const double bb = sqrt(__ldcg(&g.sync->acc[0])), bn = sqrt(__ldcg(&g.sync->acc[1]));
        s_num[0] = bb;
        s_num[1] = bn == 0.0 ? 1.0 : bn;
        s_num[2] = bb / s_num[1];
        s_num[3] = 1.0 / bb;
    }
    __syncthreads();
    const double beta = s_num[0], bnorm = s_num[1], relres = s_num[2], ib = s_num[3];
    const bool converged = relres <= g.tol;
    if (converged || iters >= g.max_iters) {
        if (manager && threadIdx.x == 0) {
            g.st->relres = relres;
            g.st->converged = converged;
            g.st->finished = 1;
        }
        return;
    }
    for (int k = threadIdx.x; k < nr; k += kThreads) {
        const double2 v = make_double2(w_s[k].x * ib, w_s[k].y * ib);
        V[k] = v;
        if (KIND == 2) g.v64[r0 + k] = v;
        else g.v32[r0 + k] = make_float2((float)v.x, (float)v.y);
    }
    if (manager && threadIdx.x == 0) gv[0] = make_double2(beta, 0.0);
    MB_WAIT();

    double hn = 0.0;  // the last step's
    int j = 0;
    for (; j < m; ++j) {
        double2* h1 = g.hsum + (int64_t)(j & 1) * 2 * (m + 1);
        double2* h2 = h1 + (m + 1);
        if (manager) {
            double2* o1 = g.hsum + (int64_t)((j - 1) & 1) * 2 * (m + 1);
            if (j > 0) givens_column(g, j - 1, o1, o1 + (m + 1), hn, bnorm, iters, col, chain, cs, sn, gv);
        } else {
            const float2* v32 = g.v32;
            const double2* v64 = g.v64;
            if constexpr (STAGED) {
                if (KIND == 2) {
                    for (int64_t k = threadIdx.x; k < g.n; k += kThreads) stage[k] = __ldcg(g.v64 + k);
                } else {
                    float4* s4 = reinterpret_cast<float4*>(stage);
                    const float4* v4 = reinterpret_cast<const float4*>(g.v32);  // padded to an even length
                    for (int64_t k = threadIdx.x; k < (g.n + 1) / 2; k += kThreads) s4[k] = __ldcg(v4 + k);
                }
                v32 = reinterpret_cast<const float2*>(stage);
                v64 = stage;
                __syncthreads();
            }
            block_product<KIND, STAGED>(g, r0, nr, v32, v64, w_s, part);
            block_dots(V, ld, w_s, nr, j + 1, h1);
        }
        MB_WAIT();
        if (threadIdx.x == 0) s_stop = atomicAdd(&g.sync->stop, 0);
        __syncthreads();
        if (s_stop) break;
        // the other step's sums were last read before this wait
        if (blockIdx.x == 0) {
            double2* o = g.hsum + (int64_t)((j + 1) & 1) * 2 * (m + 1);
            for (int i = threadIdx.x; i < 2 * (m + 1); i += kThreads) o[i] = make_double2(0.0, 0.0);
            if (threadIdx.x == 0) g.sync->w2[(j + 1) & 1] = g.sync->w2x[(j + 1) & 1] = 0.0;
        }
        if (!manager) {
            for (int i = threadIdx.x; i <= j; i += kThreads) h_s[i] = __ldcg(h1 + i);
            __syncthreads();
            block_subtract(V, ld, h_s, w_s, nr, j + 1);
            block_dots(V, ld, w_s, nr, j + 1, h2);
            const double a = block_norm2(w_s, nr);
            if (threadIdx.x == 0 && nr > 0) atomicAdd(&g.sync->w2[j & 1], a);
        }
        MB_WAIT();
        // |w - V h2|^2 = |w|^2 - |h2|^2 with V orthonormal to rounding; where the second pass took a sizable part of
        // w the norm is summed again
        for (int i = threadIdx.x; i <= j; i += kThreads) h_s[i] = __ldcg(h2 + i);
        __syncthreads();
        {
            const double s2 = block_norm2(h_s, j + 1);
            if (threadIdx.x == 0) {
                const double w2 = __ldcg(&g.sync->w2[j & 1]), d = w2 - s2, inv = rsqrt(d);
                s_num[0] = d > 0.0 ? d * inv : d;  // 0 and NaN pass through
                s_num[1] = d > 0.0 ? inv : 0.0;
                s_again = !(s2 <= 0.01 * w2);
            }
        }
        if (!manager) block_subtract(V, ld, h_s, w_s, nr, j + 1);
        __syncthreads();
        if (s_again) {
            const double a = block_norm2(w_s, nr);
            if (threadIdx.x == 0 && nr > 0) atomicAdd(&g.sync->w2x[j & 1], a);
            MB_WAIT();
            if (threadIdx.x == 0) {
                const double d = __ldcg(&g.sync->w2x[j & 1]), inv = rsqrt(d);
                s_num[0] = d > 0.0 ? d * inv : d;
                s_num[1] = d > 0.0 ? inv : 0.0;
            }
            __syncthreads();
        }
        hn = s_num[0];
        const double inv = s_num[1];
        for (int k = threadIdx.x; k < nr; k += kThreads) {
            const double2 v = make_double2(w_s[k].x * inv, w_s[k].y * inv);
            V[(int64_t)(j + 1) * ld + k] = v;
            if (KIND == 2) g.v64[r0 + k] = v;
            else g.v32[r0 + k] = make_float2((float)v.x, (float)v.y);
        }
        MB_WAIT();
    }
    if (manager) {
        if (j == m) {
            double2* o1 = g.hsum + (int64_t)((m - 1) & 1) * 2 * (m + 1);
            givens_column(g, m - 1, o1, o1 + (m + 1), hn, bnorm, iters, col, chain, cs, sn, gv);
        }
        // back substitution, column by column (one warp)
        __threadfence();
        const int jd = g.st->jdone;
        if (threadIdx.x < 32) {
            for (int i = jd - 1; i >= 0; --i) {
                const double2* hc = g.H + (int64_t)i * (m + 1);
                const double2 t = gv[i];
                const double d = hc[i].x;  // the rotated diagonal is real
                const double2 yi = make_double2(t.x / d, t.y / d);
                if (threadIdx.x == 0) g.y[i] = yi;
                for (int r = threadIdx.x; r < i; r += 32) {
                    const double2 h = hc[r];
                    gv[r].x -= h.x * yi.x - h.y * yi.y;
                    gv[r].y -= h.x * yi.y + h.y * yi.x;
                }
                __syncwarp();
            }
        }
        if (threadIdx.x == 0) {
            g.st->relres = relres;
            g.st->cycles += 1;
            g.st->iters = iters + jd;
        }
    }
    MB_WAIT();
    if (threadIdx.x == 0) s_stop = *(volatile int*)&g.st->jdone;
    __syncthreads();
    const int jd = s_stop;
    for (int i = threadIdx.x; i < jd; i += kThreads) h_s[i] = __ldcg(g.y + i);
    __syncthreads();
    for (int k = threadIdx.x; k < nr; k += kThreads) {
        double2 x = g.x[r0 + k];
        for (int i = 0; i < jd; ++i) {
            const double2 v = V[(int64_t)i * ld + k], c = h_s[i];
            x.x = fma(v.x, c.x, fma(-v.y, c.y, x.x));
            x.y = fma(v.x, c.y, fma(v.y, c.x, x.y));
        }
        g.x[r0 + k] = x;
    }
#undef MB_WAIT
}

}  // namespace

// Rows per worker block, shared memory and staging of a cycle over n unknowns with restart m; false when the
// basis does not fit the resident grid's shared memory.
static bool cycle_plan(int kind, int64_t n, int m, int sms, int smem_max, int* rows, int* pad, int* grid,
                       size_t* bytes, bool* staged) {
    if (sms < 2) return false;
    // at least 8 rows per block (fewer blocks meet faster), at most one block per SM
    const int workers = (int)std::min<int64_t>(sms - 1, (n + 7) / 8);
    *rows = (int)((n + workers - 1) / workers);
    *pad = std::max(12, *rows + ((4 - *rows % 8) + 8) % 8);  // 4 mod 8: the dots' quads meet no bank twice
    *grid = workers + 1;
    const size_t basis = 16 * ((size_t)(m + 1) * *pad + *rows + (m + 1) + kWarps);
    const size_t own = 16 * (3 * (size_t)(m + 1) + m) + 8 * (size_t)m;  // the manager's, below its h_s
    const size_t stage = (kind == 2 ? 16 : 8) * (size_t)(n + 1);
    *staged = basis + stage <= (size_t)smem_max;
    *bytes = std::max(basis + (*staged ? stage : 0), own);
    return *bytes <= (size_t)smem_max;
}

int gmres_cycle_begin(GmresCyclePlan* p, int kind, int64_t n, int m) {
    p->ok = false;
    int dev = 0, sms = 0, smem = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop || n > kMaxUnknowns ||
        !cycle_plan(kind, n, m, sms, smem - kStaticShared, &p->rows, &p->pad, &p->grid, &p->bytes, &p->staged))
        return MB_OK;
    p->kernel = kind == 0 ? (p->staged ? (const void*)gmres_cycle_kernel<0, true> : (const void*)gmres_cycle_kernel<0, false>)
              : kind == 1 ? (p->staged ? (const void*)gmres_cycle_kernel<1, true> : (const void*)gmres_cycle_kernel<1, false>)
                          : (p->staged ? (const void*)gmres_cycle_kernel<2, true> : (const void*)gmres_cycle_kernel<2, false>);
    // The limit belongs to the process, not to this solve: another thread's solve may set it between two cycles
    // of this one, so it is the same for every plan.
    int per_sm = 0;
    if (cudaFuncSetAttribute(p->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem - kStaticShared) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p->kernel, kThreads, p->bytes) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return MB_OK;
    }
    p->ok = true;
    return MB_OK;
}

int gmres_cycle_launch(const GmresCyclePlan& p, const void* a, int64_t n, const double* b, double* x, const double* r,
                       int m, double tol, long long max_iters, float* v32, double* v64, void* region, bool* refused,
                       cudaStream_t s) {
    *refused = false;
    const GmresCycleRegion q(region, m);
    // the counters and sums of a cycle start from zero
    cudaMemsetAsync(&q.head->sync, 0, GmresCycleRegion::zero_bytes(m), s);
    CycleArgs g{a, reinterpret_cast<const double2*>(b), reinterpret_cast<double2*>(x), reinterpret_cast<const double2*>(r),
                reinterpret_cast<float2*>(v32), reinterpret_cast<double2*>(v64), &q.head->sync, &q.head->st, q.hsum, q.H, q.y, n, m,
                p.rows, p.pad, tol, max_iters};
    void* args[] = {&g};
    const cudaError_t e = cudaLaunchCooperativeKernel(p.kernel, dim3((unsigned)p.grid), dim3(kThreads), args, p.bytes, s);
    if (e == cudaSuccess) return MB_OK;
    cudaGetLastError();
    // a context with fewer SMs than the device says, or one that takes no such launch
    *refused = e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported;
    return *refused ? MB_OK : set_error(MB_ERR_CUDA, "gmres cycle: %s", cudaGetErrorString(e));
}

}  // namespace mb
