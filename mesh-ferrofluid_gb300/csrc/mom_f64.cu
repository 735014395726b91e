// mom_f64.cu -- the reference-rule CFIE entries in FP64 for source rules of 1, 4, 9 and 16 points (any other
// size, and FP32 rule sizes without a kernel of their own, run mom_entry in mom_ref.cu).
//
// Bound: the FP64 pipe, 2 lanes a clock and SM, so the count of FP64 instructions per evaluation is the time.
// Vector moments with a divide, a square root and sincospi per evaluation took about 92; here 38 (46 on close
// pairs), 46.3 with all that is done per entry and test point.  2088 x 2088 entries of 9 x 4 points: 25.0 -> 13.8
// ms, the FP64 pipe active in 89 % of the cycles (5 or 6 blocks of 128 threads an SM in place of 4: the same).
// Against 80-bit sums over 17 meshes the error is 0.92 times (whole matrix), 0.95 (median entry) that of the vector
// moments.
//   * y.a, y.n1 in place of the vectors (as mom_entry_fast in mom_entry.cuh): with Y = y - B0, X = x - B0,
//     A = x - A0, c = k Y.A - 4/k, m = R^-2 ((Y.n)(X.A) - (Y.A)(X.n)), u = m kR + c and g = w / R the term is
//     g (sin, cos) combined with u and m;
//   * |x - y|^2 = |A|^2 - 2 (B0 - A0).A + |y - A0|^2 - 2 Y.A: the last product is there already.  Between close
//     pairs that sum would cancel, so a warp that holds one takes the coordinates' differences, and y.u from
//     (x - y).u, which is as small as |x - y|;
//   * the reciprocal root, sine and cosine by f64_steps.cuh, its table of angles filled by each block;
//   * the test face's values once per block and row (shared memory), the source face's length factor once per
//     thread for all its rows.
#include <algorithm>

#include "common.cuh"
#include "f64_steps.cuh"

namespace mb {

namespace {

constexpr int kF64Threads = 128;
constexpr int kF64Points = 256;  // test points: rules up to 16 x 16
constexpr int kF64Rows = 8;      // rows of a block

struct F64Rows {
    double2 angle[kAngles];  // (sin, cos) of 2 pi i / 256
    double2 r[kF64Points];   // r1 - r2, r2 of a test point
    double w[kF64Points];    // its weight; once per row, times twice the area, in a[4]
    double r0[kF64Points];   // 1 - r1
    double a[kF64Points][6]; // A = x - A0, its square, the weight on this face, and n.A; once per row
    // of each row: A0 (0-2), A1 - A0 (3-5), A2 - A0 (6-8), n1 (9-11), L / (2 area) (12), h^2 (13), 2 area (14),
    // A1 (15-17), A2 (18-20)
    double v[kF64Rows][21];
    double3 s[16];           // source points: r3 - r4, r4, weight / (4 pi)
};

__device__ __forceinline__ double dot3(const double* a, const V3<double>& b) {
    return a[0] * b.x + a[1] * b.y + a[2] * b.z;
}

// sum over the test points of w (re, im); the source point j is (p0, p1, p2, w, Y.n1) with p = Y (CLOSE) or
// (|y - A0|^2, Y.e1, Y.e2).  self: sum of w X.A.
template <int NS, bool CLOSE>
__device__ __forceinline__ void f64_sums(const F64Rows& sh, const double* rv, int nt, const double (&p0)[NS],
                                         const double (&p1)[NS], const double (&p2)[NS], const double (&wj)[NS],
                                         const double (&yn)[NS], double k, const V3<double>& c0,
                                         const V3<double>& c1, const V3<double>& c2, double be1, double be2,
                                         double xn0, bool same, double* re, double* im, double* self) {
    double ar = 0.0, ai = 0.0, sa = 0.0;
    const V3<double> n = {rv[9], rv[10], rv[11]};
    const double turn = k * (kAngles / (2.0 * kPi)), m4k = -4.0 / k;
#pragma unroll 1
    for (int i = 0; i < nt; ++i) {
        const double2 r = sh.r[i];
        const V3<double> a = {sh.a[i][0], sh.a[i][1], sh.a[i][2]};
        const double aa = sh.a[i][3];
        const double w = sh.a[i][4];
        const double xn = xn0 + sh.a[i][5];
        V3<double> x;
        double xa, x2;
        if constexpr (CLOSE) {
            // from the corners relative to B0: where one of them is B0 itself, x - B0 has no difference of
            // larger numbers in it (a - b was up to 1.5 times further off there)
            x = sh.r0[i] * c0 + (r.x * c1 + r.y * c2);
            xa = dot(x, a);
        } else {
            const double ba = fma(r.x, be1, r.y * be2);  // (B0 - A0).A
            xa = aa - ba;
            x2 = fma(-2.0, ba, aa);
        }
        double tr = 0.0, ti = 0.0;
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            double ya, r2, uy;  // uy = -(y.u), u = a (x.n) - n (x.a), orthogonal to x: y.u = -((x - y).u)
            if constexpr (CLOSE) {
                const double dx = x.x - p0[j], dy = x.y - p1[j], dz = x.z - p2[j];
                r2 = fma(dz, dz, fma(dy, dy, dx * dx));
                const double da = fma(a.x, dx, fma(a.y, dy, a.z * dz));
                const double dn = fma(n.x, dx, fma(n.y, dy, n.z * dz));
                uy = fma(da, xn, -dn * xa);
                ya = fma(a.x, p0[j], fma(a.y, p1[j], a.z * p2[j]));
            } else {
                ya = fma(r.x, p1[j], r.y * p2[j]);
                r2 = fma(-2.0, ya, x2 + p0[j]);
                uy = fma(-ya, xn, yn[j] * xa);
            }
            const double ri = rsqrt_step(r2);
            const double R = r2 * ri;
            double sn, cs;
            sincos_step(sh.angle, R, turn, &sn, &cs);
            const double g = wj[j] * ri;
            const double gr = g * cs, gs = g * sn;
            const double c = fma(k, ya, m4k);
            const double m = ri * ri * uy;
            const double u = fma(m, k * R, c);
            tr = fma(gs, u, fma(m, gr, tr));
            ti = fma(gr, u, fma(-m, gs, ti));
        }
        ar = fma(w, tr, ar);
        ai = fma(w, ti, ai);
        if (same) sa = fma(w, xa, sa);
    }
    *re = ar;
    *im = ai;
    *self = sa;
}

// block: kF64Threads columns, rows_per_block rows.  RWG: Z[fei[row], fei[col]] += entry (interleaved complex,
// caller zeroes); else split planes [batch, 3F, 3F].
template <int NS, bool RWG>
__global__ void __launch_bounds__(kF64Threads, NS <= 4 ? 4 : 2) mom_f64_kernel(
    const double* __restrict__ verts, const int32_t* __restrict__ faces, const double* __restrict__ areas,
    const double* __restrict__ normals, const int32_t* __restrict__ fei, int64_t n_edges,
    const double* __restrict__ gpx, const double* __restrict__ gwx, int nx, const double* __restrict__ gpy,
    const double* __restrict__ gwy, double k, int64_t nf, int64_t batch, int64_t row_begin, int64_t row_end,
    int rows_per_block, int64_t col_blocks, double* __restrict__ zr, double* __restrict__ zi) {
    constexpr int NY = NS == 1 ? 1 : (NS == 4 ? 2 : (NS == 9 ? 3 : 4));
    __shared__ F64Rows sh;
    const int t = threadIdx.x, nt = nx * nx;
    fill_angles(sh.angle);
    for (int i = t; i < nt; i += kF64Threads) {
        const double r1 = gpx[i / nx];
        sh.r[i] = make_double2(r1 - gpx[i % nx] * r1, gpx[i % nx] * r1);
        sh.r0[i] = 1.0 - r1;
        sh.w[i] = gwx[i / nx] * gwx[i % nx] * r1;
    }
    if (t < NS) {
        const double r3 = gpy[t / NY], r4 = gpy[t % NY] * r3;
        sh.s[t] = make_double3(r3 - r4, r4, gwy[t / NY] * gwy[t % NY] * r3 * kInv4Pi);
    }
    const int64_t ncol = 3 * nf;
    const int64_t col = ((int64_t)blockIdx.x % col_blocks) * kF64Threads + t;
    const int64_t row0 = row_begin + (int64_t)blockIdx.x / col_blocks * rows_per_block;
    const int64_t row1 = min(row0 + rows_per_block, row_end);
    const bool live = col < ncol;
    const int64_t f2 = live ? col / 3 : 0;
    const int e2 = live ? (int)(col % 3) : 0;
    const int32_t b1 = __ldg(faces + 3 * f2 + (e2 + 1) % 3), b2 = __ldg(faces + 3 * f2 + (e2 + 2) % 3);
    const V3<double> B0 = load3(verts, __ldg(faces + 3 * f2 + e2));
    const V3<double> d1 = load3(verts, b1) - B0, d2 = load3(verts, b2) - B0;
    const double area2 = __ldg(areas + f2);
    const double fac2 = (b1 < b2 ? 1.0 : -1.0) * sqrt(dot(d2 - d1, d2 - d1)) / (2.0 * area2);
    const double h2 = fmax(fmax(dot(d1, d1), dot(d2, d2)), dot(d2 - d1, d2 - d1));
    if (t < row1 - row0) {
        const int64_t f1 = (row0 + t) / 3;
        const int e1 = (int)((row0 + t) % 3);
        const int32_t a1 = __ldg(faces + 3 * f1 + (e1 + 1) % 3), a2 = __ldg(faces + 3 * f1 + (e1 + 2) % 3);
        const V3<double> A0 = load3(verts, __ldg(faces + 3 * f1 + e1));
        const V3<double> A1 = load3(verts, a1), A2 = load3(verts, a2), n1 = load3(normals, f1);
        const V3<double> u = A1 - A0, v = A2 - A1, z = A2 - A0;
        const double area1 = __ldg(areas + f1);
        double* rv = sh.v[t];
        rv[0] = A0.x, rv[1] = A0.y, rv[2] = A0.z;
        rv[3] = u.x, rv[4] = u.y, rv[5] = u.z;
        rv[6] = z.x, rv[7] = z.y, rv[8] = z.z;
        rv[9] = n1.x, rv[10] = n1.y, rv[11] = n1.z;
        rv[12] = (a1 < a2 ? 1.0 : -1.0) * sqrt(dot(v, v)) / (2.0 * area1);
        rv[13] = fmax(fmax(dot(u, u), dot(v, v)), dot(z, z));
        rv[14] = 2.0 * area1;
        rv[15] = A1.x, rv[16] = A1.y, rv[17] = A1.z;
        rv[18] = A2.x, rv[19] = A2.y, rv[20] = A2.z;
    }
    for (int64_t row = row0; row < row1; ++row) {
        const int64_t f1 = row / 3;
        const double* rv = sh.v[row - row0];
        __syncthreads();
        for (int i = t; i < nt; i += kF64Threads) {
            const double2 r = sh.r[i];
            const V3<double> a = {fma(r.x, rv[3], r.y * rv[6]), fma(r.x, rv[4], r.y * rv[7]),
                                  fma(r.x, rv[5], r.y * rv[8])};
            sh.a[i][0] = a.x, sh.a[i][1] = a.y, sh.a[i][2] = a.z, sh.a[i][3] = dot(a, a);
            sh.a[i][4] = sh.w[i] * rv[14];
            sh.a[i][5] = dot3(rv + 9, a);
        }
        __syncthreads();
        const V3<double> b = {B0.x - rv[0], B0.y - rv[1], B0.z - rv[2]};
        const double be1 = dot3(rv + 3, b), be2 = dot3(rv + 6, b);
        // x.n = n.(A0 - B0) + n.A; the second is rounding for a face's own normal, but the normals are the caller's
        const double xn = -dot3(rv + 9, b);
        const V3<double> c0 = {rv[0] - B0.x, rv[1] - B0.y, rv[2] - B0.z};  // the test corners from B0
        const V3<double> c1 = {rv[15] - B0.x, rv[16] - B0.y, rv[17] - B0.z};
        const V3<double> c2 = {rv[18] - B0.x, rv[19] - B0.y, rv[20] - B0.z};
        // Two edge lengths between the centroids (every point is within 2/3 of one of its own): |y - A0|^2
        // is then at most 6 times |x - y|^2, for the two corners nearest to each other.
        const V3<double> cd = (d1 + d2) - (c0 + c1 + c2);  // 3 times the centroids' distance
        const bool close = dot(cd, cd) <= 36.0 * fmax(h2, rv[13]);
        double p0[NS], p1[NS], p2[NS], wj[NS], yn[NS];
        double re, im, self;
        const bool same = f1 == f2;
        if (__any_sync(0xffffffffu, close)) {
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const double3 s = sh.s[j];
                p0[j] = fma(s.x, d1.x, s.y * d2.x);
                p1[j] = fma(s.x, d1.y, s.y * d2.y);
                p2[j] = fma(s.x, d1.z, s.y * d2.z);
                wj[j] = s.z * (2.0 * area2);
                yn[j] = 0.0;
            }
            f64_sums<NS, true>(sh, rv, nt, p0, p1, p2, wj, yn, k, c0, c1, c2, be1, be2, xn, same, &re, &im, &self);
        } else {
            const double n_1 = dot3(rv + 9, d1), n_2 = dot3(rv + 9, d2);
            const double u_1 = dot3(rv + 3, d1), u_2 = dot3(rv + 3, d2);
            const double v_1 = dot3(rv + 6, d1), v_2 = dot3(rv + 6, d2);
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const double3 s = sh.s[j];
                const double x = fma(s.x, d1.x, fma(s.y, d2.x, b.x)), y = fma(s.x, d1.y, fma(s.y, d2.y, b.y)),
                             z = fma(s.x, d1.z, fma(s.y, d2.z, b.z));
                p0[j] = fma(z, z, fma(y, y, x * x));
                p1[j] = fma(s.x, u_1, s.y * u_2);
                p2[j] = fma(s.x, v_1, s.y * v_2);
                wj[j] = s.z * (2.0 * area2);
                yn[j] = fma(s.x, n_1, s.y * n_2);
            }
            f64_sums<NS, false>(sh, rv, nt, p0, p1, p2, wj, yn, k, c0, c1, c2, be1, be2, xn, same, &re, &im, &self);
        }
        if (!live) continue;
        const double cc = rv[12] * fac2;
        re = cc * (same ? fma(0.5, self, re) : re);
        im *= cc;
        
        if constexpr (RWG) {
            const int64_t m = __ldg(fei + row), n = __ldg(fei + col);
            double* o = zr + 2 * (m * n_edges + n);
            atomicAdd(o, re);
            atomicAdd(o + 1, im);
        } else {
            for (int64_t q = 0; q < batch; ++q) {
                const int64_t o = (q * ncol + row) * ncol + col;
                zr[o] = re;
                zi[o] = im;
            }
        }
    }
}

template <int NS>
void launch_f64(const double* verts, const int32_t* faces, const double* areas, const double* normals,
                const int32_t* fei, int64_t n_edges, const double* gpx, const double* gwx, int nx, const double* gpy,
                const double* gwy, double k, int64_t nf, int64_t batch, int64_t row_begin, int64_t row_end,
                double* zr, double* zi, cudaStream_t stream) {
    const int64_t col_blocks = (3 * nf + kF64Threads - 1) / kF64Threads, rows = row_end - row_begin;
    // The table costs a block about a twentieth of a row of 36 evaluations, so a block takes several rows, as long
    // as there are eight blocks for each of the SMs' places (4 of 128 threads) to even out the close pairs.
    const int64_t rpb = std::min<int64_t>(kF64Rows, std::max<int64_t>(1, rows * col_blocks / (kSms * 4 * 8)));
    const unsigned blocks = (unsigned)((rows + rpb - 1) / rpb * col_blocks);
    if (fei)
        mom_f64_kernel<NS, true><<<blocks, kF64Threads, 0, stream>>>(verts, faces, areas, normals, fei, n_edges, gpx,
                                                                     gwx, nx, gpy, gwy, k, nf, batch, row_begin,
                                                                     row_end, (int)rpb, col_blocks, zr, zi);
    else
        mom_f64_kernel<NS, false><<<blocks, kF64Threads, 0, stream>>>(verts, faces, areas, normals, fei, n_edges, gpx,
                                                                      gwx, nx, gpy, gwy, k, nf, batch, row_begin,
                                                                      row_end, (int)rpb, col_blocks, zr, zi);
}

}  // namespace

// Launches the FP64 entries if the source rule has 1, 4, 9 or 16 points; returns false otherwise.
bool launch_mom_f64(const double* verts, const int32_t* faces, const double* areas, const double* normals,
                    const int32_t* fei, int64_t n_edges, const double* gpx, const double* gwx, int nx,
                    const double* gpy, const double* gwy, int ny, double k, int64_t nf, int64_t batch,
                    int64_t row_begin, int64_t row_end, double* zr, double* zi, cudaStream_t stream) {
    switch (ny) {
#define MB_F64(NYV)                                                                                              \
    case NYV:                                                                                                    \
        launch_f64<NYV * NYV>(verts, faces, areas, normals, fei, n_edges, gpx, gwx, nx, gpy, gwy, k, nf, batch,  \
                              row_begin, row_end, zr, zi, stream);                                               \
        return true;
        MB_F64(1)
        MB_F64(2)
        MB_F64(3)
        MB_F64(4)
#undef MB_F64
        default: return false;
    }
}

}  // namespace mb
