// gmres_cycle.cuh -- interface between gmres.cu's driver and the resident cycle kernel.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstddef>

namespace mb {

struct GmresSync {  // zeroed before every cycle
    unsigned count;
    int error, stop, pad;
    double acc[2], w2[2], w2x[2];
};
struct GmresState {  // zeroed before the first cycle
    long long iters, cycles;
    double relres;
    int converged, finished, jdone, pad;
};

struct GmresHead {  // copied to the host after a cycle
    GmresState st;
    GmresSync sync;
};

// Layout of the cycle's part of the workspace: head, sums, Hessenberg matrix, coefficients.
struct GmresCycleRegion {
    GmresHead* head;
    double2 *hsum, *H, *y;
    static constexpr size_t al(size_t b) { return (b + 255) & ~size_t(255); }
    static constexpr size_t zero_bytes(int m) {  // from head->sync to the end of the sums
        return al(sizeof(GmresHead)) - sizeof(GmresState) + 64 * (size_t)(m + 1);
    }
    static constexpr size_t bytes(int m) {
        return al(sizeof(GmresHead)) + al(64 * (size_t)(m + 1)) + al(16 * (size_t)m * (m + 1)) + al(16 * (size_t)m);
    }
    GmresCycleRegion(void* p, int m) {
        char* c = static_cast<char*>(p);
        head = reinterpret_cast<GmresHead*>(c);
        c += al(sizeof(GmresHead));
        hsum = reinterpret_cast<double2*>(c);
        c += al(64 * (size_t)(m + 1));
        H = reinterpret_cast<double2*>(c);
        c += al(16 * (size_t)m * (m + 1));
        y = reinterpret_cast<double2*>(c);
    }
};

struct GmresCyclePlan {
    bool ok, staged;
    int rows, pad, grid;
    size_t bytes;
    const void* kernel;
};

// Plans the resident cycle for a matrix kind (0 complex64, 1 float32, 2 float64), n unknowns and restart m;
// plan->ok false where the launch-per-operation form has to run.
int gmres_cycle_begin(GmresCyclePlan* plan, int kind, int64_t n, int m);
// One cycle from the residual r (complex128): x updated, GmresState advanced.  *refused: the driver does not
// grant the launch here and nothing ran.
int gmres_cycle_launch(const GmresCyclePlan& plan, const void* a, int64_t n, const double* b, double* x, const double* r,
                       int m, double tol, long long max_iters, float* v32, double* v64, void* region, bool* refused,
                       cudaStream_t s);

}  // namespace mb
