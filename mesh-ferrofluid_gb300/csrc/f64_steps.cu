// f64_steps.cu -- the functions of f64_steps.cuh over arrays (for their test).
#include "f64_steps.cuh"

namespace mb {

namespace {

__global__ void __launch_bounds__(256) f64_steps_kernel(int which, const double* __restrict__ x,
                                                        const double* __restrict__ y, int64_t n, double* __restrict__ out) {
    __shared__ double2 angles[kAngles];
    fill_angles(angles);
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s, c;
    switch (which) {
        case 0: out[i] = rsqrt_step(x[i]); break;
        case 1: out[i] = sqrt_step(x[i]); break;
        case 2: out[i] = quotient_step(x[i], y[i]); break;
        default:
            sincos_step(angles, x[i], y[i], &s, &c);
            out[i] = which == 3 ? s : c;
    }
}

}  // namespace

int launch_f64_steps(int which, const double* x, const double* y, int64_t n, double* out, cudaStream_t s) {
    if (n <= 0) return MB_OK;
    if ((n + 255) / 256 > 0x7fffffffLL) return set_error(MB_ERR_SIZE, "too many values for one launch");
    f64_steps_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(which, x, y, n, out);
    return check_launch("f64_steps");
}

}  // namespace mb
