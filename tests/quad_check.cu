// The arithmetic of the quad kernels beside the plain operators, element by element:
// which of n operands give other bits. Built with the library's own flags.
#include "../ifos3d-dev_b200/csrc/ifosb_corr.cuh"

#include <cuda_runtime.h>

using namespace ifosb;

namespace {

__device__ bool differ(float x, float y) {
    if (isnan(x) && isnan(y)) return false;
    return __float_as_uint(x) != __float_as_uint(y);
}

// q: 0 div4 of one quad, 1 of three quads at once, 2 a product and a sum, 3 the
// correlations' division (one divisor for all: b[0]), 4 the same for a power of two
__global__ void k_check(int what, const float *a, const float *b, int n, int in_range, int *bad, int *first) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (4 * q + 3 >= n) return;
    const float *x = a + 4 * q, *y = b + 4 * q;
    float got[4], want[4];
    if (what <= 1) {
        const F4 A = ld4(x), B = ld4(y), N = nrcp4(B);
        F4 r = A;
        if (what == 0) {
            r = div4(A, B, N, in_range != 0);
        } else {  // its neighbours in the triple are other quads of the arrays
            const int m = n / 4, p1 = 4 * ((q + 1) % m), p2 = 4 * ((q + 7) % m);
            F4 t[3] = {ld4(a + p1), A, ld4(a + p2)};
            const F4 d[3] = {ld4(b + p1), B, ld4(b + p2)}, ny[3] = {nrcp4(d[0]), N, nrcp4(d[2])};
            div4<3>(t, d, ny, in_range != 0);
            r = t[1];
        }
        for (int c = 0; c < 4; ++c) {
            got[c] = get4(r, c);
            want[c] = __fdiv_rn(x[c], y[c]);
        }
    } else if (what == 2) {
        const F4 r = ld4(x) * ld4(y) + ld4(a + 4 * ((q + 3) % (n / 4)));
        for (int c = 0; c < 4; ++c) {
            got[c] = get4(r, c);
            want[c] = __fadd_rn(__fmul_rn(x[c], y[c]), a[4 * ((q + 3) % (n / 4)) + c]);
        }
    } else {
        const float h = b[0];
        for (int c = 0; c < 4; c += 2) {
            const float2 v = make_float2(x[c], x[c + 1]);
            const float2 r = what == 3 ? dvh2<false>(v, h, __fdiv_rn(1.f, h)) : dvh2<true>(v, h, __fdiv_rn(1.f, h));
            got[c] = r.x;
            got[c + 1] = r.y;
            want[c] = __fdiv_rn(x[c], h);
            want[c + 1] = __fdiv_rn(x[c + 1], h);
        }
    }
    for (int c = 0; c < 4; ++c)
        if (differ(got[c], want[c])) {
            atomicAdd(bad, 1);
            atomicMin(first, 4 * q + c);
        }
}
__global__ void k_round(const double *x, int n, int *bad, int *first) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    if (__double_as_longlong(round24(x[q])) != __double_as_longlong((double)__double2float_rn(x[q]))) {
        atomicAdd(bad, 1);
        atomicMin(first, q);
    }
}

// every float in [2^lo, 2^hi): nrcp4 against the rounded reciprocal
__global__ void k_reciprocal(int lo, int hi, int *bad, int *first) {
    const uint32_t q0 = (uint32_t)(lo + 127) << 23, q1 = (uint32_t)(hi + 127) << 23;
    for (uint32_t q = q0 + 4 * (blockIdx.x * blockDim.x + threadIdx.x); q < q1; q += 4 * gridDim.x * blockDim.x) {
        F4 b;
        for (int c = 0; c < 4; ++c) set4(b, c, __uint_as_float(q + c));
        const F4 r = nrcp4(b);
        for (int c = 0; c < 4; ++c)
            if (differ(get4(r, c), -__frcp_rn(get4(b, c)))) {
                atomicAdd(bad, 1);
                atomicMin(first, (int)(q + c));
            }
    }
}

int outcome(cudaError_t e, int *d, int *res) {
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(res, d, 2 * sizeof(int), cudaMemcpyDeviceToHost);
    return (int)e;
}

}  // namespace

// a, b (or x): host arrays; res[0] how many differ, res[1] the first. 0, or a CUDA error.
extern "C" int quad_check(int what, const float *a, const float *b, int n, int in_range, int *res) {
    float *d = nullptr;
    int *r = nullptr;
    const int init[2] = {0, n};
    cudaError_t e = cudaMalloc((void **)&d, 2 * (size_t)n * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc((void **)&r, sizeof(init));
    if (e == cudaSuccess) e = cudaMemcpy(d, a, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(r, init, sizeof(init), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) k_check<<<(n / 4 + 127) / 128, 128>>>(what, d, d + n, n, in_range, r, r + 1);
    const int rc = outcome(e, r, res);
    cudaFree(d);
    cudaFree(r);
    return rc;
}
extern "C" int round_check(const double *x, int n, int *res) {
    double *d = nullptr;
    int *r = nullptr;
    const int init[2] = {0, n};
    cudaError_t e = cudaMalloc((void **)&d, (size_t)n * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc((void **)&r, sizeof(init));
    if (e == cudaSuccess) e = cudaMemcpy(d, x, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(r, init, sizeof(init), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) k_round<<<(n + 127) / 128, 128>>>(d, n, r, r + 1);
    const int rc = outcome(e, r, res);
    cudaFree(d);
    cudaFree(r);
    return rc;
}
extern "C" int reciprocal_check(int lo, int hi, int *res) {
    int *r = nullptr;
    const int init[2] = {0, 0x7fffffff};
    cudaError_t e = cudaMalloc((void **)&r, sizeof(init));
    if (e == cudaSuccess) e = cudaMemcpy(r, init, sizeof(init), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) k_reciprocal<<<592, 256>>>(lo, hi, r, r + 1);
    const int rc = outcome(e, r, res);
    cudaFree(r);
    return rc;
}
