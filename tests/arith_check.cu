// Device arithmetic of radiance_device.cuh against CUDA's correctly rounded operations; each check
// counts the inputs whose bits differ.  Built by test_gpu_arith.py.
#include "../lum_gb300/csrc/radiance_device.cuh"

using namespace lumrad;

__global__ void rcp_check(unsigned long long* bad, int e0, int e1) {   // every mantissa at each exponent
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    for (int e = e0; e <= e1; e++) {
        const float d = __uint_as_float(((unsigned)(e + 127) << 23) | m);
        if (rcp_normal(d) != __frcp_rn(d) || rcp_normal(-d) != __frcp_rn(-d)) atomicAdd(bad, 1ull);
    }
}
__global__ void sqrt_check(unsigned long long* bad, int e0, int e1) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    for (int e = e0; e <= e1; e++) {
        const float x = __uint_as_float(((unsigned)(e + 127) << 23) | m);
        if (sqrt_normal(x) != __fsqrt_rn(x)) atomicAdd(bad, 1ull);
    }
}
__device__ float draw(unsigned& x) {   // xorshift: sign, 16 exponents, every mantissa bit
    x ^= x << 13; x ^= x >> 17; x ^= x << 5;
    const unsigned m = x & 0x7fffffu;
    x ^= x << 13; x ^= x >> 17; x ^= x << 5;
    return __uint_as_float((x & 0x80000000u) | ((120u + ((x >> 8) & 15u)) << 23) | m);
}
__global__ void pair_check(unsigned long long* bad, unsigned seed) {
    unsigned x = (blockIdx.x * blockDim.x + threadIdx.x) * 2654435761u + seed;
    const float a = draw(x), b = draw(x), c = draw(x), d = draw(x), e = draw(x), f = draw(x);
    float lo, hi;
    unpack2(add_product2(pack2(a, b), mul2(pack2(c, d), pack2(e, f))), lo, hi);
    if (lo != fadd(a, fmul(c, e)) || hi != fadd(b, fmul(d, f))) atomicAdd(bad, 1ull);
}
__global__ void pair_sub_check(unsigned long long* bad, unsigned seed) {
    unsigned x = (blockIdx.x * blockDim.x + threadIdx.x) * 2654435761u + seed;
    const float a = draw(x), b = draw(x), c = draw(x), d = draw(x), e = draw(x), f = draw(x);
    float lo, hi;
    unpack2(sub_product2(mul2(add2(pack2(a, b), pack2(c, d)), pack2(e, f)), mul2(pack2(c, d), pack2(e, f))), lo, hi);
    if (lo != fsub(fmul(fadd(a, c), e), fmul(c, e)) || hi != fsub(fmul(fadd(b, d), f), fmul(d, f))) atomicAdd(bad, 1ull);
}

extern "C" long long arith_check(int which) {
    unsigned long long* d = nullptr;
    unsigned long long h = 0;
    if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return -1;
    const int blocks = (1 << 23) / 256;
    if (which == 0) rcp_check<<<blocks, 256>>>(d, -100, 20);
    if (which == 1) sqrt_check<<<blocks, 256>>>(d, -40, 40);
    if (which == 2) pair_check<<<blocks, 256>>>(d, 1u);
    if (which == 3) pair_sub_check<<<blocks, 256>>>(d, 2u);
    const cudaError_t e = cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? (long long)h : -1;
}
