// Compares the square roots and quotients of csrc/select_math.cuh with sqrtf and `/` on the device; each function returns how many
// results differ in any bit, and one input that does.  Built and called by test_gpu_select_math.py.
#include "select_math.cuh"

namespace {

struct Found {
    unsigned long long differ;
    float a, b;
};

__device__ unsigned scrambled(unsigned long long x) {   // splitmix64
    x += 0x9E3779B97F4A7C15ULL;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
    return (unsigned)((x ^ (x >> 31)) >> 16);
}

__device__ void compare(Found *found, float got, float want, float a, float b) {
    if (__float_as_uint(got) == __float_as_uint(want)) return;
    if (atomicAdd(&found->differ, 1ULL) == 0) {
        found->a = a;
        found->b = b;
    }
}

__global__ void roots(Found *found, int first, int count, int stride) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const int n = first + i * stride;
        compare(found, select_math::root_of_count(n), sqrtf((float)n), (float)n, 0.f);
    }
}

__device__ void quotient(Found *found, const select_math::Count &count, float a) {
    if (!select_math::Count::plain(a, a)) return;
    compare(found, count.divides(a), a / count.b, a, count.b);
    compare(found, count.divides(-a), -a / count.b, -a, count.b);
}

// every divisor from `first`: numerators anywhere in the range, next to its ends, and as close as a float can be to the middle
// between two quotients
__global__ void quotients(Found *found, int first, int count, int numerators) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const int n = first + i;
        const select_math::Count divisor(n);
        for (int k = 0; k < numerators; k++) {
            const unsigned r = scrambled((unsigned long long)n * 1000003ULL + k), s = scrambled(r);
            const int exponent = 127 - 80 + (int)(s % 180u);                       // 2^-80 .. 2^99
            quotient(found, divisor, __uint_as_float(((unsigned)exponent << 23) | (r & 0x7FFFFFu)));
            const double q = (double)(0x800000u | (r & 0x7FFFFFu)) + 0.5;          // 25 bits: the product below is exact
            const float middle = (float)(q * (double)n);
            quotient(found, divisor, middle);
            quotient(found, divisor, __uint_as_float(__float_as_uint(middle) + 1u));
            quotient(found, divisor, __uint_as_float(__float_as_uint(middle) - 1u));
            quotient(found, divisor, (float)n * (float)(1 + (r & 0xFFu)));
        }
        quotient(found, divisor, 0.f);
        quotient(found, divisor, 8.271806e-25f);
        quotient(found, divisor, 1.2676506e30f);
        quotient(found, divisor, 1.f);
    }
}

int report(Found *found, unsigned long long *differ, float *a, float *b) {
    Found host = {0, 0.f, 0.f};
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(&host, found, sizeof(host), cudaMemcpyDeviceToHost);
    cudaFree(found);
    *differ = host.differ;
    *a = host.a;
    *b = host.b;
    return (int)e;
}

}  // namespace

extern "C" int check_roots(int first, int count, int stride, unsigned long long *differ, float *a, float *b) {
    Found *found = nullptr;
    if (cudaMalloc(&found, sizeof(Found)) != cudaSuccess || cudaMemset(found, 0, sizeof(Found)) != cudaSuccess) return -1;
    roots<<<1024, 256>>>(found, first, count, stride);
    return report(found, differ, a, b);
}

extern "C" int check_quotients(int first, int count, int numerators, unsigned long long *differ, float *a, float *b) {
    Found *found = nullptr;
    if (cudaMalloc(&found, sizeof(Found)) != cudaSuccess || cudaMemset(found, 0, sizeof(Found)) != cudaSuccess) return -1;
    quotients<<<1024, 256>>>(found, first, count, numerators);
    return report(found, differ, a, b);
}
