// Quotients by one divisor (dmath.cuh) against the compiler's division, on the device.
#include <cstdint>

#include "dmath.cuh"

using namespace avbdg;

__device__ uint32_t mixed(uint64_t x) { // splitmix64, Steele, Lea and Flood 2014
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return static_cast<uint32_t>((x ^ (x >> 31)) >> 16);
}

// A float of the given exponent range; kind 0: any mantissa, 1: all ones or nearly, 2: few bits, 3: the ends of
// the range and the floats beside them.
__device__ float operand(uint32_t r, uint32_t s, int lowest, int highest, int kind) {
    uint32_t mantissa = r & 0x7fffffu, exponent = 127 + lowest + s % static_cast<uint32_t>(highest - lowest);
    if (kind == 1)
        mantissa = 0x7fffffu - (r & 15u);
    if (kind == 2)
        mantissa = (r & 0x1fu) << 18;
    uint32_t bits = exponent << 23 | mantissa;
    if (kind == 3)
        bits = (127 + (r & 1u ? lowest : highest)) * (1u << 23) + (r >> 1 & 7u) - 4u;
    return __uint_as_float(bits | (s & 0x80000000u));
}

// out: wrong quotients, operands in range that were refused, operands out of range that were taken, taken.
__global__ void compare(int kindA, int kindB, unsigned long long seed, unsigned long long *out) {
    const unsigned long long i = seed + 4ull * (blockIdx.x * blockDim.x + threadIdx.x);
    const float b = operand(mixed(i), mixed(i + 1), -40, 40, kindB), a = operand(mixed(i + 2), mixed(i + 3), -80, 80, kindA);
    bool ok = true;
    const Divisor d = divisor(b, ok);
    const float q = quotient(a, d, ok), plain = a / b;
    const bool inside = fabsf(b) >= 0x1p-40f && fabsf(b) <= 0x1p40f && fabsf(a) >= 0x1p-80f && fabsf(a) <= 0x1p80f;
    if (ok && __float_as_uint(q) != __float_as_uint(plain))
        atomicAdd(out, 1ull);
    if (ok != inside)
        atomicAdd(out + (ok ? 2 : 1), 1ull);
    if (ok)
        atomicAdd(out + 3, 1ull);
}

// Zeros of either sign by divisors of either, and what is never taken.
__global__ void special(unsigned long long *out) {
    const float divisors[] = {1.0f, -3.0f, 0x1p-40f, 0x1p40f, 0x1.fffffep-1f, 0x1.fffffep39f};
    for (float b : divisors)
        for (float a : {0.0f, -0.0f}) {
            bool ok = true;
            const Divisor d = divisor(b, ok);
            const float q = quotient(a, d, ok);
            if (!ok)
                out[1]++;
            else if (__float_as_uint(q) != __float_as_uint(a / b))
                out[0]++;
        }
    const float inf = __uint_as_float(0x7f800000u), nan = __uint_as_float(0x7fc00000u), tiny = __uint_as_float(1u);
    for (float b : {0.0f, -0.0f, inf, -inf, nan, tiny, 0x1p-41f, 0x1p41f}) {
        bool ok = true;
        const Divisor d = divisor(b, ok);
        quotient(1.0f, d, ok);
        out[2] += ok;
    }
    for (float a : {inf, -inf, nan, tiny, 0x1p-81f, 0x1p81f}) {
        bool ok = true;
        const Divisor d = divisor(3.0f, ok);
        quotient(a, d, ok);
        out[2] += ok;
    }
}

extern "C" int check_quotients(unsigned long long *host) {
    unsigned long long *out = nullptr;
    if (cudaMalloc(&out, 32) != cudaSuccess)
        return 1;
    cudaMemset(out, 0, 32);
    for (int a = 0; a < 4; a++)
        for (int b = 0; b < 4; b++)
            compare<<<4096, 256>>>(a, b, (4ull * a + b) << 40, out);
    special<<<1, 1>>>(out);
    const cudaError_t e = cudaMemcpy(host, out, 32, cudaMemcpyDeviceToHost);
    cudaFree(out);
    return e == cudaSuccess ? 0 : 2;
}
