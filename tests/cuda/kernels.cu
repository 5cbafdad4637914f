// Device code the GPU tests need beside the library: a producer that lets the
// next kernel of its stream start before it has written anything, and the
// comparison of the sampler's division by a reciprocal with the division itself.
#include <stddef.h>

#include "../../ncnn-moe-runtime_b200/csrc/moe_common.cuh"

namespace {

__device__ __forceinline__ uint64_t mix(uint64_t v) // splitmix64
{
    v += 0x9E3779B97F4A7C15ull;
    v = (v ^ (v >> 30)) * 0xBF58476D1CE4E5B9ull;
    v = (v ^ (v >> 27)) * 0x94D049BB133111EBull;
    return v ^ (v >> 31);
}

// A positive float with an exponent of [low, high]; every fourth has a mantissa next to a power of two or to the middle.
__device__ __forceinline__ float draw(uint64_t bits, int low, int high)
{
    const uint32_t exponent = static_cast<uint32_t>(low + 127) + static_cast<uint32_t>((bits >> 32) % static_cast<uint32_t>(high - low + 1));
    uint32_t mantissa = static_cast<uint32_t>(bits) & 0x7FFFFFu;
    if ((bits >> 62) == 0u)
        mantissa = (((bits >> 61) & 1u) * 0x400000u + ((bits >> 58) & 7u) - 4u) & 0x7FFFFFu;
    return __uint_as_float((exponent << 23) | mantissa);
}

__global__ void compare_divisions(uint64_t seed, uint32_t per_thread, int a_low, int a_high, int b_low, int b_high, unsigned long long* mismatches,
                                  unsigned int* largest)
{
    const uint64_t first = seed * 0x100000000ull + (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * per_thread;
    uint32_t different = 0;
    float top = 0.0f;
    for (uint32_t i = 0; i < per_thread; ++i)
    {
        const float a = draw(mix(2u * (first + i)), a_low, a_high);
        const float b = draw(mix(2u * (first + i) + 1u), b_low, b_high);
        const float q = moe::divide_by(a, b, __frcp_rn(b));
        different += __float_as_uint(q) != __float_as_uint(__fdiv_rn(a, b)) ? 1u : 0u;
        top = fmaxf(top, q == q ? q : INFINITY);
    }
    if (different != 0u)
        atomicAdd(mismatches, static_cast<unsigned long long>(different));
    atomicMax(largest, __float_as_uint(top)); // positive floats order as their bits
}

__global__ void produce_late(const uint32_t* source, uint32_t* target, size_t words, long long cycles)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); // the next kernel may start now ...
    const long long start = clock64();
    for (int i = 0; i < 100000 && clock64() - start < cycles; ++i)
        __nanosleep(100);
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < words; i += static_cast<size_t>(gridDim.x) * blockDim.x)
        target[i] = source[i]; // ... before its input exists
}

} // namespace

// Quotients of seeded operand pairs with exponents in [a_low, a_high] and [b_low, b_high]: how many differ from the
// division's (host word *mismatches), and the largest (host float *largest; infinity if one is not a number).
extern "C" int test_compare_divisions(uint64_t seed, uint32_t blocks, uint32_t per_thread, int a_low, int a_high, int b_low, int b_high,
                                      unsigned long long* mismatches, float* largest)
{
    unsigned long long* counters = nullptr;
    cudaError_t status = cudaMalloc(reinterpret_cast<void**>(&counters), 16);
    if (status != cudaSuccess)
        return status;
    status = cudaMemset(counters, 0, 16);
    if (status == cudaSuccess)
    {
        compare_divisions<<<blocks, 256>>>(seed, per_thread, a_low, a_high, b_low, b_high, counters, reinterpret_cast<unsigned int*>(counters + 1));
        status = cudaGetLastError();
    }
    if (status == cudaSuccess)
        status = cudaMemcpy(mismatches, counters, 8, cudaMemcpyDeviceToHost);
    if (status == cudaSuccess)
        status = cudaMemcpy(largest, counters + 1, 4, cudaMemcpyDeviceToHost);
    cudaFree(counters);
    return status;
}

// target[0 .. words) = source[0 .. words), about `cycles` clocks after the next kernel of the stream may have started.
extern "C" int test_produce_late(void* stream, const void* source, void* target, size_t words, long long cycles)
{
    produce_late<<<16, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint32_t*>(source), static_cast<uint32_t*>(target), words, cycles);
    return cudaGetLastError();
}
