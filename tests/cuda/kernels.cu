// Device code the GPU tests need beside the library: a producer that lets the
// next kernel of its stream start before it has written anything.
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace {

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

// target[0 .. words) = source[0 .. words), about `cycles` clocks after the next kernel of the stream may have started.
extern "C" int test_produce_late(void* stream, const void* source, void* target, size_t words, long long cycles)
{
    produce_late<<<16, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint32_t*>(source), static_cast<uint32_t*>(target), words, cycles);
    return cudaGetLastError();
}
