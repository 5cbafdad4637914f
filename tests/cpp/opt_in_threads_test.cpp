// Host-only check of what host threads see when they launch a kernel for the
// first time at once (ncnn-moe-runtime_b200/csrc/moe_internal.h): nobody goes on
// before the kernel has been allowed its shared memory, and an answer about the
// resident clusters that was never given is not remembered.  The two runtime
// calls are replaced by fakes below; no CUDA library is linked.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

#include "../../ncnn-moe-runtime_b200/csrc/moe_internal.h"

static std::atomic<int> entered{0};
static std::atomic<bool> release{false};
static std::atomic<bool> allowed{false};
static std::atomic<bool> refuse{false};

extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* device)
{
    *device = 0;
    return cudaSuccess;
}
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute, int)
{
    ++entered;
    if (refuse)
        return cudaErrorInvalidValue;
    for (int i = 0; i < 2000 && !release; ++i)
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
    allowed = true;
    return cudaSuccess;
}

static int failures = 0;
#define EXPECT(condition)                                              \
    do                                                                 \
    {                                                                  \
        if (!(condition))                                              \
        {                                                              \
            std::printf("line %d: %s\n", __LINE__, #condition);        \
            ++failures;                                                \
        }                                                              \
    } while (0)

int main()
{
    const void* const kernel = nullptr;
    moe::SharedOptIn state;
    std::thread first([&] { moe::opt_in_shared(state, kernel, 100000); });
    while (entered == 0)
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
    // the first thread is inside cudaFuncSetAttribute
    std::atomic<bool> returned{false};
    bool allowed_on_return = false;
    std::thread second([&] {
        const cudaError_t status = moe::opt_in_shared(state, kernel, 100000);
        allowed_on_return = status == cudaSuccess && allowed;
        returned = true;
    });
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
    EXPECT(!returned);
    release = true;
    first.join();
    second.join();
    EXPECT(allowed_on_return);
    EXPECT(entered == 1); // configured once

    // a refusal is handed on and not remembered
    moe::SharedOptIn refused;
    refuse = true;
    EXPECT(moe::opt_in_shared(refused, kernel, 100000) == cudaErrorInvalidValue);
    refuse = false;
    EXPECT(moe::opt_in_shared(refused, kernel, 100000) == cudaSuccess);
    EXPECT(entered == 3);

    // resident clusters: a table with a failed portable size serves this call only
    moe::ClusterOccupancyTable table;
    int asked = 0;
    const auto failing = [&](int, int*) { ++asked; return cudaErrorInvalidValue; };
    const auto answering = [&](int size_index, int* clusters) {
        ++asked;
        if (size_index == 4)
            return cudaErrorInvalidValue; // no clusters of 16 CTAs here
        *clusters = 148 >> size_index;
        return cudaSuccess;
    };
    moe::ClusterOccupancy found = moe::cluster_occupancy(table, 0, failing);
    EXPECT(found.active[0] == 1 && found.active[3] == 0);
    asked = 0;
    found = moe::cluster_occupancy(table, 0, answering);
    EXPECT(asked == moe::kClusterSizes);
    EXPECT(found.active[0] == 148 && found.active[1] == 74 && found.active[3] == 18 && found.active[4] == 0);
    asked = 0;
    found = moe::cluster_occupancy(table, 0, failing); // known: not asked again
    EXPECT(asked == 0 && found.active[0] == 148 && found.active[2] == 37);
    found = moe::cluster_occupancy(table, 1, answering); // per device
    EXPECT(asked == moe::kClusterSizes && found.active[0] == 148);
    asked = 0;
    (void)moe::cluster_occupancy(table, moe::kMaxDevices, answering); // untracked ordinals are asked every time
    (void)moe::cluster_occupancy(table, -1, answering);
    EXPECT(asked == 2 * moe::kClusterSizes);

    if (failures == 0)
        std::puts("concurrent opt-in ok");
    return failures == 0 ? 0 : 1;
}
