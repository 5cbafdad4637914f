// Host-side declarations shared by the translation units of the library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>

#include "../../include/moe_b200_sampler.h"

#define MOE_SLICE_SLOT_RECORDS 1024u
// largest top_k the small-buffer kernel instantiation serves (the 4 * k + 64 records a slice expects above its sampled
// threshold must fit the 2048-record buffer with room for their spread)
#define MOE_SAMPLER_TOPK_SMALL_MAX 448u
// kept lists up to this length are verified in shared memory; longer ones need the dense residual scratch
#define MOE_SPECULATIVE_SHORT_LIST 1024u
// entries of the router's [expert][block] count table (expert_count * blocks of the select kernel never exceeds it)
#define MOE_ROUTER_BLOCK_TABLE_ENTRIES 262144u

namespace moe {

// Device workspace shared by the kernels of one handle.
struct Workspace
{
    // rows the streaming kernel could not finish; consumed (and reset to 0) by
    // the exact kernel of the same call
    uint32_t* exact_count = nullptr;   // [1]
    uint32_t* exact_done = nullptr;    // [1] CTAs of the exact kernel that have finished
    uint32_t* exact_next = nullptr;    // [1] next entry of exact_rows nobody has taken yet
    uint32_t* exact_rows = nullptr;    // [max_rows]
    // rows the clusters left to the one-CTA kernel of the same call (with a mark in the high bit), and their number
    uint32_t* exact_deferred = nullptr;       // [max_rows]
    uint32_t* exact_deferred_count = nullptr; // [1]
    // what the clusters did since it was last read, for tests (a row they leave has the same result): rows finished, rows
    // left, sums repeated with a corrected accumulator, sums repeated with better exponents
    uint32_t* cluster_counts = nullptr; // [4]
    uint32_t cluster_ctas = 0;          // CTAs per row; 0: chosen by the launcher
    // per-slot scratch of the exact kernels, stride = max_vocab rounded up to a multiple of 4 entries: two buffers of
    // 64-bit items for the one-CTA kernel; the cluster kernel before it keeps its items there (see ClusterSlice)
    uint32_t* sort_keys = nullptr;     // [slots][4][stride]
    // publication slots of the streaming kernel when a row is cut into slices:
    // one per CTA, MOE_SLICE_SLOT_RECORDS records and a 4-word header each
    uint64_t* slice_records = nullptr; // [slice_slots][MOE_SLICE_SLOT_RECORDS]
    uint32_t* slice_header = nullptr;  // [slice_slots][4]: count, needs-exact flag, max key, pad
    uint32_t* row_arrivals = nullptr;  // [max_rows] slices of the row that have published (self-resetting)
    uint32_t slice_slots = 0;
    uint32_t slots = 0;
    uint32_t max_rows = 0;
    uint32_t max_vocab = 0;
};

// The part [begin, end) of a row that one CTA of a cluster owns.  Slices begin at multiples of four logits and their items
// are written in whole groups of four, so a cluster's items end at the row's length rounded up to four: the numerators
// (4 B) fill at most the first of a slot's four arrays, the value groups (2 B) at most half of the second.
struct ClusterSlice
{
    uint32_t begin;
    uint32_t end;
};
__host__ __device__ inline ClusterSlice cluster_slice(uint32_t vocab, uint32_t cluster_size, uint32_t rank)
{
    const uint32_t per = ((vocab + cluster_size - 1u) / cluster_size + 3u) & ~3u;
    const uint64_t begin = static_cast<uint64_t>(rank) * per;
    if (begin >= vocab)
        return ClusterSlice{vocab, vocab}; // nothing left for it
    return ClusterSlice{static_cast<uint32_t>(begin), vocab - static_cast<uint32_t>(begin) < per ? vocab : static_cast<uint32_t>(begin) + per};
}

struct SampleArgs
{
    const void* logits;
    // a second logit matrix of the same stride that holds the rows from second_begin on (null: all rows are in `logits`)
    const void* logits_second;
    uint32_t second_begin;
    int dtype;
    uint32_t rows;
    uint32_t vocab;
    size_t row_stride;
    const moe_row_params* params; // device
    uint64_t step_offset;
    const int32_t* stop_offsets; // device or null
    const int32_t* stop_tokens;  // device or null
    int32_t* token_id;
    float* probability;
    uint32_t* row_flags;   // may be null
    int32_t* row_status;   // may be null
    // the four results above as one record per row instead (host-mapped memory of moe_sample_tokens); null: the arrays
    moe_sampled_row* packed;
    int32_t* topk_index;   // may be null
    uint32_t topk_stride;
    // optional: every row's kept candidates with their renormalised probabilities
    // (the vector sampling_distribution returns, session.cpp:76-136)
    int32_t* kept_token;     // [rows x kept_stride] or null
    float* kept_probability; // [rows x kept_stride] or null
    uint32_t* kept_count;    // [rows] or null: candidates kept (may exceed kept_stride; the list is cut there)
    uint32_t kept_stride;
    // vocabulary-sharded local pass: write the slice's Top-K records instead of sampling
    uint64_t* candidates_out; // may be null
    uint32_t candidates_k;
    uint32_t vocab_begin;
    // some row has a Top-K too large for the small record buffer: use the
    // large-buffer instantiation (fewer CTAs per SM)
    bool large_top_k;
    // moe_sampler_set_overlap: the streaming kernel reads its parameters and logits while the kernel before it is still
    // running and waits for that kernel (griddepcontrol.wait) before it touches anything else; without it the wait is
    // the first thing it does
    bool overlap_previous;
    // the exact kernels follow in the same call and may take their places on the SMs while this one runs
    bool release_exact;
};

cudaError_t launch_sample_rows(const SampleArgs& args, const Workspace& ws, uint32_t splits, cudaStream_t stream);
// untruncated_rows: how many rows of the batch have no Top-K (clusters take those; the other rows a batch may hand
// over have a Top-K above MOE_SAMPLER_TOPK_FAST_MAX)
cudaError_t launch_sample_exact(const SampleArgs& args, const Workspace& ws, uint32_t untruncated_rows, cudaStream_t stream);
cudaError_t launch_merge_candidates(const uint64_t* gathered, uint32_t shards, uint32_t rows, uint32_t top_k, const moe_row_params* params,
                                    uint64_t step_offset, int32_t* token_id, float* probability, uint32_t* row_flags, int32_t* row_status,
                                    int32_t* topk_index, uint32_t topk_stride, cudaStream_t stream);

// Speculative verification of `sessions` Sessions with draft_count proposals each.  Rows of the row
// outputs and kept lists: Session b's target positions are rows b*(draft_count+1) .. +draft_count,
// its draft positions rows sessions*(draft_count+1) + b*draft_count .. +draft_count-1.
struct SpeculativeArgs
{
    uint32_t sessions;
    uint32_t draft_count;
    uint32_t vocab;
    const moe_row_params* params; // device, by row; a Session's options and counters are those of its first target row
    const int32_t* proposed;      // device, [sessions * draft_count]
    const int32_t* token;         // per-row sampler outputs
    const float* probability;
    const uint32_t* row_flags;
    const int32_t* row_status;
    const int32_t* kept_token;
    const float* kept_probability;
    const uint32_t* kept_count;
    uint32_t kept_stride;
    float* dense;             // [sessions * vocab] scratch: the residual by token id
    int32_t* residual_token;  // [sessions * vocab] scratch: its positive entries in token-id order
    float* residual_value;
    float* accepted_probability; // [sessions * draft_count]
    moe_speculative_result* result; // [sessions]
};

cudaError_t launch_speculative_verify(const SpeculativeArgs& args, cudaStream_t stream);

struct RouterArgs
{
    const float* logits;
    uint32_t token_count;
    moe_router_options options; // pointers are device pointers
    uint32_t* expert_offsets;
    uint32_t* route_token;
    uint32_t* route_rank;
    float* route_weight;
    int32_t* plan_status;
    // scratch
    uint32_t* selected_expert; // [token_count * top_k]
    float* selected_weight;    // [token_count * top_k]
    uint32_t* block_counts;    // [MOE_ROUTER_BLOCK_TABLE_ENTRIES]: routes per (expert, block of the select kernel)
    uint32_t tokens_per_block; // filled in by the launcher
};
struct RouterPartition
{
    uint32_t tokens_per_block;
    uint32_t blocks;
};
// blocks of the select kernel: about four per SM (148 SMs, four warps of one token each per block), fewer when
// the [expert][block] table would outgrow MOE_ROUTER_BLOCK_TABLE_ENTRIES
inline RouterPartition router_partition_host(uint32_t token_count, uint32_t experts)
{
    constexpr uint32_t kWarpsPerBlock = 4;
    RouterPartition part;
    part.tokens_per_block = kWarpsPerBlock * ((token_count + kWarpsPerBlock * 592u - 1u) / (kWarpsPerBlock * 592u));
    if (part.tokens_per_block == 0)
        part.tokens_per_block = kWarpsPerBlock;
    part.blocks = (token_count + part.tokens_per_block - 1u) / part.tokens_per_block;
    while (static_cast<uint64_t>(part.blocks) * experts > MOE_ROUTER_BLOCK_TABLE_ENTRIES)
    {
        part.tokens_per_block *= 2u;
        part.blocks = (token_count + part.tokens_per_block - 1u) / part.tokens_per_block;
    }
    if (part.blocks == 0)
        part.blocks = 1;
    return part;
}
// expert_counts: [expert_count] scratch; scan_done: one word that is 0 between calls; error_word: ~0 between calls
cudaError_t launch_router_dispatch_kernels(const RouterArgs& args, uint32_t* expert_counts, uint32_t* scan_done, unsigned long long* error_word,
                                           cudaStream_t stream);
// out_of_range: one device word, set to 1 when a route_token entry is >= token_count (its row is zero-filled)
cudaError_t launch_regroup_gather(const float* hidden, uint32_t token_count, uint32_t columns, const uint32_t* route_token, uint32_t route_count,
                                  float* gathered, int32_t* out_of_range, cudaStream_t stream);

// Kernels that need more than 48 KiB of dynamic shared memory must opt in with
// cudaFuncSetAttribute, which applies to the current device only: what has been
// configured is remembered per device ordinal (one SharedOptIn per kernel).
constexpr int kMaxDevices = 64;
struct SharedOptIn
{
    std::mutex guard; // held from the look at `bytes` until the attribute is set: nobody launches in between
    size_t bytes[kMaxDevices] = {};
};
// true when `shared_bytes` still has to be configured on `device`; records it as configured (the caller holds the guard
// and configures it)
inline bool opt_in_needed(SharedOptIn& state, int device, size_t shared_bytes)
{
    if (device < 0 || device >= kMaxDevices)
        return true; // untracked ordinal: configure on every launch
    if (state.bytes[device] >= shared_bytes)
        return false;
    state.bytes[device] = shared_bytes;
    return true;
}
template<typename Kernel>
cudaError_t opt_in_shared(SharedOptIn& state, Kernel kernel, size_t shared_bytes)
{
    int device = 0;
    cudaError_t status = cudaGetDevice(&device);
    if (status != cudaSuccess)
        return status;
    const std::lock_guard<std::mutex> lock(state.guard);
    if (!opt_in_needed(state, device, shared_bytes))
        return cudaSuccess;
    status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared_bytes));
    if (status != cudaSuccess && device >= 0 && device < kMaxDevices)
        state.bytes[device] = 0;
    return status;
}

// Clusters of 1, 2, 4, 8 and 16 CTAs of one kernel that a device holds at once; 0: none of that size.
constexpr int kClusterSizes = 5;
struct ClusterOccupancy
{
    int active[kClusterSizes] = {};
};
struct ClusterOccupancyTable
{
    std::mutex guard;
    bool known[kMaxDevices] = {};
    ClusterOccupancy found[kMaxDevices];
};
// query(size_index, &clusters) -> cudaError_t.  Asked once per device, unless a size up to the portable 8 was not
// answered: then the call makes do with what it has (clusters of one CTA at least) and the next one asks again.
template<typename Query>
ClusterOccupancy cluster_occupancy(ClusterOccupancyTable& table, int device, Query query)
{
    const bool tracked = device >= 0 && device < kMaxDevices;
    const std::lock_guard<std::mutex> lock(table.guard);
    if (tracked && table.known[device])
        return table.found[device];
    ClusterOccupancy found;
    bool answered = true;
    for (int i = 0; i < kClusterSizes; ++i)
    {
        if (query(i, &found.active[i]) == cudaSuccess)
            continue;
        found.active[i] = 0;
        answered = answered && (1 << i) > 8;
    }
    if (found.active[0] < 1)
        found.active[0] = 1;
    if (tracked && answered)
    {
        table.found[device] = found;
        table.known[device] = true;
    }
    return found;
}

// All kernels but the router's three launches (and the reset before them in moe_router_dispatch_static) are launched while
// the kernel before them in the stream may still run (programmatic stream serialization) and wait for it before they
// touch memory (wait_for_previous_kernel): the launch itself is out of the way when the earlier kernel ends.
// 1 to 3 us per launch.  The loads behind the wait are coherent ones: ld.global.nc and __ldg are for data that nobody
// writes while the kernel is resident.
inline cudaLaunchAttribute follow_closely()
{
    cudaLaunchAttribute attribute = {};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    return attribute;
}
template<typename... Parameters, typename... Arguments>
cudaError_t launch_following(void (*kernel)(Parameters...), uint32_t grid, uint32_t block, size_t shared_bytes, cudaStream_t stream, Arguments... arguments)
{
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(block, 1, 1);
    config.dynamicSmemBytes = shared_bytes;
    config.stream = stream;
    cudaLaunchAttribute attribute = follow_closely();
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Parameters>(arguments)...);
}

// Stable Top-K of every row of `scores` (score descending, index ascending): out_index [rows x top_k] in that
// order, 0xFFFFFFFF beyond min(top_k, count); out_score may be null.  top_k <= MOE_INDEXER_TOPK_MAX.
cudaError_t launch_indexer_topk(const float* scores, uint32_t rows, uint32_t count, size_t row_stride, uint32_t top_k, uint32_t* out_index,
                                float* out_score, int sm_count, cudaStream_t stream);

uint32_t choose_splits(uint32_t rows, uint32_t vocab, int dtype, int sm_count, uint32_t slice_slots, bool large_top_k, bool overlapped);

} // namespace moe

// ---- for tests; not part of the ABI ----
// Fixes the CTAs per row of the handle's clusters (1, 2, 4, 8 or 16; 0: chosen by the launcher).
extern "C" int moe_internal_set_cluster_ctas(moe_sampler* sampler, uint32_t ctas);
// Synchronises `stream`, copies Workspace::cluster_counts to the host and clears them.
extern "C" int moe_internal_cluster_counts(moe_sampler* sampler, void* stream, uint32_t* counts);
