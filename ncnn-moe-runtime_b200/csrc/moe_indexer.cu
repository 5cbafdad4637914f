// Stable Top-K over rows of scores: the latent-attention indexer's choice of
// compressed history entries (src/kernels/cpu_latent_attention.cpp:377-425 of
// the reference: std::partial_sort of {index, score} pairs with
// scored_index_precedes, :257-262 — score descending, index ascending on equal
// scores — and the first index_top_k indices in that order).
//
// Rows of up to 1024 scores are put in order whole, one record per thread (indexer_short_rows_kernel).
// Longer ones: one CTA per row.  The row is read once: as much of it as fits stays in shared
// memory (40 000 scores), later passes read the rest again from L2.  The 32-bit
// order-preserving keys are counted by their upper 14 bits, which spreads
// ordinary scores over a hundred counters and more (a byte digit leaves them in a
// few).  Entries above the digit the k-th largest key falls into are taken; those
// inside it are ranked against each other while they are few, and by two more
// digits (14 and 4 bits) otherwise — equal scores, lowest indices first.  The
// taken (key, index) records — the record and ordering primitive of the sampler —
// are put in order by a monotone map of their keys onto 4096 or 8192 buckets and a look
// inside each bucket, or, where keys pile up, by a bitonic network that runs in
// registers for strides inside a warp and through shared memory for the others.
//
// What bounds it: latency and shared-memory instructions of one SM per row.  With
// byte digits, match.any aggregation, six passes over L2 and a bitonic sort in
// shared memory, before and after: 64 rows x 40000 scores, top 2048 82.0 -> 27.3 us;
// 64 x 131072, top 2048 260 -> 72; 64 x 2300, top 2048 30.0 -> 11.4; 1000 x 2300, top
// 512 75.7 -> 50.7; 64 x 1024, top 512 13.3 -> 6.6; 4000 x 300, top 64 130 -> 55.  What
// got slower: rows between 1024 and some 9000 scores that nearly all agree in the upper
// 14 key bits take all three digits and the network (1000 x 2300, top 512, 1 + 1e-6 N(0,1)
// 76.8 -> 87.3; 64 of them 16.8 -> 16.6; top 64 12.7 -> 15.7).

#include "moe_common.cuh"
#include "moe_internal.h"

namespace moe {

namespace {

constexpr int kIndexThreads = 1024;
constexpr int kIndexWarps = kIndexThreads / 32;

constexpr uint32_t kDigitBits = 14;
constexpr uint32_t kDigits = 1u << kDigitBits;
// scores of the row kept in shared memory: what is left of 227 KiB beside the counters
constexpr uint32_t kResidentScores = (227u * 1024u - 5u * 1024u - kDigits * 4u) / 16u * 4u;
constexpr uint32_t kZeroDigit = 0x80000000u >> (32 - kDigitBits); // zeros, the most common score by far
constexpr uint32_t kCandidates = 512;   // entries of the boundary digit that are ranked directly
// buckets of the final order; fewer of them where two CTAs share an SM
template<int kCtas>
constexpr uint32_t kOrderKeysFor = kCtas == 1 ? 8192u : 4096u;
// Records a bucket may hold (else the bitonic network): a look inside costs n / 32 x records shared loads, and the
// network for 1024 to 2048 records as much as about 4000 of them.
__device__ __forceinline__ uint32_t order_limit(uint32_t n)
{
    return min(256u, 131072u / max(n, 1u));
}
constexpr size_t kHalfSharedBytes = 113u * 1024u; // of an SM's 228 KiB, with 1 KiB per CTA for the system
constexpr size_t kRowOffset = sizeof(uint32_t) * kDigits + 5u * 1024u; // of the resident scores in shared memory

struct IndexerShared
{
    uint32_t warp_total[kIndexWarps];
    uint32_t digit;
    uint32_t above;
    uint32_t in_digit;
    uint32_t taken;
    uint32_t candidates;
    uint32_t max_key;
    uint32_t largest;
    uint32_t tiny; // some score shares the zeros' digit
};
static_assert(sizeof(IndexerShared) <= 1024, "the candidates start 1 KiB behind the counters");

// NaN scores make the reference's comparator inconsistent; here they rank last.
__device__ __forceinline__ uint32_t score_key(float value)
{
    return (value == value) ? ordered_key(value) : 0u;
}

// A row as groups of four scores.  Behind `count` stands a NaN: it ranks below everything, and callers that
// must not see it check the index.
struct ScoreRow
{
    const float* row;
    const float4* resident; // the first `resident_fours` groups, in shared memory
    uint32_t resident_fours;
    uint32_t count;
    bool aligned;

    __device__ __forceinline__ float4 global_four(uint32_t q) const
    {
        const uint32_t i = 4u * q;
        if (aligned && i + 4u <= count)
            return *reinterpret_cast<const float4*>(row + i);
        const float nothing = __uint_as_float(0x7FC00000u);
        float4 v = make_float4(nothing, nothing, nothing, nothing);
        if (i < count)
            v.x = row[i];
        if (i + 1u < count)
            v.y = row[i + 1u];
        if (i + 2u < count)
            v.z = row[i + 2u];
        if (i + 3u < count)
            v.w = row[i + 3u];
        return v;
    }
    __device__ __forceinline__ float4 four(uint32_t q) const
    {
        return q < resident_fours ? resident[q] : global_four(q);
    }
};

// Counts one digit per lane; `active` lanes only.  The digit of the first active lane is counted for all
// lanes that share it by one atomic: equal scores (the many zeros) would otherwise queue on one counter.
__device__ __forceinline__ void count_digit(uint32_t* hist, uint32_t digit, bool active)
{
    const unsigned voters = __ballot_sync(kFullMask, active);
    if (voters == 0u)
        return;
    const int first = __ffs(static_cast<int>(voters)) - 1;
    const uint32_t common = __shfl_sync(kFullMask, digit, first);
    const unsigned same = __ballot_sync(kFullMask, active && digit == common);
    const int lane = static_cast<int>(threadIdx.x & 31u);
    if (lane == first)
        atomicAdd(hist + common, static_cast<uint32_t>(__popc(same)));
    else if (active && digit != common)
        atomicAdd(hist + digit, 1u);
}

// Descending order of kItems * kThreads records, thread-major by warp: element j of a thread is
// position warp * 32 * kItems + 32 * j + lane.  `buffer` holds two images of the list.
template<int kItems, int kThreads>
__device__ void bitonic_descending(uint64_t (&v)[kItems], uint64_t* buffer)
{
    constexpr uint32_t kWarpSpan = 32u * kItems;
    constexpr uint32_t kTotal = kThreads * kItems;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t first = (threadIdx.x >> 5) * kWarpSpan + lane;
    uint32_t image = 0;
#pragma unroll 1
    for (uint32_t size = 2; size <= kTotal; size <<= 1)
    {
#pragma unroll 1
        for (uint32_t stride = size >> 1; stride >= kWarpSpan; stride >>= 1)
        {
            uint64_t* const list = buffer + image * kTotal; // alternating images: one barrier per stage
            image ^= 1u;
#pragma unroll
            for (int j = 0; j < kItems; ++j)
                list[first + 32u * j] = v[j];
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kItems; ++j)
            {
                const uint32_t position = first + 32u * j;
                const uint64_t other = list[position ^ stride];
                const bool take_larger = ((position & size) == 0u) == ((position & stride) == 0u);
                v[j] = (v[j] > other) == take_larger ? v[j] : other;
            }
        }
#pragma unroll
        for (int span = kItems / 2; span > 0; span >>= 1)
        {
            if (size < 64u * span)
                continue;
#pragma unroll
            for (int j = 0; j < kItems; ++j)
            {
                if ((j & span) != 0)
                    continue;
                const bool descending = ((first + 32u * j) & size) == 0u;
                const uint64_t a = v[j], b = v[j + span];
                if ((a < b) == descending)
                {
                    v[j] = b;
                    v[j + span] = a;
                }
            }
        }
#pragma unroll 1
        for (uint32_t stride = min(size >> 1, 16u); stride > 0; stride >>= 1)
        {
#pragma unroll
            for (int j = 0; j < kItems; ++j)
            {
                const uint32_t position = first + 32u * j;
                const uint64_t other = __shfl_xor_sync(kFullMask, v[j], static_cast<int>(stride));
                const bool take_larger = ((position & size) == 0u) == ((position & stride) == 0u);
                v[j] = (v[j] > other) == take_larger ? v[j] : other;
            }
        }
    }
}

// A short row (at most kThreads scores): the network puts all of it in rank order, one record per thread; the scores decide
// nothing about the time.  What bounds it: shuffles and barriers.  The digits' counters cost the same whatever the row's
// length and fill most of an SM: 4000 rows x 300, top 64 took 231 us, 130 with byte digits.
template<int kThreads>
__global__ void __launch_bounds__(kThreads) indexer_short_rows_kernel(const float* scores, uint32_t count, size_t row_stride, uint32_t top_k, uint32_t* out_index,
                                                                      float* out_score)
{
    __shared__ uint64_t buffer[2 * kThreads];
    const uint32_t tid = threadIdx.x;
    wait_for_previous_kernel();
    const float* row = scores + static_cast<size_t>(blockIdx.x) * row_stride;
    const uint32_t selected = min(top_k, count);
    out_index += static_cast<size_t>(blockIdx.x) * top_k;
    if (out_score != nullptr)
        out_score += static_cast<size_t>(blockIdx.x) * top_k;
    uint64_t v[1] = {tid < count ? make_record(score_key(row[tid]), tid) : 0ull};
    bitonic_descending<1, kThreads>(v, buffer);
    if (tid < selected)
    {
        const uint32_t index = record_index(v[0]);
        out_index[tid] = index;
        if (out_score != nullptr)
            out_score[tid] = row[index];
    }
    for (uint32_t position = selected + tid; position < top_k; position += kThreads)
    {
        out_index[position] = 0xFFFFFFFFu;
        if (out_score != nullptr)
            out_score[position] = 0.0f;
    }
}

// kCtas: CTAs per SM.
template<int kItems, int kCtas>
__global__ void __launch_bounds__(kIndexThreads, kCtas) indexer_topk_kernel(const float* scores, uint32_t count, size_t row_stride, uint32_t top_k,
                                                                     uint32_t resident_fours, uint32_t* out_index, float* out_score)
{
    constexpr uint32_t kOrderKeys = kOrderKeysFor<kCtas>;
    extern __shared__ __align__(16) unsigned char shared_raw[];
    uint32_t* const hist = reinterpret_cast<uint32_t*>(shared_raw);
    IndexerShared& sh = *reinterpret_cast<IndexerShared*>(shared_raw + sizeof(uint32_t) * kDigits);
    uint64_t* const candidates = reinterpret_cast<uint64_t*>(shared_raw + sizeof(uint32_t) * kDigits + 1024u);
    float4* const resident = reinterpret_cast<float4*>(shared_raw + kRowOffset);
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    wait_for_previous_kernel();
    const float* row = scores + static_cast<size_t>(blockIdx.x) * row_stride;
    const uint32_t selected = min(top_k, count);
    out_index += static_cast<size_t>(blockIdx.x) * top_k;
    if (out_score != nullptr)
        out_score += static_cast<size_t>(blockIdx.x) * top_k;
    for (uint32_t position = selected + tid; position < top_k; position += kIndexThreads)
    {
        out_index[position] = 0xFFFFFFFFu;
        if (out_score != nullptr)
            out_score[position] = 0.0f;
    }
    if (selected == 0)
        return;
    const auto write = [&](uint32_t position, uint64_t record) {
        const uint32_t key = record_key(record);
        const uint32_t index = record_index(record);
        out_index[position] = index;
        // the key has lost the sign of a zero and the bits of a NaN
        if (out_score != nullptr)
            out_score[position] = key == 0x80000000u || key == 0u ? row[index] : key_to_float(key);
    };
    const uint32_t fours = (count + 3u) / 4u;
    const ScoreRow in{row, resident, resident_fours, count, (reinterpret_cast<uintptr_t>(row) & 15u) == 0u};
    const uint32_t trips = (fours + kIndexThreads - 1u) / kIndexThreads; // every lane of a warp takes part in every trip

    // ---- the selected-th largest key, digit by digit -----------------------------------
    uint32_t threshold = 0;         // digits decided so far (high bits)
    uint32_t remaining = selected;  // rank still looked for among the keys that match them
    uint32_t equal_total = count;   // keys that match them
    bool few = false;               // only the first digit is decided, and few keys have it
    if (tid == 0)
        sh.tiny = 0u;
#pragma unroll 1
    for (int level = 0; level < 3; ++level)
    {
        const int shift = level == 0 ? 18 : (level == 1 ? 4 : 0);
        const uint32_t digits = level == 2 ? 16u : kDigits;
        const uint32_t decided = level == 0 ? 0u : (level == 1 ? 0xFFFC0000u : 0xFFFFFFF0u);
        for (uint32_t d = tid; d < kDigits / 4u; d += kIndexThreads)
            reinterpret_cast<uint4*>(hist)[d] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        if (level == 0)
        {
            uint32_t zeros = 0; // of the warp's lanes: counted once, at the end
            bool tiny = false;
            for (uint32_t trip = 0; trip < trips; trip += 5u)
            {
                float4 v[5];
                const float nothing = __uint_as_float(0x7FC00000u);
#pragma unroll
                for (uint32_t t = 0; t < 5u; ++t)
                {
                    const uint32_t q = (trip + t) * kIndexThreads + tid;
                    v[t] = q < fours ? in.global_four(q) : make_float4(nothing, nothing, nothing, nothing);
                }
#pragma unroll
                for (uint32_t t = 0; t < 5u; ++t)
                {
                    const uint32_t q = (trip + t) * kIndexThreads + tid;
                    if (q < resident_fours)
                        resident[q] = v[t];
                    const float s[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
#pragma unroll
                    for (uint32_t u = 0; u < 4u; ++u)
                    {
                        const uint32_t key = score_key(s[u]);
                        const uint32_t digit = key >> 18;
                        zeros += digit == kZeroDigit ? 1u : 0u; // the padding is no zero
                        tiny |= digit == kZeroDigit && key != 0x80000000u;
                        count_digit(hist, digit, digit != kZeroDigit && 4u * q + u < count);
                    }
                }
            }
            zeros = __reduce_add_sync(kFullMask, zeros);
            if (lane == 0 && zeros != 0u)
                atomicAdd(hist + kZeroDigit, zeros);
            if (tiny)
                sh.tiny = 1u;
        }
        else
        {
#pragma unroll 1
            for (uint32_t trip = 0; trip < trips; ++trip)
            {
                const uint32_t q = trip * kIndexThreads + tid;
                float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (q < fours)
                {
                    const float4 v = in.four(q);
                    s[0] = v.x;
                    s[1] = v.y;
                    s[2] = v.z;
                    s[3] = v.w;
                }
                bool match[4];
#pragma unroll
                for (uint32_t u = 0; u < 4u; ++u)
                    match[u] = 4u * q + u < count && (score_key(s[u]) & decided) == threshold;
                if (__any_sync(kFullMask, match[0] || match[1] || match[2] || match[3]))
                {
#pragma unroll
                    for (uint32_t u = 0; u < 4u; ++u)
                        count_digit(hist, (score_key(s[u]) >> shift) & (digits - 1u), match[u]);
                }
            }
        }
        __syncthreads();
        // thread t owns sixteen digits, thread 0 the largest ones
        const uint32_t lowest = kDigits - 16u * (tid + 1u);
        uint32_t counts[16];
        uint32_t sum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const uint4 four = reinterpret_cast<const uint4*>(hist + lowest)[k];
            counts[4 * k] = four.x;
            counts[4 * k + 1] = four.y;
            counts[4 * k + 2] = four.z;
            counts[4 * k + 3] = four.w;
            sum += four.x + four.y + four.z + four.w;
        }
        uint32_t scan = sum;
#pragma unroll
        for (int offset = 1; offset < 32; offset <<= 1)
        {
            const uint32_t other = __shfl_up_sync(kFullMask, scan, offset);
            if (lane >= static_cast<uint32_t>(offset))
                scan += other;
        }
        if (lane == 31)
            sh.warp_total[warp] = scan;
        __syncthreads();
        const uint32_t warp_total = sh.warp_total[lane];
        const uint32_t before_warp = __reduce_add_sync(kFullMask, lane < warp ? warp_total : 0u);
        uint32_t above = before_warp + scan - sum;
        if (above < remaining && above + sum >= remaining)
        {
#pragma unroll
            for (int k = 15; k >= 0; --k)
            {
                if (above < remaining && above + counts[k] >= remaining)
                {
                    sh.digit = lowest + k;
                    sh.above = above;
                    sh.in_digit = counts[k];
                }
                above += counts[k];
            }
        }
        __syncthreads();
        threshold |= sh.digit << shift;
        remaining -= sh.above;
        equal_total = sh.in_digit;
        few = level == 0 && equal_total <= kCandidates;
        if (few || (level == 0 && sh.digit == kZeroDigit && sh.tiny == 0u))
            break; // ... or every key of that digit is a zero
    }

    // ---- the records of the selection: their order of arrival does not matter, the sort decides ----
    uint64_t* const records = reinterpret_cast<uint64_t*>(hist); // kItems * 1024 records; the counters have served
    static_assert(sizeof(uint64_t) * 8u * kIndexThreads <= sizeof(uint32_t) * kDigits, "the records reuse the counters' memory");
    // The entries above the boundary: its digit, when only that is decided (then those inside it are candidates), or
    // its key (then the rest of the selection are equal keys, lowest indices first).
    const uint32_t boundary = threshold >> 18;
    const uint32_t cut = few ? threshold | 0x3FFFFu : threshold;
    const uint32_t above_total = selected - remaining;
    if (tid == 0)
    {
        sh.taken = 0;
        sh.candidates = 0;
        sh.max_key = 0;
        sh.largest = 0;
    }
    __syncthreads();
    uint32_t max_key = 0;
#pragma unroll 1
    for (uint32_t trip = 0; trip < trips; ++trip)
    {
        const uint32_t q = trip * kIndexThreads + tid;
        const float nothing = __uint_as_float(0x7FC00000u);
        const float4 v = q < fours ? in.four(q) : make_float4(nothing, nothing, nothing, nothing);
        const float s[4] = {v.x, v.y, v.z, v.w};
        uint32_t key[4];
        unsigned takers[4];
        uint32_t total = 0, mine = 0;
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u)
        {
            key[u] = score_key(s[u]);
            const bool take = key[u] > cut; // never the padding
            takers[u] = __ballot_sync(kFullMask, take);
            mine |= (take ? 1u : 0u) << u;
            total += __popc(takers[u]);
            if (few && (key[u] >> 18) == boundary && 4u * q + u < count)
                candidates[atomicAdd(&sh.candidates, 1u)] = make_record(key[u], 4u * q + u);
        }
        if (total == 0u)
            continue;
        uint32_t slot = 0;
        if (lane == 0)
            slot = atomicAdd(&sh.taken, total);
        slot = __shfl_sync(kFullMask, slot, 0);
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u)
        {
            if ((mine >> u) & 1u)
            {
                max_key = max(max_key, key[u]);
                records[slot + __popc(takers[u] & ((1u << lane) - 1u))] = make_record(key[u], 4u * q + u);
            }
            slot += __popc(takers[u]);
        }
    }
    max_key = __reduce_max_sync(kFullMask, max_key);
    if (lane == 0)
        atomicMax(&sh.max_key, max_key);
    if (!few)
    {
        // entries equal to the threshold: the `remaining` lowest indices.  Each warp owns a contiguous part of the row.
        const uint32_t part = (fours + kIndexWarps * 32u - 1u) / (kIndexWarps * 32u) * 32u;
        const uint32_t begin = min(fours, warp * part);
        const uint32_t end = min(fours, begin + part);
        const auto equal_mask = [&](uint32_t q) {
            uint32_t mask = 0;
            if (q < end)
            {
                const float4 v = in.four(q);
                const float s[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (uint32_t u = 0; u < 4u; ++u)
                    mask |= (4u * q + u < count && score_key(s[u]) == threshold ? 1u : 0u) << u;
            }
            return mask;
        };
        uint32_t here = 0;
        for (uint32_t base = begin; base < end; base += 32u)
            here += __popc(equal_mask(base + lane));
        here = __reduce_add_sync(kFullMask, here);
        if (lane == 0)
            sh.warp_total[warp] = here;
        __syncthreads();
        const uint32_t warp_total = sh.warp_total[lane];
        uint32_t before = __reduce_add_sync(kFullMask, lane < warp ? warp_total : 0u);
        for (uint32_t base = begin; base < end && before < remaining; base += 32u)
        {
            uint32_t mask = equal_mask(base + lane);
            const uint32_t mine = __popc(mask);
            uint32_t scan = mine;
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1)
            {
                const uint32_t other = __shfl_up_sync(kFullMask, scan, offset);
                if (lane >= static_cast<uint32_t>(offset))
                    scan += other;
            }
            uint32_t rank = before + scan - mine;
            for (; mask != 0u && rank < remaining; mask &= mask - 1u, ++rank)
                write(above_total + rank, make_record(threshold, 4u * (base + lane) + static_cast<uint32_t>(__ffs(static_cast<int>(mask))) - 1u));
            before += __shfl_sync(kFullMask, scan, 31);
        }
    }
    __syncthreads();
    // the row's scores have served: bucket counters, then the records in bucket order
    uint32_t* const bucket_end = reinterpret_cast<uint32_t*>(shared_raw + kRowOffset);
    uint64_t* const ordered = reinterpret_cast<uint64_t*>(shared_raw + kRowOffset + sizeof(uint32_t) * kOrderKeys);
    const uint32_t top = sh.max_key;
    const uint32_t range = top - cut - 1u; // of the taken keys, wraps only when none is taken
    const bool dense = range < kOrderKeys;
    const uint32_t scale = dense ? 0u : static_cast<uint32_t>((static_cast<uint64_t>(kOrderKeys) << 32) / (static_cast<uint64_t>(range) + 1u));
    const auto bucket_of = [&](uint64_t record) {
        const uint32_t below = top - record_key(record);
        return dense ? below : __umulhi(below, scale);
    };
    for (uint32_t i = tid; i < kOrderKeys / 4u; i += kIndexThreads)
        reinterpret_cast<uint4*>(bucket_end)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (uint32_t i = tid; i < above_total; i += kIndexThreads)
        atomicAdd(bucket_end + bucket_of(records[i]), 1u);
    if (few) // the candidates, two threads each, in the meantime
    {
        const uint64_t mine = tid / 2u < equal_total ? candidates[tid / 2u] : 0ull;
        uint32_t rank = 0;
#pragma unroll 4
        for (uint32_t j = tid & 1u; j < equal_total; j += 2u)
            rank += candidates[j] > mine ? 1u : 0u;
        rank += __shfl_xor_sync(kFullMask, rank, 1);
        if ((tid & 1u) == 0u && tid / 2u < equal_total && rank < remaining)
            write(above_total + rank, mine);
    }
    __syncthreads();
    uint32_t counts[kOrderKeys / kIndexThreads];
    uint32_t sum = 0, largest = 0;
#pragma unroll
    for (uint32_t k = 0; k < kOrderKeys / kIndexThreads / 4u; ++k)
    {
        const uint4 four = reinterpret_cast<const uint4*>(bucket_end + kOrderKeys / kIndexThreads * tid)[k];
        counts[4u * k] = four.x;
        counts[4u * k + 1u] = four.y;
        counts[4u * k + 2u] = four.z;
        counts[4u * k + 3u] = four.w;
        sum += four.x + four.y + four.z + four.w;
        largest = max(max(max(four.x, four.y), max(four.z, four.w)), largest);
    }
    uint32_t scan = sum;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1)
    {
        const uint32_t other = __shfl_up_sync(kFullMask, scan, offset);
        if (lane >= static_cast<uint32_t>(offset))
            scan += other;
    }
    largest = __reduce_max_sync(kFullMask, largest);
    if (lane == 31)
    {
        sh.warp_total[warp] = scan;
        atomicMax(&sh.largest, largest);
    }
    __syncthreads();
    if (sh.largest <= order_limit(above_total))
    {
        const uint32_t warp_total = sh.warp_total[lane];
        uint32_t before = __reduce_add_sync(kFullMask, lane < warp ? warp_total : 0u) + scan - sum;
#pragma unroll
        for (uint32_t k = 0; k < kOrderKeys / kIndexThreads; ++k)
        {
            bucket_end[kOrderKeys / kIndexThreads * tid + k] = before;
            before += counts[k];
        }
        __syncthreads();
        for (uint32_t i = tid; i < above_total; i += kIndexThreads)
        {
            const uint64_t record = records[i];
            ordered[atomicAdd(bucket_end + bucket_of(record), 1u)] = record;
        }
        __syncthreads();
        for (uint32_t i = tid; i < above_total; i += kIndexThreads)
        {
            const uint64_t record = ordered[i];
            const uint32_t bucket = bucket_of(record);
            const uint32_t begin = bucket == 0u ? 0u : bucket_end[bucket - 1u];
            const uint32_t end = bucket_end[bucket];
            uint32_t rank = begin;
#pragma unroll 4
            for (uint32_t j = begin; j < end; ++j)
                rank += ordered[j] > record ? 1u : 0u;
            write(rank, record);
        }
        return;
    }
    for (uint32_t i = above_total + tid; i < kItems * kIndexThreads; i += kIndexThreads)
        records[i] = 0ull;
    __syncthreads();
    uint64_t v[kItems];
    const uint32_t first = warp * 32u * kItems + lane;
#pragma unroll
    for (int j = 0; j < kItems; ++j)
        v[j] = records[first + 32u * j];
    __syncthreads();
    bitonic_descending<kItems, kIndexThreads>(v, reinterpret_cast<uint64_t*>(shared_raw + kRowOffset));
#pragma unroll
    for (int j = 0; j < kItems; ++j)
        if (first + 32u * j < above_total)
            write(first + 32u * j, v[j]);
}

// groups of four scores kept in shared memory
uint32_t resident_fours_of(uint32_t count)
{
    const uint32_t fours = count / 4u + (count % 4u != 0u ? 1u : 0u);
    return fours < kResidentScores / 4u ? fours : kResidentScores / 4u;
}
template<int kItems, int kCtas>
size_t indexer_shared_bytes(uint32_t count)
{
    // the buckets and the ordered records, or the network's two images of the list, take the place of the resident scores
    const size_t list_bytes = sizeof(uint64_t) * kItems * kIndexThreads;
    const size_t bucket_bytes = sizeof(uint32_t) * kOrderKeysFor<kCtas>;
    const size_t sort_bytes = list_bytes + (list_bytes > bucket_bytes ? list_bytes : bucket_bytes);
    const size_t row_bytes = sizeof(float) * 4u * resident_fours_of(count);
    return kRowOffset + (row_bytes > sort_bytes ? row_bytes : sort_bytes);
}

template<int kItems, int kCtas>
cudaError_t launch_indexer(const float* scores, uint32_t rows, uint32_t count, size_t row_stride, uint32_t top_k, uint32_t* out_index, float* out_score,
                           int sm_count, cudaStream_t stream)
{
    if constexpr (kCtas == 1 && kItems <= 2)
    {
        // More rows than SMs: two CTAs share one, if their rows and lists fit.  A CTA alone is a little faster with all the
        // registers and buckets (64 x 40000, top 2048: 27.3 us, 29.1 without), but waits a good part of its time: 1000 rows x
        // 2300, top 512 62.7 -> 50.7 us, 1000 x 9000, top 2048 91.5 -> 79.4.
        if (rows > static_cast<uint32_t>(sm_count) && indexer_shared_bytes<kItems, 2>(count) <= kHalfSharedBytes)
            return launch_indexer<kItems, 2>(scores, rows, count, row_stride, top_k, out_index, out_score, sm_count, stream);
    }
    const size_t shared_bytes = indexer_shared_bytes<kItems, kCtas>(count);
    static SharedOptIn opt_in;
    if (cudaError_t status = opt_in_shared(opt_in, indexer_topk_kernel<kItems, kCtas>, shared_bytes))
        return status;
    return launch_following(indexer_topk_kernel<kItems, kCtas>, rows, kIndexThreads, shared_bytes, stream, scores, count, row_stride, top_k,
                            resident_fours_of(count), out_index, out_score);
}

template<int kThreads>
cudaError_t launch_short_rows(const float* scores, uint32_t rows, uint32_t count, size_t row_stride, uint32_t top_k, uint32_t* out_index, float* out_score,
                              cudaStream_t stream)
{
    if constexpr (kThreads < kIndexThreads)
    {
        if (count > kThreads)
            return launch_short_rows<2 * kThreads>(scores, rows, count, row_stride, top_k, out_index, out_score, stream);
    }
    return launch_following(indexer_short_rows_kernel<kThreads>, rows, kThreads, 0, stream, scores, count, row_stride, top_k, out_index, out_score);
}

} // namespace

cudaError_t launch_indexer_topk(const float* scores, uint32_t rows, uint32_t count, size_t row_stride, uint32_t top_k, uint32_t* out_index,
                                float* out_score, int sm_count, cudaStream_t stream)
{
    if (rows == 0 || top_k == 0)
        return cudaSuccess;
    if (count <= kIndexThreads) // one record per thread
        return launch_short_rows<32>(scores, rows, count, row_stride, top_k, out_index, out_score, stream);
    const uint32_t selected = top_k < count ? top_k : count;
    if (selected <= kIndexThreads)
        return launch_indexer<1, 1>(scores, rows, count, row_stride, top_k, out_index, out_score, sm_count, stream);
    if (selected <= 2u * kIndexThreads)
        return launch_indexer<2, 1>(scores, rows, count, row_stride, top_k, out_index, out_score, sm_count, stream);
    if (selected <= 4u * kIndexThreads)
        return launch_indexer<4, 1>(scores, rows, count, row_stride, top_k, out_index, out_score, sm_count, stream);
    return launch_indexer<8, 1>(scores, rows, count, row_stride, top_k, out_index, out_score, sm_count, stream);
}

} // namespace moe
