// An fp32 row without Top-K finished by a thread-block cluster, without sorting the row.
// Included by moe_sample_exact.cu only (uses its helpers).
//
// While the accumulator of a left-to-right fp32 sum stays in one binade it is an integer multiple of
// its unit u, and an addend x moves it by the integer rn(x / u), whatever stood before it — except
// for a tie (x / u exactly between two integers), whose rounding depends on the accumulator's
// parity.  So inside one binade the order of the addends does not matter, and the rank order is only
// needed at a few places: where a tie, the end of a binade or the bound of the sum lies.
//
//   * The live logits are mapped to kGroups value groups (monotone, group 0 = the maximum); the row
//     is never reordered.  Every CTA of the cluster owns a contiguous slice of the row.
//   * The best kHead or more candidates (whole groups) are gathered, sorted and added literally: the
//     accumulator passes most of its binades there.
//   * For each of the three sums, every item adds its integer step — in the unit its group's binade
//     was guessed to have — to its group's counter in shared memory; the CTAs reduce the counters over
//     the cluster and scan them into the exact accumulator before every group (a 64-bit integer).
//   * Groups with a tie, near the end of a binade, near the bound, or entered in another binade than
//     guessed are "literal": their items are gathered, sorted, and added one by one; one warp walks
//     them in order and checks that every stretch between two of them stays in its binade and
//     below the bound.  A guess can therefore cost time, never a different result.
//   * What the method does not cover (Top-K rows, groups above kGroupLimit items, outcomes that reach below
//     the live window, a check that fails) is listed for the one-CTA kernel that runs behind this one.
//
// What bounds it: for one to twenty rows latency (about twenty cluster barriers and block scans, the
// sequential adds of the head); for hundreds of rows the issue slots of the item passes.  The one-CTA path
// it replaces for these rows put all live items in rank order first.  Calls of rows of 151936 logits
// 3 N(0,1), T 0.9, Top-P 0.95, streaming kernel included: 1 row 433 -> 123 us, 8 rows 450 -> 139, 64 rows
// 517 -> 313, 256 rows 1378 -> 734.

#include <cooperative_groups.h>

namespace moe {

namespace {

namespace cg = cooperative_groups;

// Debug builds: phases of rank 0, and sums of what happened (see moe_debug_exact_cycles).
#ifdef MOE_PHASE_TIMERS
#define CL_MARK(slot)                 \
    do                                \
    {                                 \
        if (rank == 0)                \
            MOE_EXACT_MARK(slot);     \
    } while (0)
#define CL_COUNT(slot, v)                                                                     \
    do                                                                                        \
    {                                                                                         \
        if (rank == 0 && threadIdx.x == 0)                                                    \
            atomicAdd(&g_exact_cycles[slot], static_cast<unsigned long long>(v));             \
    } while (0)
#else
#define CL_MARK(slot) do {} while (0)
#define CL_COUNT(slot, v) do {} while (0)
#endif

constexpr uint32_t kGroups = 16384;
// Items per group: as many as the literal list takes (equal logits, such as those of a padded vocabulary, share a group).
// An item behind the head is at most 1/kHead of the accumulator, which is below 2^24 units: its step is below kStepLimit
// unless the unit was guessed far too small, and kGroupLimit such steps fit the 31 bits of a counter.  The limit ends in
// one half, so that an item that reaches it looks like a tie and makes its group literal.
// With 120 items per group rows with 267 equal logits were left after two passes: 8 of them took 629 us, 604 without
// the clusters, 138 now; 256 of them 2690, 2280 and 730.
constexpr uint32_t kGroupLimit = 3072;
constexpr float kStepLimit = 131071.5f;
constexpr uint32_t kHead = 192;          // candidates added literally, rounded up to whole groups
constexpr uint32_t kHeadCapacity = 512;
constexpr uint32_t kLiteralGroups = 96;
constexpr uint32_t kLiteralItems = 3072; // dense rows (90 items a group) mark up to thirty groups that refining does not spare
constexpr uint32_t kFewLiteralItems = 256;
constexpr uint32_t kMaxCluster = 16;
constexpr uint32_t kDeadGroup = 0xFFFFu;
constexpr int kGuardUnits = 64;          // a group this close to the end of a binade or to the bound is literal
constexpr int kMaxGuesses = 5;
constexpr uint32_t kTieBit = 0x80000000u; // of a group's step counter: some item is a tie
static_assert(kGroupLimit <= kLiteralItems, "a group that has to be added literally fits the list");
static_assert((1u << 24) / kHead < 131071u && static_cast<uint64_t>(kGroupLimit) * 131072u < kTieBit, "the steps of a group fit its counter");

struct LiteralGroup
{
    uint64_t before; // accumulator before the group, in units of 2^(base_exponent - 23), ties rounded to even integers
    uint64_t after;
    uint32_t group;
    uint32_t pad;
};

enum ClusterAction : int
{
    kActionContinue = 0,
    kActionDone = 1,    // rank 0 has written the row's result
    kActionFallback = 2, // the one-CTA path takes the row
    kActionRepeat = 3    // the same sum once more, with the accumulator corrected behind `repeat_group`
};

// What rank 0 tells the others after a sum.
struct SumState
{
    int action;
    float total;
    float kept_total;
    float head_acc;        // accumulator of the next sum behind the head
    float floor_probability;
    uint32_t repeat_group;
    int64_t repeat_delta;
    uint64_t threshold;    // record of the last kept candidate (0: the list was not cut by Top-P)
};

// A correction of the scanned accumulators: `delta` for every group behind `group`.
struct Jump
{
    uint32_t group;
    int64_t delta;
};

struct ClusterStats
{
    uint32_t max_key, min_key, finite, pos_inf, low_bits;
};

struct alignas(16) ClusterShared
{
    uint32_t table[kGroups];   // per group: count, then steps of the current sum
    uint16_t count[kGroups];   // items of the group over the whole cluster
    uint8_t exponent[kGroups]; // guessed exponent of the accumulator before the group, biased by 127
    uint32_t literal_bits[kGroups / 32];
    // rank 0 only
    uint64_t head_in[kHeadCapacity];
    uint64_t head[kHeadCapacity];
    float head_value[kHeadCapacity];
    uint64_t item[kLiteralItems];          // as they come; many of them in rank order too
    uint64_t item_by_group[kLiteralItems]; // many: group by group; few: in rank order
    float item_value[kLiteralItems];
    LiteralGroup literal_in[kLiteralGroups];
    LiteralGroup literal[kLiteralGroups];
    uint32_t literal_begin[kLiteralGroups]; // where the group's items stand in the list
    uint32_t literal_end[kLiteralGroups];
    uint32_t head_count, item_count, literal_count;
    uint32_t literal_items; // items of the literal groups
    // every CTA
    ClusterStats stats[kMaxCluster];
    uint64_t cta_total[kMaxCluster];
    uint64_t warp_total[kExactWarps];
    float warp_sum[kExactWarps];
    uint32_t overfull;
    uint32_t head_end;
    uint32_t head_total; // candidates of the head
    uint32_t entry;
    Jump jump[kMaxGuesses];
    SumState state;
    SumState next_state; // rank 0: under construction
    uint32_t counts[4];  // Workspace::cluster_counts of this cluster
};
constexpr size_t kClusterSharedBytes = sizeof(ClusterShared);

__device__ __forceinline__ int high_bit(uint64_t v)
{
    return 63 - __clzll(static_cast<long long>(v));
}

// 2^e as a float, -126 <= e <= 127.
__device__ __forceinline__ float power_of_two(int e)
{
    return __uint_as_float(static_cast<uint32_t>(e + 127) << 23);
}

__device__ __forceinline__ double power_of_two_double(int e)
{
    return __longlong_as_double(static_cast<long long>(e + 1023) << 52);
}

__device__ __forceinline__ int exponent_of(float v)
{
    return static_cast<int>((__float_as_uint(v) >> 23) & 0xFFu) - 127;
}

// Calls visit(q, logits) for every group q of four consecutive logits of row[begin, end); NaN stands behind
// `end`.  Four 16-byte loads in flight per thread while the row is 16-byte aligned.
template<typename Visit>
__device__ __forceinline__ void for_each_four(const float* row, uint32_t begin, uint32_t end, Visit visit)
{
    const uint32_t vectors = (end - begin + 3u) / 4u;
    const bool aligned = (reinterpret_cast<uintptr_t>(row + begin) & 15u) == 0u;
    uint32_t q = threadIdx.x;
    if (aligned)
    {
        const float4* whole = reinterpret_cast<const float4*>(row + begin);
        const uint32_t whole_count = (end - begin) / 4u;
        for (; q + 3u * kExactThreads < whole_count; q += 4u * kExactThreads)
        {
            float4 v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u)
                v[u] = whole[q + u * kExactThreads];
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u)
                visit(q + u * kExactThreads, v[u]);
        }
    }
#pragma unroll 2
    for (; q < vectors; q += kExactThreads)
    {
        const uint32_t i = begin + 4u * q;
        float v[4];
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u)
            v[u] = i + u < end ? row[i + u] : __uint_as_float(0x7FC00000u);
        visit(q, make_float4(v[0], v[1], v[2], v[3]));
    }
}

// out[rank] = in[i] with rank = the number of larger records: four lanes per record.
__device__ __noinline__ void rank_records(const uint64_t* in, uint64_t* out, uint32_t n)
{
    const uint32_t part = threadIdx.x & 3u;
    for (uint32_t base = 0; base < n; base += kExactThreads / 4u)
    {
        const uint32_t i = base + (threadIdx.x >> 2);
        const uint64_t mine = i < n ? in[i] : 0ull;
        uint32_t rank = 0;
#pragma unroll 4
        for (uint32_t j = part; j < n; j += 4u)
            rank += in[j] > mine ? 1u : 0u;
        rank += __shfl_xor_sync(kFullMask, rank, 1);
        rank += __shfl_xor_sync(kFullMask, rank, 2);
        if (part == 0 && i < n)
            out[rank] = mine;
    }
}

// Literal fp32 adds of value[0..n) onto acc by one warp, every lane doing the same.
struct LiteralSum
{
    float acc;
    uint32_t stopped; // the sum met its bound at `index`
    uint32_t ended;   // value[index] no longer belongs to the list (negative)
    uint32_t index;
};
__device__ __noinline__ LiteralSum literal_sum(const float* value, uint32_t n, float acc, int kind, float bound)
{
    const uint32_t base = shared_address(value);
    const auto met = [&](float sum) { return kind == kSeqReachBound ? sum >= bound : (kind == kSeqExceedBound ? bound < sum : false); };
    uint32_t i = 0;
    float x[8];
#pragma unroll
    for (uint32_t u = 0; u < 8u; ++u)
        x[u] = u < n ? load_shared_f32(base + 4u * u) : 0.0f;
    while (i + 8u <= n)
    {
        // eight adds, one test: the addends are not negative, so a bound met on the way is met at the end
        float next[8];
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u)
            next[u] = i + 8u + u < n ? load_shared_f32(base + 4u * (i + 8u + u)) : 0.0f;
        float running = acc;
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u)
            running = __fadd_rn(running, x[u]);
        const float least = fminf(fminf(fminf(x[0], x[1]), fminf(x[2], x[3])), fminf(fminf(x[4], x[5]), fminf(x[6], x[7])));
        if (least < 0.0f || met(running))
            break;
        acc = running;
        i += 8u;
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u)
            x[u] = next[u];
    }
#pragma unroll 1
    for (; i < n; ++i)
    {
        const float addend = load_shared_f32(base + 4u * i);
        if (addend < 0.0f)
            return LiteralSum{acc, 0u, 1u, i};
        acc = __fadd_rn(acc, addend);
        if (met(acc))
            return LiteralSum{acc, 1u, 0u, i};
    }
    return LiteralSum{acc, 0u, 0u, n};
}

// Inclusive block scans (kExactThreads threads, all of them call).
__device__ __forceinline__ uint64_t block_scan_u64(uint64_t v, uint64_t* warp_total, uint64_t& block_total)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1)
    {
        const uint64_t other = __shfl_up_sync(kFullMask, v, offset);
        if (lane >= static_cast<uint32_t>(offset))
            v += other;
    }
    if (lane == 31)
        warp_total[warp] = v;
    __syncthreads();
    uint64_t w = warp_total[lane];
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1)
    {
        const uint64_t other = __shfl_up_sync(kFullMask, w, offset);
        if (lane >= static_cast<uint32_t>(offset))
            w += other;
    }
    block_total = __shfl_sync(kFullMask, w, 31);
    const uint64_t before = __shfl_sync(kFullMask, w, warp == 0 ? 0 : static_cast<int>(warp) - 1);
    __syncthreads();
    return warp == 0 ? v : v + before;
}
__device__ __forceinline__ float block_scan_float(float v, float* warp_sum)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1)
    {
        const float other = __shfl_up_sync(kFullMask, v, offset);
        if (lane >= static_cast<uint32_t>(offset))
            v += other;
    }
    if (lane == 31)
        warp_sum[warp] = v;
    __syncthreads();
    float w = warp_sum[lane];
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1)
    {
        const float other = __shfl_up_sync(kFullMask, w, offset);
        if (lane >= static_cast<uint32_t>(offset))
            w += other;
    }
    const float before = __shfl_sync(kFullMask, w, warp == 0 ? 0 : static_cast<int>(warp) - 1);
    __syncthreads();
    return warp == 0 ? v : v + before;
}

// Guesses the accumulator's exponent before every group from the group counts alone: the prefix sums
// of (count x the addend in the middle), four groups at a time, first in real numbers, then twice with
// the addends rounded to the unit of the exponent guessed before.  Every CTA computes the same table.
__device__ __noinline__ void guess_exponents(ClusterShared& cs, uint32_t first_group, float start, float factor, float log2_step)
{
    static_assert(kGroups == 16u * kExactThreads, "a thread guesses for sixteen groups");
    const uint32_t tid = threadIdx.x;
    const uint2* const words = reinterpret_cast<const uint2*>(cs.count + 16u * tid);
    float items[4], addend[4];
    int exponent[4] = {0, 0, 0, 0};
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k)
    {
        const uint32_t g = 16u * tid + 4u * k;
        const uint2 four = words[k];
        const uint32_t n = (g >= first_group ? four.x & 0xFFFFu : 0u) + (g + 1u >= first_group ? four.x >> 16 : 0u)
                           + (g + 2u >= first_group ? four.y & 0xFFFFu : 0u) + (g + 3u >= first_group ? four.y >> 16 : 0u);
        items[k] = static_cast<float>(n);
        addend[k] = factor * exp2f(-static_cast<float>(g + 2u) * log2_step);
    }
#pragma unroll
    for (int round = 0; round < 3; ++round)
    {
        float mass[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            mass[k] = items[k] * (round == 0 ? addend[k] : rintf(addend[k] * power_of_two(23 - exponent[k])) * power_of_two(exponent[k] - 23));
        const float sum = (mass[0] + mass[1]) + (mass[2] + mass[3]);
        float before = start + (block_scan_float(sum, cs.warp_sum) - sum);
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            exponent[k] = min(90, max(-90, exponent_of(before)));
            before += mass[k];
        }
    }
    uint32_t out[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        out[k] = static_cast<uint32_t>(exponent[k] + 127) * 0x01010101u;
    *reinterpret_cast<uint4*>(cs.exponent + 16u * tid) = make_uint4(out[0], out[1], out[2], out[3]);
    __syncthreads();
}

// Adds the peers' counters of this CTA's groups to its own (the tie bits are joined).  Sixteen bytes per
// remote load, at most four loads per thread, all of them in flight together.
__device__ __forceinline__ void reduce_table(ClusterShared& cs, cg::cluster_group& cluster, uint32_t owned_begin, uint32_t owned)
{
    const uint32_t cluster_size = cluster.num_blocks();
    if (cluster_size == 1u)
        return;
    const uint32_t rank = cluster.block_rank();
    const uint32_t quads = owned / 4u;
    const uint32_t sharers = quads < kExactThreads ? kExactThreads / quads : 1u; // threads that share a quad's peers
    for (uint32_t quad = threadIdx.x % quads; quad < quads; quad += kExactThreads)
    {
        uint4 sum = make_uint4(0u, 0u, 0u, 0u), tie = sum;
#pragma unroll 4
        for (uint32_t r = threadIdx.x / quads % sharers; r < cluster_size; r += sharers)
        {
            if (r == rank)
                continue;
            const uint4 peer = reinterpret_cast<const uint4*>(cluster.map_shared_rank(cs.table, r) + owned_begin)[quad];
            sum.x += peer.x & ~kTieBit;
            sum.y += peer.y & ~kTieBit;
            sum.z += peer.z & ~kTieBit;
            sum.w += peer.w & ~kTieBit;
            tie.x |= peer.x;
            tie.y |= peer.y;
            tie.z |= peer.z;
            tie.w |= peer.w;
        }
        uint32_t* own = cs.table + owned_begin + 4u * quad;
        const uint32_t sums[4] = {sum.x, sum.y, sum.z, sum.w};
        const uint32_t ties[4] = {tie.x, tie.y, tie.z, tie.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            if (sums[u] != 0u)
                atomicAdd(own + u, sums[u]);
            if ((ties[u] & kTieBit) != 0u)
                atomicOr(own + u, kTieBit);
        }
    }
    __syncthreads();
}

// What the items of a slice need to know for their steps.
struct StepArgs
{
    const float* row;
    float* item_x;
    const uint16_t* item_group;
    uint32_t begin, end;
    uint32_t vectors;
    uint32_t head_end;
    uint32_t active_last;
    float total, total_reciprocal;
    float kept_total, kept_reciprocal;
    float floor_probability;
    uint64_t threshold;
    float temperature, peak;
    bool aligned; // row + begin is 16-byte aligned
};

// Every item of the slice adds its integer step to its group's counter.  kFirst: the numerators are computed
// (and kept for the later passes) and the items of the head are handed to the first CTA.
template<int kSum, bool kFirst>
__device__ __forceinline__ void add_steps(const StepArgs& s, ClusterShared& cs, ClusterShared& first_cta)
{
    const uint32_t active_range = s.active_last - s.head_end; // wraps when nothing is left behind the head
    const bool any = s.active_last >= s.head_end;
    const uint32_t table_base = shared_address(cs.table);
    const uint32_t exponent_base = shared_address(cs.exponent);
    uint32_t q = threadIdx.x;
    if (q >= s.vectors)
        return;
    ushort4 gv = *reinterpret_cast<const ushort4*>(s.item_group + 4u * q);
    float4 xv;
    const auto load = [&]() {
        if (!kFirst)
        {
            xv = *reinterpret_cast<const float4*>(s.item_x + 4u * q);
            return;
        }
        float logit[4];
        const uint32_t i = s.begin + 4u * q;
        if (s.aligned && i + 4u <= s.end)
        {
            xv = *reinterpret_cast<const float4*>(s.row + i);
            return;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u)
            logit[u] = i + u < s.end ? s.row[i + u] : 0.0f;
        xv = make_float4(logit[0], logit[1], logit[2], logit[3]);
    };
    load();
    while (q < s.vectors)
    {
        const uint32_t g[4] = {gv.x, gv.y, gv.z, gv.w};
        float x[4] = {xv.x, xv.y, xv.z, xv.w};
        const uint32_t at = s.begin + 4u * q;
        float* const keep = s.item_x + 4u * q;
        q += kExactThreads;
        if (q < s.vectors)
        {
            gv = *reinterpret_cast<const ushort4*>(s.item_group + 4u * q);
            load();
        }
        if (kFirst)
        {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                x[u] = exact_expf(scaled_offset(x[u], s.temperature, s.peak)); // of no meaning for a dead item
            *reinterpret_cast<float4*>(keep) = make_float4(x[0], x[1], x[2], x[3]);
        }
        float t[4];
        bool active[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            active[u] = any && g[u] - s.head_end <= active_range; // dead items have the largest group number
            float value = x[u];
            // For numerators below the range of divide_by (a peak of 1e7 temperatures and more widens the live window to
            // them) the quotient may be off in its last bits: it is below 2^-70 then, the accumulators start above
            // 2^-25, so the item takes no step whatever they are, in or out of the Min-P list.
            if (kSum >= 1)
            {
                value = divide_by(value, s.total, s.total_reciprocal);
                active[u] = active[u] && value >= s.floor_probability; // 0 without Min-P
            }
            if (kSum == 2)
                value = divide_by(value, s.kept_total, s.kept_reciprocal);
            uint32_t exponent;
            asm("ld.shared.u8 %0, [%1];" : "=r"(exponent) : "r"(exponent_base + (active[u] ? g[u] : 0u)));
            t[u] = fminf(value * __uint_as_float((277u - exponent) << 23), kStepLimit); // value / unit
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            if (kFirst && g[u] < s.head_end)
            {
                const uint32_t slot = atomicAdd(&first_cta.head_count, 1u);
                if (slot < kHeadCapacity)
                    first_cta.head_in[slot] = make_record(ordered_key(s.row[at + u]), at + u);
            }
            if (!active[u] || t[u] < 0.5f)
                continue;
            if (kSum == 2 && g[u] == s.active_last && s.threshold != 0 && make_record(ordered_key(s.row[at + u]), at + u) < s.threshold)
                continue;
            const uint32_t address = table_base + 4u * g[u];
            asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(address), "r"(__float2uint_rn(t[u])) : "memory");
            if (t[u] - truncf(t[u]) == 0.5f)
                asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(address), "r"(kTieBit) : "memory");
        }
    }
}

// The walk of one sum over its literal groups, by one warp of rank 0 (every lane the same).
struct WalkResult
{
    float acc;
    uint32_t stopped;
    uint32_t ended;
    uint32_t failed;
    uint32_t item;       // position of the stopping item
    uint32_t last_group; // failed: the last literal group before the stretch that failed ...
    int64_t delta;       // ... and the accumulator behind it minus what the scan had
};

__device__ WalkResult walk_literal_groups(const ClusterShared& cs, uint32_t groups, uint32_t first_group, uint32_t last_group, uint64_t start, uint64_t end,
                                          int base_exponent, int kind, float bound, uint64_t bound_fixed, const Jump* jumps, uint32_t jump_count)
{
    const uint32_t lane = threadIdx.x & 31u;
    const double to_float = power_of_two_double(base_exponent - 23);
    const double to_fixed = power_of_two_double(23 - base_exponent);
    WalkResult result{0.0f, 0u, 0u, 0u, 0u, 0u, 0};
    uint32_t between_begin = first_group; // groups of the current stretch
    int64_t delta = 0;
    uint64_t previous = start;
    uint32_t position = 0;
    float acc = 0.0f;
    for (uint32_t j = 0;; ++j)
    {
        const bool last = j == groups;
        const uint64_t next = last ? end : cs.literal[j].before;
        const uint64_t first_fixed = previous + delta;
        const uint64_t last_fixed = next + delta;
        acc = static_cast<float>(static_cast<double>(last_fixed) * to_float);
        // the stretch of groups that were added as integers has to lie in the binade its steps were taken in
        const int e = high_bit(previous);
        const bool met = kind == kSeqReachBound ? acc >= bound : (kind == kSeqExceedBound ? bound < acc : false);
        // groups behind the bound are not looked at: the walk has to end before them
        const bool overran = last && kind != kSeqSumOnly && end > bound_fixed;
        if (overran || high_bit(first_fixed) != e || high_bit(last_fixed) != e || met || static_cast<uint64_t>(static_cast<double>(acc) * to_fixed) != last_fixed)
        {
            // ... unless it holds no items
            bool occupied = false;
            const uint32_t between_end = last ? last_group + 1u : cs.literal[j].group;
            for (uint32_t g = between_begin + lane; g < between_end; g += 32u)
                occupied |= cs.count[g] != 0;
            if (overran || __any_sync(kFullMask, occupied))
            {
                result.failed = 1u;
                result.last_group = between_begin - 1u;
                result.delta = delta;
                return result;
            }
        }
        if (last)
            break;
        const uint32_t items = cs.count[cs.literal[j].group];
        const LiteralSum sum = literal_sum(cs.item_value + position, items, acc, kind, bound);
        if (sum.stopped || sum.ended)
        {
            result.acc = sum.acc;
            result.stopped = sum.stopped;
            result.ended = sum.ended;
            result.item = position + sum.index;
            return result;
        }
        position += items;
        previous = cs.literal[j].after;
        delta = static_cast<int64_t>(static_cast<uint64_t>(static_cast<double>(sum.acc) * to_fixed)) - static_cast<int64_t>(previous);
        between_begin = cs.literal[j].group + 1u;
        for (uint32_t k = 0; k < jump_count; ++k)
            if (jumps[k].group == cs.literal[j].group)
            {
                previous += jumps[k].delta;
                delta -= jumps[k].delta;
            }
    }
    result.acc = acc;
    return result;
}

// One row by one cluster.  Every CTA takes the same decisions (they depend on published values only).
// Returns false when the row has to go through the one-CTA path.  `outcome` is valid in rank 0.
__device__ __noinline__ bool exact_row_cluster(const SampleArgs& a, uint32_t row, const moe_row_params& p, float* item_x, uint16_t* item_group, ClusterShared& cs,
                                  cg::cluster_group& cluster, RowOutcome& outcome)
{
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    const uint32_t cluster_size = cluster.num_blocks();
    const uint32_t rank = cluster.block_rank();
    const float* row_pointer = row_logits<float>(a, row);
    const ClusterSlice slice = cluster_slice(a.vocab, cluster_size, rank);
    const uint32_t begin = slice.begin;
    const uint32_t end = slice.end;
    const uint32_t vectors = (end - begin + 3u) / 4u;
    outcome = RowOutcome{MOE_ROW_OK, -1, 0.0f, 0u, false};

    MOE_EXACT_BEGIN();
    // ---- maximum, finite range, +inf ------------------------------------------------------
    for (uint32_t g = tid; g < kGroups; g += kExactThreads)
        cs.table[g] = 0;
    if (tid == 0)
    {
        cs.overfull = 0;
        cs.head_count = 0;
        cs.item_count = 0;
        cs.literal_count = 0;
        cs.head_end = kGroups;
        cs.head_total = 0;
        cs.stats[rank] = ClusterStats{0u, 0xFFFFFFFFu, 0u, 0u, 0u};
    }
    __syncthreads();
    {
        uint32_t max_key = 0, min_key = 0xFFFFFFFFu, finite = 0, low_bits = 0;
        bool pos_inf = false;
        const auto see = [&](float v) {
            pos_inf |= v == INFINITY;
            if (fabsf(v) < INFINITY)
            {
                const uint32_t key = ordered_key(v);
                max_key = max(max_key, key);
                min_key = min(min_key, key);
                ++finite;
                low_bits |= __float_as_uint(v);
            }
            else if (v != v && (__float_as_uint(v) & 0x007F0000u) == 0u)
            {
                low_bits |= 1u; // a NaN whose upper half alone would be an infinity
            }
        };
        for_each_four(row_pointer, begin, end, [&](uint32_t, const float4& v) {
            see(v.x);
            see(v.y);
            see(v.z);
            see(v.w);
        });
        max_key = __reduce_max_sync(kFullMask, max_key);
        min_key = __reduce_min_sync(kFullMask, min_key);
        finite = __reduce_add_sync(kFullMask, finite);
        low_bits = __reduce_or_sync(kFullMask, low_bits) & 0xFFFFu;
        const bool warp_pos_inf = __any_sync(kFullMask, pos_inf);
        if (lane == 0)
        {
            atomicMax(&cs.stats[rank].max_key, max_key);
            atomicMin(&cs.stats[rank].min_key, min_key);
            atomicAdd(&cs.stats[rank].finite, finite);
            if (low_bits != 0u)
                atomicOr(&cs.stats[rank].low_bits, low_bits);
            if (warp_pos_inf)
                cs.stats[rank].pos_inf = 1;
        }
    }
    __syncthreads();
    if (tid < cluster_size && tid != rank)
        *cluster.map_shared_rank(&cs.stats[rank], tid) = cs.stats[rank];
    cluster.sync();
    uint32_t max_key = 0, min_key = 0xFFFFFFFFu, finite_total = 0, pos_inf = 0, low_bits = 0;
    for (uint32_t r = 0; r < cluster_size; ++r)
    {
        max_key = max(max_key, cs.stats[r].max_key);
        min_key = min(min_key, cs.stats[r].min_key);
        finite_total += cs.stats[r].finite;
        pos_inf |= cs.stats[r].pos_inf;
        low_bits |= cs.stats[r].low_bits;
    }
    if (pos_inf != 0 || finite_total == 0)
    {
        outcome.status = MOE_ROW_NO_FINITE_LOGIT; // session.cpp:84-85,399
        return true;
    }
    if (low_bits == 0)
    {
        outcome.defer = true; // bf16 values widened to fp32: the one-CTA path replays them over value runs
        return false;
    }
    const float top = key_to_float(max_key);
    const float window_floor = live_window_floor(top, p.temperature);
    const float least = key_to_float(min_key);
    const float floor_value = window_floor > least ? window_floor : least;
    BucketMap map;
    map.top = top;
    const float range = __fsub_rn(top, floor_value);
    if (!(range > 0.0f) || !(range < INFINITY))
        return false; // one value, or a span fp32 cannot hold
    map.scale = __fdiv_rn(static_cast<float>(kGroups - 1u), range);
    const float log2_step = 1.44269504f / (map.scale * p.temperature); // exponent (base 2) per group
    if (!(map.scale < INFINITY) || !(log2_step > 0.0f) || !(log2_step < 1.0f))
        return false;
    static_assert(kGroups == kOrderBuckets, "order_bucket maps onto the groups");
    const auto group_of = [&](float v) { return min(kGroups - 1u, __float2uint_rz(__fmul_rn(__fsub_rn(map.top, v), map.scale))); };

    CL_MARK(16);
    // ---- groups and their counts ---------------------------------------------------------------
    const float peak = __fdiv_rn(top, p.temperature);
    for_each_four(row_pointer, begin, end, [&](uint32_t q, const float4& v) {
        const float logit[4] = {v.x, v.y, v.z, v.w};
        uint32_t g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const bool live = fabsf(logit[u]) < INFINITY && logit[u] >= floor_value;
            g[u] = live ? group_of(logit[u]) : kDeadGroup;
            if (live)
                atomicAdd(&cs.table[g[u]], 1u);
        }
        *reinterpret_cast<ushort4*>(item_group + 4u * q) = make_ushort4(static_cast<unsigned short>(g[0]), static_cast<unsigned short>(g[1]),
                                                                        static_cast<unsigned short>(g[2]), static_cast<unsigned short>(g[3]));
    });
    cluster.sync();
    CL_MARK(17);
    const uint32_t owned = kGroups / cluster_size; // groups whose counters this CTA reduces
    const uint32_t owned_begin = rank * owned;
    const uint32_t per_thread = owned / kExactThreads;
    {
        reduce_table(cs, cluster, owned_begin, owned);
        bool over = false;
        for (uint32_t i = tid; i < owned; i += kExactThreads)
        {
            const uint32_t n = cs.table[owned_begin + i];
            over |= n > kGroupLimit;
            cs.count[owned_begin + i] = static_cast<uint16_t>(min(n, 65535u));
        }
        __syncthreads();
        // my counts to every peer, two stores of sixteen bytes per thread
        const uint32_t packs = owned / 8u;
        static_assert(kGroups / 8u == 2u * kExactThreads, "two stores per thread");
#pragma unroll
        for (uint32_t i = tid; i < kGroups / 8u; i += kExactThreads)
        {
            const uint32_t peer = i / packs;
            if (peer != rank)
                reinterpret_cast<uint4*>(cluster.map_shared_rank(cs.count, peer) + owned_begin)[i % packs] =
                    reinterpret_cast<const uint4*>(cs.count + owned_begin)[i % packs];
        }
        if (__any_sync(kFullMask, over) && lane < cluster_size)
            *cluster.map_shared_rank(&cs.overfull, lane) = 1u;
    }
    cluster.sync();
    if (cs.overfull != 0)
        return false;

    // ---- the head: the first groups that hold kHead candidates or more -----------------------
    uint32_t live_total;
    {
        constexpr uint32_t kPerThread = kGroups / kExactThreads;
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < kPerThread / 2u; ++j)
        {
            const uint32_t two = reinterpret_cast<const uint32_t*>(cs.count + tid * kPerThread)[j];
            sum += (two & 0xFFFFu) + (two >> 16);
        }
        uint64_t total;
        const uint32_t inclusive = static_cast<uint32_t>(block_scan_u64(sum, cs.warp_total, total));
        uint32_t before = inclusive - sum;
        if (before < kHead && inclusive >= kHead)
        {
            for (uint32_t j = 0; j < kPerThread; ++j)
            {
                before += cs.count[tid * kPerThread + j];
                if (before >= kHead)
                {
                    cs.head_end = tid * kPerThread + j + 1u;
                    cs.head_total = before;
                    break;
                }
            }
        }
        live_total = static_cast<uint32_t>(total);
        __syncthreads();
    }
    CL_MARK(18);
    const uint32_t head_end = cs.head_end; // groups below it are the head
    if (cs.head_total > kHeadCapacity)
        return false; // its last group piles up
    const bool all_listed = live_total == finite_total;

    // groups behind this one hold nobody that passes the Min-P floor (the slack covers every rounding)
    uint32_t last_group = kGroups - 1u;
    if (p.min_p > 0.0f)
    {
        const float reach = -logf(p.min_p) * p.temperature + 0.1f * p.temperature + 9.5367431640625e-07f * fabsf(top);
        const float bounded = fminf(reach * map.scale + 2.0f, static_cast<float>(kGroups - 1u));
        last_group = __float2uint_rz(bounded);
    }
    const float uniform = philox_uniform(p.seed, p.row_id, p.step + a.step_offset);

    float total = 0.0f, kept_total = 0.0f, floor_probability = 0.0f;
    uint64_t threshold = 0;
    float head_acc = 0.0f;
    uint32_t active_last = kGroups - 1u; // groups behind it take no part in the current sum
    for (int sum = 0; sum < 3; ++sum)
    {
        const int kind = sum == 0 ? kSeqSumOnly : (sum == 1 ? kSeqReachBound : kSeqExceedBound);
        const float bound = sum == 0 ? 0.0f : (sum == 1 ? p.top_p : uniform);
        if (sum == 1)
            active_last = last_group;
        if (sum == 2 && threshold != 0)
            active_last = min(last_group, group_of(key_to_float(record_key(threshold))));
        const float factor = sum == 0 ? 1.0f : (sum == 1 ? 1.0f / total : 1.0f / total / kept_total);
        guess_exponents(cs, sum == 0 ? 0u : head_end, sum == 0 ? 0.0f : head_acc, factor, log2_step);
        if (sum == 0 && head_end < 4u)
        {
            // nothing stands before the first four groups, but the head may end among them: its addends are close to one
            if (tid < 4u)
                cs.exponent[tid] = static_cast<uint8_t>(exponent_of(static_cast<float>(cs.head_total) * exp2f(-2.0f * log2_step)) + 127);
            __syncthreads();
        }
        CL_MARK(19);
        // the fixed-point unit: one binade below the first guess while the head's sum is not known yet
        const int base_exponent = sum == 0 ? (head_end < kGroups ? static_cast<int>(cs.exponent[head_end]) - 128 : -1) : exponent_of(head_acc);
        uint32_t jump_count = 0;
        for (int guess = 0;; ++guess)
        {
            if (guess == kMaxGuesses)
                return false;
            // ---- integer steps of the items -------------------------------------------------
            for (uint32_t g = tid; g < kGroups / 4u; g += kExactThreads)
                reinterpret_cast<uint4*>(cs.table)[g] = make_uint4(0u, 0u, 0u, 0u);
            if (tid < kGroups / 32u)
                cs.literal_bits[tid] = 0;
            if (tid == 0)
            {
                cs.item_count = 0;
                cs.literal_count = 0;
                cs.literal_items = 0;
            }
            __syncthreads();
            const bool gather_head = sum == 0 && guess == 0;
            const StepArgs step_args{row_pointer, item_x, item_group, begin, end, vectors, head_end, active_last, total, __frcp_rn(total), kept_total,
                                     __frcp_rn(kept_total), floor_probability, threshold, p.temperature, peak,
                                     (reinterpret_cast<uintptr_t>(row_pointer + begin) & 15u) == 0u};
            ClusterShared& first_cta = *cluster.map_shared_rank(&cs, 0);
            if (gather_head)
                add_steps<0, true>(step_args, cs, first_cta);
            else if (sum == 0)
                add_steps<0, false>(step_args, cs, first_cta);
            else if (sum == 1)
                add_steps<1, false>(step_args, cs, first_cta);
            else
                add_steps<2, false>(step_args, cs, first_cta);
            cluster.sync();

            CL_MARK(20);
            // ---- reduction over the cluster, exact accumulator before every group ----------------
            reduce_table(cs, cluster, owned_begin, owned);
            uint64_t own = 0;
            for (uint32_t j = 0; j < per_thread; ++j)
            {
                const uint32_t g = owned_begin + tid * per_thread + j;
                const int shift = static_cast<int>(cs.exponent[g]) - 127 - base_exponent;
                own += shift >= 0 ? static_cast<uint64_t>(cs.table[g] & ~kTieBit) << min(shift, 32) : 0ull;
            }
            uint64_t cta_total;
            const uint64_t inclusive = block_scan_u64(own, cs.warp_total, cta_total);
            if (tid < cluster_size)
                *cluster.map_shared_rank(&cs.cta_total[rank], tid) = cta_total;
            if (gather_head && rank == 0)
            {
                const uint32_t heads = min(cs.head_count, kHeadCapacity);
                rank_records(cs.head_in, cs.head, heads);
                __syncthreads();
                for (uint32_t i = tid; i < heads; i += kExactThreads)
                    cs.head_value[i] = exact_expf(scaled_offset(key_to_float(record_key(cs.head[i])), p.temperature, peak));
                __syncthreads();
                if (warp == 0)
                {
                    const float acc = literal_sum(cs.head_value, heads, 0.0f, kSeqSumOnly, 0.0f).acc;
                    if (lane < cluster_size)
                        cluster.map_shared_rank(&cs.state, lane)->head_acc = acc;
                }
            }
            cluster.sync();
            CL_MARK(21);
            if (gather_head)
                head_acc = cs.state.head_acc;
            if (exponent_of(head_acc) < base_exponent)
                return false; // the first guess was off by more than a binade
            const uint64_t start = static_cast<uint64_t>(static_cast<double>(head_acc) * power_of_two_double(23 - base_exponent));
            uint64_t running = start + inclusive - own;
            uint64_t finish = start;
            for (uint32_t r = 0; r < cluster_size; ++r)
            {
                if (r < rank)
                    running += cs.cta_total[r];
                finish += cs.cta_total[r];
            }
            const uint64_t bound_fixed = sum == 0 ? ~0ull : static_cast<uint64_t>(static_cast<double>(bound) * power_of_two_double(23 - base_exponent));
            const uint64_t first_running = running;
            // corrections that hold for group g
            const auto jumped = [&](uint32_t g) {
                int64_t delta = 0;
                for (uint32_t k = 0; k < jump_count; ++k)
                    if (cs.jump[k].group < g)
                        delta += cs.jump[k].delta;
                return delta;
            };
            finish += jumped(kGroups);
            for (uint32_t j = 0; j < per_thread; ++j)
            {
                const uint32_t g = owned_begin + tid * per_thread + j;
                if (g < head_end || g > active_last || cs.count[g] == 0)
                    continue;
                const uint32_t steps = cs.table[g] & ~kTieBit;
                const int shift = static_cast<int>(cs.exponent[g]) - 127 - base_exponent;
                const int64_t correction = jump_count != 0 ? jumped(g) : 0;
                const uint64_t before = running + correction;
                if (shift >= 0)
                    running += static_cast<uint64_t>(steps) << min(shift, 32);
                if (sum != 0 && before > bound_fixed + (static_cast<uint64_t>(kGuardUnits) << max(shift, 0)))
                    continue; // the sum ends before this group (the walk checks that)
                const bool tied = cs.table[g] >= kTieBit;
                bool literal = tied || shift < 0 || high_bit(before) != 23 + shift;
                if (!literal && steps != 0)
                {
                    const uint64_t guard = static_cast<uint64_t>(kGuardUnits) << shift;
                    const uint64_t after = running + correction;
                    literal = high_bit(after + guard) != 23 + shift || high_bit(before - guard) != 23 + shift
                              || (sum != 0 && after + guard >= bound_fixed);
                }
                if (literal)
                {
                    const uint32_t slot = atomicAdd(&first_cta.literal_count, 1u);
                    atomicAdd(&first_cta.literal_items, static_cast<uint32_t>(cs.count[g]));
                    if (slot < kLiteralGroups)
                        cluster.map_shared_rank(cs.literal_in, 0)[slot] = LiteralGroup{before, running + correction, g, 0u};
                }
            }
            cluster.sync();
            const uint32_t literal_groups = first_cta.literal_count;
            const uint32_t literal_items = first_cta.literal_items;
            CL_MARK(22);
            CL_COUNT(27, literal_groups);
            CL_COUNT(28, 1);
            // exponents of my groups behind `from`, taken from the accumulators found
            const auto publish_exponents = [&](uint32_t from) {
                running = first_running;
                for (uint32_t j = 0; j < per_thread; ++j)
                {
                    const uint32_t g = owned_begin + tid * per_thread + j;
                    const int shift = static_cast<int>(cs.exponent[g]) - 127 - base_exponent;
                    const uint64_t before = running + jumped(g);
                    if (g >= head_end && shift >= 0)
                        running += static_cast<uint64_t>(cs.table[g] & ~kTieBit) << min(shift, 32);
                    if (g <= from && from != 0u)
                        continue;
                    const uint8_t exponent = static_cast<uint8_t>(min(217, max(37, base_exponent + high_bit(before) - 23 + 127)));
                    for (uint32_t r = 0; r < cluster_size; ++r)
                        cluster.map_shared_rank(cs.exponent, r)[g] = exponent;
                }
            };
            if (literal_groups > kLiteralGroups || literal_items > kLiteralItems)
            {
                // the guess was too far off: repeat with the exponents of the accumulators just found; a better guess that
                // marks few groups with too many items shows that refining does not help
                if (guess > 0 && literal_groups <= kLiteralGroups)
                    return false;
                publish_exponents(0u);
                jump_count = 0;
                if (tid == 0)
                    ++cs.counts[3];
                cluster.sync();
                continue;
            }

            // ---- gather the items of the literal groups ------------------------------------------
            if (literal_groups != 0)
            {
                for (uint32_t j = tid; j < literal_groups; j += kExactThreads)
                {
                    const uint32_t g = cluster.map_shared_rank(cs.literal_in, 0)[j].group;
                    atomicOr(&cs.literal_bits[g >> 5], 1u << (g & 31u));
                }
                __syncthreads();
#pragma unroll 4
                for (uint32_t q = tid; q < vectors; q += kExactThreads)
                {
                    const ushort4 gv = *reinterpret_cast<const ushort4*>(item_group + 4u * q);
                    const uint32_t g[4] = {gv.x, gv.y, gv.z, gv.w};
                    uint32_t hits = 0;
#pragma unroll
                    for (uint32_t u = 0; u < 4u; ++u)
                    {
                        const uint32_t in_range = g[u] <= active_last ? g[u] : 0u; // group 0 is part of the head, never literal
                        hits |= ((cs.literal_bits[in_range >> 5] >> (in_range & 31u)) & 1u) << u;
                    }
                    while (hits != 0u)
                    {
                        const uint32_t i = begin + 4u * q + static_cast<uint32_t>(__ffs(static_cast<int>(hits))) - 1u;
                        hits &= hits - 1u;
                        const uint32_t slot = atomicAdd(&first_cta.item_count, 1u);
                        if (slot < kLiteralItems)
                            first_cta.item[slot] = make_record(ordered_key(row_pointer[i]), i);
                    }
                }
            }
            cluster.sync();

            CL_MARK(23);
            CL_COUNT(29, cs.item_count);
            // ---- rank 0 walks them ----------------------------------------------------------------
            if (rank == 0)
            {
                SumState state{kActionContinue, total, kept_total, 0.0f, floor_probability, 0u, 0, threshold};
                const uint32_t items = cs.item_count;
                const uint32_t heads = cs.head_count;
                if (items > kLiteralItems || heads > kHeadCapacity)
                {
                    state.action = kActionFallback;
                }
                else
                {
                    // the literal groups in rank order, and where the items of each stand
                    if (tid < literal_groups)
                    {
                        uint32_t before = 0, items_before = 0;
                        for (uint32_t j = 0; j < literal_groups; ++j)
                        {
                            const bool earlier = cs.literal_in[j].group < cs.literal_in[tid].group;
                            before += earlier ? 1u : 0u;
                            items_before += earlier ? cs.count[cs.literal_in[j].group] : 0u;
                        }
                        cs.literal[before] = cs.literal_in[tid];
                        cs.literal_begin[before] = items_before;
                        cs.literal_end[before] = items_before; // grows to the end as the items come in
                    }
                    // Rank order: a few items are compared all with all; more of them inside their groups, behind two more
                    // barriers (half a microsecond), where all with all grows to 180 us for a dense row's 2400.
                    const bool few = items <= kFewLiteralItems;
                    const uint64_t* const ranked = few ? cs.item_by_group : cs.item;
                    if (few)
                        rank_records(cs.item, cs.item_by_group, items);
                    __syncthreads();
                    // place in `literal` of an item's group
                    const auto literal_of = [&](uint64_t record) {
                        const uint32_t g = group_of(key_to_float(record_key(record)));
                        uint32_t low = 0, high = literal_groups;
                        while (high - low > 1u)
                        {
                            const uint32_t middle = (low + high) / 2u;
                            if (cs.literal[middle].group <= g)
                                low = middle;
                            else
                                high = middle;
                        }
                        return low;
                    };
                    if (!few)
                    {
                        for (uint32_t i = tid; i < items; i += kExactThreads)
                        {
                            const uint64_t record = cs.item[i];
                            cs.item_by_group[atomicAdd(&cs.literal_end[literal_of(record)], 1u)] = record;
                        }
                        __syncthreads();
                        for (uint32_t i = tid; i < items; i += kExactThreads)
                        {
                            const uint64_t record = cs.item_by_group[i];
                            const uint32_t at = literal_of(record);
                            uint32_t rank_in_group = 0;
#pragma unroll 4
                            for (uint32_t j = cs.literal_begin[at]; j < cs.literal_end[at]; ++j)
                                rank_in_group += cs.item_by_group[j] > record ? 1u : 0u;
                            cs.item[cs.literal_begin[at] + rank_in_group] = record;
                        }
                        __syncthreads();
                    }
                    for (uint32_t i = tid; i < items; i += kExactThreads)
                    {
                        const uint64_t record = ranked[i];
                        float value = exact_expf(scaled_offset(key_to_float(record_key(record)), p.temperature, peak));
                        bool listed = true;
                        if (sum >= 1)
                        {
                            value = __fdiv_rn(value, total);
                            listed = !(p.min_p > 0.0f) || value >= floor_probability;
                        }
                        if (sum == 2)
                        {
                            listed = listed && record >= threshold;
                            value = __fdiv_rn(value, kept_total);
                        }
                        cs.item_value[i] = listed ? value : -1.0f;
                    }
                    __syncthreads();
                    CL_MARK(25);
                    if (warp == 0)
                    {
                        const WalkResult walk = walk_literal_groups(cs, literal_groups, head_end, active_last, start, finish, base_exponent, kind, bound, bound_fixed, cs.jump,
                                                                    jump_count);
                        if (walk.failed)
                        {
                            state.action = walk.delta != 0 ? kActionRepeat : kActionFallback;
                            state.repeat_group = walk.last_group;
                            state.repeat_delta = walk.delta;
                        }
                        else if (sum == 0)
                        {
                            state.total = walk.acc;
                            if (!(walk.acc - walk.acc == 0.0f) || walk.acc <= 0.0f)
                            {
                                outcome.status = MOE_ROW_INVALID_DISTRIBUTION; // session.cpp:102-103
                                state.action = kActionDone;
                            }
                        }
                        else if (sum == 1)
                        {
                            state.kept_total = walk.acc;
                            state.threshold = walk.stopped ? ranked[walk.item] : 0ull;
                        }
                        else
                        {
                            outcome.flags = MOE_ROW_FLAG_USED_UNIFORM;
                            state.action = kActionDone;
                            uint64_t chosen = 0;
                            if (walk.stopped)
                                chosen = ranked[walk.item];
                            else if (threshold != 0)
                                chosen = threshold; // session.cpp:441-442: the last candidate if the sum never passes the uniform
                            else
                                state.action = kActionFallback; // the last candidate of the list is not known here
                            if (chosen != 0)
                            {
                                const float x = exact_expf(scaled_offset(key_to_float(record_key(chosen)), p.temperature, peak));
                                outcome.token = static_cast<int32_t>(record_index(chosen));
                                outcome.probability = __fdiv_rn(__fdiv_rn(x, total), kept_total);
                            }
                        }
                        if (lane == 0)
                            cs.next_state = state;
                    }
                    __syncthreads();
                    CL_MARK(26);
                    state = cs.next_state;
                    // the head's part of the next sum; a row whose list or draw ends inside the head is finished here
                    if (state.action == kActionContinue && sum == 0)
                    {
                        for (uint32_t i = tid; i < heads; i += kExactThreads)
                            cs.head_value[i] = __fdiv_rn(cs.head_value[i], state.total);
                        __syncthreads();
                        state.floor_probability = __fmul_rn(cs.head_value[0], p.min_p);
                        __syncthreads();
                        if (p.min_p > 0.0f)
                            for (uint32_t i = tid; i < heads; i += kExactThreads)
                                if (!(cs.head_value[i] >= state.floor_probability))
                                    cs.head_value[i] = -1.0f; // not listed: a suffix, probabilities do not increase
                        __syncthreads();
                        if (warp == 0)
                        {
                            const LiteralSum nucleus = literal_sum(cs.head_value, heads, 0.0f, kSeqReachBound, p.top_p);
                            state.head_acc = nucleus.acc;
                            if (nucleus.stopped || nucleus.ended || (head_end == kGroups && all_listed))
                            {
                                state.action = kActionDone;
                                const uint32_t kept = nucleus.stopped ? nucleus.index + 1u : nucleus.index;
                                if (kept == 1u)
                                {
                                    outcome.token = static_cast<int32_t>(record_index(cs.head[0]));
                                    outcome.probability = 1.0f; // session.cpp:429-430: no uniform drawn
                                }
                                else
                                {
                                    outcome.flags = MOE_ROW_FLAG_USED_UNIFORM;
                                    for (uint32_t i = lane; i < kept; i += 32u)
                                        cs.head_value[i] = __fdiv_rn(cs.head_value[i], nucleus.acc);
                                    __syncwarp();
                                    const LiteralSum draw = literal_sum(cs.head_value, kept, 0.0f, kSeqExceedBound, uniform);
                                    const uint32_t chosen = draw.stopped ? draw.index : kept - 1u;
                                    outcome.token = static_cast<int32_t>(record_index(cs.head[chosen]));
                                    outcome.probability = cs.head_value[chosen];
                                }
                            }
                            if (lane == 0)
                                cs.next_state = state;
                        }
                    }
                    else if (state.action == kActionContinue && sum == 1)
                    {
                        for (uint32_t i = tid; i < heads; i += kExactThreads)
                            cs.head_value[i] = __fdiv_rn(cs.head_value[i], state.kept_total);
                        __syncthreads();
                        if (warp == 0)
                        {
                            const LiteralSum draw = literal_sum(cs.head_value, heads, 0.0f, kSeqExceedBound, uniform);
                            state.head_acc = draw.acc;
                            if (draw.stopped)
                            {
                                state.action = kActionDone;
                                outcome.flags = MOE_ROW_FLAG_USED_UNIFORM;
                                outcome.token = static_cast<int32_t>(record_index(cs.head[draw.index]));
                                outcome.probability = cs.head_value[draw.index];
                            }
                            if (lane == 0)
                                cs.next_state = state;
                        }
                    }
                    __syncthreads();
                    state = cs.next_state;
                }
                if (tid < cluster_size)
                    *cluster.map_shared_rank(&cs.state, tid) = state;
            }
            cluster.sync();
            CL_MARK(24);
            if (cs.state.action != kActionRepeat)
                break;
            // a stretch left the binade (or met the bound) because ties and binade ends before it had moved the
            // accumulator: the same literal groups up to there, the rest with the corrected accumulator
            if (guess + 1 == kMaxGuesses)
                return false;
            if (tid == 0)
            {
                cs.jump[jump_count] = Jump{cs.state.repeat_group, cs.state.repeat_delta};
                ++cs.counts[2];
            }
            ++jump_count;
            __syncthreads();
            publish_exponents(cs.state.repeat_group);
            cluster.sync();
        }
        const SumState state = cs.state;
        if (state.action == kActionFallback)
            return false;
        if (state.action == kActionDone)
            return true;
        total = state.total;
        kept_total = state.kept_total;
        floor_probability = state.floor_probability;
        threshold = state.threshold;
        head_acc = state.head_acc;
    }
    return false; // not reached: the third sum ends the row
}

// Clusters take rows from the hand-over list; nobody waits on another cluster.
__global__ void __launch_bounds__(kExactThreads, 1) sample_exact_cluster_kernel(const SampleArgs a, Workspace ws)
{
    extern __shared__ __align__(16) uint32_t cluster_words[];
    ClusterShared& cs = *reinterpret_cast<ClusterShared*>(cluster_words);
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const uint32_t cluster_size = cluster.num_blocks();
    const uint32_t tid = threadIdx.x;
    grid_dependency_release(); // every cluster is resident: the one-CTA kernel behind takes no place from any
    wait_for_previous_kernel();
    const uint32_t pending = *ws.exact_count;
    if (pending == 0)
        return; // the counters are as the next call needs them
    const uint32_t slot_stride = (ws.max_vocab + 3u) & ~3u;
    // the cluster's items (numerators, then group numbers) in the slot of its number, every CTA its slice
    const uint32_t cluster_index = blockIdx.x / cluster_size;
    uint32_t* items = ws.sort_keys + static_cast<size_t>(cluster_index) * 4u * slot_stride;
    const uint32_t item_begin = cluster_slice(a.vocab, cluster_size, rank).begin;
    if (tid < 4u)
        cs.counts[tid] = 0;
    cluster.sync(); // every CTA of the cluster runs before its shared memory is written to
    for (;;)
    {
        if (rank == 0 && tid == 0)
        {
            const uint32_t next = atomicAdd(ws.exact_next, 1u);
            for (uint32_t r = 0; r < cluster_size; ++r)
                *cluster.map_shared_rank(&cs.entry, r) = next;
        }
        cluster.sync();
        const uint32_t entry = cs.entry;
        if (entry >= pending)
            break;
        const uint32_t row = ws.exact_rows[entry];
        const moe_row_params p = a.params[row];
        bool handled = false;
        RowOutcome outcome{MOE_ROW_OK, -1, 0.0f, 0u, false};
        if (p.top_k == 0 && a.kept_count == nullptr)
            handled = exact_row_cluster(a, row, p, reinterpret_cast<float*>(items) + item_begin,
                                        reinterpret_cast<uint16_t*>(items + slot_stride) + item_begin, cs, cluster, outcome);
        if (rank == 0)
        {
            __syncthreads();
            if (!handled)
            {
                if (tid == 0)
                {
                    ws.exact_deferred[atomicAdd(ws.exact_deferred_count, 1u)] = row | (outcome.defer ? kBf16ValuedRow : 0u);
                    ++cs.counts[1];
                }
            }
            else
            {
                if (a.topk_index != nullptr)
                    for (uint32_t i = tid; i < a.topk_stride; i += kExactThreads)
                        a.topk_index[static_cast<size_t>(row) * a.topk_stride + i] = -1;
                if (tid == 0)
                {
                    if (outcome.status == MOE_ROW_OK && is_stop_token(a.stop_offsets, a.stop_tokens, row, outcome.token))
                        outcome.flags |= MOE_ROW_FLAG_STOP_TOKEN;
                    write_row_result(a, row, outcome.token, outcome.probability, outcome.flags, outcome.status);
                    ++cs.counts[0];
                }
            }
        }
        cluster.sync();
    }
    if (rank == 0 && tid < 4u && cs.counts[tid] != 0u)
        atomicAdd(ws.cluster_counts + tid, cs.counts[tid]);
    if (tid == 0)
    {
        __threadfence();
        if (atomicAdd(ws.exact_done, 1u) == gridDim.x - 1)
        {
            *ws.exact_count = 0; // every CTA has read it: ready for the next call
            *ws.exact_done = 0;
            *ws.exact_next = 0;
            __threadfence();
        }
    }
}

// CTAs per row.  A row costs a part that does not shrink with the cluster (barriers, scans, sequential adds) and a
// part that does (the passes over its items); clusters run side by side as far as the device holds them.  The size with the
// smallest rounds x (fixed + passes / size) wins.  Alone, a call of one row fits 110 + 214 / size us; the 45 and 200 below
// count a further round as what it adds while others run, and they choose the best measured size at every batch but one
// (80 rows: 400 against 376).  Clusters of 1, 2, 4, 8, 16 CTAs, us per call, 151936 logits a row:
// 1 row 324, 211, 161, 132, 124; 8 rows 331, 219, 167, 138, 182; 20 rows 333, 224, 170, 218, 313; 64 rows 352, 244, 317, 493,
// 878; 100 rows 376, 397, 473, 719, 1315; 160 rows 605, 556, 692, 1119, 2101; 256 rows 736, 793, 1072, 1778, 3378.
// The rows counted are those without Top-K; how many of them the streaming kernel hands over is not known here.
cudaError_t launch_sample_exact_cluster(const SampleArgs& args, const Workspace& ws, uint32_t untruncated_rows, cudaStream_t stream)
{
    static SharedOptIn opt_in;
    static ClusterOccupancyTable occupancy;
    if (cudaError_t status = opt_in_shared(opt_in, sample_exact_cluster_kernel, kClusterSharedBytes))
        return status;
    int device = 0;
    if (cudaError_t status = cudaGetDevice(&device))
        return status;
    cudaLaunchConfig_t config = {};
    config.blockDim = dim3(kExactThreads, 1, 1);
    config.dynamicSmemBytes = kClusterSharedBytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    const ClusterOccupancy known = cluster_occupancy(occupancy, device, [&](int size_index, int* clusters) {
        cudaError_t status = cudaFuncSetAttribute(sample_exact_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (status == cudaSuccess)
        {
            attribute[0].val.clusterDim.x = 1u << size_index;
            config.gridDim = dim3(1u << size_index, 1, 1);
            status = cudaOccupancyMaxActiveClusters(clusters, sample_exact_cluster_kernel, &config);
        }
        if (status != cudaSuccess)
            (void)cudaGetLastError(); // this size is not available
        return status;
    });
    const uint32_t rows = untruncated_rows < args.rows ? untruncated_rows : args.rows;
    const double passes = 200.0 * static_cast<double>(args.vocab) / 150000.0;
    const double fixed = 45.0;
    uint32_t best = 0;
    double best_cost = 0.0;
    for (uint32_t i = 0; i < kClusterSizes; ++i)
    {
        const uint32_t size = 1u << i;
        const uint32_t resident = known.active[i] < static_cast<int>(ws.slots) ? static_cast<uint32_t>(known.active[i]) : ws.slots;
        if (resident == 0)
            continue;
        const double rounds = static_cast<double>((rows + resident - 1u) / resident);
        const double cost = rounds * (fixed + passes / size);
        if (best_cost == 0.0 || cost < best_cost)
        {
            best = i;
            best_cost = cost;
        }
    }
    for (uint32_t i = 0; i < kClusterSizes; ++i)
        if (ws.cluster_ctas == 1u << i && known.active[i] > 0)
            best = i;
    const uint32_t size = 1u << best;
    const uint32_t resident = known.active[best] < static_cast<int>(ws.slots) ? static_cast<uint32_t>(known.active[best]) : ws.slots;
    const uint32_t clusters = rows < resident ? rows : resident;
    attribute[0].val.clusterDim.x = size;
    config.gridDim = dim3(clusters * size, 1, 1);
    attribute[1] = follow_closely();
    config.numAttrs = 2;
    return cudaLaunchKernelEx(&config, sample_exact_cluster_kernel, args, ws);
}

} // namespace

} // namespace moe
