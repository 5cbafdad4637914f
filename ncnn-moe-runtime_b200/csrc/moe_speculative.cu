// Verification step of speculative decoding, one CTA per Session
// (src/engine/session.cpp:776-880): walk the proposed tokens, accept each with
// probability min(1, p_target / p_draft) (:800-835), and produce the token
// that follows the accepted prefix — a draw from the residual distribution
// max(0, target - draft) after a rejection (sample_residual_distribution,
// :150-202), else the sample of the next target row.
//
// The distributions come from the sampler kernels (kept-candidate lists, the
// vectors sampling_distribution returns); this kernel is the control flow on
// top of them.  One CTA per Session: the walk is sequential by nature (position j is only
// looked at when 0..j-1 were accepted), the look-ups and the residual are
// spread over the threads.  The residual sums run in token-id order like the
// reference's std::accumulate over its dense vector; zeros change nothing in
// an fp32 sum, so only the positive entries are added, in that order.

#include "moe_common.cuh"
#include "moe_internal.h"
#include "moe_seqscan.cuh"

namespace moe {

namespace {

constexpr int kVerifyThreads = 1024;
constexpr int kVerifyWarps = kVerifyThreads / 32;
// Kept lists up to this length (every Session has a Top-K up to it) are looked up by one warp each and
// their residual is built in shared memory; longer ones (rows without Top-K) take the whole block and a
// dense vector over the vocabulary.
constexpr uint32_t kShortList = MOE_SPECULATIVE_SHORT_LIST;

struct VerifyShared
{
    SeqShared<kVerifyThreads> seq;
    float found[2];
    float found_all[2 * MOE_SPECULATIVE_MAX_DRAFT]; // short lists: the proposal's probability, target then draft of each position
    int32_t list_token[2][kShortList];              // short lists: the rejected position's target and draft candidates
    float list_value[2][kShortList];
    float residual[kShortList];                     // ... and its residual in token-id order
    int32_t residual_id[kShortList];
    uint32_t warp_count[kVerifyWarps];
    uint32_t cursor;
    uint32_t decision; // 0 accepted, 1 rejected, 2 error
};

// candidate_probability (session.cpp:138-148): the probability listed for `token`, 0 if absent.
// Token ids are unique in a list, so at most one thread writes.
__device__ float list_probability(const int32_t* tokens, const float* probabilities, uint32_t count, int32_t token, float* slot)
{
    if (threadIdx.x == 0)
        *slot = 0.0f;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < count; i += kVerifyThreads)
        if (tokens[i] == token)
            *slot = probabilities[i];
    __syncthreads();
    return *slot;
}

} // namespace

__global__ void __launch_bounds__(kVerifyThreads, 1) speculative_verify_kernel(const SpeculativeArgs s)
{
    __shared__ VerifyShared sh;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const uint32_t n = s.draft_count;
    const uint32_t session = blockIdx.x;
    wait_for_previous_kernel();
    // rows of the sampler outputs: every Session's draft_count + 1 target positions first, then every Session's draft positions
    const uint32_t target_first = session * (n + 1u);
    const uint32_t draft_first = s.sessions * (n + 1u) + session * n;
    const moe_row_params p = s.params[target_first];
    const int32_t* const proposed_tokens = s.proposed + static_cast<size_t>(session) * n;
    float* const accepted_probability = s.accepted_probability + static_cast<size_t>(session) * n;
    float* const dense = s.dense + static_cast<size_t>(session) * s.vocab;
    int32_t* const residual_token = s.residual_token + static_cast<size_t>(session) * s.vocab;
    float* const residual_value = s.residual_value + static_cast<size_t>(session) * s.vocab;
    const bool greedy = p.temperature == 0.0f;

    const bool short_lists = s.kept_stride <= kShortList;
    if (short_lists && !greedy)
    {
        // What the walk may look up, all positions at once: one warp per list.  The walk below then costs
        // no memory latency per position (it used to take two dependent list scans and four barriers each).
        for (uint32_t pair = warp; pair < 2u * n; pair += kVerifyWarps)
        {
            const uint32_t row = (pair & 1u) == 0u ? target_first + (pair >> 1) : draft_first + (pair >> 1);
            const int32_t token = proposed_tokens[pair >> 1];
            const uint32_t count = min(s.kept_count[row], s.kept_stride);
            const int32_t* tokens = s.kept_token + static_cast<size_t>(row) * s.kept_stride;
            const float* probabilities = s.kept_probability + static_cast<size_t>(row) * s.kept_stride;
            float found = 0.0f; // candidate_probability (session.cpp:138-148): 0 if absent
            for (uint32_t i = lane; i < count; i += 32)
                if (tokens[i] == token)
                    found = probabilities[i];
            const unsigned holder = __ballot_sync(kFullMask, found != 0.0f); // token ids are unique in a list
            found = __shfl_sync(kFullMask, found, holder != 0u ? __ffs(holder) - 1 : 0);
            if (lane == 0)
                sh.found_all[pair] = found;
        }
        __syncthreads();
    }

    uint32_t accepted = 0;
    uint32_t used = 0;
    int32_t status = MOE_ROW_OK;
    bool rejected = false;
    while (accepted < n)
    {
        const uint32_t target_row = target_first + accepted;
        const uint32_t draft_row = draft_first + accepted;
        const int32_t proposed = proposed_tokens[accepted];
        if (s.row_status[target_row] != MOE_ROW_OK)
        {
            status = s.row_status[target_row];
            break;
        }
        if (greedy)
        {
            if (s.token[target_row] != proposed)
                break; // session.cpp:790-794
            if (tid == 0)
                accepted_probability[accepted] = 1.0f;
        }
        else
        {
            if (s.row_status[draft_row] != MOE_ROW_OK)
            {
                status = s.row_status[draft_row];
                break;
            }
            const size_t stride = s.kept_stride;
            float target_probability, draft_probability;
            if (short_lists)
            {
                target_probability = sh.found_all[2u * accepted];
                draft_probability = sh.found_all[2u * accepted + 1u];
            }
            else
            {
                target_probability = list_probability(s.kept_token + target_row * stride, s.kept_probability + target_row * stride,
                                                      min(s.kept_count[target_row], s.kept_stride), proposed, &sh.found[0]);
                draft_probability = list_probability(s.kept_token + draft_row * stride, s.kept_probability + draft_row * stride,
                                                     min(s.kept_count[draft_row], s.kept_stride), proposed, &sh.found[1]);
            }
            if (!(draft_probability > 0.0f))
            {
                status = MOE_ROW_DRAFT_ZERO_PROBABILITY; // session.cpp:813-821
                break;
            }
            const float ratio = __fdiv_rn(target_probability, draft_probability);
            const float acceptance = ratio < 1.0f ? ratio : 1.0f; // std::min(1.0f, ratio)
            const float uniform = philox_uniform(p.seed, p.row_id, p.step + used);
            ++used;
            if (uniform >= acceptance)
            {
                rejected = true; // session.cpp:827-833
                break;
            }
            if (tid == 0)
                accepted_probability[accepted] = target_probability;
        }
        ++accepted;
    }

    int32_t next_token = -1;
    float next_probability = 0.0f;
    if (status == MOE_ROW_OK && rejected)
    {
        // ---- residual distribution of the rejected position (session.cpp:150-202) ----
        const uint32_t target_row = target_first + accepted;
        const uint32_t draft_row = draft_first + accepted;
        const size_t stride = s.kept_stride;
        const int32_t* target_token = s.kept_token + target_row * stride;
        const float* target_probability = s.kept_probability + target_row * stride;
        const int32_t* draft_token = s.kept_token + draft_row * stride;
        const float* draft_probability = s.kept_probability + draft_row * stride;
        const uint32_t target_count = min(s.kept_count[target_row], s.kept_stride);
        const uint32_t draft_count = min(s.kept_count[draft_row], s.kept_stride);
        const float* residual = residual_value;
        const int32_t* residual_ids = residual_token;
        if (short_lists)
        {
            // max(0, target - draft) is only positive on target candidates: one thread per candidate finds the
            // draft's probability of its token and its place among the positive ones by token id, in shared memory
            // (a dense vector over the vocabulary cost three passes of vocab * 4 bytes by one CTA: 190 us at 201088)
            residual = sh.residual;
            residual_ids = sh.residual_id;
            static_assert(kShortList <= kVerifyThreads, "one thread per candidate");
            if (static_cast<uint32_t>(tid) < target_count)
            {
                sh.list_token[0][tid] = target_token[tid];
                sh.list_value[0][tid] = target_probability[tid];
            }
            if (static_cast<uint32_t>(tid) < draft_count)
            {
                sh.list_token[1][tid] = draft_token[tid];
                sh.list_value[1][tid] = draft_probability[tid];
            }
            if (tid == 0)
                sh.cursor = 0;
            __syncthreads();
            float value = 0.0f;
            int32_t id = 0;
            if (static_cast<uint32_t>(tid) < target_count)
            {
                id = sh.list_token[0][tid];
                value = sh.list_value[0][tid];
                for (uint32_t i = 0; i < draft_count; ++i)
                    if (sh.list_token[1][i] == id)
                    {
                        const float reduced = __fsub_rn(value, sh.list_value[1][i]);
                        value = reduced > 0.0f ? reduced : 0.0f; // std::max(0.0f, ...)
                        break;
                    }
            }
            const bool positive = value > 0.0f;
            __syncthreads();
            if (static_cast<uint32_t>(tid) < target_count)
                sh.list_value[0][tid] = value;
            const unsigned voters = __ballot_sync(kFullMask, positive);
            if (lane == 0 && voters != 0u)
                atomicAdd(&sh.cursor, static_cast<uint32_t>(__popc(voters)));
            __syncthreads();
            if (positive)
            {
                uint32_t place = 0;
                for (uint32_t i = 0; i < target_count; ++i)
                    place += (sh.list_value[0][i] > 0.0f && sh.list_token[0][i] < id) ? 1u : 0u;
                sh.residual[place] = value;
                sh.residual_id[place] = id;
            }
        }
        else
        {
            for (uint32_t i = tid; i < s.vocab; i += kVerifyThreads)
                dense[i] = 0.0f;
            __syncthreads();
            for (uint32_t i = tid; i < target_count; i += kVerifyThreads)
                dense[target_token[i]] = target_probability[i];
            __syncthreads();
            for (uint32_t i = tid; i < draft_count; i += kVerifyThreads)
            {
                const int32_t id = draft_token[i];
                const float reduced = __fsub_rn(dense[id], draft_probability[i]);
                dense[id] = reduced > 0.0f ? reduced : 0.0f; // std::max(0.0f, ...)
            }
            if (tid == 0)
                sh.cursor = 0;
            __syncthreads();
            // positive entries in token-id order
            for (uint32_t base = 0; base < s.vocab; base += kVerifyThreads)
            {
                const uint32_t id = base + tid;
                const float value = id < s.vocab ? dense[id] : 0.0f;
                const bool positive = value > 0.0f;
                const unsigned voters = __ballot_sync(kFullMask, positive);
                if (lane == 0)
                    sh.warp_count[warp] = __popc(voters);
                __syncthreads();
                uint32_t before = sh.cursor;
                for (int w = 0; w < warp; ++w)
                    before += sh.warp_count[w];
                if (positive)
                {
                    const uint32_t slot = before + __popc(voters & ((1u << lane) - 1u));
                    residual_token[slot] = static_cast<int32_t>(id);
                    residual_value[slot] = value;
                }
                __syncthreads();
                if (tid == kVerifyThreads - 1)
                    sh.cursor = before + __popc(voters);
                __syncthreads();
            }
        }
        __syncthreads();
        const uint32_t positives = sh.cursor;
        __syncthreads();
        // std::accumulate over the dense vector (session.cpp:171-176) = the positive entries added in token-id
        // order; replayed bit-exactly by the whole block (the entries are not sorted by value)
        const float normalizer = block_sequential_sum<kVerifyThreads, 8, false>(residual, positives, kSeqSumOnly, 0.0f, sh.seq).acc;
        if (positives == 0 || !(normalizer - normalizer == 0.0f) || normalizer <= 0.0f)
        {
            if (tid == 0)
            {
                sh.decision = 2;
                sh.found[0] = 0.0f;
                sh.cursor = 0;
            }
        }
        else
        {
            const float uniform = philox_uniform(p.seed, p.row_id, p.step + used);
            const float sample_value = __fmul_rn(uniform, normalizer); // uniform_real_distribution<float>(0, normalizer)
            const SeqResult draw = block_sequential_sum<kVerifyThreads, 8, false>(residual, positives, kSeqExceedBound, sample_value, sh.seq);
            // session.cpp:189-197: the last positive entry if the sum never passes the draw
            const uint32_t chosen = draw.stopped ? draw.taken - 1u : positives - 1u;
            if (tid == 0)
            {
                sh.decision = 0;
                sh.cursor = static_cast<uint32_t>(residual_ids[chosen]);
                sh.found[0] = __fdiv_rn(residual[chosen], normalizer);
            }
        }
        __syncthreads();
        ++used;
        if (sh.decision == 2)
        {
            status = MOE_ROW_RESIDUAL_EMPTY;
            --used; // the reference returns before it draws
        }
        else
        {
            next_token = static_cast<int32_t>(sh.cursor);
            next_probability = sh.found[0];
        }
    }
    else if (status == MOE_ROW_OK)
    {
        // every proposal accepted, or greedy: the sample of the next target row (session.cpp:871-874);
        // its uniform is number `used` of this step, which is draft_count when all were accepted
        const uint32_t row = target_first + accepted;
        status = s.row_status[row];
        if (status == MOE_ROW_OK)
        {
            next_token = s.token[row];
            next_probability = s.probability[row];
            if (s.row_flags[row] & MOE_ROW_FLAG_USED_UNIFORM)
                ++used;
        }
    }
    if (tid == 0)
    {
        moe_speculative_result result;
        result.accepted = accepted;
        result.next_token = next_token;
        result.next_probability = next_probability;
        result.uniforms_used = used;
        result.status = status;
        result.flags = 0;
        s.result[session] = result;
    }
}

cudaError_t launch_speculative_verify(const SpeculativeArgs& args, cudaStream_t stream)
{
    return launch_following(speculative_verify_kernel, args.sessions, kVerifyThreads, 0, stream, args);
}

} // namespace moe
