// Host-only check of how a cluster cuts a row and where it keeps the items of the
// slices (ncnn-moe-runtime_b200/csrc/moe_internal.h): the slices partition the
// row, start 16-byte aligned relative to it, and their items stay inside the
// slot of the one-CTA kernel's scratch.  No CUDA call is made.
#include <cstdio>

#include "../../ncnn-moe-runtime_b200/csrc/moe_internal.h"

int main()
{
    int failures = 0;
    const auto check = [&](uint32_t vocab) {
        for (uint32_t size = 1; size <= 16; size *= 2)
        {
            const uint64_t stride = (static_cast<uint64_t>(vocab) + 3u) & ~3ull; // the smallest handle that takes the row
            uint32_t covered = 0;
            for (uint32_t rank = 0; rank < size; ++rank)
            {
                const moe::ClusterSlice slice = moe::cluster_slice(vocab, size, rank);
                bool good = slice.begin == covered && slice.end >= slice.begin && slice.end <= vocab;
                if (slice.begin < slice.end)
                {
                    const uint64_t items_end = slice.begin + 4ull * ((slice.end - slice.begin + 3u) / 4u); // whole groups of four are written
                    good = good && slice.begin % 4u == 0 && items_end <= stride;                            // numerators: array 0
                    good = good && 4u * stride + 2u * items_end <= 16u * stride;                            // groups: from array 1 on
                }
                if (!good)
                {
                    std::printf("vocab %u size %u rank %u: [%u, %u)\n", vocab, size, rank, slice.begin, slice.end);
                    ++failures;
                }
                covered = slice.end;
            }
            if (covered != vocab)
            {
                std::printf("vocab %u size %u: covers %u\n", vocab, size, covered);
                ++failures;
            }
        }
    };
    for (uint32_t vocab = 1; vocab <= 600; ++vocab)
        check(vocab);
    for (uint32_t vocab : {1023u, 1024u, 1025u, 40001u, 129280u, 151936u, 201088u, 1048575u, 0x7FFFFFFCu, 0x7FFFFFFFu})
        check(vocab);
    if (failures == 0)
        std::puts("scratch layout ok");
    return failures == 0 ? 0 : 1;
}
