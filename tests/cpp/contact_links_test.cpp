// Shared memory of the key-ordered contact passes' links: whatever a schedule's
// layout leaves, layout and links fit the launch.
#include "../../simwing_b200/csrc/cluster_schedule.h"

#include <cstdio>

int main() {
    int failed = 0;
    for (uint32_t cap : {226304u, 227584u, 218u * 1024u, 100u * 1024u})
        for (uint64_t rows : {1ull, 100ull, 4500ull, 12000ull, 60000ull})
            for (uint32_t layout = 16; layout <= cap; layout += layout + 4096 < cap ? 1008 : 16) {
                const uint32_t links = swb::contact_link_bytes(layout, rows, cap);
                if (uint64_t{layout} + links > cap || links % 16 != 0) {
                    if (failed++ < 5)
                        std::printf("FAIL layout %u rows %llu cap %u: %u\n", layout,
                                    static_cast<unsigned long long>(rows), cap, links);
                }
            }
    // what a landed 24 x 24 sheet has room for: its 4,500 rows
    if (swb::contact_link_bytes(40000, 4500, 227584) < 4500 * swb::kContactLinkBytes) {
        std::printf("FAIL room\n");
        ++failed;
    }
    return failed ? 1 : 0;
}
