// The line iteration's window for blocks of any width: as many of the last
// stages as leave the suspension CTA's last warp without a record, two or none.
#include "../../simwing_b200/csrc/cluster_schedule.h"
#include "../../simwing_b200/csrc/schedule.h"

#include <cstdio>

using namespace swb;

static uint32_t owner_records(const ClusterSchedule& S, int g) {
    int k, s;
    global_stage(S, g, k, s);
    const size_t o = static_cast<size_t>(S.susp_cta) * (S.kinds[k].stages + 1) + s;
    return S.kinds[k].offsets[o + 1] - S.kinds[k].offsets[o];
}

int main() {
    int failed = 0, shorter = 0;
    for (int ctas : {1, 4, 16}) {
        swb_wing_params p;
        swb_default_wing_params(&p);
        p.cells = 6;
        p.chordwise = 20;
        swb_definition* d = nullptr;
        if (swb_generate_wing(&p, &d) != SWB_OK) return 1;
        OwnedDefinition def;
        def.assign(*swb_definition_view(d));
        ClusterSchedule S;
        if (!build_cluster_schedule(def, suspension_endpoint_nodes(def), ctas, S) || S.line_stage < 0) return 1;
        const int G = total_stages(S);
        for (int threads = 32; threads <= 1024; threads += 32) {
            const LineWindow w = line_window(S, threads);
            auto fits = [&](int g) { return static_cast<int>(owner_records(S, g)) <= threads - 32; };
            int first = G;
            while (first > S.line_stage && fits(first - 1)) --first;
            uint32_t records = 0;
            for (int g = first; g < G; ++g) records = std::max(records, owner_records(S, g));
            const bool any = G - first >= 2;
            if (w.first != (any ? first : -1) || w.records != (any ? records : 0u)) {
                std::printf("FAIL %d CTAs, %d threads: %d with %u records\n", ctas, threads, w.first, w.records);
                ++failed;
            }
            shorter += any && first > S.line_stage;
        }
        swb_definition_destroy(d);
    }
    std::printf("%d shorter windows\n", shorter);
    return failed || shorter == 0 ? 1 : 0;
}
