// Which sweeps hand nodes over and which reach foreign nodes in place: nets of
// springs between random nodes, nine and five a node (nine: no room for the
// ghosts; five: room in the forward sweep, not in the reverse one, which keeps
// more per record), two a node (room in both), and stars, whose hub receives
// a node in most of some thousand stages.
#include "../../simwing_b200/csrc/cluster_schedule.h"

#include <cstdio>
#include <set>

using namespace swb;

static uint32_t draw(uint64_t& s) {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    return static_cast<uint32_t>(s >> 33);
}

static OwnedDefinition net(uint32_t nodes, int per_node, uint32_t hub) {
    OwnedDefinition d;
    uint64_t seed = 7;
    for (uint32_t i = 0; i < nodes; ++i) {
        swb_node_def n{};
        n.position = {draw(seed) % 1000 * 0.01, draw(seed) % 1000 * 0.01, draw(seed) % 1000 * 0.01};
        n.mass = 1.0;
        d.nodes.push_back(n);
    }
    std::set<std::pair<uint32_t, uint32_t>> seen;
    auto add = [&](uint32_t a, uint32_t b) {
        if (a == b || !seen.insert({std::min(a, b), std::max(a, b)}).second) return;
        swb_constraint_def c{};
        c.kind = SWB_CONSTRAINT_DISTANCE;
        c.first_node = a;
        c.second_node = b;
        c.rest_length = 1.0;
        d.constraints.push_back(c);
    };
    for (uint32_t i = 0; i < nodes; ++i)
        for (int k = 0; k < per_node; ++k) add(i, draw(seed) % nodes);
    for (uint32_t i = 1; i <= hub; ++i) add(0, i);
    return d;
}

static int check(const char* what, const OwnedDefinition& d, int ctas, bool forward_direct, bool reverse_direct) {
    const size_t limit = 227 * 1024 - 6144;
    ClusterSchedule S;
    if (!build_cluster_schedule(d, {}, ctas, S)) {
        std::printf("FAIL %s: no schedule\n", what);
        return 1;
    }
    verify_flow(d, S, S.forward, false);
    const ClusterFlow r = build_reverse_flow(d, S, limit);
    verify_flow(d, S, r, true);
    const bool ok = S.forward.direct == forward_direct && r.direct == reverse_direct;
    std::printf("%s %s: forward %s, reverse %s, %d stages, %u and %u barriers\n", ok ? "ok  " : "FAIL", what,
                S.forward.direct ? "direct" : "handed over", r.direct ? "direct" : "handed over", total_stages(S),
                S.forward.max_barriers, r.max_barriers);
    return !ok;
}

int main() {
    int failed = 0;
    failed += check("nine springs a node", net(24000, 9, 0), 16, true, true);
    failed += check("five springs a node", net(24000, 5, 0), 16, false, true);
    failed += check("two springs a node", net(6000, 2, 0), 16, false, false);
    failed += check("a star of 3,000", net(3100, 0, 3000), 2, false, false);
    failed += check("a star of 5,900", net(6000, 0, 5900), 2, false, true);
    return failed;
}
