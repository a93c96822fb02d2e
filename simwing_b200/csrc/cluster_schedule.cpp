// Host construction and checking of the cluster sweep schedule.
#include "cluster_schedule.h"

#include <algorithm>
#include <cmath>
#include <limits>
#include <numeric>

namespace swb {

namespace {

uint32_t make_ref(const ClusterSchedule& s, uint32_t node) {
    const uint32_t slot = s.slot_of_node[node];
    const uint32_t cta = static_cast<uint32_t>(
        std::upper_bound(s.patch_begin.begin(), s.patch_begin.end(), slot) - s.patch_begin.begin() - 1);
    return (cta << 12) | (slot - s.patch_begin[cta]);
}

// Tries to colour with one colour fewer, repeatedly: the constraints of the
// last colour are spread over the others and the conflicts that causes are
// repaired by min-conflicts local search with a tabu list (each move puts a
// conflicting constraint into the colour with the fewest conflicts for it,
// not undoing a recent move unless that reaches a new best).  Stops at the
// first count it cannot reach within `budget` moves and keeps the last
// proper colouring.  Deterministic (fixed seed).  Returns the colour count.
int reduce_colours(const std::vector<std::array<uint32_t, 4>>& nodes, const std::vector<int>& counts,
                   uint32_t node_count, int colours, std::vector<int>& colour, long budget) {
    const size_t m = nodes.size();
    if (m == 0 || colours <= 1) return colours;
    // conflict graph (constraints sharing a node)
    std::vector<uint32_t> off(node_count + 1, 0);
    for (size_t i = 0; i < m; ++i)
        for (int q = 0; q < counts[i]; ++q) ++off[nodes[i][q] + 1];
    for (uint32_t v = 0; v < node_count; ++v) off[v + 1] += off[v];
    std::vector<uint32_t> inc(off.back());
    {
        std::vector<uint32_t> cur(off.begin(), off.end() - 1);
        for (size_t i = 0; i < m; ++i)
            for (int q = 0; q < counts[i]; ++q) inc[cur[nodes[i][q]]++] = static_cast<uint32_t>(i);
    }
    std::vector<uint32_t> nb_off(m + 1, 0), nb;
    {
        std::vector<uint32_t> tmp;
        for (size_t i = 0; i < m; ++i) {
            tmp.clear();
            for (int q = 0; q < counts[i]; ++q)
                for (uint32_t k = off[nodes[i][q]]; k < off[nodes[i][q] + 1]; ++k)
                    if (inc[k] != i) tmp.push_back(inc[k]);
            std::sort(tmp.begin(), tmp.end());
            tmp.erase(std::unique(tmp.begin(), tmp.end()), tmp.end());
            nb.insert(nb.end(), tmp.begin(), tmp.end());
            nb_off[i + 1] = static_cast<uint32_t>(nb.size());
        }
    }
    uint64_t state = 0x9e3779b97f4a7c15ull;
    auto rnd = [&]() {
        state ^= state << 13;
        state ^= state >> 7;
        state ^= state << 17;
        return state;
    };
    // the constraints at one node form a clique: no colouring has fewer
    // colours than the largest incidence count
    uint32_t clique = 0;
    for (uint32_t v = 0; v < node_count; ++v) clique = std::max(clique, off[v + 1] - off[v]);
    for (int k = colours - 1; k >= static_cast<int>(std::max<uint32_t>(clique, 1)); --k) {
        std::vector<int> c2 = colour;
        for (size_t i = 0; i < m; ++i)
            if (c2[i] >= k) c2[i] = static_cast<int>(rnd() % k);
        std::vector<uint16_t> cnt(m * static_cast<size_t>(k), 0);
        for (size_t i = 0; i < m; ++i)
            for (uint32_t e = nb_off[i]; e < nb_off[i + 1]; ++e) ++cnt[i * k + c2[nb[e]]];
        long conflicts = 0;
        for (size_t i = 0; i < m; ++i) conflicts += cnt[i * k + c2[i]];
        conflicts /= 2;
        long best = conflicts;
        std::vector<long> tabu(m * static_cast<size_t>(k), 0);
        std::vector<uint32_t> open;
        std::vector<int64_t> pos(m, -1);
        auto update = [&](uint32_t i) {
            const bool bad = cnt[i * k + c2[i]] > 0;
            if (bad && pos[i] < 0) {
                pos[i] = static_cast<int64_t>(open.size());
                open.push_back(i);
            } else if (!bad && pos[i] >= 0) {
                const uint32_t last = open.back();
                open[pos[i]] = last;
                pos[last] = pos[i];
                open.pop_back();
                pos[i] = -1;
            }
        };
        for (size_t i = 0; i < m; ++i) update(static_cast<uint32_t>(i));
        for (long it = 0; it < budget && !open.empty(); ++it) {
            const uint32_t i = open[rnd() % open.size()];
            const int cur = c2[i];
            int bc = -1, bv = 1 << 30;
            for (int c = 0; c < k; ++c) {
                if (c == cur) continue;
                const int v = cnt[i * k + c];
                const bool aspiration = conflicts - cnt[i * k + cur] + v < best;
                if (tabu[i * k + c] > it && !aspiration) continue;
                if (v < bv || (v == bv && (rnd() & 1))) {
                    bv = v;
                    bc = c;
                }
            }
            if (bc < 0) continue;
            conflicts += bv - cnt[i * k + cur];
            tabu[i * k + cur] = it + 7 + static_cast<long>(rnd() % 10) + static_cast<long>(open.size() / 10);
            c2[i] = bc;
            for (uint32_t e = nb_off[i]; e < nb_off[i + 1]; ++e) {
                const uint32_t j = nb[e];
                --cnt[j * k + cur];
                ++cnt[j * k + bc];
                update(j);
            }
            update(i);
            best = std::min(best, conflicts);
        }
        if (!open.empty()) return k + 1;
        colour = c2;
        colours = k;
    }
    return colours;
}

// Evens out, CTA by CTA, how many records each colour gives the CTA, without
// adding colours: a constraint whose colour holds more than the CTA's mean
// moves to the colour with the fewest of the CTA's records that none of its
// conflicting constraints (shared nodes) has, as long as that colour holds
// at least two fewer.  Stages then carry similar record counts on every CTA,
// so the largest colours no longer need two rounds of the CTA's threads
// while the small ones leave them idle.
void balance_colours(const std::vector<std::array<uint32_t, 4>>& nodes, const std::vector<int>& counts,
                     const std::vector<int>& cta_of, int ctas, uint32_t node_count, int colours,
                     std::vector<int>& colour) {
    const size_t m = nodes.size();
    if (colours < 2 || colours > 64 || m == 0) return;
    std::vector<uint32_t> off(node_count + 1, 0);
    for (size_t i = 0; i < m; ++i)
        for (int q = 0; q < counts[i]; ++q) ++off[nodes[i][q] + 1];
    for (uint32_t v = 0; v < node_count; ++v) off[v + 1] += off[v];
    std::vector<uint32_t> inc(off.back());
    {
        std::vector<uint32_t> cur(off.begin(), off.end() - 1);
        for (size_t i = 0; i < m; ++i)
            for (int q = 0; q < counts[i]; ++q) inc[cur[nodes[i][q]]++] = static_cast<uint32_t>(i);
    }
    std::vector<int64_t> size(static_cast<size_t>(ctas) * colours, 0), total(ctas, 0);
    for (size_t i = 0; i < m; ++i) {
        ++size[static_cast<size_t>(cta_of[i]) * colours + colour[i]];
        ++total[cta_of[i]];
    }
    for (int pass = 0; pass < 8; ++pass) {
        bool moved = false;
        for (size_t i = 0; i < m; ++i) {
            const int c = colour[i];
            int64_t* sz = size.data() + static_cast<size_t>(cta_of[i]) * colours;
            const int64_t mean = (total[cta_of[i]] + colours - 1) / colours;
            if (sz[c] <= mean) continue;
            uint64_t used = 0;
            for (int q = 0; q < counts[i]; ++q)
                for (uint32_t k = off[nodes[i][q]]; k < off[nodes[i][q] + 1]; ++k)
                    if (inc[k] != i) used |= 1ull << colour[inc[k]];
            int best = -1;
            for (int t = 0; t < colours; ++t)
                if (!((used >> t) & 1ull) && sz[t] + 1 < sz[c] && (best < 0 || sz[t] < sz[best])) best = t;
            if (best < 0) continue;
            --sz[c];
            ++sz[best];
            colour[i] = best;
            moved = true;
        }
        if (!moved) break;
    }
}

}  // namespace

// Nodes of element i (definition index) of kind k: 2 (distance), 4
// (dihedral) or 3 (membrane: its triangle's corners); returns the count.
static int element_nodes(const OwnedDefinition& d, int k, size_t i, uint32_t* nodes) {
    if (k == 0) {
        nodes[0] = static_cast<uint32_t>(d.constraints[i].first_node);
        nodes[1] = static_cast<uint32_t>(d.constraints[i].second_node);
        return 2;
    }
    if (k == 1) {
        for (int q = 0; q < 4; ++q) nodes[q] = static_cast<uint32_t>(d.dihedrals[i].nodes[q]);
        return 4;
    }
    const swb_triangle_def& t = d.triangles[d.membranes[i].triangle];
    for (int q = 0; q < 3; ++q) nodes[q] = static_cast<uint32_t>(t.nodes[q]);
    return 3;
}

// Load-path order of the cables and ties (loadPathConstraintOrder,
// soft_body.cpp:528-629) in sweep order, then the level schedule of one
// cable pair (reverse pass, forward pass) over the distance records.
static void build_load_path(const OwnedDefinition& d, ClusterSchedule& S) {
    const size_t N = d.nodes.size();
    std::vector<uint8_t> structural(N, 0);
    std::vector<std::vector<uint32_t>> adj(N);
    for (size_t v = 0; v < N; ++v) structural[v] = d.nodes[v].fixed ? 1 : 0;
    for (const auto& t : d.triangles)
        for (int k = 0; k < 3; ++k) structural[t.nodes[k]] = 1;
    std::vector<uint64_t> seq;
    for (uint64_t i : S.distance_order) {  // the device sweep order
        const auto& c = d.constraints[i];
        if (c.kind == SWB_CONSTRAINT_DISTANCE || c.kind == SWB_CONSTRAINT_SEAM_STITCH) continue;
        seq.push_back(i);
    }
    for (const auto& c : d.constraints) {
        if (c.kind == SWB_CONSTRAINT_DISTANCE || c.kind == SWB_CONSTRAINT_SEAM_STITCH) {
            structural[c.first_node] = structural[c.second_node] = 1;
            continue;
        }
        adj[c.first_node].push_back(static_cast<uint32_t>(c.second_node));
        adj[c.second_node].push_back(static_cast<uint32_t>(c.first_node));
    }
    for (const auto& h : d.dihedrals)
        for (int k = 0; k < 4; ++k) structural[h.nodes[k]] = 1;
    S.pair_stages = 0;
    S.pair_offsets.assign(static_cast<size_t>(S.ctas), 0);
    S.pair_rec.clear();
    if (seq.empty()) return;
    // breadth-first depth from the structural skin; a component without a
    // structural node is rooted at its heaviest node (first of the smallest
    // inverse mass)
    const uint64_t unknown = ~uint64_t{0};
    std::vector<uint64_t> depth(N, unknown);
    std::vector<uint32_t> queue;
    for (size_t v = 0; v < N; ++v)
        if (structural[v] && !adj[v].empty()) {
            depth[v] = 0;
            queue.push_back(static_cast<uint32_t>(v));
        }
    size_t head = 0;
    for (;;) {
        while (head < queue.size()) {
            const uint32_t v = queue[head++];
            for (uint32_t u : adj[v])
                if (depth[u] == unknown) {
                    depth[u] = depth[v] + 1;
                    queue.push_back(u);
                }
        }
        size_t root = N;
        double smallest = std::numeric_limits<double>::infinity();
        for (size_t v = 0; v < N; ++v) {
            const double w = d.nodes[v].fixed ? 0.0 : 1.0 / d.nodes[v].mass;
            if (depth[v] == unknown && !adj[v].empty() && w < smallest) {
                root = v;
                smallest = w;
            }
        }
        if (root == N) break;
        depth[root] = 0;
        queue.push_back(static_cast<uint32_t>(root));
    }
    auto cdepth = [&](uint64_t i) {
        return std::max(depth[d.constraints[i].first_node], depth[d.constraints[i].second_node]);
    };
    std::stable_sort(seq.begin(), seq.end(), [&](uint64_t a, uint64_t b) { return cdepth(a) < cdepth(b); });
    // distance record and executing CTA of each definition index
    const ClusterKind& K = S.kinds[0];
    std::vector<uint32_t> rec_of(d.constraints.size(), ~0u);
    std::vector<int> cta_of_rec(K.def_index.size(), 0);
    for (int c = 0; c < S.ctas; ++c)
        for (uint32_t r = K.offsets[static_cast<size_t>(c) * (K.stages + 1)];
             r < K.offsets[static_cast<size_t>(c) * (K.stages + 1) + K.stages]; ++r) {
            rec_of[K.def_index[r]] = r;
            cta_of_rec[r] = c;
        }
    // levels of the reverse pass, then of the forward pass
    struct Item { int level, cta; uint32_t rec; };
    std::vector<Item> items;
    int levels = 0;
    for (int pass = 0; pass < 2; ++pass) {
        std::vector<int> last(N, -1);
        int top = -1;
        for (size_t k = 0; k < seq.size(); ++k) {
            const uint64_t i = pass == 0 ? seq[seq.size() - 1 - k] : seq[k];
            const auto& c = d.constraints[i];
            const int level = std::max(last[c.first_node], last[c.second_node]) + 1;
            last[c.first_node] = last[c.second_node] = level;
            top = std::max(top, level);
            items.push_back({levels + level, cta_of_rec[rec_of[i]], rec_of[i]});
        }
        levels += top + 1;
    }
    S.pair_stages = levels;
    std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) {
        if (a.cta != b.cta) return a.cta < b.cta;
        return a.level < b.level;
    });
    S.pair_offsets.assign(static_cast<size_t>(S.ctas) * (levels + 1), 0);
    size_t at = 0;
    for (int c = 0; c < S.ctas; ++c) {
        for (int l = 0; l <= levels; ++l) {
            while (at < items.size() && items[at].cta == c && items[at].level < l) ++at;
            S.pair_offsets[static_cast<size_t>(c) * (levels + 1) + l] = static_cast<uint32_t>(at);
        }
        while (at < items.size() && items[at].cta == c) ++at;
    }
    for (const Item& it : items) S.pair_rec.push_back(it.rec);
}

// True when a record of global stage g has a node flagged in `attached`.
static bool stage_touches(const OwnedDefinition& d, const ClusterSchedule& S, const std::vector<uint8_t>& attached,
                          int g) {
    int k, s;
    global_stage(S, g, k, s);
    const ClusterKind& K = S.kinds[k];
    for (int c = 0; c < S.ctas; ++c)
        for (uint32_t r = K.offsets[static_cast<size_t>(c) * (K.stages + 1) + s];
             r < K.offsets[static_cast<size_t>(c) * (K.stages + 1) + s + 1]; ++r) {
            uint32_t nodes[4];
            const int cnt = element_nodes(d, k, K.def_index[r], nodes);
            for (int q = 0; q < cnt; ++q)
                if (attached[nodes[q]]) return true;
        }
    return false;
}

// Global stage of stage `s` of kind k.
static int global_stage_of(const ClusterSchedule& S, int k, int s) {
    return k == 0 ? s : (k == 2 ? S.kinds[0].stages + s : S.kinds[0].stages + S.kinds[2].stages + s);
}

// Homes, patches and slots.  A node's home is the CTA of its first touch in
// an iteration (its bisection part when nothing touches it, when that
// patch is full, and in direct schedules); ghosts are the foreign nodes a
// CTA's records touch, in node order.  `patch_limit`: nodes a patch may hold.
static void place_nodes(ClusterSchedule& S, const std::vector<int>& part,
                        const std::array<std::vector<std::array<uint32_t, 4>>, 3>& nodes,
                        const std::array<std::vector<int>, 3>& counts, const std::array<std::vector<int>, 3>& cta,
                        const std::array<std::vector<int>, 3>& colour, const std::vector<uint8_t>& attached,
                        uint32_t patch_limit, bool direct) {
    const uint32_t N = S.node_count;
    const int C = S.ctas;
    std::vector<int> home = part, first(N, -1), first_stage(N, std::numeric_limits<int>::max());
    std::vector<uint16_t> touched(N, 0);  // CTAs that touch the node
    for (int k = 0; k < 3; ++k)
        for (size_t i = 0; i < counts[k].size(); ++i) {
            const int g = global_stage_of(S, k, colour[k][i]);
            for (int q = 0; q < counts[k][i]; ++q) {
                const uint32_t n = nodes[k][i][q];
                touched[n] |= static_cast<uint16_t>(1u << cta[k][i]);
                if (g < first_stage[n]) {
                    first_stage[n] = g;
                    first[n] = cta[k][i];
                }
            }
        }
    std::vector<uint32_t> size(C, 0);
    for (uint32_t n = 0; n < N; ++n) ++size[part[n]];
    if (!direct)
        for (uint32_t n = 0; n < N; ++n)
            if (first[n] >= 0 && first[n] != part[n] && !attached[n] && size[first[n]] < patch_limit) {
                --size[part[n]];
                ++size[first[n]];
                home[n] = first[n];
            }
    S.patch_begin.assign(C + 1, 0);
    S.max_patch = 0;
    for (int c = 0; c < C; ++c) {
        S.max_patch = std::max(S.max_patch, size[c]);
        S.patch_begin[c + 1] = S.patch_begin[c] + size[c];
    }
    S.node_of_slot.assign(N, 0);
    S.slot_of_node.assign(N, 0);
    std::vector<uint32_t> cur(S.patch_begin.begin(), S.patch_begin.end() - 1);
    for (uint32_t n = 0; n < N; ++n) {
        const uint32_t s = cur[home[n]]++;
        S.node_of_slot[s] = n;
        S.slot_of_node[n] = s;
    }
    S.ghost_begin.assign(C + 1, 0);
    S.ghost_node.clear();
    S.max_local = S.max_patch;
    for (int c = 0; c < C; ++c) {
        if (!direct)
            for (uint32_t n = 0; n < N; ++n)
                if (home[n] != c && (touched[n] >> c & 1)) S.ghost_node.push_back(n);
        S.ghost_begin[c + 1] = static_cast<uint32_t>(S.ghost_node.size());
        S.max_local = std::max(S.max_local, size[c] + S.ghost_begin[c + 1] - S.ghost_begin[c]);
    }
}

// Home CTA of a node.
static int home_of(const ClusterSchedule& S, uint32_t node) {
    return static_cast<int>(std::upper_bound(S.patch_begin.begin(), S.patch_begin.end(), S.slot_of_node[node]) -
                            S.patch_begin.begin() - 1);
}

// Slot of a node in CTA c's array (its own patch, then its ghosts).
static uint32_t local_slot(const ClusterSchedule& S, int c, uint32_t node) {
    const uint32_t s = S.slot_of_node[node];
    if (s >= S.patch_begin[c] && s < S.patch_begin[c + 1]) return s - S.patch_begin[c];
    const auto lo = S.ghost_node.begin() + S.ghost_begin[c], hi = S.ghost_node.begin() + S.ghost_begin[c + 1];
    const auto at = std::lower_bound(lo, hi, node);
    if (at == hi || *at != node) return 0;  // direct schedules: read in place
    return S.patch_begin[c + 1] - S.patch_begin[c] + static_cast<uint32_t>(at - lo);
}

// Records of every kind in schedule order.
static void emit_records(const OwnedDefinition& d, ClusterSchedule& S,
                         const std::array<std::vector<std::array<uint32_t, 4>>, 3>& kind_nodes,
                         const std::array<std::vector<int>, 3>& kind_counts,
                         const std::array<std::vector<int>, 3>& kind_cta,
                         const std::array<std::vector<int>, 3>& kind_colour, bool direct) {
    const int ctas = S.ctas;
    // a boundary node: its home and every CTA that touches it are not one
    std::vector<int> home(S.node_count);
    std::vector<uint8_t> shared(S.node_count, 0);
    for (int c = 0; c < ctas; ++c)
        for (uint32_t s = S.patch_begin[c]; s < S.patch_begin[c + 1]; ++s) home[S.node_of_slot[s]] = c;
    for (int k = 0; k < 3; ++k)
        for (size_t i = 0; i < kind_counts[k].size(); ++i)
            for (int q = 0; q < kind_counts[k][i]; ++q)
                if (home[kind_nodes[k][i][q]] != kind_cta[k][i]) shared[kind_nodes[k][i][q]] = 1;
    for (int k = 0; k < 3; ++k) {
        ClusterKind& K = S.kinds[k];
        const auto& nodes = kind_nodes[k];
        const auto& counts = kind_counts[k];
        const auto& cta_of = kind_cta[k];
        const auto& colour = kind_colour[k];
        const size_t m = counts.size();
        const int stages = K.stages;
        std::vector<uint8_t> edge(m, 0);
        for (size_t i = 0; i < m; ++i)
            for (int q = 0; q < counts[i]; ++q)
                // in a direct schedule only the records with foreign nodes
                edge[i] |= direct ? home[nodes[i][q]] != cta_of[i] : shared[nodes[i][q]] != 0;
        // CTA-major, stage within, boundary records first, definition order within
        std::vector<uint32_t> idx(m);
        std::iota(idx.begin(), idx.end(), 0u);
        std::stable_sort(idx.begin(), idx.end(), [&](uint32_t x, uint32_t y) {
            if (cta_of[x] != cta_of[y]) return cta_of[x] < cta_of[y];
            if (colour[x] != colour[y]) return colour[x] < colour[y];
            return edge[x] > edge[y];
        });
        K.offsets.assign(static_cast<size_t>(ctas) * (stages + 1), 0);
        K.boundary.assign(static_cast<size_t>(ctas) * stages, 0);
        K.boundary_first.assign(static_cast<size_t>(ctas) * stages, 0);
        std::vector<uint32_t> count(static_cast<size_t>(ctas) * std::max(stages, 1), 0);
        for (size_t i = 0; i < m; ++i) {
            ++count[static_cast<size_t>(cta_of[i]) * stages + colour[i]];
            K.boundary[static_cast<size_t>(cta_of[i]) * stages + colour[i]] += edge[i];
        }
        K.max_cta_records = 0;
        K.boundary_total = 0;
        uint32_t off = 0;
        for (int c = 0; c < ctas; ++c) {
            const uint32_t cta_start = off;
            for (int s = 0; s < stages; ++s) {
                K.offsets[static_cast<size_t>(c) * (stages + 1) + s] = off;
                off += count[static_cast<size_t>(c) * stages + s];
                K.boundary_first[static_cast<size_t>(c) * stages + s] = K.boundary_total;
                K.boundary_total += K.boundary[static_cast<size_t>(c) * stages + s];
            }
            K.offsets[static_cast<size_t>(c) * (stages + 1) + stages] = off;
            K.max_cta_records = std::max(K.max_cta_records, off - cta_start);
        }
        for (auto* v : {&K.ab, &K.cd, &K.lab, &K.lcd, &K.def_index}) v->clear();
        K.rest.clear();
        K.comp.clear();
        for (uint32_t i : idx) {
            const int c = cta_of[i];
            K.ab.push_back(make_ref(S, nodes[i][0]) | (make_ref(S, nodes[i][1]) << 16));
            K.lab.push_back(local_slot(S, c, nodes[i][0]) | (local_slot(S, c, nodes[i][1]) << 16));
            if (k == 2) {
                K.cd.push_back(make_ref(S, nodes[i][2]));
                K.lcd.push_back(local_slot(S, c, nodes[i][2]));
                K.rest.push_back(0.0f);
                K.comp.push_back(0.0f);
            } else if (k == 1) {
                K.cd.push_back(make_ref(S, nodes[i][2]) | (make_ref(S, nodes[i][3]) << 16));
                K.lcd.push_back(local_slot(S, c, nodes[i][2]) | (local_slot(S, c, nodes[i][3]) << 16));
                K.rest.push_back(static_cast<float>(d.dihedrals[i].rest_angle));
                K.comp.push_back(static_cast<float>(d.dihedrals[i].compliance));
            } else {
                const auto& dc = d.constraints[i];
                const bool stitch = dc.kind == SWB_CONSTRAINT_SEAM_STITCH;
                K.lcd.push_back(0);
                K.rest.push_back(stitch ? 0.0f : static_cast<float>(dc.rest_length));
                float cp = stitch ? 0.0f : static_cast<float>(dc.compliance);
                if (dc.kind == SWB_CONSTRAINT_CABLE) cp = std::copysign(std::fabs(cp), -1.0f);
                K.comp.push_back(cp);
            }
            K.def_index.push_back(i);
        }
    }
}

ClusterFlow build_flow(const OwnedDefinition& d, const ClusterSchedule& S, bool reverse, bool direct) {
    const int C = S.ctas, G = total_stages(S);
    ClusterFlow F;
    F.direct = direct;
    for (int k = 0; k < 3; ++k) F.send[k].assign(S.kinds[k].boundary_total, {0, 0, 0, 0});
    F.barrier.assign(static_cast<size_t>(C) * G, 0);
    F.out_begin.assign(C + 1, 0);
    F.bytes_begin.assign(C + 1, 0);
    std::vector<int> home(S.node_count);
    for (int c = 0; c < C; ++c)
        for (uint32_t s = S.patch_begin[c]; s < S.patch_begin[c + 1]; ++s) home[S.node_of_slot[s]] = c;
    std::vector<std::vector<uint32_t>> bytes(C, std::vector<uint32_t>(1, 0));
    auto receive = [&](int c, int g) {  // the barrier of CTA c's stage g, one more node on it
        uint32_t& b = F.barrier[static_cast<size_t>(c) * G + g];
        if (b == 0) {
            b = static_cast<uint32_t>(bytes[c].size());
            bytes[c].push_back(0);
        }
        bytes[c][b] += 16;
        return b;
    };
    // each boundary node's last touch so far: CTA and its send word
    struct Touch { int cta = -1; uint32_t* word = nullptr; };
    std::vector<Touch> last(S.node_count);
    std::vector<std::vector<std::array<uint32_t, 2>>> out(C);
    for (int step = 0; step < G; ++step) {
        const int g = reverse ? G - 1 - step : step;
        int k, s;
        global_stage(S, g, k, s);
        const ClusterKind& K = S.kinds[k];
        for (int c = 0; c < C; ++c) {
            const uint32_t lo = K.offsets[static_cast<size_t>(c) * (K.stages + 1) + s];
            const size_t cs = static_cast<size_t>(c) * K.stages + s;
            for (uint32_t j = 0; j < K.boundary[cs]; ++j) {
                uint32_t nodes[4];
                const int cnt = element_nodes(d, k, K.def_index[lo + j], nodes);
                std::array<uint32_t, 4>& words = F.send[k][K.boundary_first[cs] + j];
                for (int q = 0; q < cnt; ++q) {
                    const uint32_t n = nodes[q];
                    if (direct) {
                        if (home[n] != c)
                            words[q] = send_word(static_cast<uint32_t>(home[n]), 0,
                                                 S.slot_of_node[n] - S.patch_begin[home[n]]);
                        continue;
                    }
                    Touch& t = last[n];
                    if (t.cta < 0) {
                        if (home[n] != c)
                            out[home[n]].push_back({local_slot(S, home[n], n),
                                                    send_word(static_cast<uint32_t>(c), receive(c, g),
                                                              local_slot(S, c, n))});
                    } else if (t.cta != c) {
                        *t.word = send_word(static_cast<uint32_t>(c), receive(c, g), local_slot(S, c, n));
                    }
                    t = {c, &words[q]};
                }
            }
        }
    }
    for (uint32_t n = 0; n < S.node_count; ++n)
        if (last[n].cta >= 0 && last[n].cta != home[n]) {
            bytes[home[n]][0] += 16;
            *last[n].word = send_word(static_cast<uint32_t>(home[n]), 0, local_slot(S, home[n], n));
        }
    for (int c = 0; c < C; ++c) {
        F.out.insert(F.out.end(), out[c].begin(), out[c].end());
        F.out_begin[c + 1] = static_cast<uint32_t>(F.out.size());
        F.bytes.insert(F.bytes.end(), bytes[c].begin(), bytes[c].end());
        F.bytes_begin[c + 1] = static_cast<uint32_t>(F.bytes.size());
        F.max_barriers = std::max(F.max_barriers, static_cast<uint32_t>(bytes[c].size()));
    }
    return F;
}

std::vector<std::array<uint32_t, 4>> stage_descriptors(const ClusterSchedule& S, const ClusterFlow& F) {
    const int G = total_stages(S);
    std::vector<std::array<uint32_t, 4>> out(static_cast<size_t>(S.ctas) * G);
    uint32_t record_first[3] = {0, 0, 0}, send_first[3] = {0, 0, 0};
    for (int k = 1; k < 3; ++k) {
        record_first[k] = record_first[k - 1] + static_cast<uint32_t>(S.kinds[k - 1].ab.size());
        send_first[k] = send_first[k - 1] + S.kinds[k - 1].boundary_total;
    }
    for (int c = 0; c < S.ctas; ++c)
        for (int g = 0; g < G; ++g) {
            int k, s;
            global_stage(S, g, k, s);
            const ClusterKind& K = S.kinds[k];
            const size_t o = static_cast<size_t>(c) * (K.stages + 1), cs = static_cast<size_t>(c) * K.stages + s;
            out[static_cast<size_t>(c) * G + g] = {record_first[k] + K.offsets[o + s],
                                                   K.offsets[o + s + 1] - K.offsets[o + s],
                                                   send_first[k] + K.boundary_first[cs],
                                                   K.boundary[cs] | F.barrier[static_cast<size_t>(c) * G + g] << 16};
        }
    return out;
}

ClusterLayout layout_of(const ClusterSchedule& s) {
    auto align = [](uint64_t v) { return (v + 15) & ~uint64_t{15}; };
    ClusterLayout L;
    uint64_t off = align(s.max_local * 16ull);
    L.velocity = static_cast<uint32_t>(off);
    uint64_t lam = off;
    for (int k = 0; k < 3; ++k) {
        L.lambda[k] = static_cast<uint32_t>(lam);
        lam = align(lam + s.kinds[k].max_cta_records * (k == 2 ? 12ull : 4ull));
    }
    off = std::max(lam, align(off + s.max_patch * 16ull));
    L.stages = kStagesInGlobal;
    if (total_stages(s) <= kSharedStages) {
        L.stages = static_cast<uint32_t>(off);
        off = align(off + total_stages(s) * 16ull);
    }
    L.barriers = static_cast<uint32_t>(off);
    if (!s.forward.direct) off = align(off + s.forward.max_barriers * 8ull);
    L.bytes = static_cast<uint32_t>(off);
    if (!s.forward.direct) off = align(off + s.forward.max_barriers * 4ull);
    L.total = static_cast<uint32_t>(std::min<uint64_t>(off, 0xffffffffu));
    return L;
}

LineWindow line_window(const ClusterSchedule& S, int threads) {
    LineWindow w;
    if (S.line_stage < 0) return w;
    const int G = total_stages(S);
    for (int g = G - 1; g >= S.line_stage; --g) {
        int k, s;
        global_stage(S, g, k, s);
        const ClusterKind& K = S.kinds[k];
        const size_t o = static_cast<size_t>(S.susp_cta) * (K.stages + 1) + s;
        const uint32_t n = K.offsets[o + 1] - K.offsets[o];
        if (static_cast<int64_t>(n) > threads - 32) break;
        if (G - g >= 2) w.first = g;
        w.records = std::max(w.records, n);
    }
    if (w.first < 0) w.records = 0;
    return w;
}

bool build_cluster_schedule(const OwnedDefinition& d, const std::vector<uint32_t>& suspension_nodes, int ctas,
                            ClusterSchedule& S, bool split, size_t shared_limit) {
    S = ClusterSchedule{};
    const uint32_t N = static_cast<uint32_t>(d.nodes.size());
    ctas = std::clamp(ctas, 1, kClusterMaxCtas);
    if (N == 0) ctas = 1;
    S.ctas = ctas;
    S.node_count = N;
    const std::vector<int> part = bisect_nodes(d, suspension_nodes, ctas, 0.03);
    {
        std::vector<uint32_t> size(ctas, 0);
        for (uint32_t n = 0; n < N; ++n) ++size[part[n]];
        S.max_part = *std::max_element(size.begin(), size.end());
        if (S.max_part > kClusterPatchNodes) {
            S = ClusterSchedule{};
            return false;
        }
    }
    std::vector<uint8_t> attached(N, 0);
    for (uint32_t n : suspension_nodes) attached[n] = 1;
    if (!suspension_nodes.empty()) S.susp_cta = part[suspension_nodes[0]];

    // per kind: nodes, executing CTA and stage of every element
    std::array<std::vector<std::array<uint32_t, 4>>, 3> kind_nodes;
    std::array<std::vector<int>, 3> kind_counts, kind_cta, kind_colour;
    for (int k = 0; k < 3; ++k) {
        ClusterKind& K = S.kinds[k];
        const size_t m = k == 0 ? d.constraints.size() : (k == 1 ? d.dihedrals.size() : d.membranes.size());
        std::vector<std::array<uint32_t, 4>>& nodes = kind_nodes[k];
        std::vector<int>& counts = kind_counts[k];
        nodes.resize(m);
        counts.assign(m, 0);
        for (size_t i = 0; i < m; ++i) {
            nodes[i] = {0, 0, 0, 0};
            counts[i] = element_nodes(d, k, i, nodes[i].data());
        }
        // executing CTA: owner of most of the constraint's nodes (ties: first)
        std::vector<int>& cta_of = kind_cta[k];
        cta_of.assign(m, 0);
        std::vector<uint8_t> interior(m, 0);
        for (size_t i = 0; i < m; ++i) {
            int best = part[nodes[i][0]], best_count = 0;
            for (int q = 0; q < counts[i]; ++q) {
                int cnt = 0;
                for (int r = 0; r < counts[i]; ++r) cnt += part[nodes[i][r]] == part[nodes[i][q]];
                if (cnt > best_count) {
                    best_count = cnt;
                    best = part[nodes[i][q]];
                }
            }
            cta_of[i] = best;
            interior[i] = best_count == counts[i];
        }
        std::vector<int>& colour = kind_colour[k];  // becomes the stage
        colour.assign(m, 0);
        if (!split || ctas == 1 || k == 2) {  // membranes: classic stages
            K.stages = dsatur_colour(nodes, counts, colour);
            K.stages = reduce_colours(nodes, counts, N, K.stages, colour, kColourSearchMoves);
            balance_colours(nodes, counts, cta_of, ctas, N, K.stages, colour);
            K.sync_stages = K.stages;
        } else {
            // Split stages.  A record whose nodes all lie in its CTA's patch
            // is interior; the others (boundary records) are coloured first
            // and alone, so they take only as many colours as the most
            // boundary records at one node need.  Interior records then
            // take the smallest colour free at all of their nodes,
            // boundary colours included, and open a colour of their own
            // only where none is.  The stages of interior-only colours run
            // first (a CTA touches its own patch only), then the stages with
            // boundary records.
            std::vector<size_t> ids;
            std::vector<std::array<uint32_t, 4>> sub;
            std::vector<int> subc;
            for (size_t i = 0; i < m; ++i)
                if (!interior[i]) {
                    ids.push_back(i);
                    sub.push_back(nodes[i]);
                    subc.push_back(counts[i]);
                }
            std::vector<int> col;
            int B = dsatur_colour(sub, subc, col);
            if (B > 1) B = reduce_colours(sub, subc, N, B, col, kColourSearchMoves);
            // colours in use at each node (bit c: colour c), boundary first
            std::vector<std::vector<uint64_t>> used(N);
            auto taken = [&](uint32_t n, int c) {
                const auto& u = used[n];
                return static_cast<size_t>(c >> 6) < u.size() && ((u[c >> 6] >> (c & 63)) & 1ull);
            };
            auto take = [&](uint32_t n, int c) {
                auto& u = used[n];
                if (u.size() <= static_cast<size_t>(c >> 6)) u.resize((c >> 6) + 1, 0ull);
                u[c >> 6] |= 1ull << (c & 63);
            };
            for (size_t j = 0; j < ids.size(); ++j) {
                colour[ids[j]] = col[j];
                for (int q = 0; q < subc[j]; ++q) take(sub[j][q], col[j]);
            }
            // interior records, most constrained first (largest node degree sum)
            std::vector<uint32_t> degree(N, 0);
            for (size_t i = 0; i < m; ++i)
                for (int q = 0; q < counts[i]; ++q) ++degree[nodes[i][q]];
            std::vector<size_t> inner;
            for (size_t i = 0; i < m; ++i)
                if (interior[i]) inner.push_back(i);
            auto weight = [&](size_t i) {
                uint32_t w = 0;
                for (int q = 0; q < counts[i]; ++q) w += degree[nodes[i][q]];
                return w;
            };
            std::stable_sort(inner.begin(), inner.end(), [&](size_t a, size_t b) { return weight(a) > weight(b); });
            int total = B;
            for (size_t i : inner) {
                int c = 0;
                for (;; ++c) {
                    bool free = true;
                    for (int q = 0; q < counts[i] && free; ++q) free = !taken(nodes[i][q], c);
                    if (free) break;
                }
                colour[i] = c;
                for (int q = 0; q < counts[i]; ++q) take(nodes[i][q], c);
                total = std::max(total, c + 1);
            }
            // stage order: interior-only colours, then the boundary colours
            std::vector<int> stage_of(total);
            const int inner_only = total - B;
            for (int c = 0; c < total; ++c) stage_of[c] = c >= B ? c - B : inner_only + c;
            for (size_t i = 0; i < m; ++i) colour[i] = stage_of[colour[i]];
            K.stages = total;
            K.sync_stages = B + std::min(inner_only, 1);
        }
        // sweep order: stage-major, CTA of the bisection, definition order
        auto& order = k == 0 ? S.distance_order : (k == 1 ? S.dihedral_order : S.membrane_order);
        order.resize(m);
        std::iota(order.begin(), order.end(), uint64_t{0});
        std::stable_sort(order.begin(), order.end(), [&](uint64_t x, uint64_t y) {
            if (colour[x] != colour[y]) return colour[x] < colour[y];
            return cta_of[x] < cta_of[y];
        });
        // the suspension nodes are the suspension CTA's alone: the line
        // iteration works on its shared memory
        for (size_t i = 0; i < m; ++i)
            for (int q = 0; q < counts[i]; ++q)
                if (attached[nodes[i][q]]) cta_of[i] = S.susp_cta;
    }

    // Patches may outgrow the bisection's parts by the homes they take, as far
    // as the reverse sweep of a rollout (nodes, their start adjoints, three
    // values per distance record, two per dihedral) keeps its room.
    uint64_t records[2] = {0, 0};
    for (int k = 0; k < 2; ++k) {
        std::vector<uint64_t> count(ctas, 0);
        for (int c : kind_cta[k]) ++count[c];
        records[k] = *std::max_element(count.begin(), count.end());
    }
    const uint64_t reverse = 32ull * S.max_part + 12 * records[0] + 8 * records[1] + 4ull * (total_stages(S) + 2) + 112;
    const uint64_t room = reverse < shared_limit ? (shared_limit - reverse) / 32 : 0;
    const uint32_t patch_limit = static_cast<uint32_t>(std::min<uint64_t>(kClusterPatchNodes, S.max_part + room));
    bool direct = false;
    for (;;) {
        place_nodes(S, part, kind_nodes, kind_counts, kind_cta, kind_colour, attached, patch_limit, direct);
        emit_records(d, S, kind_nodes, kind_counts, kind_cta, kind_colour, direct);
        S.forward = build_flow(d, S, false, direct);
        if (direct || (S.max_local <= kSendSlots && S.forward.max_barriers <= kSendBarriers &&
                       layout_of(S).total <= shared_limit))
            break;
        direct = true;
    }

    // line iteration window: the last stages of the iteration that touch no
    // suspension endpoint node, two at least
    if (S.susp_cta >= 0 && !(split && ctas > 1) && !direct) {
        const int Sg = total_stages(S);
        int first = Sg;
        while (first > 0 && Sg - first < kLineWindow && !stage_touches(d, S, attached, first - 1)) --first;
        if (Sg - first >= 2) {
            S.line_stage = first;
            S.line_owner_records = line_window(S, std::numeric_limits<int>::max()).records;
        }
    }

    build_load_path(d, S);

    // seam closing pass: level scheduling in sweep order, executing CTA =
    // owner of the first node
    {
        std::vector<int32_t> node_stage(N, -1);
        struct Rec { int stage, cta; uint64_t index; };
        std::vector<Rec> recs;
        for (uint64_t i : S.distance_order) {
            const auto& c = d.constraints[i];
            if (c.kind != SWB_CONSTRAINT_SEAM_STITCH) continue;
            const int s = std::max(node_stage[c.first_node], node_stage[c.second_node]) + 1;
            node_stage[c.first_node] = node_stage[c.second_node] = s;
            recs.push_back({s, home_of(S, static_cast<uint32_t>(c.first_node)), i});
        }
        S.seam_stages = 0;
        for (const Rec& r : recs) S.seam_stages = std::max(S.seam_stages, r.stage + 1);
        std::stable_sort(recs.begin(), recs.end(), [](const Rec& x, const Rec& y) {
            if (x.cta != y.cta) return x.cta < y.cta;
            return x.stage < y.stage;
        });
        S.seam_offsets.assign(static_cast<size_t>(ctas) * (S.seam_stages + 1), 0);
        size_t at = 0;
        for (int c = 0; c < ctas; ++c) {
            for (int s = 0; s <= S.seam_stages; ++s) {
                while (at < recs.size() && recs[at].cta == c && recs[at].stage < s) ++at;
                S.seam_offsets[static_cast<size_t>(c) * (S.seam_stages + 1) + s] = static_cast<uint32_t>(at);
            }
            while (at < recs.size() && recs[at].cta == c) ++at;
        }
        for (const Rec& r : recs) {
            const auto& c = d.constraints[r.index];
            S.seam_ab.push_back(make_ref(S, static_cast<uint32_t>(c.first_node)) |
                                (make_ref(S, static_cast<uint32_t>(c.second_node)) << 16));
        }
    }
    return true;
}

ReverseLayout reverse_layout_of(const ClusterSchedule& s, const ClusterFlow& f, size_t limit) {
    auto align = [](uint64_t v) { return (v + 15) & ~uint64_t{15}; };
    const uint64_t m[2] = {s.kinds[0].max_cta_records * 4ull, s.kinds[1].max_cta_records * 4ull};
    ReverseLayout L;
    uint64_t off = align((f.direct ? s.max_patch : s.max_local) * 16ull);
    auto take = [&](uint64_t bytes) {
        const uint64_t at = off;
        off = align(off + bytes);
        return static_cast<uint32_t>(at);
    };
    L.start = take(s.max_patch * 16ull);
    L.lambda[0] = take(m[0]);
    L.lambda[1] = take(m[1]);
    L.rest = take(m[0]);
    L.compliance[0] = take(m[0]);
    L.compliance[1] = take(m[1]);
    L.barriers = take(f.direct ? 0 : f.max_barriers * 8ull);
    L.bytes = take(f.direct ? 0 : f.max_barriers * 4ull);
    const int G = total_stages(s);
    L.stages = G <= kSharedStages && off + G * 16ull <= limit ? take(G * 16ull) : kStagesInGlobal;
    L.total = static_cast<uint32_t>(std::min<uint64_t>(off, 0xffffffffu));
    return L;
}

ClusterFlow build_reverse_flow(const OwnedDefinition& d, const ClusterSchedule& s, size_t limit) {
    if (!s.forward.direct) {
        ClusterFlow f = build_flow(d, s, true, false);
        if (f.max_barriers <= kSendBarriers && reverse_layout_of(s, f, limit).total <= limit) return f;
    }
    return build_flow(d, s, true, true);
}

// Checks a flow: walking the stages, every record finds each of its nodes in
// its own CTA's array (or, in a direct schedule, marked with the node's
// home), counted on the barrier its stage waits on; every node ends at home;
// each barrier receives exactly the bytes it is armed with.
void verify_flow(const OwnedDefinition& d, const ClusterSchedule& S, const ClusterFlow& F, bool reverse) {
    auto fail = [](const std::string& what) { raise(SWB_INVALID_ARGUMENT, "cluster schedule hand-overs: " + what); };
    const int C = S.ctas, G = total_stages(S);
    std::vector<int> at(S.node_count);
    std::vector<uint32_t> slot(S.node_count);
    std::vector<int64_t> pending(S.node_count, -1);  // the barrier that counts the node's last send
    std::vector<std::vector<uint32_t>> got(C);
    for (int c = 0; c < C; ++c) got[c].assign(F.bytes_begin[c + 1] - F.bytes_begin[c], 0);
    for (int c = 0; c < C; ++c)
        for (uint32_t s = S.patch_begin[c]; s < S.patch_begin[c + 1]; ++s) {
            at[S.node_of_slot[s]] = c;
            slot[S.node_of_slot[s]] = s - S.patch_begin[c];
        }
    const std::vector<int> home = at;
    auto node_at_local = [&](int c, uint32_t local) {
        const uint32_t own = S.patch_begin[c + 1] - S.patch_begin[c];
        if (local < own) return S.node_of_slot[S.patch_begin[c] + local];
        if (local - own >= S.ghost_begin[c + 1] - S.ghost_begin[c]) fail("local reference past the ghosts");
        return S.ghost_node[S.ghost_begin[c] + local - own];
    };
    auto send = [&](uint32_t n, uint32_t word) {
        const int to = static_cast<int>(word >> 27 & 15u);
        const uint32_t bar = word >> 14 & (kSendBarriers - 1), local = word & (kSendSlots - 1);
        if (!(word & kSendValid) || to >= C || bar >= got[to].size()) fail("send word");
        if (node_at_local(to, local) != n) fail("a send names another node's slot");
        got[to][bar] += 16;
        at[n] = to;
        slot[n] = local;
        pending[n] = bar;
    };
    for (int c = 0; c < C; ++c)
        for (uint32_t e = F.out_begin[c]; e < F.out_begin[c + 1]; ++e) {
            const uint32_t n = node_at_local(c, F.out[e][0]);
            if (at[n] != c) fail("a node is sent out from a CTA that does not hold it");
            send(n, F.out[e][1]);
        }
    for (int step = 0; step < G; ++step) {
        const int g = reverse ? G - 1 - step : step;
        int k, s;
        global_stage(S, g, k, s);
        const ClusterKind& K = S.kinds[k];
        for (int c = 0; c < C; ++c) {
            const size_t o = static_cast<size_t>(c) * (K.stages + 1) + s, cs = static_cast<size_t>(c) * K.stages + s;
            const uint32_t barrier = F.barrier[static_cast<size_t>(c) * G + g];
            for (uint32_t r = K.offsets[o]; r < K.offsets[o + 1]; ++r) {
                uint32_t nodes[4];
                const int cnt = element_nodes(d, k, K.def_index[r], nodes);
                const bool edge = r - K.offsets[o] < K.boundary[cs];
                const uint32_t local[4] = {K.lab[r] & 0xffffu, K.lab[r] >> 16, K.lcd[r] & 0xffffu, K.lcd[r] >> 16};
                for (int q = 0; q < cnt; ++q) {
                    const uint32_t n = nodes[q];
                    const uint32_t word = edge ? F.send[k][K.boundary_first[cs] + (r - K.offsets[o])][q] : 0u;
                    if (F.direct) {
                        const uint32_t want = home[n] == c ? 0u : send_word(static_cast<uint32_t>(home[n]), 0, slot[n]);
                        if (word != want || (!want && local[q] != slot[n])) fail("direct record's node");
                        continue;
                    }
                    if (at[n] != c || slot[n] != local[q]) fail("a record's node is not in its CTA's array");
                    if (pending[n] >= 0 && (!edge || pending[n] != static_cast<int64_t>(barrier) || barrier == 0))
                        fail("a stage does not wait for a node it receives");
                    pending[n] = -1;
                    if (word) send(n, word);
                }
            }
        }
    }
    if (F.direct) return;
    for (uint32_t n = 0; n < S.node_count; ++n)
        if (at[n] != home[n] || (pending[n] >= 0 && pending[n] != 0)) fail("a node does not come home");
    for (int c = 0; c < C; ++c)
        for (size_t b = 0; b < got[c].size(); ++b)
            if (got[c][b] != F.bytes[F.bytes_begin[c] + b]) fail("bytes of a barrier");
}

void verify_cluster_schedule(const OwnedDefinition& d, const std::vector<uint32_t>& suspension_nodes,
                             const ClusterSchedule& S) {
    verify_flow(d, S, S.forward, false);
    auto fail = [](const std::string& what) { raise(SWB_INVALID_ARGUMENT, "cluster schedule invariant: " + what); };
    const uint32_t N = static_cast<uint32_t>(d.nodes.size());
    const int C = S.ctas;
    if (C < 1 || C > kClusterMaxCtas) fail("cta count");
    if (S.patch_begin.size() != static_cast<size_t>(C) + 1 || S.patch_begin[C] != N) fail("patch ranges");
    for (uint32_t n = 0; n < N; ++n)
        if (S.node_of_slot[S.slot_of_node[n]] != n) fail("slot map");
    auto node_of_ref = [&](uint32_t ref) {
        const uint32_t cta = ref >> 12, local = ref & 0xfffu;
        if (static_cast<int>(cta) >= C || S.patch_begin[cta] + local >= S.patch_begin[cta + 1])
            fail("reference outside its patch");
        return S.node_of_slot[S.patch_begin[cta] + local];
    };
    for (uint32_t n : suspension_nodes) {
        const uint32_t slot = S.slot_of_node[n];
        if (slot < S.patch_begin[S.susp_cta] || slot >= S.patch_begin[S.susp_cta + 1])
            fail("suspension node outside the owner patch");
    }
    if (S.line_stage >= 0) {
        const int Sg = total_stages(S);
        if (S.susp_cta < 0 || S.line_stage > Sg - 2 || S.line_stage < Sg - kLineWindow)
            fail("line iteration window position");
        std::vector<uint8_t> attached(N, 0);
        for (uint32_t n : suspension_nodes) attached[n] = 1;
        for (int g = S.line_stage; g < Sg; ++g) {
            int k, s;
            global_stage(S, g, k, s);
            if (stage_touches(d, S, attached, g)) fail("line iteration window touches a suspension node");
            const size_t o = static_cast<size_t>(S.susp_cta) * (S.kinds[k].stages + 1) + s;
            if (S.kinds[k].offsets[o + 1] - S.kinds[k].offsets[o] > S.line_owner_records)
                fail("line iteration window record count");
        }
    }
    std::vector<int64_t> stamp(N, -1);
    int64_t epoch = 0;
    for (int k = 0; k < 3; ++k) {
        const ClusterKind& K = S.kinds[k];
        const size_t m = k == 0 ? d.constraints.size() : (k == 1 ? d.dihedrals.size() : d.membranes.size());
        std::vector<uint8_t> seen(m, 0);
        for (int s = 0; s < K.stages; ++s) {
            ++epoch;
            for (int c = 0; c < C; ++c)
                for (uint32_t r = K.offsets[static_cast<size_t>(c) * (K.stages + 1) + s];
                     r < K.offsets[static_cast<size_t>(c) * (K.stages + 1) + s + 1]; ++r) {
                    const uint32_t i = K.def_index[r];
                    if (seen[i]++) fail("constraint scheduled twice");
                    const uint32_t refs[4] = {K.ab[r] & 0xffffu, K.ab[r] >> 16, k ? (K.cd[r] & 0xffffu) : 0u,
                                              k ? (K.cd[r] >> 16) : 0u};
                    uint32_t want[4];
                    const int cnt = element_nodes(d, k, i, want);
                    if (k == 2 && (K.cd[r] >> 16) != 0) fail("membrane record's fourth reference");
                    for (int q = 0; q < cnt; ++q) {
                        const uint32_t n = node_of_ref(refs[q]);
                        if (n != want[q]) fail("reference does not name the constraint's node");
                        if (stamp[n] == epoch) fail("stage is not node-disjoint");
                        stamp[n] = epoch;
                    }
                }
        }
        for (size_t i = 0; i < m; ++i)
            if (!seen[i]) fail("constraint not scheduled");
    }
    // cable pairs: node-disjoint levels, each record run by the CTA owning
    // it, every cable and tie once per pass
    {
        const ClusterKind& K = S.kinds[0];
        std::vector<int> owner_of(K.def_index.size(), -1);
        for (int c = 0; c < C; ++c)
            for (uint32_t r = K.offsets[static_cast<size_t>(c) * (K.stages + 1)];
                 r < K.offsets[static_cast<size_t>(c) * (K.stages + 1) + K.stages]; ++r)
                owner_of[r] = c;
        size_t load_path = 0;
        for (const auto& c : d.constraints)
            load_path += !(c.kind == SWB_CONSTRAINT_DISTANCE || c.kind == SWB_CONSTRAINT_SEAM_STITCH);
        if (S.pair_stages > 0 && S.pair_offsets.size() != static_cast<size_t>(C) * (S.pair_stages + 1))
            fail("pair offsets");
        if (S.pair_rec.size() != 2 * load_path) fail("every cable and tie once per pass of a pair");
        std::vector<uint8_t> visits(K.def_index.size(), 0);
        for (int l = 0; l < S.pair_stages; ++l) {
            ++epoch;
            for (int c = 0; c < C; ++c)
                for (uint32_t i = S.pair_offsets[static_cast<size_t>(c) * (S.pair_stages + 1) + l];
                     i < S.pair_offsets[static_cast<size_t>(c) * (S.pair_stages + 1) + l + 1]; ++i) {
                    const uint32_t r = S.pair_rec[i];
                    if (r >= K.def_index.size() || owner_of[r] != c) fail("pair record run by another CTA");
                    const auto& con = d.constraints[K.def_index[r]];
                    if (con.kind == SWB_CONSTRAINT_DISTANCE || con.kind == SWB_CONSTRAINT_SEAM_STITCH)
                        fail("pair record is not a cable or tie");
                    ++visits[r];
                    for (uint64_t n : {con.first_node, con.second_node}) {
                        if (stamp[n] == epoch) fail("pair level is not node-disjoint");
                        stamp[n] = epoch;
                    }
                }
        }
        for (size_t r = 0; r < visits.size(); ++r) {
            const auto& con = d.constraints[K.def_index[r]];
            const bool lp = !(con.kind == SWB_CONSTRAINT_DISTANCE || con.kind == SWB_CONSTRAINT_SEAM_STITCH);
            if (visits[r] != (lp ? 2 : 0)) fail("cable pair visits");
        }
    }
    for (int s = 0; s < S.seam_stages; ++s) {
        ++epoch;
        for (int c = 0; c < C; ++c)
            for (uint32_t r = S.seam_offsets[static_cast<size_t>(c) * (S.seam_stages + 1) + s];
                 r < S.seam_offsets[static_cast<size_t>(c) * (S.seam_stages + 1) + s + 1]; ++r)
                for (uint32_t ref : {S.seam_ab[r] & 0xffffu, S.seam_ab[r] >> 16}) {
                    const uint32_t n = node_of_ref(ref);
                    if (stamp[n] == epoch) fail("seam stage is not node-disjoint");
                    stamp[n] = epoch;
                }
    }
}

}  // namespace swb
