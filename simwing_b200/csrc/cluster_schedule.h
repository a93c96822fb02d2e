// Cluster sweep schedule: one thread-block cluster solves one structure.
//
// The nodes are split into one patch per CTA of the cluster (recursive
// bisection, suspension endpoint nodes kept together) and live in that
// CTA's shared memory for the whole step.  Each constraint kind is
// coloured over the whole mesh (DSatur); a colour is one stage, and every
// constraint of a stage is executed by the CTA that owns most of its nodes
// (the suspension CTA where it touches a suspension endpoint).
//
// Between stages a CTA waits only for itself (a CTA barrier): a node that
// several CTAs touch is handed from one to the next.  Within an iteration a
// node is touched by at most one record per stage, so its touches form a
// sequence; where two touches in turn belong to different CTAs, the record
// that finishes the first sends the node to the second CTA (a store into
// its shared memory that counts on a barrier there, see cluster_kernel.cuh),
// which waits for what its stage receives before the stage's boundary
// records.  Every CTA keeps a copy slot (ghost) for each foreign node it
// touches and reads its own shared memory only.  After its last touch of an
// iteration a node returns home, to the CTA whose patch holds it: the first
// to touch it in an iteration, so that the way home is also the way to its
// next touch.  At the end of an iteration every node's value is at home,
// where the passes between iterations (ground plane, contacts, seams) and
// the kernel's epilogue find it.
//
// Direct flows (fallback, when the ghosts do not fit in shared memory: meshes
// whose constraints join nodes at random over the patches): no ghosts; a
// record reads and writes foreign nodes in place through distributed shared
// memory, and a cluster barrier closes every stage.  A schedule's forward
// sweep may hand over while its reverse, which needs more shared memory per
// record, is direct.
//
// Node references are 16-bit: the home rank in the top 4 bits and the index
// in its patch in the low 12 bits (home references), or the index in the
// executing CTA's node array, ghosts after the patch (local references).
//
// Split stages (optional, SWB_OPT_SPLIT_STAGES): a constraint whose
// nodes all lie in one CTA's patch is interior.  Per kind, the interior
// constraints run first, coloured per CTA; the constraints that span CTAs
// are coloured together and their stages follow.
//
// Sweep order per kind: stage-major, then the CTA that owns most of a
// constraint's nodes in the bisection, then definition order -- the
// reference serial solver run on the definition permuted into this
// order performs exactly the device sweep: constraints of one stage share
// no node, and every node meets its stages in order.
#pragma once

#include "common.h"

#include <array>
#include <cstdint>
#include <vector>

namespace swb {

constexpr int kClusterMaxCtas = 16;
constexpr uint32_t kClusterPatchNodes = 4096;

struct ClusterKind {
    int stages = 0;
    // [ctas * (stages + 1)]: record offsets of (cta, stage); records are
    // stored CTA-major, stage within, boundary records first.
    std::vector<uint32_t> offsets;
    // [ctas * stages]: boundary records of (cta, stage), those that touch a
    // node another CTA touches too, and the first of their entries in the
    // flows' send tables (one entry per boundary record, in record order)
    std::vector<uint32_t> boundary, boundary_first;
    uint32_t boundary_total = 0;
    std::vector<uint32_t> ab;    // home ref(a) | ref(b) << 16
    std::vector<uint32_t> cd;    // dihedral: home ref(c) | ref(d) << 16
    std::vector<uint32_t> lab, lcd;  // the same as local references
    std::vector<float> rest;
    std::vector<float> comp;     // distance: sign bit = cable
    std::vector<uint32_t> def_index;
    uint32_t max_cta_records = 0;  // multipliers held in shared memory per CTA
    int sync_stages = 0;  // stages after which nodes may change hands (split stages: those with
                          // records that span CTAs, and the last one before them)
};

// Where a record sends a node after its projection: 0 = nowhere (the node
// stays in the executing CTA's array), else kSendValid | rank << 27 | the
// barrier that counts it there << 14 | its slot in that CTA's node array.
// In a direct flow the word marks a foreign node: its home rank and slot
// (barrier 0), read and written in place.
constexpr uint32_t kSendValid = 1u << 31;
constexpr uint32_t kSendSlots = 1u << 14, kSendBarriers = 1u << 13;
constexpr uint32_t send_word(uint32_t rank, uint32_t barrier, uint32_t slot) {
    return kSendValid | rank << 27 | barrier << 14 | slot;
}

// The hand-overs of a sweep through the iteration's stages, forward or in
// reverse.  Barriers are numbered per CTA: 0 counts the nodes that come home
// at the end of an iteration, the others one receiving stage each.
struct ClusterFlow {
    bool direct = false;                  // foreign nodes in place, cluster barriers (see above)
    std::array<std::vector<std::array<uint32_t, 4>>, 3> send;  // per kind, per boundary record, per node
    std::vector<uint32_t> barrier;        // [ctas * stages]: the stage's barrier, 0 when it receives nothing
    std::vector<uint32_t> bytes_begin;    // [ctas + 1] into bytes
    std::vector<uint32_t> bytes;          // per barrier: bytes received per iteration
    // nodes whose first touch of an iteration is not at home: the home CTA
    // sends them out at the iteration's start ([ctas + 1] offsets; slot, word)
    std::vector<uint32_t> out_begin;
    std::vector<std::array<uint32_t, 2>> out;
    uint32_t max_barriers = 0;            // per CTA
};

struct ClusterSchedule {
    int ctas = 0;
    // [ctas + 1] into ghost_node: the foreign nodes a CTA touches, in the
    // order of their slots after its patch; the largest patch with ghosts
    std::vector<uint32_t> ghost_begin, ghost_node;
    uint32_t max_local = 0;
    ClusterFlow forward;
    uint32_t node_count = 0;
    std::vector<uint32_t> node_of_slot, slot_of_node;  // slots: patch-major
    std::vector<uint32_t> patch_begin;                 // [ctas + 1]
    uint32_t max_patch = 0;
    uint32_t max_part = 0;                             // the bisection's largest part
    // kinds[0] distance-type constraints, kinds[1] dihedrals, kinds[2]
    // membrane elements; an iteration runs distance, membrane, then dihedral
    // stages (soft_body.cpp:1318-1369)
    std::array<ClusterKind, 3> kinds;
    // seam closing pass: level-scheduled in sweep order, per (cta, stage)
    int seam_stages = 0;
    std::vector<uint32_t> seam_offsets;  // [ctas * (seam_stages + 1)]
    std::vector<uint32_t> seam_ab;
    int susp_cta = -1;
    // Line iteration window (classic stages only): the last stages of an
    // iteration, two to kLineWindow of them, that touch no suspension endpoint
    // node.  The iteration's line iteration runs beside them on the last warp
    // of the suspension CTA, which has no record in any, instead of after
    // them.  line_stage = the first of them (global stage index), -1 without
    // a window; line_owner_records = the suspension CTA's largest record count
    // in the window.
    int line_stage = -1;
    uint32_t line_owner_records = 0;
    std::vector<uint64_t> distance_order, dihedral_order, membrane_order;
    // Load-path cable sweeps (soft_body.cpp:528-629, 1265-1317): one pair is
    // a reverse then a forward pass over the cables and ties in graph-depth
    // order; each pass is level-scheduled (a constraint one level after the
    // last earlier one sharing a node), so a level's constraints share no
    // node and the levels reproduce the serial pass.  pair_stages = levels of
    // both passes; pair_offsets [ctas * (pair_stages + 1)] index pair_rec,
    // the distance records (kind 0) each CTA runs per level (its own: their
    // multipliers are the general sweep's).
    int pair_stages = 0;
    std::vector<uint32_t> pair_offsets, pair_rec;
};

// Colour stages per iteration, all kinds.
inline int total_stages(const ClusterSchedule& s) {
    return s.kinds[0].stages + s.kinds[1].stages + s.kinds[2].stages;
}
// Kind and stage within the kind of global stage g of an iteration
// (distance stages, membrane stages, dihedral stages).
inline void global_stage(const ClusterSchedule& s, int g, int& kind, int& local) {
    const int S0 = s.kinds[0].stages, S2 = s.kinds[2].stages;
    if (g < S0) {
        kind = 0;
        local = g;
    } else if (g < S0 + S2) {
        kind = 2;
        local = g - S0;
    } else {
        kind = 1;
        local = g - S0 - S2;
    }
}

// Stages of an iteration after which nodes may change hands, plus the line
// iteration where it follows the stages.
inline int cluster_barriers_per_iteration(const ClusterSchedule& s) {
    int n = s.susp_cta >= 0 && s.line_stage < 0 ? 1 : 0;
    for (const ClusterKind& k : s.kinds) n += k.sync_stages;
    return n;
}

// Shared memory a schedule is admitted by: nodes and velocities of the
// bisection's largest part, every multiplier, stage offsets.  A schedule that
// passes runs whatever its boundary is (a direct schedule takes no more).
inline size_t cluster_shared_bytes(const ClusterSchedule& s) {
    return s.max_part * 32ull + s.kinds[0].max_cta_records * 4ull + s.kinds[1].max_cta_records * 4ull +
           s.kinds[2].max_cta_records * 12ull + (total_stages(s) + 3) * 4ull + 80;
}

// Dynamic shared memory of the step kernel, byte offsets: the node array
// (patch and ghosts) at 0; the multipliers, three per membrane element, and
// in the same place, before and after the iterations, the patch's forces or
// velocities; the stage descriptors (none above kSharedStages, read from
// global memory then); the barriers and the bytes each receives.
constexpr int kSharedStages = 256;
constexpr uint32_t kStagesInGlobal = ~0u;  // ClusterFlowDev::smem_stages
struct ClusterLayout {
    uint32_t lambda[3] = {0, 0, 0};
    uint32_t velocity = 0, stages = 0, barriers = 0, bytes = 0, total = 0;
};
ClusterLayout layout_of(const ClusterSchedule& s);

// Shared memory of a contact launch with the key-ordered passes' links (11
// bytes a candidate in contact, contact_phase.cuh).  Shared memory comes off
// the L1 cache in steps, and the detection phases read through that cache
// (with 192 KB of links the row passes of 24 x 24 sheets take 2.0 ms a step
// against 1.1 ms), but links that do not fit cost more still (40 x 40 sheets:
// 22 ms of rounds against 13 ms).  So: the smallest step that holds one
// candidate in contact per candidate row, about what a landed sheet has (24 x
// 24 sheets: 4,500 rows, 3,900 in contact), and the first step when none does.
constexpr uint32_t kContactSharedSteps[] = {124 * 1024, 156 * 1024, 188 * 1024, 218 * 1024};
constexpr uint32_t kContactLinkBytes = 11;
// Their bytes behind a layout of `layout` bytes in a launch that may take `cap`;
// 0 where it leaves none (the links stay in global memory).
inline uint32_t contact_link_bytes(uint32_t layout, uint64_t rows, uint64_t cap) {
    const uint64_t want = layout + rows * kContactLinkBytes + 256;
    uint64_t limit = kContactSharedSteps[0];
    for (uint32_t step : kContactSharedSteps)
        if (limit < want && step >= want) limit = step;
    limit = limit < cap ? limit : cap;
    return limit > layout ? static_cast<uint32_t>(limit - layout) & ~15u : 0u;
}

// Stages a line iteration may run beside: one takes about 5 us, a stage of a
// wing 0.5 to 1 us.
constexpr int kLineWindow = 8;

// The stages of the schedule's line iteration window that a block of `threads`
// threads leaves a warp idle in (the suspension CTA's records fit the others),
// from the last one back: the first of them, -1 when they are fewer than two,
// and the suspension CTA's largest record count in them.
struct LineWindow {
    int first = -1;
    uint32_t records = 0;
};
LineWindow line_window(const ClusterSchedule& s, int threads);

// Returns false (and leaves `out` empty) when the mesh does not fit one
// cluster of `ctas` CTAs (a patch over kClusterPatchNodes nodes).  The
// forward flow is direct when its layout with ghosts would exceed
// `shared_limit` bytes.
bool build_cluster_schedule(const OwnedDefinition& d, const std::vector<uint32_t>& suspension_nodes, int ctas,
                            ClusterSchedule& out, bool split = false, size_t shared_limit = 227 * 1024 - 6144);

// The hand-overs of one sweep direction (see ClusterFlow).
ClusterFlow build_flow(const OwnedDefinition& d, const ClusterSchedule& s, bool reverse, bool direct);

// Dynamic shared memory of the reverse kernel with hand-overs `f`, byte
// offsets: the node adjoints (with ghosts unless direct) at 0, their start
// adjoints, the records' multiplier and parameter adjoints (rest lengths of
// distances, compliances), then as in ClusterLayout; the stage descriptors are
// left in global memory where they would exceed `limit`.
struct ReverseLayout {
    uint32_t start = 0, lambda[2] = {0, 0}, rest = 0, compliance[2] = {0, 0};
    uint32_t stages = 0, barriers = 0, bytes = 0, total = 0;
};
ReverseLayout reverse_layout_of(const ClusterSchedule& s, const ClusterFlow& f, size_t limit);

// The reverse sweep's hand-overs: direct where the forward's are, where
// handing over would exceed `limit` bytes of shared memory, or where a CTA has
// more receiving stages than a send word can name.
ClusterFlow build_reverse_flow(const OwnedDefinition& d, const ClusterSchedule& s, size_t limit);

// Checks a flow of a schedule; raises on failure (verify_cluster_schedule
// checks the forward one, a planned schedule's reverse ones are checked too).
void verify_flow(const OwnedDefinition& d, const ClusterSchedule& s, const ClusterFlow& f, bool reverse);

// Stage descriptors of a flow, [ctas * stages] (global stages): the first
// record, the record count, the first boundary record's entry in the send
// table, boundary records | barrier << 16.  Records and send entries of all
// kinds are numbered together, kind after kind.
std::vector<std::array<uint32_t, 4>> stage_descriptors(const ClusterSchedule& s, const ClusterFlow& f);

// Move budget of the search for a colouring with fewer colours (per colour
// count tried).
constexpr long kColourSearchMoves = 300000;

// Checks the invariants the cluster kernel relies on; raises on failure.
void verify_cluster_schedule(const OwnedDefinition& d, const std::vector<uint32_t>& suspension_nodes,
                             const ClusterSchedule& s);

// Colouring helper shared with the grid schedule: DSatur over constraints
// given as node lists (2 or 4 nodes), conflicts = shared nodes.
int dsatur_colour(const std::vector<std::array<uint32_t, 4>>& nodes, const std::vector<int>& counts,
                  std::vector<int>& colour);

// Recursive coordinate bisection of nodes into `parts` (see schedule.cpp).
std::vector<int> bisect_nodes(const OwnedDefinition& d, const std::vector<uint32_t>& grouped_nodes, int parts,
                              double tolerance);

}  // namespace swb
