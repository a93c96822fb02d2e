// Hand-over of nodes between the CTAs of a cluster (ClusterFlow,
// cluster_schedule.h): a CTA's barriers, one per stage that receives nodes
// and one for the nodes that come home at an iteration's end, each armed
// with the bytes it receives per iteration.  A send is one st.async: the
// node's 16 bytes into the receiver's node array and their count on the
// receiver's barrier, with no fence and no wait at the sender.
//
// A barrier's phase p is iteration p (reverse sweeps count their own): it
// is armed again for the next iteration only after the CTA barrier that
// closes the receiving stage (for the nodes that come home, the next
// iteration's first barrier of the whole block), when every thread has passed
// its wait.  The next iteration's first nodes may be counted before that (a transaction
// count may run ahead of its arming); the phase cannot end before the
// arming, which is its only arrival.  A node is not overwritten before its
// reader is done: its next value exists only after the reader's result.
//
// A wait has a limit.  A CTA in which one has run out goes on to the end of
// the step, so that every barrier of the block and of the cluster is met, but
// it arms none of its own again (the phase that did not end has had its
// arrival), and from the next iteration on it leaves out the stages and sends
// nothing, so that the CTAs that wait for it run out in turn.  Before it
// leaves it lets what is under way to it arrive (flow_drain).  The status word
// makes the host drop the trial state.
#pragma once

#include "cluster_params.h"
#include "device_common.cuh"

namespace swb {
namespace dev {

constexpr long long kFlowDrain = 200000;     // cycles, about 0.1 ms

// The CTA's waits, in shared memory: what one that runs out works on.
struct FlowLimit {
    long long budget;      // cycles a wait may take
    int* status;
    uint32_t* bytes;       // Flow::bytes, set to 0 when a wait has run out
    uint32_t barriers;
    uint32_t home;         // shared address of the barrier of the nodes that come home
    int ran_out;           // first iteration with a wait that ran out (one for the nodes that come
                           // home counts to the next), kFlowNever, or -1: FlowWait::held
};
constexpr int kFlowNever = 0x7fffffff;

struct Flow {
    uint32_t x_base;       // shared address of the node array
    uint32_t bar_base;     // shared address of the barriers
    uint32_t rank_base;    // the structure's first rank in the cluster
    const uint32_t* bytes; // per barrier (shared memory); [0]: the nodes that come home
    uint32_t out_lo, out_hi;
    FlowLimit* limit;
    bool home;             // nodes come home to this CTA from others
};

__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    return remote;
}

// The CTA barrier between two stages, for `threads` of the block: all, or all
// but a warp that works across several stages (barriers of their own, so that
// the two counts never meet on one).
__device__ __forceinline__ void stage_sync(uint32_t id, uint32_t threads) {
    asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void flow_arm(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Arms this CTA's barrier `index` for the next iteration (one thread, behind a
// barrier that follows every wait for this one), unless a wait has run out.
__device__ __forceinline__ void flow_arm_again(const Flow& f, uint32_t index) {
    const uint32_t bytes = f.bytes[index];
    if (bytes) flow_arm(f.bar_base + index * 8u, bytes);
}

// This CTA's barriers (every thread; a cluster barrier must follow before
// the first send).
__device__ __forceinline__ void flow_setup(Flow& f, const ClusterFlowDev& F, uint32_t me, unsigned char* smem,
                                           uint32_t x_base, uint32_t rank_base, FlowLimit* limit, int* status,
                                           const FlowWait& wait) {
    uint32_t* bytes = reinterpret_cast<uint32_t*>(smem + F.smem_bytes);
    f.x_base = x_base;
    f.bar_base = smem_addr(smem + F.smem_barriers);
    f.rank_base = rank_base;
    f.bytes = bytes;
    f.out_lo = __ldg(F.out_begin + me);
    f.out_hi = __ldg(F.out_begin + me + 1);
    f.limit = limit;
    f.home = false;
    const uint32_t lo = __ldg(F.bytes_begin + me), n = F.direct ? 0u : __ldg(F.bytes_begin + me + 1) - lo;
    // (direct schedules have no waits to run out)
    const bool held = static_cast<int>(me) == wait.held && !F.direct;
    if (threadIdx.x == 0) *limit = FlowLimit{wait.budget, status, bytes, n, f.bar_base, held ? -1 : kFlowNever};
    if (F.direct) return;
    for (uint32_t b = threadIdx.x; b < n; b += blockDim.x) {
        const uint32_t v = __ldg(F.bytes + lo + b);
        bytes[b] = v;
        const uint32_t bar = f.bar_base + b * 8u;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        flow_arm(bar, v);
    }
    f.home = n > 0 && __ldg(F.bytes + lo) > 0;
}

__device__ __forceinline__ bool flow_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

__device__ __noinline__ void flow_wait_slow(uint32_t bar, uint32_t iteration, FlowLimit* limit) {
    volatile FlowLimit& l = *limit;
    const long long start = clock64(), budget = l.budget;
    while (l.ran_out == kFlowNever && !flow_test(bar, iteration & 1u)) {
        // (a structure with a wait that has run out in another CTA waits no longer)
        if (clock64() - start > budget || (ld_relaxed_status(l.status) & kStatusFlowTimeout)) {
            for (uint32_t b = 0; b < l.barriers; ++b) *static_cast<volatile uint32_t*>(l.bytes + b) = 0;
            atomicMin(&limit->ran_out, static_cast<int>(iteration + (bar == l.home ? 1u : 0u)));
            atomicOr(l.status, kStatusFlowTimeout);
            return;
        }
    }
}

// Waits for phase `iteration` of this CTA's barrier `index`.
__device__ __forceinline__ void flow_wait(const Flow& f, uint32_t index, uint32_t iteration) {
    const uint32_t bar = f.bar_base + index * 8u;
    if (!flow_test(bar, iteration & 1u)) flow_wait_slow(bar, iteration, f.limit);
}

// Before iteration `iteration`: a wait of the ones before ran out (those for
// the nodes of the last home-coming apart).  The same for every thread: all
// that could answer otherwise lies behind a barrier of the block.
__device__ __forceinline__ bool flow_ran_out(const Flow& f, uint32_t iteration) {
    return static_cast<volatile FlowLimit*>(f.limit)->ran_out < static_cast<int>(iteration);
}

// Before this CTA leaves (one thread, behind a cluster barrier that follows
// the iterations): where a wait has run out, nodes sent here may still be under
// way.  They take a microsecond or two.
__device__ __forceinline__ void flow_drain(const Flow& f) {
    if (static_cast<volatile FlowLimit*>(f.limit)->ran_out == kFlowNever) return;
    for (const long long start = clock64(); clock64() - start < kFlowDrain;) __nanosleep(1000);
}

// Sends a node where its word says (cluster_schedule.h, send_word).
__device__ __forceinline__ void flow_send(const Flow& f, uint32_t word, float4 v) {
    const uint32_t rank = ((word >> 27) & 15u) + f.rank_base;
    const uint32_t to = map_rank(f.x_base + (word & 0x3fffu) * 16u, rank);
    const uint32_t bar = map_rank(f.bar_base + ((word >> 14) & 0x1fffu) * 8u, rank);
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}

// The same where `word` may be 0 (no send): predicated, so that a warp whose
// lanes send different nodes of their records does not branch on each.
__device__ __forceinline__ void flow_send_if(const Flow& f, uint32_t word, float4 v) {
    const uint32_t rank = ((word >> 27) & 15u) + f.rank_base;
    const uint32_t to = map_rank(f.x_base + (word & 0x3fffu) * 16u, rank);
    const uint32_t bar = map_rank(f.bar_base + ((word >> 14) & 0x1fffu) * 8u, rank);
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %6, 0;\n"
        " @p st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];\n}\n" ::"r"(to),
        "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar), "r"(word)
        : "memory");
}

// Direct schedules: the address of a foreign node.
__device__ __forceinline__ uint32_t flow_address(const Flow& f, uint32_t word) {
    return map_rank(f.x_base + (word & 0x3fffu) * 16u, ((word >> 27) & 15u) + f.rank_base);
}

// The nodes this CTA sends out at the start of an iteration (every thread;
// their values are final and visible to the block).
__device__ __forceinline__ void flow_send_out(const Flow& f, const ClusterFlowDev& F, const float4* x) {
    for (uint32_t e = f.out_lo + threadIdx.x; e < f.out_hi; e += blockDim.x) {
        const uint2 o = __ldg(F.out + e);
        flow_send(f, o.y, x[o.x]);
    }
}

}  // namespace dev
}  // namespace swb
