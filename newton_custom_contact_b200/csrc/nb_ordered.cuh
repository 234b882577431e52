// Ordered accumulation of per-body deltas within one world, for a group of G
// threads.
//
// The reference sums the deltas its constraint kernels produce into per-body
// accumulators with float atomics (solve_body_contact_positions,
// solve_body_joints, apply_rigid_restitution in
// newton/_src/solvers/xpbd/kernels.py): run sequentially, every body's delta is
// the float sum of its contributions in item order (contact index, joint
// index), starting from zero.  ordered_pass reproduces exactly that sum, in
// parallel and deterministically:
//
//   1. test: the group tests items in rounds of G (thread t takes item
//      base + t) and appends the active ones to a shared ring in item order
//      (warp ballots; across warps a prefix of the per-warp counts);
//   2. solve: whenever the ring holds G entries, every thread solves one of the
//      G oldest into its row of deltas (A side, B side); the rest stay for the
//      next round, so only a pass's last solve has idle threads;
//   3. gather: body i belongs to thread i % G.  The solve marks, per owner
//      thread, which entries touch its bodies (a bit per entry, shared-memory
//      atomicOr, one word per 32 entries), and every owner adds the rows of its
//      own entries in ring order -- in registers where it owns one body (at most
//      G bodies), else in the accumulators entry by entry.
//
// No atomics touch the accumulators, and because the ring is solved and walked
// in item order, each body sees its contributions in item order.
//
// Why a full round per solve: a one-warp group's test round finds 10 to 20
// active contacts, and solving whatever a 48-entry batch held when it could
// overflow ran the solve (the longest code of the step) on about 60 % of the
// lanes.  Why marks for every group size: an owner that walks all entries costs
// a wide group more than the solve itself.
#pragma once

#include "nb_math.cuh"

namespace nb {

// the active items of a group of G threads waiting to be solved, and the rows of the ones being solved
template <int G>
struct OrderedBatch {
    static constexpr int kRing = 2 * G;   // fewer than G wait when a round of G is tested
    static constexpr int kWords = G / 32;
    float d[G][12];            // A side (lin 3, ang 3), B side (lin 3, ang 3)
    int item[kRing];
    int ends[kRing];           // (la + 1) | (lb + 1) << 16
    unsigned own_a[kWords][G];  // bit (a & 31) of word a >> 5: entry a touches a body of the thread on side A
    unsigned own_b[kWords][G];  // ... on side B
    int wcnt[2][8];            // per-warp counts of the last two test rounds (G > 32)
};

__device__ __forceinline__ int ends_pack(int la, int lb) { return (la + 1) | ((lb + 1) << 16); }
__device__ __forceinline__ int ends_a(int e) { return (e & 0xFFFF) - 1; }
__device__ __forceinline__ int ends_b(int e) { return ((e >> 16) & 0xFFFF) - 1; }

// barrier of a group of G threads (group g of the CTA): a warp, a named
// barrier over the group's warps, or the whole CTA
template <int G, int kCTA>
__device__ __forceinline__ void ordered_sync(int g) {
    if constexpr (G == 32) {
        __syncwarp();
    } else if constexpr (G == kCTA) {
        __syncthreads();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(G) : "memory");
    }
}

// Appends the active items of one test round behind the n waiting entries (the first at ring place
// `head`), in item order; n is uniform over the group.  `round` alternates the per-warp counts, so one
// barrier per round separates a round's reads from the next but one's writes.
template <int G, int kCTA>
__device__ __forceinline__ void ordered_append(OrderedBatch<G>& B, bool active, int k, int ends, int g, int t,
                                               int head, int round, int& n) {
    const unsigned lane = (unsigned)t & 31u;
    const unsigned ball = __ballot_sync(0xffffffffu, active);
    int off = head + n + __popc(ball & ((1u << lane) - 1u));
    if constexpr (G == 32) {
        n += __popc(ball);
    } else {
        const int warp = t >> 5;
        if (lane == 0) B.wcnt[round & 1][warp] = __popc(ball);
        ordered_sync<G, kCTA>(g);
#pragma unroll
        for (int w = 0; w < G / 32; ++w) {
            const int c = B.wcnt[round & 1][w];
            if (w < warp) off += c;
            n += c;
        }
    }
    if (active) {
        const int pos = off & (OrderedBatch<G>::kRing - 1);
        B.item[pos] = k;
        B.ends[pos] = ends;
    }
}

// Solves the m <= G oldest entries (ring places head, head + 1, ...) and adds their rows to the owners'
// accumulators in entry (= item) order.  solve(item, d[12]) fills a row; load(i, a6) reads body i's
// accumulator and store(i, a6, n) writes it after n rows were added (called by body i's owner thread only).
template <int G, int kCTA, class Solve, class Load, class Store>
__device__ __forceinline__ void ordered_flush(OrderedBatch<G>& B, int head, int m, int n_bodies, int g, int t,
                                              Solve& solve, Load& load, Store& store) {
    constexpr int kW = OrderedBatch<G>::kWords, kMask = OrderedBatch<G>::kRing - 1;
#pragma unroll
    for (int w = 0; w < kW; ++w) {
        B.own_a[w][t] = 0u;
        B.own_b[w][t] = 0u;
    }
    ordered_sync<G, kCTA>(g);  // the entries and the cleared marks are visible
    if (t < m) {
        const int pos = (head + t) & kMask;
        solve(B.item[pos], B.d[t]);
        const int e = B.ends[pos];
        const int la = ends_a(e), lb = ends_b(e);
        const unsigned bit = 1u << (t & 31);
        if (la >= 0) atomicOr(&B.own_a[t >> 5][la & (G - 1)], bit);
        if (lb >= 0) atomicOr(&B.own_b[t >> 5][lb & (G - 1)], bit);
    }
    // Never taken (m > 0).  With a single call site the compiler inlines the solve and contracts other pairs
    // of its products into FMAs than in the other kernels that call it (3e-7 relative per step); with a second
    // one the product build's plain step gives the same bits on every schedule.  That is how this compiler
    // behaves, not a rule of the language: tests/test_gpu_schedule_bits.py compares the schedules.  The
    // warm-started step is not covered: groups of 32 with the compact slab round a few values differently (4e-9
    // relative over a step's velocities).  The parity build, which contracts nothing, needs none of this.
    if (m < 0) solve(t, B.d[t]);
    ordered_sync<G, kCTA>(g);  // the rows and the marks are visible
    float acc[6];
    if (n_bodies <= G) {
        // body t: one loop over all of its entries, whichever word they are in.  The lanes' loops end
        // together only once per flush, not once per word, and no entry waits for the one before to reach
        // shared memory: 256 stacks of 16 boxes, about 12 contact ends per box, 84 -> 65 us per step; 4096
        // mixed worlds (with the loop below for the larger of them) 355 -> 323 us
        int w = 0, n = 0;
        unsigned mb = B.own_b[0][t], rest = B.own_a[0][t] | mb;
        for (;;) {
            while (rest == 0u && ++w < kW) {
                mb = B.own_b[w][t];
                rest = B.own_a[w][t] | mb;
            }
            if (rest == 0u) break;
            const int j = __ffs(rest) - 1;
            rest &= rest - 1u;
            if (n++ == 0) load(t, acc);
            const float* row = &B.d[(w << 5) + j][(mb >> j) & 1u ? 6 : 0];
#pragma unroll
            for (int k = 0; k < 6; ++k) acc[k] = acc[k] + row[k];
        }
        if (n > 0) store(t, acc, n);
    } else {
#pragma unroll
        for (int w = 0; w < kW; ++w) {
            unsigned ma = B.own_a[w][t], mb = B.own_b[w][t];
            while (ma | mb) {
                // the entry's A side first, then its B side (another body)
                const int j = __ffs(ma | mb) - 1;
                const unsigned bit = 1u << j;
                const bool side_a = (ma & bit) != 0u;
                if (side_a) ma &= ~bit;
                else mb &= ~bit;
                const int e = B.ends[(head + (w << 5) + j) & kMask];
                const int i = side_a ? ends_a(e) : ends_b(e);
                const float* row = &B.d[(w << 5) + j][side_a ? 0 : 6];
                load(i, acc);
#pragma unroll
                for (int k = 0; k < 6; ++k) acc[k] = acc[k] + row[k];
                store(i, acc, 1);
            }
        }
    }
    ordered_sync<G, kCTA>(g);  // the rows, the marks and the solved ring places may be rewritten
}

// The pass over items 0 .. n_items - 1.  test(k, ends) -> bool decides whether
// item k contributes (and to which bodies); every thread of the group must
// call this with the same n_items.
template <int G, int kCTA, class Test, class Solve, class Load, class Store>
__device__ __forceinline__ void ordered_pass(OrderedBatch<G>& B, int n_items, int n_bodies, int g, int t, Test& test,
                                             Solve& solve, Load& load, Store& store) {
    int n = 0, head = 0, round = 0;
    int base = 0;
    // one flush for full rounds and the last, partial one: the solve is the step's longest code, and two
    // live copies of it cost instruction fetches (4096 mixed worlds: 396 against 355 us per step)
    for (;;) {
        while (n < G && base < n_items) {
            const int k = base + t;
            int ends = 0;
            const bool active = k < n_items && test(k, ends);
            ordered_append<G, kCTA>(B, active, k, ends, g, t, head, round, n);
            base += G;
            ++round;
        }
        if (n == 0) break;
        const int m = n < G ? n : G;
        ordered_flush<G, kCTA>(B, head, m, n_bodies, g, t, solve, load, store);
        head += m;
        n -= m;
    }
}

// n_bodies of a pass whose owners always add in the accumulators (see ordered_flush)
constexpr int kManyBodies = 1 << 30;

}  // namespace nb
