// The IDA* search kernel, one search per warp.
//
// Same method, queue and admission as search_kernel.cuh, but a warp's 32 lanes share one search: the
// warp keeps a pool of nodes (six frames, bounds, frame order, path) in shared memory and a queue of
// their children; every lane evaluates up to two children and takes the next ones when they are
// decided, and each pass of the loop probes the table once for each.  A child that passes all its
// frames waits in a stash, with its bounds but without frames, until the queue runs short: then
// five of them, the deepest first, become nodes at once (six lanes a node, a frame each).  Nothing is
// undone on the way back: a node's place is free when no lane, queue or stash entry refers to it.
//
// What bounds it: random 32-byte sectors of the table (44 G/s of them on B200).  With one search per
// lane (search_phased.cuh) a pass took 20.5 warp instructions per probe at 18 of 32 lanes, since
// pushes, pops and fetches run for a few lanes at a time, and a call of few cubes was 75,776 lanes
// each alone on a subtree of very uneven size.  Here 59 of 64 places hold a child, control is
// uniform, and 2,960 warps share an iteration's items and search a subtree 32 lanes wide.  Measured
// on B200, d4t, cubes/s before (the lane kernels' defaults) and now: one cube per call 57 -> 203, 16 at a
// time 131 -> 299, 100 at a time 179 -> 354, 1,024 at a time 334 -> 418, 4,096 with 5% hard 235 -> 283; a lone
// superflip on d4 0.65 -> 0.43 s, on d4t, 73 G probes of a tree that hardly narrows, 2.53-2.76 -> 2.45 s.
// 640 threads a block, one block an SM: 92 registers, and with 32 nodes a warp some 50 KB stay L1; when
// 640 threads gave 351 cubes/s at 1,024, 512 (116 registers) gave 313 and 768 (80 registers, spills) 329.
#pragma once

#include "search_kernel.cuh"
#include "warp_tables.cuh"

namespace ccs {

// (the CPU test builds them small)
#ifndef CCS_WARP_POOL
#define CCS_WARP_POOL 32
#define CCS_WARP_STACK 6
#endif
#ifndef CCS_WARP_SPILL
#define CCS_WARP_SPILL 24
#endif
#ifndef CCS_WARP_FULL
#define CCS_WARP_FULL (CCS_WARP_SPILL > 10 ? 32u * CCS_WARP_SPILL - 324u : 0u)
#endif
#ifndef CCS_WARP_BARREN
#define CCS_WARP_BARREN (1u << 16)
#endif

constexpr uint32_t WN_E2 = 24;      // frame k: c0 c1 e0 e1 at 4k, e2 here + k
constexpr uint32_t WN_H = 30;       // bounds, 5 bits per frame
constexpr uint32_t WN_META = 31;    // budget (moves to the bound) | depth << 8 | prefix length << 16
constexpr uint32_t WN_ORD = 32;     // frame order (18 bits) | budget of its children << 18
constexpr uint32_t WN_PATH = 33;    // moves from the root, six per word
constexpr uint32_t WN_STRIDE = 40;  // words of a node
constexpr uint32_t WN_POOL = CCS_WARP_POOL;       // nodes of a warp (at most 32)
constexpr uint32_t WARP_STACK = CCS_WARP_STACK;   // passed children a lane holds until they are opened
                                                  // (two words each, see PUSH)
constexpr uint32_t WARP_QUEUE = 256;              // children of open nodes (node | move << 6 | axis << 11, 16 bits)
constexpr uint32_t WARP_WORDS = WN_POOL * WN_STRIDE + 64u * WARP_STACK + WARP_QUEUE / 2u + 96u;  // shared memory of a warp
constexpr uint32_t WARP_RATIO = 4, WARP_COOL = 4;  // see OPEN
constexpr uint32_t WARP_WIDE = 11;  // budgets held to be wide before they are counted (most entries are 11 or less)
constexpr uint32_t WARP_BARREN = CCS_WARP_BARREN;  // passes without a probe or a poll after which a warp gives
                                                   // its work up
constexpr uint32_t WARP_HOLD = 2048;  // passes (about 10 ms) after which a warp takes its next item from the
                                      // queue again, so that a long iteration does not keep warps from others
constexpr int WARP_SPILL = CCS_WARP_SPILL;  // spilled nodes per lane (with 24 the launch's stacks, 56 MB, stay below
                                            // the 57 MB of 256 x 2 lanes: a server's budget counts them)
// Children stashed or spilled from which on a warp opens no more of them, so that the spill list cannot
// overflow.  Up to here at most 64 children are under evaluation and 235 queued (160 and five nodes of 15), which
// may all pass.  Beyond, all of them go to the list, and the last one of the list is searched alone, one of its
// children at a time: what is left of it waits in its place, which adds at most one node to each of 22 depths.
constexpr uint32_t WARP_FULL = CCS_WARP_FULL;

__device__ __forceinline__ State node_frame(const uint32_t* n, uint32_t k) {
    const Word4 a = reinterpret_cast<const Word4*>(n)[k];
    return State{a.x, a.y, a.z, a.w, n[WN_E2 + k]};
}

__device__ __forceinline__ void set_node_frame(uint32_t* n, uint32_t k, const State& s) {
    reinterpret_cast<Word4*>(n)[k] = Word4{s.c0, s.c1, s.e0, s.e1};
    n[WN_E2 + k] = s.e2;
}

template <int THREADS>
constexpr size_t warp_dyn_smem() {
    return (size_t)THREADS / 32u * WARP_WORDS * 4u;
}

// Sum over the warp of 32-bit counts, in 64 bits.
__device__ __forceinline__ unsigned long long warp_sum(uint32_t v) {
    const unsigned long long hi = __reduce_add_sync(0xFFFFFFFFu, v >> 16);
    return (hi << 16) + __reduce_add_sync(0xFFFFFFFFu, v & 0xFFFFu);
}

// Bounds of a new cube's six frames, one per lane, and its first iteration.
template <int MODE, int NEC, int FMT>
__device__ __forceinline__ void admit_slot_warp(const WarpTables& T, const SearchParams& P, uint32_t s, uint32_t lane) {
    Slot& sl = P.slots[s];
    uint32_t v = 0;
    bool solved = false;
    if (lane < 6u) {
        const State f = slot_frame(sl, lane);
        const bool second = __ldcg(&sl.table) != 0u;
        v = min(warp_probe<MODE, NEC, FMT>(T, P.classidx, second ? P.table2 : P.table, f, second), 31u);
        solved = lane == 0u && is_solved(f);
    }
    const uint32_t h = __reduce_or_sync(0xFFFFFFFFu, lane < 6u ? v << (5u * lane) : 0u);
    uint32_t bound = __reduce_max_sync(0xFFFFFFFFu, v);
    if (lane == 0u) {
        atomicAdd(&sl.probes, 6ull);
        atomicAdd(&P.q->probes, 6ull);
        sl.h0 = h;
        sl.t_admit = globaltimer_ns();
        if (solved) {
            sl.sol_len = 0;
            sl.found = 1;
            finish_slot(P, s, SLOT_SOLVED);
        } else {
            if (bound == 0u) bound = 1u;  // not solved, so at least one move
            publish_epoch(P, s, next_plen(P, 0ull, bound), bound, 1u);
        }
    }
    __syncwarp();
}

// A warp leaves with units in hand: the cube ends as SLOT_ERROR (unless another warp has solved it).
static __device__ __noinline__ void give_up(const SearchParams& P, uint32_t slot, uint32_t held) {
    Slot& sl = P.slots[slot];
    atomicOr(&P.q->error, ERR_STUCK);
    atomicCAS(&sl.found, 0u, FOUND_FAILED);
    __threadfence();
    if (atomicSub(&sl.open, held) == held) {
        __threadfence();
        finish_slot(P, slot, *(volatile uint32_t*)&sl.found == FOUND_FAILED ? SLOT_ERROR : SLOT_SOLVED);
    }
}

// Up to two children per lane are under evaluation.  k: frame to probe next, 6 = passed (see PUSH),
// 7 = none.  budget: moves the child leaves to the bound.
struct WarpChild {
    uint32_t node = 0, m = 0, k = 7, rem = 0, c = 0, budget = 0;
};

template <int MODE, int NEC, int FMT, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB)
search_kernel_warp(const WarpTables* __restrict__ gT, const __grid_constant__ SearchParams P) {  // (else every thread copies it)
    __shared__ WarpTables T;
    extern __shared__ Word4 pool_smem[];
    stage_tables(T, gT);
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    constexpr uint32_t POOL_ALL = WN_POOL < 32u ? (1u << (WN_POOL & 31u)) - 1u : FULL;
    constexpr uint32_t NONE = (1u << (5u * WARP_STACK)) - 1u;  // an empty stash
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    uint32_t* const pool = reinterpret_cast<uint32_t*>(pool_smem) + (threadIdx.x >> 5) * WARP_WORDS;
    uint32_t* const stash = pool + WN_POOL * WN_STRIDE;  // entry j of a lane: words 64 j + lane, 64 j + 32 + lane
    uint32_t* const handed = stash + 64u * WARP_STACK;  // by budget of the parent, sampled: children taken up, passed
    uint32_t* const passed = handed + 32;
    uint32_t* const refs = passed + 32;  // stashed children of a node
    uint16_t* const queue = reinterpret_cast<uint16_t*>(refs + 32);
    // (every place holds a state, be it none, so that lanes without a child compute harmless indexes)
    for (uint32_t i = lane; i < WARP_WORDS; i += 32u) pool[i] = 0u;
    const uint32_t seed0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 0x9E3779B1u >> 7;
    const uint32_t team = lane / 6u, tk = lane % 6u;  // OPEN: lane builds frame tk of the team-th node

    // The warp's unit of work: `held` items (or donated subtrees) of one iteration of one cube.
    uint32_t slot = 0, bound = 0, held = 0;
    bool dry = true;                   // the iteration has no more items (or this warp takes no more)
    const uint32_t* table = P.table;
    bool second = false;
    uint32_t mine = NONE, ns = 0;      // budgets of the lane's stash entries (5 bits each, 31: free); entries in all
    uint32_t wide_at = ~0u << WARP_WIDE, cool = 0;  // budgets of wide nodes (mask); passes since one was opened
    uint32_t head = 0, tail = 0;       // the queue's children
    uint32_t spilled = 0;              // nodes in the lanes' spill lists (most recent last)
    unsigned long long sw1[WARP_SPILL], sw2[WARP_SPILL], sw3[WARP_SPILL];

    WarpChild ch[2];
    uint32_t nodes = 0, probes = 0;
    uint32_t barren = 0;  // passes in a row without a probe
    uint32_t iter = 0, iter0 = 0, idle_polls = 0, backoff = 32, fetches = 0;

    // Places of nodes without a child stashed, queued or under evaluation.
    auto free_places = [&]() {
        uint32_t used = (ch[0].k < 7u ? 1u << ch[0].node : 0u) | (ch[1].k < 7u ? 1u << ch[1].node : 0u);
        for (uint32_t i = head + lane; (int)(tail - i) > 0; i += 32u) used |= 1u << (queue[i % WARP_QUEUE] & 31u);
        used = __reduce_or_sync(FULL, used);
        return __ballot_sync(FULL, refs[lane] == 0u) & ~used & POOL_ALL;
    };
    // A stash entry (bounds; node | move << 6 | children << 11)
    // ... as a node of its own: bounds | depth << 32 | budget << 37 | children << 42 | prefix
    // length << 60, and its path.
    auto pack_entry = [&](uint32_t owner, uint32_t j, unsigned long long& w1, unsigned long long& w2, unsigned long long& w3) {
        const uint32_t e0 = stash[64u * j + owner], e1 = stash[64u * j + 32u + owner], mv = (e1 >> 6) & 31u;
        const uint32_t* n = pool + (e1 & 63u) * WN_STRIDE;
        const uint32_t meta = n[WN_META], g = (meta >> 8) & 255u, plen = meta >> 16;
        uint32_t w[4] = {n[WN_PATH], n[WN_PATH + 1], n[WN_PATH + 2], n[WN_PATH + 3]};
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)
            if (i == g / 6u && g >= plen) w[i] |= mv << (5u * (g % 6u));
        w1 = (unsigned long long)e0 | ((unsigned long long)(g + 1u) << 32) |
             ((unsigned long long)((meta & 255u) - 1u) << 37) | ((unsigned long long)(e1 >> 11) << 42) |
             ((unsigned long long)plen << 60);
        w2 = w[0] | ((unsigned long long)w[1] << 30);
        w3 = w[2] | ((unsigned long long)w[3] << 30);
    };
    // The lane's deepest stash entry, as budget << 3 | entry (31 << 3 and above: none); the warp's
    // shallowest, as budget << 8 | lane << 3 | entry (0: none).
    auto deepest = [&]() {
        uint32_t best = mine & 31u;
        best <<= 3;
#pragma unroll
        for (uint32_t j = 1; j < WARP_STACK; ++j) best = min(best, (((mine >> (5u * j)) & 31u) << 3) | j);
        return best;
    };
    auto shallowest = [&]() {
        uint32_t best = 0;
#pragma unroll
        for (uint32_t j = 0; j < WARP_STACK; ++j) {
            const uint32_t b = (mine >> (5u * j)) & 31u;
            if (b != 31u) best = max(best, (b << 8) | (lane << 3) | j);
        }
        return __reduce_max_sync(FULL, best);
    };

    for (;;) {
        __syncwarp();
        const bool sample = (iter & 7u) == 0u;  // passes whose children are counted
        // PUSH a child that passed all its frames (one per lane and pass): at the bound it is a
        // solution or nothing; a dead end is dropped; the others go into the lane's stash.
        if (__ballot_sync(FULL, ch[0].k == 6u || ch[1].k == 6u)) {
            const bool s1 = ch[0].k != 6u;
            bool keep = !s1 || ch[1].k == 6u;
            const uint32_t xn = s1 ? ch[1].node : ch[0].node, xm = s1 ? ch[1].m : ch[0].m, xc = s1 ? ch[1].c : ch[0].c;
            const uint32_t budget = s1 ? ch[1].budget : ch[0].budget;
            uint32_t todo = 0;
            bool gone = false;
            if (keep) {
                const uint32_t* n = pool + xn * WN_STRIDE;
                const uint32_t meta = n[WN_META], g = ((meta >> 8) & 255u) + 1u, plen = meta >> 16;
                if (budget == 0u) {
                    const State t = warp_step(T, node_frame(n, 0u), 0u, xm);
                    Slot& sl = P.slots[slot];
                    if (is_solved(t) && atomicCAS(&sl.found, 0u, 1u) == 0u) {
                        sl.sol_len = g;
                        for (uint32_t j = 0; j + 1u < g; ++j)
                            sl.sol[j] = (uint8_t)((n[WN_PATH + j / 6u] >> (5u * (j % 6u))) & 31u);
                        sl.sol[g - 1u] = (uint8_t)xm;
                    }
                } else if (!all_axes_tight(xc, budget)) {
                    const uint32_t allow = g < plen ? 1u << ((n[WN_PATH] >> (5u * g)) & 31u) : T.amask[xm + 1u];
                    todo = allow & ~axis_move_mask(excluded_axes(xc, budget));
                }
                gone = todo == 0u;
                keep = !gone;
            }
            uint32_t j = WARP_STACK;  // a free entry
#pragma unroll
            for (uint32_t i = 0; i < WARP_STACK; ++i)
                if (((mine >> (5u * i)) & 31u) == 31u) j = i;
            keep = keep && j < WARP_STACK;
            ns += __popc(__ballot_sync(FULL, keep));
            if (keep) {
                stash[64u * j + lane] = xc;
                stash[64u * j + 32u + lane] = xn | (xm << 6) | (todo << 11);
                mine ^= (budget ^ 31u) << (5u * j);
                atomicAdd(&refs[xn], 1u);
                if (sample) atomicAdd(&passed[budget + 1u], 1u);
                gone = true;
            }
            if (gone) {
                if (s1) ch[1].k = 7u;
                else ch[0].k = 7u;
            }
            __syncwarp();
        }

        if (held) ++iter;
        if (held && (iter & (P.don_period - 1u)) == 0u) {
            // One look at the words of others, a lane each: found elsewhere, or the host is stopping
            // (drop everything this warp holds); warps starving, and donations waiting.
            uint32_t look = 0;
            if (lane == 0u) look = *(volatile uint32_t*)&P.slots[slot].found;
            if (lane == 1u) look = ((volatile QueueState*)P.q)->yield;
            if (lane == 2u && P.don_cap) look = ((volatile QueueState*)P.q)->starving;
            if (lane == 3u && P.don_cap) look = (int)((volatile QueueState*)P.q)->don_count < (int)P.don_target;
            if (lane == 4u)
                look = P.don_min_prev == 0ull || *(volatile unsigned long long*)&P.slots[slot].iter_nodes[
                                                     bound - 1u < 24u ? bound - 1u : 23u] >= P.don_min_prev;
            look = __ballot_sync(FULL, look != 0u);
            if (handed[lane] >= 1u << 20) handed[lane] >>= 1, passed[lane] >>= 1;  // (counts of late)
            wide_at = __ballot_sync(FULL, handed[lane] < 16u ? lane >= WARP_WIDE : WARP_RATIO * passed[lane] >= handed[lane]);
            if (look & 3u) ns = spilled = 0, mine = NONE, head = tail, refs[lane] = 0u, dry = true, ch[0].k = ch[1].k = 7u;
            if ((look & 12u) == 4u && lane == 0u) ((volatile QueueState*)P.q)->starving = 0u;  // enough wait
            // DONATE while warps starve (the rule of search_phased.cuh): the last spilled node, else the
            // shallowest stashed child.  (Without the spilled ones a wide search ends on a few warps: the superflip on d4t
            // with base_plen 3 took 3.8 s, with them 2.7.)
            if ((look & 28u) == 28u && (ns > 1u || spilled)) {
                const uint32_t best = shallowest(), j = best & 7u, at = spilled - 1u;
                const uint32_t owner = spilled ? at & 31u : (best >> 3) & 31u;
                uint32_t give = 0;
                if (lane == owner) {
                    unsigned long long w1, w2, w3;
                    if (spilled) w1 = sw1[at >> 5], w2 = sw2[at >> 5], w3 = sw3[at >> 5];
                    else pack_entry(owner, j, w1, w2, w3);
                    const uint32_t hb = (uint32_t)w1 & 0x3FFFFFFFu, g = (uint32_t)(w1 >> 32) & 31u, budget = (uint32_t)(w1 >> 37) & 31u;
                    uint32_t hmax = 0;
#pragma unroll
                    for (int i = 0; i < 6; ++i) hmax = max(hmax, hget(hb, i));
                    if (g >= (uint32_t)(w1 >> 60) && budget >= hmax + P.don_min_depth) {
                        atomicAdd(&P.slots[slot].open, 1u);  // before the post: the count never runs short
                        w1 = (w1 & ~((31ull << 37) | (15ull << 60))) | ((unsigned long long)bound << 37);
                        give = post_donation(P, seed0 + iter, slot, w1, w2, w3);
                        if (!give) atomicSub(&P.slots[slot].open, 1u);
                        else if (!spilled) mine |= 31u << (5u * j), refs[stash[64u * j + 32u + lane] & 63u] -= 1u;
                    }
                }
                give = __shfl_sync(FULL, give, owner);
                if (spilled) spilled -= give;
                else ns -= give;
            }
        }

        const uint32_t idle0 = __ballot_sync(FULL, ch[0].k == 7u), idle1 = __ballot_sync(FULL, ch[1].k == 7u);
        const uint32_t n_idle = __popc(idle0) + __popc(idle1);
        const uint32_t probing = __popc(__ballot_sync(FULL, ch[0].k < 6u)) + __popc(__ballot_sync(FULL, ch[1].k < 6u));
        barren = probing ? 0u : barren + 1u;
        if (barren > WARP_BARREN) {  // (never reached: a warp that makes no probe has work to finish or polls)
            if (lane == 0) give_up(P, slot, held);
            break;
        }

        // OPEN up to five stashed children, the deepest first, when fewer children are queued than
        // there are places for: six lanes build a node's frames and queue its children.  A wide node
        // (more than one in WARP_RATIO of its children are to pass, by the counts of its budget) is
        // opened alone or last, and not again for some passes: its children take a pass per frame,
        // and more of them opened meanwhile would turn the search breadth-first and fill the stash.
        ++cool;
        const uint32_t supply = tail - head;
        const bool full = ns + spilled > WARP_FULL;
        if (ns && (supply < n_idle || !probing)) {
            uint32_t room = free_places();
            if (!probing && (!room || supply > WARP_QUEUE - 96u || full) && (!n_idle || !supply)) {
                // Nothing is on its way and nothing can be opened -- every place holds the parent of a
                // stashed or queued child, or the queue is full and no lane with a passed child has a
                // free entry, or see WARP_FULL: the shallowest ones go to the spill list.
                for (uint32_t i = 0; i < 16u && ns; ++i) {
                    const uint32_t best = shallowest(), owner = (best >> 3) & 31u, j = best & 7u;
                    if (spilled < 32u * WARP_SPILL) {
                        if (lane == (spilled & 31u)) pack_entry(owner, j, sw1[spilled >> 5], sw2[spilled >> 5], sw3[spilled >> 5]);
                        ++spilled;
                    } else if (lane == 0) {  // the subtree is dropped: this iteration cannot prove its bound
                        atomicOr(&P.q->error, ERR_STACK);
                        atomicCAS(&P.slots[slot].found, 0u, FOUND_FAILED);
                    }
                    if (lane == owner) mine |= 31u << (5u * j), refs[stash[64u * j + 32u + lane] & 63u] -= 1u;
                    --ns;
                    __syncwarp();
                }
                room = free_places();
            }
            const bool open_wide = (cool >= WARP_COOL && supply < 64u) || (!supply && probing < 32u) || !probing;
            const uint32_t most = supply > WARP_QUEUE - 96u || full ? 0u : min((uint32_t)__popc(room), 5u);
            const uint32_t best = deepest(), level = best >> 3;
            const bool wide = level == 31u || ((wide_at >> level) & 1u);
            const uint32_t low = __reduce_min_sync(FULL, wide ? 31u : level);  // deepest narrow one
            uint32_t take = __ballot_sync(FULL, !wide && level <= low + 1u);
            if ((uint32_t)__popc(take) < most) take = __ballot_sync(FULL, !wide);
            uint32_t cnt = 0, from = 0, to = 0;
#pragma unroll
            for (uint32_t i = 0; i < 5; ++i)
                if (i < most && take) {  // (from a lane that moves on with the passes: no stash stays full)
                    const uint32_t l = (__ffs(__funnelshift_r(take, take, iter)) - 1u + iter) & 31u;
                    if (team == i) from = l, to = __ffs(room) - 1u;
                    if (lane == l) mine |= 31u << (5u * (best & 7u));
                    take &= ~(1u << l);
                    room &= room - 1u;
                    ++cnt;
                }
            if (cnt < most && open_wide) {
                const uint32_t at = __reduce_min_sync(FULL, wide ? level : 31u);
                if (at != 31u) {
                    const uint32_t l = __ffs(__ballot_sync(FULL, wide && level == at)) - 1u;
                    if (team == cnt) from = l, to = __ffs(room) - 1u;
                    if (lane == l) mine |= 31u << (5u * (best & 7u));
                    ++cnt;
                    cool = 0u;
                }
            }
            const uint32_t entry = __shfl_sync(FULL, best, from) & 7u;
            uint32_t todo = 0, h = 0, budget = 0;
            if (team < cnt) {
                const uint32_t e1 = stash[64u * entry + 32u + from], mv = (e1 >> 6) & 31u;
                const uint32_t* a = pool + (e1 & 63u) * WN_STRIDE;
                uint32_t* b = pool + to * WN_STRIDE;
                set_node_frame(b, tk, warp_step(T, node_frame(a, tk), tk, mv));
                const uint32_t meta = a[WN_META], g = (meta >> 8) & 255u;
                todo = e1 >> 11;
                h = stash[64u * entry + from];
                budget = (meta & 255u) - 1u;
                if (tk < 4u) {
                    uint32_t w = a[WN_PATH + tk];
                    if (tk == g / 6u && g >= (meta >> 16)) w |= mv << (5u * (g % 6u));
                    b[WN_PATH + tk] = w;
                } else if (tk == 4u) {
                    b[WN_H] = h;
                } else {
                    b[WN_META] = meta + 255u;  // one move deeper, one less to the bound
                    atomicSub(&refs[e1 & 63u], 1u);
                }
            }
            // frame order, a frame per lane: at the bound, one below, the rest
            const uint32_t v = hget(h, (int)tk);
            const uint32_t at_edge = (__ballot_sync(FULL, v >= budget) >> (6u * team)) & 63u;
            const uint32_t below_it = (__ballot_sync(FULL, v + 1u == budget) >> (6u * team)) & 63u;
            // queue the children (a lane those of its face): a team's start is the number of children of
            // the teams before it
            const uint32_t kids = __popc(todo);
            uint32_t start = tail, all = 0;
#pragma unroll
            for (uint32_t i = 0; i < 5; ++i) {
                const uint32_t x = __shfl_sync(FULL, kids, 6u * i);
                if (i < team) start += x;
                all += x;
            }
            const uint32_t entry_of = to | ((tk % 3u) << 11);
#pragma unroll
            for (uint32_t i = 0; i < 3; ++i) {
                const uint32_t mv = 3u * tk + i;
                if (team < 5u && ((todo >> mv) & 1u))
                    queue[(start + __popc(todo & ((1u << mv) - 1u))) % WARP_QUEUE] = (uint16_t)(entry_of | (mv << 6));
            }
            if (tk == 0u && team < cnt) {
                pool[to * WN_STRIDE + WN_ORD] = at_edge | (below_it << 6) | ((~(at_edge | below_it) & 63u) << 12) | ((budget - 1u) << 18);
            }
            tail += all;
            ns -= cnt;
            __syncwarp();
        }

        // REFILL: places without a child take the next queued ones.
        uint32_t left = n_idle;
        if (tail != head) {
            const uint32_t r[2] = {(uint32_t)__popc(idle0 & below), __popc(idle0) + (uint32_t)__popc(idle1 & below)};
            const uint32_t have = tail - head;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                if (ch[s].k == 7u && r[s] < have) {
                    const uint32_t e = queue[(head + r[s]) % WARP_QUEUE];
                    const uint32_t* n = pool + (e & 63u) * WN_STRIDE;
                    const uint32_t order = n[WN_ORD];
                    ch[s].node = e & 63u;
                    ch[s].m = (e >> 6) & 31u;
                    ch[s].c = n[WN_H];
                    ch[s].budget = order >> 18;
                    // (the inverse frame on the move's axis is in the parent's coset: same bound)
                    ch[s].rem = order & 0x3FFFFu & ~(0x41041u << (3u + (e >> 11)));
                    ch[s].k = (uint32_t)next_frame(ch[s].rem);
                    ++nodes;
                    if (sample) atomicAdd(&handed[ch[s].budget + 1u], 1u);
                }
            }
            const uint32_t take = min(n_idle, have);
            head += take;
            left -= take;
        }

        // More work for idle places: a spilled node, else the next item of the iteration, else (when
        // everything held is done) another iteration's item, a donated subtree or a new cube.
        if (left && !ns) {
            // (node to build: root frames and path, from a spilled node, a donation or an item)
            unsigned long long w1 = 0, w2 = 0, w3 = 0;
            uint32_t build = 0;
            const bool all_idle = left == 64u;
            if (spilled) {
                if ((!full || all_idle) && free_places()) {
                    const int l = (int)((spilled - 1u) & 31u), i = (int)((spilled - 1u) >> 5);
                    w1 = __shfl_sync(FULL, sw1[i], l);
                    w2 = __shfl_sync(FULL, sw2[i], l);
                    w3 = __shfl_sync(FULL, sw3[i], l);
                    build = 1;
                    const uint32_t kids = (uint32_t)(w1 >> 42) & 0x3FFFFu, rest = full ? kids & (kids - 1u) : 0u;
                    if (rest) {  // (its other children wait for this one's)
                        if (lane == (uint32_t)l) sw1[i] ^= (unsigned long long)(kids ^ rest) << 42;
                        w1 ^= (unsigned long long)rest << 42;
                    } else {
                        --spilled;
                    }
                }
            } else if (held && !dry && free_places()) {
                uint32_t idx = 0, plen = 0, ok = 0;
                if (lane == 0 && iter - iter0 < WARP_HOLD) {
                    const unsigned long long t = atomicAdd(&P.slots[slot].ticket, 1ull);
                    idx = (uint32_t)t;
                    plen = (uint32_t)(t >> 56);
                    ok = plen <= (uint32_t)MAX_PLEN && idx < P.n_prefix[plen];
                }
                ok = __shfl_sync(FULL, ok, 0);
                if (ok) {
                    idx = __shfl_sync(FULL, idx, 0);
                    plen = __shfl_sync(FULL, plen, 0);
                    ++held;
                    w1 = (unsigned long long)plen << 60 | ((unsigned long long)bound << 37);
                    w2 = plen ? __ldg(P.prefixes[plen] + idx) : 0u;
                    build = 2;
                } else {
                    dry = true;
                }
            }
            if (!build && all_idle && !spilled) {
                if (held) {  // FINISH
                    const unsigned long long ns = warp_sum(nodes), ps = warp_sum(probes);
                    nodes = probes = 0;
                    if (lane == 0) {
                        Slot& sl = P.slots[slot];
                        atomicAdd(&sl.nodes, ns);
                        atomicAdd(&sl.probes, ps);
                        atomicAdd(&sl.iter_nodes[bound < 24u ? bound : 23u], ns);
                        atomicAdd(&P.q->probes, ps);
                        __threadfence();
                        const bool final_unit = atomicSub(&sl.open, held) == held;
                        if (final_unit) {
                            __threadfence();
                            if (const uint32_t found = *(volatile uint32_t*)&sl.found) {
                                finish_slot(P, slot, found == FOUND_FAILED ? SLOT_ERROR : SLOT_SOLVED);
                            } else if (bound + 1u > MAX_BOUND) {
                                atomicOr(&P.q->error, ERR_BOUND);
                                finish_slot(P, slot, SLOT_ERROR);
                            } else {
                                const unsigned long long last = *(volatile unsigned long long*)&sl.iter_nodes[bound];
                                const uint32_t epoch = (uint32_t)(*(volatile unsigned long long*)&sl.ticket >> 32) & 0xFFFFu;
                                publish_epoch(P, slot, next_plen(P, last, bound + 1u), bound + 1u, epoch + 1u);
                            }
                        }
                    }
                    held = 0;
                    dry = true;
                }
                // FETCH
                uint32_t idx = 0, plen = 0, epoch = 0;
                int r = FETCH_EMPTY;
                if (lane == 0) {
                    const uint32_t seed = seed0 + (fetches++) * 0x2545F491u;
                    r = fetch_item(P, seed, slot, idx, plen, bound, epoch);
                    if (r == FETCH_EMPTY && P.don_cap && take_donation(P, seed, slot, w1, w2, w3)) r = 4;
                }
                r = __shfl_sync(FULL, r, 0);
                slot = __shfl_sync(FULL, slot, 0);
                if (r == FETCH_FINISHED) break;
                if (r == FETCH_ADMIT) {
                    admit_slot_warp<MODE, NEC, FMT>(T, P, slot, lane);
                    barren = 0;
                    continue;
                }
                if (r == FETCH_EMPTY) {
                    // Nothing queued: ask for donated subtrees, back off, leave after too many polls.
                    if (lane == 0 && P.don_cap && !*(volatile uint32_t*)&P.q->starving)
                        *(volatile uint32_t*)&P.q->starving = 1u;
                    if (++idle_polls > P.idle_limit) {
                        if (!P.persistent) {
                            if (lane == 0) atomicOr(&P.q->error, ERR_IDLE_LIMIT);
                            break;
                        }
                        if (__shfl_sync(FULL, (int)server_idle(P), 0)) break;
                        idle_polls = 0;
                    }
                    if ((idle_polls & 1023u) == 64u && lane == 0) requeue_stranded(P);
                    __syncwarp();
                    __nanosleep(backoff);
                    barren = 0;
                    backoff = backoff < 4096u ? backoff * 2u : 4096u;
                    continue;
                }
                idle_polls = 0;
                backoff = 32;
                barren = 0;
                const Slot& sl = P.slots[slot];
                const uint32_t found = __shfl_sync(FULL, *(const volatile uint32_t*)&sl.found, 0);
                second = __ldcg(&sl.table) != 0u;
                table = second ? P.table2 : P.table;
                held = 1;
                iter0 = iter;
                if (r == 4) {  // a donated subtree
                    w1 = __shfl_sync(FULL, w1, 0);
                    w2 = __shfl_sync(FULL, w2, 0);
                    w3 = __shfl_sync(FULL, w3, 0);
                    bound = (uint32_t)(w1 >> 37) & 31u;
                    const uint32_t g = (uint32_t)(w1 >> 32) & 31u;
                    if (g >= (uint32_t)MAX_DEPTH || bound > MAX_BOUND || g > bound) {
                        if (lane == 0) {  // a malformed cell (never written by a donor)
                            atomicOr(&P.q->error, ERR_STACK);
                            if (finish_unit(P, slot)) finish_slot(P, slot, SLOT_ERROR);
                        }
                        held = 0;
                        continue;
                    }
                    w1 = (w1 & ~(31ull << 37)) | ((unsigned long long)(bound - g) << 37);
                    dry = true;
                    build = 1;
                } else {
                    bound = __shfl_sync(FULL, bound, 0);
                    plen = __shfl_sync(FULL, plen, 0);
                    idx = __shfl_sync(FULL, idx, 0);
                    w1 = (unsigned long long)plen << 60 | ((unsigned long long)bound << 37);
                    w2 = plen ? __ldg(P.prefixes[plen] + idx) : 0u;
                    dry = false;
                    build = 2;
                }
                if (found) {  // solved by another unit: this one only counts as done ...
                    build = 0;
                    dry = true;
                    if (r == FETCH_OK) {  // ... and with it all items not handed out yet, up to 10 M of them
                        // (the iteration cannot end meanwhile, so its ticket is the one that was drawn from)
                        const uint32_t items = P.n_prefix[plen];
                        uint32_t next = items;
                        if (lane == 0) next = (uint32_t)atomicMax(&P.slots[slot].ticket, ticket_make(plen, bound, epoch) | items);
                        next = __shfl_sync(FULL, next, 0);
                        held += next < items ? items - next : 0u;
                    }
                }
            }
            if (build) {
                const uint32_t at = __ffs(free_places()) - 1u;
                uint32_t* n = pool + at * WN_STRIDE;
                const Slot& sl = P.slots[slot];
                const uint32_t plen = (uint32_t)(w1 >> 60), budget = (uint32_t)(w1 >> 37) & 31u;
                const uint32_t g = build == 2u ? 0u : (uint32_t)(w1 >> 32) & 31u;
                uint32_t todo = (uint32_t)(w1 >> 42) & 0x3FFFFu;
                const uint32_t h = build == 2u ? __ldcg(&sl.h0) : (uint32_t)w1 & 0x3FFFFFFFu;
                if (build == 2u)
                    todo = (plen ? 1u << ((uint32_t)w2 & 31u) : T.amask[0]) & ~axis_move_mask(excluded_axes(h, budget));
                if (lane < 6u) {
                    State t = slot_frame(sl, lane);
                    for (uint32_t j = 0; j < g; ++j)
                        t = warp_step(T, t, lane, (uint32_t)((j < 12u ? w2 : w3) >> (5u * (j % 12u))) & 31u);
                    set_node_frame(n, lane, t);
                } else if (lane < 10u) {
                    const uint32_t j = lane - 6u;
                    n[WN_PATH + j] = (uint32_t)((j < 2u ? w2 : w3) >> (30u * (j & 1u))) & 0x3FFFFFFFu;
                } else if (lane == 10u) {
                    n[WN_H] = h;
                    n[WN_META] = budget | (g << 8) | (plen << 16);
                    n[WN_ORD] = frame_order(h, budget) | ((budget - 1u) << 18);
                }
                const uint32_t kids = __popc(todo);
                if (lane < 18u && ((todo >> lane) & 1u))
                    queue[(tail + __popc(todo & below)) % WARP_QUEUE] = (uint16_t)(at | (lane << 6) | (((lane / 3u) % 3u) << 11));
                tail += kids;
                __syncwarp();
            }
        }

        // PROBE FEW: with no more children than teams, six lanes probe all remaining frames of a child at
        // once (one pass, where a child that passes takes up to six).  The passes of a near-empty warp are a
        // serial chain -- an item's walk, the end of an iteration, all of a short scramble's search.  Measured
        // on B200, d4t: a search of 6 to 12 moves 110 -> 70 us on the device, 16 and 100 cubes per call
        // within 1% either way (a warp with more children fills its lanes as it is).
        if (left >= 59u && tail == head) {
            const uint32_t live0 = __ballot_sync(FULL, ch[0].k < 6u), live1 = __ballot_sync(FULL, ch[1].k < 6u);
            uint32_t src = 0, from1 = 0, have = 0, l0 = live0, l1 = live1;
#pragma unroll
            for (uint32_t i = 0; i < 5; ++i) {
                const uint32_t l = l0 ? l0 : l1;
                if (team == i) src = l ? __ffs(l) - 1u : 0u, from1 = l0 == 0u, have = l != 0u;
                if (l0) l0 &= l0 - 1u;
                else l1 &= l1 - 1u;
            }
            uint32_t a[2];
#pragma unroll
            for (int s = 0; s < 2; ++s)
                a[s] = ch[s].node | (ch[s].m << 6) | (ch[s].budget << 11) |
                       (((ch[s].rem | (ch[s].rem >> 6) | (ch[s].rem >> 12) | (1u << ch[s].k)) & 63u) << 16);
            const uint32_t a0 = __shfl_sync(FULL, a[0], src), a1 = __shfl_sync(FULL, a[1], src);
            const uint32_t h0 = __shfl_sync(FULL, ch[0].c, src), h1 = __shfl_sync(FULL, ch[1].c, src);
            const uint32_t x = from1 ? a1 : a0, h = from1 ? h1 : h0, parent = hget(h, (int)tk);
            uint32_t v = parent;
            bool over = false;
            if (have && ((x >> (16u + tk)) & 1u)) {
                v = warp_probe<MODE, NEC, FMT>(T, P.classidx, table, warp_step(T, node_frame(pool + (x & 63u) * WN_STRIDE, tk), tk, (x >> 6) & 31u), second);
                if (tk < 3u && parent) v = max(v, parent - 1u);
                v = min(v, 31u);
                over = v > ((x >> 11) & 31u);
                ++probes;
            }
            const uint32_t out = __ballot_sync(FULL, over), part = v << (5u * tk);
            const uint32_t at[2] = {(uint32_t)__popc(live0 & below), (uint32_t)__popc(live0) + (uint32_t)__popc(live1 & below)};
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const uint32_t first = min(at[s], 4u) * 6u;
                uint32_t c = 0;
#pragma unroll
                for (uint32_t i = 0; i < 6; ++i) c |= __shfl_sync(FULL, part, first + i);
                if (ch[s].k < 6u) ch[s].c = c, ch[s].k = (out >> first) & 63u ? 7u : 6u;
            }
            continue;
        }

        // PROBE: the next frame of each lane's children.  The index arithmetic runs for every lane,
        // the table is read for the lanes with a child.
        uint32_t sector[2], entry[2], w[2][8];
        {
            State t[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const uint32_t kk = min(ch[s].k, 5u);
                t[s] = warp_step(T, node_frame(pool + ch[s].node * WN_STRIDE, kk), kk, ch[s].m);
            }
            uint32_t packed[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) packed[s] = __ldg(P.classidx + warp_corner_raw(T, t[s].c0, t[s].c1));
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                split_sector<FMT, KindTraits<MODE, NEC>::N_EDGE>(
                    packed[s] >> 4, warp_edge_coord<MODE, NEC>(T, t[s], packed[s] & 15u, second), sector[s], entry[s]);
                if (ch[s].k < 6u) {
                    load_sector(table + (uint64_t)sector[s] * 8u, w[s]);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[s][i] = 0u;
                }
            }
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            WarpChild& x = ch[s];
            uint32_t v = warp_decode<FMT>(w[s], entry[s]);
            if (x.k < 6u) {
                ++probes;
                const uint32_t parent = hget(x.c, (int)x.k);  // (c still holds the parent's value of this frame)
                if (x.k < 3u && parent) v = max(v, parent - 1u);  // a right move changes the coset distance by <= 1
                v = min(v, 31u);
                x.c = hset(x.c, (int)x.k, v);
                x.k = v > x.budget ? 7u : (uint32_t)next_frame(x.rem);  // pruned, next frame, or passed (6)
            }
        }
    }
}

}  // namespace ccs
