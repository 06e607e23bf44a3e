// The LBVH build's device arrays and the enqueue functions that run it
// (bvh.cu), shared with the tracer, which builds its tree over face boxes.
#pragma once

#include <cfloat>

#include "internal.cuh"

namespace phx {

constexpr int LBVH_TILE = 4096;  // radix-sort tile (256 threads x 16 keys)
constexpr int LBVH_PASSES = 4;   // 8-bit digits over the 30-bit Morton code

// A device-side switch on a launch: the kernel does its work only when
// *word == want (word NULL: always). A captured CUDA graph can then hold
// both a rebuild and a refit and choose per replay by one word in device
// memory, which every gated kernel reads before doing anything else.
struct Gate {
    const uint32_t* word = nullptr;
    uint32_t want = 0;
#ifdef __CUDACC__
    __device__ __forceinline__ bool off() const { return word != nullptr && *word != want; }
#endif
};

#ifdef __CUDACC__
// Decoupled look-back words of the radix sort: a tile's count for one digit
// with a flag — its own count only (AGG) or the inclusive prefix (INC).
constexpr uint32_t LOOKBACK_AGG = 1u << 30;
constexpr uint32_t LOOKBACK_INC = 2u << 30;
constexpr uint32_t LOOKBACK_VALUE = (1u << 30) - 1;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The exclusive prefix of digit d for tile `tile` (> 0): walks back over
// the earlier tiles' words (256 per tile), adding aggregates until an
// inclusive prefix. A word not yet written is polled again, at most `limit`
// times in all; past that the wait gives up, sets STATUS_SPIN_LIMIT in
// *status and returns what it has (the caller's result is then wrong and the
// host reports the status instead of it).
__device__ __forceinline__ uint32_t lookback_prefix(const uint32_t* lookback, uint32_t tile, uint32_t d,
                                                    uint32_t limit, uint32_t* status) {
    uint32_t prefix = 0, spins = 0;
    int t = (int)tile - 1;
    while (t >= 0) {
        const uint32_t v = ld_relaxed(lookback + (size_t)t * 256 + d);
        const uint32_t flag = v & ~LOOKBACK_VALUE;
        if (flag == 0) {
            if (++spins > limit) {
                atomicOr(status, STATUS_SPIN_LIMIT);
                break;
            }
            if (spins > 32) __nanosleep(64);
            continue;
        }
        prefix += v & LOOKBACK_VALUE;
        if (flag == LOOKBACK_INC) break;
        t--;
    }
    return prefix;
}

// The climb of the atomic bottom-up refit (Bvh::refit's bounds, build.rs:
// 180-194) from node i, whose box (lx .. hz) is already stored: at each
// parent the first arriving child stops and the second unions its box with
// its sibling's (left box first) and carries on up. counters[] start even
// and every reachable inner node gets exactly two arrivals, so they need no
// reset between refits. A climb longer than any Karras tree (65 levels)
// means a corrupt parent array: STATUS_BAD_INDEX, and the climb stops.
__device__ __forceinline__ void refit_climb(uint32_t i, float lx, float ly, float lz, float hx, float hy, float hz,
                                            const uint32_t* __restrict__ parent, float4* nodes, uint32_t* counters,
                                            uint32_t* status) {
    uint32_t p = __ldg(parent + i);
    for (int hops = 0; i != 0; hops++) {
        if (hops > 80) {
            atomicOr(status, STATUS_BAD_INDEX);
            return;
        }
        // p's child links and parent (fixed during a refit) are read before the
        // arrival count, so the sibling is known when the count returns
        const uint32_t above = __ldg(parent + p);
        const uint32_t l = __ldcg((const uint32_t*)(nodes + 2 * (size_t)p) + 3);
        const uint32_t r = __ldcg((const uint32_t*)(nodes + 2 * (size_t)p + 1) + 3);
        // the count releases this box and acquires the sibling's
        uint32_t old;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(counters + p) : "memory");
        if ((old & 1u) == 0) return;  // first child here: the sibling finishes p
        const bool is_left = (l == i);
        const uint32_t sib = is_left ? r : l;
        const float4 sa = __ldcg(nodes + 2 * (size_t)sib), sb = __ldcg(nodes + 2 * (size_t)sib + 1);
        if (is_left) {
            lx = fminf(lx, sa.x);
            ly = fminf(ly, sa.y);
            lz = fminf(lz, sa.z);
            hx = fmaxf(hx, sb.x);
            hy = fmaxf(hy, sb.y);
            hz = fmaxf(hz, sb.z);
        } else {
            lx = fminf(sa.x, lx);
            ly = fminf(sa.y, ly);
            lz = fminf(sa.z, lz);
            hx = fmaxf(sb.x, hx);
            hy = fmaxf(sb.y, hy);
            hz = fmaxf(sb.z, hz);
        }
        nodes[2 * (size_t)p] = make_float4(lx, ly, lz, __uint_as_float(l));
        nodes[2 * (size_t)p + 1] = make_float4(hx, hy, hz, __uint_as_float(r));
        i = p;
        p = above;
    }
}

// A block's part of the refit: the leaves and the subtrees that lie wholly in
// its REFIT_SLOTS sorted slots, in shared memory.
//
// A Karras node's id is one end of the slots it covers, so the inner nodes
// [s0, s0 + REFIT_SLOTS) include every node whose leaves are all in the
// block's slots, and one thread a slot and inner node loads and stores them in
// order. The subtrees rise in rounds: a node whose children were made in
// earlier rounds takes the union of their boxes (one barrier a round, `stamp`
// holds the round). What has no parent made here climbs through memory as
// refit_climb does. A climb from every leaf had two atomics, two fences and
// three dependent reads a node, all through L2: 89 us at 1M boxes, 137 at 2M
// and 21 of latency at 1,000; now 70, 114 and 16. The smallest bytes are the
// boxes, the inner nodes' links and all the nodes written, 0.14 GB at 1M or 22
// us; what keeps it from that is the climbs' chain (29 us), shared memory's
// pipe and the rounds' barriers. A box is one 16- and one 8-byte word there: six
// words of 4 took 45 us at 1M without the climbs, this takes 41. With the six
// words: blocks of 256 slots 41 + 30 us at 1M, 83 + 43 at 2M. Steps of a warp
// alone between barriers cost more than the barriers: two 47, four 56, six 65.
//
// `slot(s, last, write)` gives slot s's box; write: also what goes with the
// slot (once a slot), last: the slot ends its leaf. owner[s]: the leaf (an
// inner node cut short or a leaf node) that begins at slot s, or NO_OWNER.
struct RefitBox {
    float lx, ly, lz, hx, hy, hz;
};

__device__ __forceinline__ void grow(RefitBox& a, const RefitBox& b) {
    a.lx = fminf(a.lx, b.lx);
    a.ly = fminf(a.ly, b.ly);
    a.lz = fminf(a.lz, b.lz);
    a.hx = fmaxf(a.hx, b.hx);
    a.hy = fmaxf(a.hy, b.hy);
    a.hz = fmaxf(a.hz, b.hz);
}

constexpr int REFIT_SLOTS = 512;  // threads of a refit block too
constexpr uint32_t NO_OWNER = 0xFFFFFFFFu;

// Nodes a block leaves to climb from: each has a parent that crosses one of
// the block's two edges, at most one a depth and edge (32 depths, the root's
// not counted), and a leaf across the end.
constexpr int REFIT_OPEN = 64;

// From this many slots on (more blocks than the chip holds at once) the climbs
// are left to a launch of their own: a block that climbed stayed on its SM for
// the climb's latency (about 1.3 us a level, some twenty levels) and kept the
// next from starting, 88 us against 45 + 29 at 1M boxes. Below, all blocks are
// resident and the second launch would only add its own latency.
constexpr uint32_t REFIT_LIST_MIN = 1u << 18;

__device__ __forceinline__ void refit_climb_from(uint32_t id, const uint32_t* __restrict__ parent, float4* nodes,
                                                 uint32_t* counters, uint32_t* status) {
    const float4 a = __ldcg(nodes + 2 * (size_t)id), b = __ldcg(nodes + 2 * (size_t)id + 1);
    refit_climb(id, a.x, a.y, a.z, b.x, b.y, b.z, parent, nodes, counters, status);
}

template <class Slot>
__device__ __forceinline__ void refit_block(uint32_t n, const uint32_t* __restrict__ owner,
                                            const uint32_t* __restrict__ parent, float4* nodes, uint32_t* counters,
                                            uint32_t* status, uint32_t* list, const Slot& slot) {
    constexpr uint32_t SB = REFIT_SLOTS, CUT = 0x80000000u;  // CUT: a record's leaf bit
    __shared__ float4 box4[2 * SB];         // lx ly lz hx of inner nodes, then of leaf nodes
    __shared__ float2 box2[2 * SB];         // hy hz
    __shared__ uint8_t stamp[2 * SB];       // the round a node was made in; 0: not here
    __shared__ uint8_t taken[2 * SB];       // its parent was made here
    __shared__ uint32_t open[REFIT_OPEN], nopen;  // the nodes to climb from
    const uint32_t t = threadIdx.x, s0 = blockIdx.x * SB, s = s0 + t;
    const uint32_t first_leaf = n - 1;      // node ids below are inner nodes
    auto put = [&](uint32_t k, const RefitBox& b) {
        box4[k] = make_float4(b.lx, b.ly, b.lz, b.hx);
        box2[k] = make_float2(b.hy, b.hz);
    };
    auto get = [&](uint32_t k) {
        const float4 a = box4[k];
        const float2 b = box2[k];
        return RefitBox{a.x, a.y, a.z, a.w, b.x, b.y};
    };
    auto store = [&](uint32_t id, const RefitBox& b, uint32_t lo, uint32_t hi) {
        nodes[2 * (size_t)id] = make_float4(b.lx, b.ly, b.lz, __uint_as_float(lo));
        nodes[2 * (size_t)id + 1] = make_float4(b.hx, b.hy, b.hz, __uint_as_float(hi));
    };

    uint32_t own = NO_OWNER, lo = CUT, hi = 0;
    RefitBox mine{FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
    if (s < n) {
        own = __ldg(owner + s);
        const bool last = s + 1 == n || __ldg(owner + s + 1) != NO_OWNER;
        if (s < first_leaf) {
            lo = __ldcg((const uint32_t*)(nodes + 2 * (size_t)s) + 3);
            hi = __ldcg((const uint32_t*)(nodes + 2 * (size_t)s + 1) + 3);
        }
        grow(mine, slot(s, last, true));
        put(SB + t, mine);
    }
    const bool leaf_node = own != NO_OWNER && own >= first_leaf;
    if (t == 0) nopen = 0;
    if (t < REFIT_OPEN) open[t] = NO_OWNER;
    stamp[t] = 0;
    taken[t] = 0;
    stamp[SB + t] = leaf_node ? 1 : 0;
    taken[SB + t] = 0;
    __syncthreads();
    bool far = false;  // the leaf's record is another block's inner node
    if (own != NO_OWNER && !leaf_node) {
        const uint32_t end = __ldcg((const uint32_t*)(nodes + 2 * (size_t)own + 1) + 3);
        for (uint32_t k = s + 1; k < end; k++)
            grow(mine, k < s0 + SB ? get(SB + (k - s0)) : slot(k, false, false));
        far = own - s0 >= SB;
        if (far) {
            store(own, mine, s | CUT, end);
        } else {
            put(own - s0, mine);
            stamp[own - s0] = 1;
        }
    }
    __syncthreads();

    // this thread's inner node, of two children here
    auto here = [&](uint32_t c) {
        if (c >= first_leaf) {
            const uint32_t k = c - first_leaf - s0;
            return k < SB ? SB + k : 2 * SB;
        }
        return c - s0 < SB ? c - s0 : 2 * SB;
    };
    bool pending = false;
    uint32_t l = 0, r = 0;
    if (!(lo & CUT)) {
        l = here(lo);
        r = here(hi);
        pending = l < 2 * SB && r < 2 * SB;
    }
    for (uint32_t round = 2; round < 255; round++) {
        const uint32_t a = pending ? stamp[l] : 0u, b = pending ? stamp[r] : 0u;
        const bool ready = a != 0 && b != 0 && a < round && b < round;
        if (ready) {
            RefitBox m = get(l);
            grow(m, get(r));
            put(t, m);
            stamp[t] = (uint8_t)round;
            taken[l] = 1;
            taken[r] = 1;
            pending = false;
        }
        if (!__syncthreads_or(ready)) break;
    }

    auto climb_from = [&](uint32_t id) {
        const uint32_t k = atomicAdd(&nopen, 1u);
        if (k < REFIT_OPEN) open[k] = id;
        else atomicOr(status, STATUS_BAD_INDEX);
    };
    if (stamp[t]) {
        store(s, get(t), lo, hi);
        if (!taken[t]) climb_from(s);
    }
    if (leaf_node) {
        store(own, mine, s | CUT, s + 1);
        if (!taken[SB + t]) climb_from(own);
    }
    if (far) climb_from(own);
    __syncthreads();
    if (t >= REFIT_OPEN) return;
    if (list) list[blockIdx.x * REFIT_OPEN + t] = open[t];
    else if (open[t] != NO_OWNER) refit_climb_from(open[t], parent, nodes, counters, status);
}
#endif

struct BvhWork {
    uint32_t cap = 0;  // prims the arrays hold
    DevMem prims, codes, sorted, order, alt_keys, alt_vals, partial, zeroed, links, parent, nodes, starts, counters,
        scalars, scene;
    uint32_t tiles = 0, nparts = 0;

    int32_t reserve(uint32_t n, int sms);
    // [hist 4*256][tickets 4][pad to 16][look-back 4 * tiles * 256]
    size_t zeroed_bytes() const { return (size_t)(LBVH_PASSES * 256 + 16) * 4 + (size_t)LBVH_PASSES * tiles * 256 * 4; }
    uint32_t* hist() const { return (uint32_t*)zeroed.ptr; }
    uint32_t* tickets() const { return (uint32_t*)zeroed.ptr + LBVH_PASSES * 256; }
    uint32_t* lookback(int pass) const {
        return (uint32_t*)zeroed.ptr + LBVH_PASSES * 256 + 16 + (size_t)pass * tiles * 256;
    }
    uint32_t* depth() const { return (uint32_t*)scalars.ptr; }
    uint32_t* nstarts() const { return (uint32_t*)scalars.ptr + 1; }
    // The list for the climbs of a large refit (refit_block), else none.
    uint32_t* climbs(uint32_t n) const { return n >= REFIT_LIST_MIN ? (uint32_t*)alt_keys.ptr : nullptr; }
    uint32_t* owner() const { return (uint32_t*)codes.ptr; }  // refit_block's; the codes are sorted out of here by then
};

// The stable radix sort of `codes` over caller-provided work arrays (see
// bvh.cu): order and sorted codes out. Stream-ordered; no allocation.
int32_t enqueue_sort_raw(Ctx* c, const uint32_t* codes, uint32_t n, uint32_t* order, uint32_t* sorted,
                         uint32_t* alt_keys, uint32_t* alt_vals, uint32_t* hist, uint32_t* tickets, uint32_t* lookback,
                         uint32_t stride);

// Every stage of Bvh::build over w.prims[0..n) on the context's stream;
// refit = false leaves out the last one, the bounds (the caller runs a
// refit of its own, which must climb as refit_climb does).
int32_t enqueue_build(Ctx* c, BvhWork& w, uint32_t n, uint32_t leaf, Gate gate = Gate{}, bool refit = true);
// The climbs a large refit_block left in w.climbs(n).
int32_t enqueue_climbs(Ctx* c, BvhWork& w, uint32_t n, Gate gate = Gate{});
// Bvh::refit (slots = false: prims through order; true: prims already in
// slot order, Bvh::refit_slots).
int32_t enqueue_refit(Ctx* c, BvhWork& w, uint32_t n, bool slots, Gate gate = Gate{});

}  // namespace phx
