// Whole subtrees of the SAH build's seeds, a warp each: the kernels that
// phx_bvh_build_sah launches (sah.cu). They use nothing but warp operations, so a
// host build can run a warp's lanes as threads and hold them to the reference.
#pragma once

#include "sah_core.cuh"

namespace phx {
namespace {

using sah::TNode;

constexpr uint32_t SUB = 128;  // nodes under this many slots are seeds

// The most nodes a build of n slots opens above and with its seeds: only nodes of
// SUB slots or more open two others, those of a level share the slots out, and
// no more than MAX_DEPTH - 1 levels have them.
constexpr uint32_t open_nodes(uint32_t n) {
    const uint64_t all = 2ull * n - 1, some = 1 + 2ull * (sah::MAX_DEPTH - 1) * (n / SUB);
    return (uint32_t)(some < all ? some : all);
}

// Floats as words whose unsigned order is the floats' order (for atomic min
// and max; a NaN has no place among them and is left out).
__device__ __forceinline__ uint32_t ord(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unord(uint32_t w) {
    return __uint_as_float((w & 0x80000000u) ? (w & 0x7FFFFFFFu) : ~w);
}

// ---- whole subtrees of the seeds, a warp each ----
//
// A thread a node and a launch a level spent 2.9 of the 8.1 ms a 1.3 M-box
// build took: serial loops over scattered slots, 12 levels of them (now 1.7 in
// one launch, of a 4.9 ms build; seeds of 64 slots 1.5, with two more levels
// of blocks above them, 5.2). What bounds it now is instructions: about 400 a
// node and 54 a slot and node. Here a
// seed's boxes and centres are read once into shared memory and the subtree
// is built there, in the reference's depth-first order: each lane holds four
// slots, the planes of the three axes are priced by a lane each (a loop over
// the node's slots, every lane reading the same box), and the partition is
// the queue model by bit masks. Depth-first numbering makes a node's final
// index a function of the seed's rank. The nodes of a seed of n slots at
// `start` are records loc[2 start ..): (start, end, parent's inner rank * 2 +
// side or NONE, own inner rank or SUB_LEAF | depth << 8).
constexpr uint32_t SUB_WARPS = 4;
constexpr uint32_t SUB_LEAF = 255u;
constexpr uint32_t SUB_LANE = SUB / 32;  // positions a lane holds

struct SubShared {
    float c[3][SUB], lo[3][SUB], hi[3][SUB];
    uint32_t slot[SUB];
    uint32_t stack[SUB];  // start | end << 8 | depth << 16; the parent's rank beside it
    uint8_t rank_of[SUB];
    uint8_t idx[SUB];     // position -> the slot's place in the arrays above
    uint8_t bin[3][SUB];
    uint32_t lefts[SUB_LANE], before[SUB_LANE];  // the left slots' mask, lefts before each word
};

// Left slots before position x.
__device__ __forceinline__ uint32_t lefts_before(const SubShared& w, uint32_t x) {
    return w.before[x >> 5] + __popc(w.lefts[x >> 5] & ((1u << (x & 31u)) - 1u));
}

// Area of the box (lo, hi) (sah.rs:32-35).
__device__ __forceinline__ float area_of(const float* lo, const float* hi) {
    sah::Box b;
    for (int k = 0; k < 3; k++) {
        b.lo[k] = lo[k];
        b.hi[k] = hi[k];
    }
    return sah::area(b);
}

// A plane's two sides over positions j0, j0 + step, .. < j1: boxes and counts.
struct Sides {
    float llo[3], lhi[3], rlo[3], rhi[3];
    uint32_t lc, rc;
};

__device__ __forceinline__ Sides sides_of(const SubShared& w, uint32_t axis, uint32_t at, uint32_t j0, uint32_t j1,
                                          uint32_t step) {
    constexpr float BIGF = 3.402823466e38f;
    Sides s;
    for (int k = 0; k < 3; k++) {
        s.llo[k] = s.rlo[k] = BIGF;
        s.lhi[k] = s.rhi[k] = -BIGF;
    }
    s.lc = s.rc = 0;
    for (uint32_t j = j0; j < j1; j += step) {
        const uint32_t i = w.idx[j];
        const bool left = w.bin[axis][i] <= at;
        for (int k = 0; k < 3; k++) {
            const float lo = w.lo[k][i], hi = w.hi[k][i];
            s.llo[k] = fminf(s.llo[k], left ? lo : BIGF);
            s.lhi[k] = fmaxf(s.lhi[k], left ? hi : -BIGF);
            s.rlo[k] = fminf(s.rlo[k], left ? BIGF : lo);
            s.rhi[k] = fmaxf(s.rhi[k], left ? -BIGF : hi);
        }
        s.lc += left ? 1u : 0u;
        s.rc += left ? 0u : 1u;
    }
    return s;
}

// An axis's sweep (sweep_axis) from its planes' costs, plane `at` in lane
// first + at: the first plane with two sides if its cost is no number, else
// the lowest cost, the lower plane on a tie. Every lane calls.
__device__ __forceinline__ sah::AxisBest axis_best(bool priced, float cost, uint32_t first, uint32_t lane) {
    const bool mine = lane >= first && lane < first + 15u && priced;
    const uint32_t planes = __ballot_sync(0xffffffffu, mine);
    const float c0 = __shfl_sync(0xffffffffu, cost, planes ? __ffs(planes) - 1 : 0);
    if (!planes) return sah::AxisBest{false, 0.0f, 0u};
    if (c0 != c0) return sah::AxisBest{true, c0, (uint32_t)__ffs(planes) - 1u - first};
    // costs are sums of products of areas and counts: none is negative
    const uint32_t key = mine && cost == cost ? __float_as_uint(cost) : 0xFFFFFFFFu;
    const uint32_t low = __reduce_min_sync(0xffffffffu, key);
    const uint32_t who = __ballot_sync(0xffffffffu, key == low);
    return sah::AxisBest{true, __uint_as_float(low), (uint32_t)__ffs(who) - 1u - first};
}

__global__ void __launch_bounds__(32 * SUB_WARPS) k_sah_subtree(const uint32_t* __restrict__ seeds, uint32_t nseeds,
                                                                const TNode* __restrict__ tn,
                                                                const float* __restrict__ prims,
                                                                const float* __restrict__ centres, uint32_t* order,
                                                                uint32_t leaf, uint4* __restrict__ loc,
                                                                uint32_t* __restrict__ loc_count, uint32_t* inner,
                                                                uint32_t* max_depth, bool vec_prims) {
    __shared__ SubShared shared[SUB_WARPS];
    const uint32_t lane = threadIdx.x & 31u, k0 = blockIdx.x * SUB_WARPS + (threadIdx.x >> 5);
    if (k0 >= nseeds) return;
    SubShared& w = shared[threadIdx.x >> 5];
    const uint32_t t = seeds[k0];
    const TNode seed = tn[t];
    const uint32_t total = seed.end - seed.start;
    uint4* out = loc + 2 * (uint64_t)seed.start;
    if (seed.depth + 1 >= sah::MAX_DEPTH || total <= 1u) {
        if (lane == 0) {
            out[0] = make_uint4(seed.start, seed.end, sah::NONE, SUB_LEAF | seed.depth << 8);
            loc_count[k0] = 1u;
            inner[t] = 0u;
            atomicMax(max_depth, seed.depth);
        }
        return;
    }
    for (uint32_t j = lane; j < total; j += 32u) {
        const uint32_t i = order[seed.start + j];
        w.slot[j] = i;
        w.idx[j] = (uint8_t)j;
        if (vec_prims) {
            const float4 a = __ldg((const float4*)prims + 2 * (uint64_t)i), b = __ldg((const float4*)prims + 2 * (uint64_t)i + 1);
            w.lo[0][j] = a.x;
            w.lo[1][j] = a.y;
            w.lo[2][j] = a.z;
            w.hi[0][j] = b.x;
            w.hi[1][j] = b.y;
            w.hi[2][j] = b.z;
        } else {
            for (int k = 0; k < 3; k++) {
                w.lo[k][j] = __ldg(prims + 8 * (uint64_t)i + k);
                w.hi[k][j] = __ldg(prims + 8 * (uint64_t)i + 4 + k);
            }
        }
        for (int k = 0; k < 3; k++) w.c[k][j] = __ldg(centres + 3 * (uint64_t)i + k);
    }
    __syncwarp();
    uint32_t sp = 0, ninner = 0, nrec = 0, deepest = seed.depth;
    uint32_t s = 0, e = total, depth = seed.depth, code = sah::NONE;
    for (;;) {
        const uint32_t n = e - s;
        uint32_t m = sah::NONE;
        if (depth + 1 < sah::MAX_DEPTH && n > 1u) {
            // this lane's positions s + lane, s + 32 + lane, ..
            uint32_t mine[SUB_LANE];
            bool held[SUB_LANE];
            float lo[3], scale[3];
            sah::Box cbox;
#pragma unroll
            for (uint32_t q = 0; q < SUB_LANE; q++) {
                held[q] = q * 32u + lane < n;
                mine[q] = 0u;
                if (q * 32u < n && held[q]) mine[q] = w.idx[s + q * 32u + lane];  // (most nodes need one word)
            }
            for (int k = 0; k < 3; k++) {
                uint32_t l = ord(3.402823466e38f), h = ord(-3.402823466e38f);
#pragma unroll
                for (uint32_t q = 0; q < SUB_LANE; q++) {
                    if (q * 32u >= n) break;
                    const float c = w.c[k][mine[q]];
                    if (held[q] && c == c) {
                        l = min(l, ord(c));
                        h = max(h, ord(c));
                    }
                }
                cbox.lo[k] = unord(__reduce_min_sync(0xffffffffu, l));
                cbox.hi[k] = unord(__reduce_max_sync(0xffffffffu, h));
            }
            if (!sah::grid_of(cbox, lo, scale)) {
                if (n > leaf) m = n / 2u;
            } else {
#pragma unroll
                for (uint32_t q = 0; q < SUB_LANE; q++)
                    if (q * 32u < n && held[q]) {
                        const float c[3] = {w.c[0][mine[q]], w.c[1][mine[q]], w.c[2][mine[q]]};
                        for (int k = 0; k < 3; k++) w.bin[k][mine[q]] = (uint8_t)sah::bin_of(c, lo, scale, k);
                    }
                __syncwarp();
                // axes 0 and 1: a lane a plane; axis 2: two lanes a plane, each half the slots
                sah::AxisBest axes[3];
                sah::Box bounds;
                {
                    const uint32_t axis = lane < 15u ? 0u : 1u;
                    const Sides d = sides_of(w, axis, lane < 30u ? lane - 15u * axis : 0u, s, e, 1u);
                    const bool priced = d.lc != 0u && d.rc != 0u && (axis ? scale[1] : scale[0]) != 0.0f;
                    const float cost = area_of(d.llo, d.lhi) * (float)d.lc + area_of(d.rlo, d.rhi) * (float)d.rc;
                    axes[0] = axis_best(priced, cost, 0u, lane);
                    axes[1] = axis_best(priced, cost, 15u, lane);
                    for (int k = 0; k < 3; k++) {
                        bounds.lo[k] = fminf(d.llo[k], d.rlo[k]);
                        bounds.hi[k] = fmaxf(d.lhi[k], d.rhi[k]);
                    }
                }
                {
                    Sides d = sides_of(w, 2u, lane & 15u, s + (lane >> 4), e, 2u);
                    for (int k = 0; k < 3; k++) {
                        d.llo[k] = fminf(d.llo[k], __shfl_xor_sync(0xffffffffu, d.llo[k], 16));
                        d.lhi[k] = fmaxf(d.lhi[k], __shfl_xor_sync(0xffffffffu, d.lhi[k], 16));
                        d.rlo[k] = fminf(d.rlo[k], __shfl_xor_sync(0xffffffffu, d.rlo[k], 16));
                        d.rhi[k] = fmaxf(d.rhi[k], __shfl_xor_sync(0xffffffffu, d.rhi[k], 16));
                    }
                    d.lc += __shfl_xor_sync(0xffffffffu, d.lc, 16);
                    d.rc += __shfl_xor_sync(0xffffffffu, d.rc, 16);
                    const bool priced = d.lc != 0u && d.rc != 0u && scale[2] != 0.0f;
                    const float cost = area_of(d.llo, d.lhi) * (float)d.lc + area_of(d.rlo, d.rhi) * (float)d.rc;
                    axes[2] = axis_best(priced, cost, 0u, lane);
                }
                const sah::Decision cut = sah::decide_from(axes, scale, bounds, n, leaf);
                if (cut.cut == sah::CUT_HALF) m = n / 2u;
                if (cut.cut == sah::CUT_PLANE) {
                    uint32_t count = 0;
#pragma unroll
                    for (uint32_t q = 0; q < SUB_LANE; q++) {
                        if (q * 32u >= n) break;
                        const uint32_t word =
                            __ballot_sync(0xffffffffu, held[q] && w.bin[cut.axis][mine[q]] <= cut.at);
                        if (lane == 0) {
                            w.lefts[q] = word;
                            w.before[q] = count;
                        }
                        count += __popc(word);
                    }
                    __syncwarp();
                    if (count == 0u || count == n) {
                        m = n / 2u;  // no left slot or no right one: the swap loop moved nothing
                    } else {
                        m = count;
                        uint8_t put[SUB_LANE];
#pragma unroll
                        for (uint32_t q = 0; q < SUB_LANE; q++) {
                            // position x of the result: the x-th left slot, or (with
                            // the log shifted by the first right slot) entry x,
                            // chased to the slot it carries
                            const uint32_t x = q * 32u + lane;
                            put[q] = 0;
                            if (q * 32u >= n) break;
                            if (x >= n || x < m) continue;
                            uint32_t j = x;
                            while ((w.lefts[j >> 5] >> (j & 31u)) & 1u) j = lefts_before(w, j);
                            put[q] = w.idx[s + j];
                        }
                        __syncwarp();
#pragma unroll
                        for (uint32_t q = 0; q < SUB_LANE; q++) {
                            const uint32_t x = q * 32u + lane;
                            if (q * 32u >= n) break;
                            if (x < n && x >= m) w.idx[s + x] = put[q];
                            if (held[q] && ((w.lefts[q] >> lane) & 1u)) w.idx[s + lefts_before(w, x)] = (uint8_t)mine[q];
                        }
                        __syncwarp();
                    }
                }
            }
        }
        deepest = max(deepest, depth);
        if (lane == 0)
            out[nrec] = make_uint4(seed.start + s, seed.start + e, code, (m == sah::NONE ? SUB_LEAF : ninner) | depth << 8);
        nrec++;
        if (m != sah::NONE) {
            if (lane == 0) {
                w.stack[sp] = (s + m) | e << 8 | (depth + 1u) << 16;
                w.rank_of[sp] = (uint8_t)ninner;
            }
            sp++;
            code = ninner * 2u;
            ninner++;
            e = s + m;
            depth++;
            continue;
        }
        if (sp == 0u) break;
        sp--;
        __syncwarp();
        const uint32_t top = w.stack[sp];
        code = (uint32_t)w.rank_of[sp] * 2u + 1u;
        s = top & 255u;
        e = (top >> 8) & 255u;
        depth = top >> 16;
        __syncwarp();
    }
    for (uint32_t j = lane; j < total; j += 32u) order[seed.start + j] = w.slot[w.idx[j]];
    if (lane == 0) {
        loc_count[k0] = nrec;
        inner[t] = ninner;
        atomicMax(max_depth, deepest);
    }
}

// The seeds' nodes at their final indices, with their bounds: leaves from
// their primitives in slot order, inner nodes from their children, deepest
// first (sah_core.cuh emit).
__global__ void __launch_bounds__(32 * SUB_WARPS) k_sah_subtree_emit(
    const uint32_t* __restrict__ seeds, uint32_t nseeds, const TNode* __restrict__ tn, const uint4* __restrict__ loc,
    const uint32_t* __restrict__ loc_count, const uint32_t* __restrict__ rank, const uint32_t* __restrict__ final_index,
    const float* __restrict__ prims, const uint32_t* __restrict__ order, sah::Box* boxes, float* nodes,
    bool vec_nodes) {
    __shared__ float s_box[SUB_WARPS][6][2 * SUB];  // 24 KB
    __shared__ uint8_t s_child[SUB_WARPS][2 * SUB];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, k0 = blockIdx.x * SUB_WARPS + warp;
    if (k0 >= nseeds) return;
    float(*box)[2 * SUB] = s_box[warp];
    uint8_t* child = s_child[warp];
    const uint32_t t = seeds[k0], count = loc_count[k0], R = rank[t];
    const uint4* rec = loc + 2 * (uint64_t)tn[t].start;
    uint4 mine[2 * SUB_LANE];
    uint32_t low = sah::MAX_DEPTH, high = 0;
#pragma unroll
    for (uint32_t q = 0; q < 2u * SUB_LANE; q++) {
        const uint32_t k = q * 32u + lane;
        if (k >= count) continue;
        mine[q] = rec[k];
        if (mine[q].z != sah::NONE) child[mine[q].z] = (uint8_t)k;
        if ((mine[q].w & 255u) == SUB_LEAF) {
            sah::Box b = sah::empty_box();
            for (uint32_t j = mine[q].x; j < mine[q].y; j++) sah::grow(b, sah::prim_box(prims + 8 * (uint64_t)order[j]));
            for (int f = 0; f < 3; f++) {
                box[f][k] = b.lo[f];
                box[3 + f][k] = b.hi[f];
            }
        } else {
            low = min(low, mine[q].w >> 8);
            high = max(high, mine[q].w >> 8);
        }
    }
    low = __reduce_min_sync(0xffffffffu, low);
    high = __reduce_max_sync(0xffffffffu, high);
    __syncwarp();
    for (uint32_t d = high; d + 1u > low; d--) {
#pragma unroll
        for (uint32_t q = 0; q < 2u * SUB_LANE; q++) {
            const uint32_t k = q * 32u + lane;
            if (k >= count || (mine[q].w & 255u) == SUB_LEAF || mine[q].w >> 8 != d) continue;
            const uint32_t r = mine[q].w & 255u, l = child[2 * r], h = child[2 * r + 1];
            for (int f = 0; f < 3; f++) {
                box[f][k] = sah::rmin(box[f][l], box[f][h]);
                box[3 + f][k] = sah::rmax(box[3 + f][l], box[3 + f][h]);
            }
        }
        __syncwarp();
        if (d == 0u) break;
    }
#pragma unroll
    for (uint32_t q = 0; q < 2u * SUB_LANE; q++) {
        const uint32_t k = q * 32u + lane;
        if (k >= count) continue;
        const uint32_t code = mine[q].z, r = mine[q].w & 255u;
        const uint32_t at = code == sah::NONE ? final_index[t] : 2u * (R + (code >> 1)) + 1u + (code & 1u);
        const bool is_leaf = r == SUB_LEAF;
        const uint32_t lo_i = is_leaf ? mine[q].x | sah::LEAF_BIT : 2u * (R + r) + 1u;
        const uint32_t hi_i = is_leaf ? mine[q].y : 2u * (R + r) + 2u;
        if (vec_nodes) {
            float4* o = (float4*)nodes + 2 * (uint64_t)at;
            o[0] = make_float4(box[0][k], box[1][k], box[2][k], __uint_as_float(lo_i));
            o[1] = make_float4(box[3][k], box[4][k], box[5][k], __uint_as_float(hi_i));
        } else {
            float* o = nodes + 8 * (uint64_t)at;
            for (int f = 0; f < 3; f++) {
                o[f] = box[f][k];
                o[4 + f] = box[3 + f][k];
            }
            o[3] = __uint_as_float(lo_i);
            o[7] = __uint_as_float(hi_i);
        }
        if (code == sah::NONE) {
            sah::Box b;
            for (int f = 0; f < 3; f++) {
                b.lo[f] = box[f][k];
                b.hi[f] = box[3 + f][k];
            }
            boxes[t] = b;
        }
    }
}

}  // namespace
}  // namespace phx
