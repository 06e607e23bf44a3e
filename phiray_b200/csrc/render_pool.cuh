// The pooled render: each block keeps a pool of sample paths and alternates
// between tracing all of its paths' rays and shading all of its paths' hits.
//
// What bounds the megakernel is divergence and instruction fetch: a lane owns
// a pixel, the paths of a warp's 32 pixels end at different bounces and take
// different lobes, and the warps of an SM run different parts of a long code
// (on the 1.3 M-face mesh 9.7 of 32 lanes were active in an instruction, and
// waiting for instructions was the largest stall). Here a path's state sits
// in memory (PW_WORDS words in the pool of its block), so
// lanes are not bound to paths: in the trace phase they take the next ray of
// the block's list as soon as theirs is done, and the shading phase runs each
// kind of hit over the slots that hold it, 32 at a time. A block's warps run
// the same phase at the same time, so they fetch the same code. Samples of
// one pixel are separate paths, so a small frame of many samples fills the
// chip too. One launch, no grid barrier, no host round trip.
//
// Measured (B200, against the fastest megakernel form): the 1.3 M-face mesh at
// 1080p, 16 spp, 8 bounces on its SAH tree 48.7 -> 27.8 ms (2.72 Grays/s);
// the 65,536-face cloud at 256 x 256, 16 spp on its LBVH 26.5 -> 4.9 ms.
// What is left (that mesh at 960 x 540, 4 spp, one launch): 52 % of issue slots
// used, 17 of 32 lanes active, the rest waiting on memory past L1 (tree,
// triangles, path state; 5.2 of 14.7 cycles an instruction) and at the phases'
// barriers (2.7). A large frame's pools, 296 MB, go through DRAM: 1.1 TB/s.
// At many samples blocks of 512 threads, two an SM, beat 256 x 4 and 128 x 8
// (27.8 against 28.6 and 31.5 ms at 16 spp; 2.71, 2.67 and 2.83 at 1) and 1,024 x
// 1 (31.7): more warps in one phase, but two phases an SM to overlap; 64
// registers beat 80 (31.8, 768 threads an SM) and 40 (34.4). Frames of few
// samples take 256 (rules.cuh). A warp-sized pool (64-256 slots) ran 41-117 ms:
// small groups, and an SM's warps spread over all phases.
//
// A sample's arithmetic and its draws are those of render.cuh's `sample` in
// the same order, one exception apart: a shadow ray is traced beside the
// path's next ray instead of before it, and its result enters the sum when
// the path is next shaded. The draws do not depend on it and the sums keep
// their order, so a sample's light is the same bit for bit. Samples finish in
// any order: each leaves its terms in `out`, and k_pool_resolve adds them to
// its pixel's sums in sample order.
//
// Scenes: single-instance ones whose materials transmit no light (no glass:
// a path then has one camera hit that is shaded); the caller checks.
#pragma once

#include "render.cuh"

namespace phx {
namespace {

// Words of a path's state. A pool's slots lie in groups of 32, a group's words
// one after another for its slots (Pool::w), so that a pool takes the memory of
// the slots it uses.
enum : uint32_t {
    PW_SEED = 0,
    PW_PIX,       // pixel
    PW_OUT,       // result index
    PW_RO,        // the ray to trace (closest hit, or any hit: ambient occlusion)
    PW_RD = PW_RO + 3,
    PW_HIT = PW_RD + 3,    // its hit: t, slot, u, v
    PW_SP = PW_HIT + 4,    // where the shadow rays start
    PW_Q = PW_SP + 3,      // up to three light queries: direction, distance, light
    PW_D0 = PW_Q + 21,     // the studio rig's fill light
    PW_COL = PW_D0 + 3,
    PW_C = PW_COL + 3,     // light of the camera hit
    PW_IB = PW_C + 3,      // indirect bounce
    PW_IACC,               // indirect light so far        | the glossy lobe's Fresnel
    PW_ITHR = PW_IACC + 3, // throughput                   | bounce light's albedo
    PW_ITP = PW_ITHR + 3,  // throughput the queries meet  | bounce light's emission
    PW_IPB = PW_ITP + 3,   // the ray's cosine pdf         | the lobe's weight
    PW_DW,                 // diffuse weight
    PW_P = PW_DW + 3,      // chance of the diffuse lobe
    PW_WORDS
};

// What a slot waits for; ST_MISS is set beside it when the slot's ray met
// nothing, so that hits and misses are shaded apart.
enum : uint32_t { ST_FREE = 0, ST_CAM, ST_IND, ST_GLS, ST_AO, ST_END, ST_MISS = 8, ST_UNUSED = 15 };
// Whose light queries are pending (`own` bits of a slot's info word).
enum : uint32_t { OWN_CAM = 0, OWN_IND = 1, OWN_BL = 2 };

// A slot's info word: bits 0-1 pending queries, 2-4 a query's shadow ray met
// something, 5-6 the owner, 7 the occlusion ray's near light (0.25),
// 8-15 faces seen through so far, 16 whether a diffuse bounce is under way.
constexpr uint32_t INFO_BLOCKED = 4u, INFO_OWN = 32u, INFO_NEAR = 128u, INFO_SEEN = 256u, INFO_DIFFUSE = 65536u;

// Ray list entries: slot, and which of the slot's rays.
constexpr uint32_t RAY_SLOT = 4095u;
constexpr uint32_t RAY_KIND = 12;  // bits 12-13: 0 the path's ray, 1-3 shadow ray k - 1
constexpr uint32_t RAY_AO = 1u << 14;  // the path's ray is an any-hit ray of range F.ao

constexpr int POOL_STEPS = 6;    // node visits between looks at the warp's other lanes (2: 29.9 ms, 4: 28.1, 6: 28.0)
constexpr int POOL_REFILL = 12;  // idle lanes that make a refill (8: 28.4 ms, 12: 28.1)
// A leaf's triangles are tested once this share of the lanes that hold an
// inner node (1 / POOL_LEAF) waits at one.
constexpr int POOL_LEAF = 2;

// The kinds of slot the shading phase takes, the longest code first.
constexpr uint32_t POOL_KINDS = 9;
__constant__ const uint8_t POOL_ORDER[POOL_KINDS] = {ST_CAM,           ST_IND,           ST_GLS,
                                                     ST_END,           ST_CAM | ST_MISS, ST_IND | ST_MISS,
                                                     ST_GLS | ST_MISS, ST_AO,            ST_AO | ST_MISS};

template <int P>
struct PoolShared {
    Scene S;
    Frame F;
    uint32_t info[P];
    uint16_t ray[P], shadow[3 * P], pick[P + 32 * POOL_KINDS];
    uint8_t stage[P];
    uint32_t nray, nshadow, head;  // the ray lists' lengths, the next ray to trace
    uint32_t count[16];            // slots of each stage
    uint32_t unit, group;          // first unit of a fill; next group of 32 to shade
};

template <int P>
struct Pool {
    uint32_t* st;  // this block's pool
    PoolShared<P>* sh;
    uint32_t lane;

    __device__ __forceinline__ uint32_t& w(uint32_t k, uint32_t s) const {
        return st[(s >> 5) * (PW_WORDS * 32u) + (s & 31u) + k * 32u];
    }
    __device__ __forceinline__ float f(uint32_t k, uint32_t s) const { return __uint_as_float(w(k, s)); }
    __device__ __forceinline__ f3 f3at(uint32_t k, uint32_t s) const { return mk(f(k, s), f(k + 1, s), f(k + 2, s)); }
    __device__ __forceinline__ void put(uint32_t k, uint32_t s, float v) const { w(k, s) = __float_as_uint(v); }
    __device__ __forceinline__ void put(uint32_t k, uint32_t s, f3 v) const {
        put(k, s, v.x);
        put(k + 1, s, v.y);
        put(k + 2, s, v.z);
    }
    // `n` places on a shared counter for the warp's lanes in `m`; this lane's.
    __device__ __forceinline__ uint32_t take(uint32_t* counter, uint32_t m) const {
        uint32_t base = 0;
        const uint32_t leader = __ffs(m) - 1u;
        if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
        return __shfl_sync(0xffffffffu, base, leader) + __popc(m & ((1u << lane) - 1u));
    }
    // Appends the lanes' entries to the lists (every lane of the warp calls).
    __device__ __forceinline__ void push_ray(bool on, uint32_t e) const {
        const uint32_t m = __ballot_sync(0xffffffffu, on);
        if (!m) return;
        const uint32_t k = take(&sh->nray, m);
        if (on) sh->ray[k] = (uint16_t)e;
    }
    __device__ __forceinline__ void push_shadows(bool on, uint32_t s) const {
        const uint32_t nq = on ? sh->info[s] & 3u : 0u;
#pragma unroll 1
        for (uint32_t q = 0; q < 3u; q++) {
            const uint32_t m = __ballot_sync(0xffffffffu, nq > q);
            if (!m) return;
            const uint32_t k = take(&sh->nshadow, m);
            if (nq > q) sh->shadow[k] = (uint16_t)(s | ((q + 1u) << RAY_KIND));
        }
    }
};

// The trace phase: every ray of the block's lists, the path rays first (they
// run longest). Hits go to the slots, a blocked shadow ray to its slot's info
// bit. A ray's walk is walk_tree's (shade.cuh), step by step; what the warp
// does next is one step for the lanes at an inner node or one triangle for
// the lanes at a leaf. Taking both for whichever lanes were there cost a leaf
// test in nearly every step; the lanes at a leaf wait until they are half as many
// as those at inner nodes (1 spp of the mesh at 1080p 5.3 -> 3.6 ms). A ray's own
// order is not changed, so ties of two triangles at one t fall as before.
template <int STATS, int P>
__device__ __forceinline__ void pool_trace(const Scene& S, const Frame& F, const Pool<P>& of, Count& cnt) {
    const Tree T = tree_of(S);
    const Pool<P> pool = of;  // a copy whose fields stay in registers across the walk
    const float ao = F.ao;
    const uint32_t lane = pool.lane, nray = pool.sh->nray, total = nray + pool.sh->nshadow;
    bool drained = total == 0u;
    bool active = false, any = false;
    uint32_t entry = 0, nd = 0;
    uint32_t stack[STACK];
    int sp = 0;
    f3 o = mk(0.0f), inv = mk(0.0f);
    RaySpace rs{2u, false, mk(0.0f)};
    Hit best{0.0f, NONE, 0.0f, 0.0f, 0u};
    for (;;) {
        const uint32_t inner = __ballot_sync(0xffffffffu, active && !(nd & LEAF));
        const uint32_t leaf = __ballot_sync(0xffffffffu, active && (nd & LEAF));
        const uint32_t need = ~(inner | leaf);
        if (!drained && __popc(need) >= POOL_REFILL) {
            const uint32_t k = pool.take(&pool.sh->head, need);
            if (!active && k < total) {
                entry = k < nray ? pool.sh->ray[k] : pool.sh->shadow[k - nray];
                const uint32_t s = entry & RAY_SLOT, kind = (entry >> RAY_KIND) & 3u;
                f3 d;
                if (kind == 0u) {
                    o = pool.f3at(PW_RO, s);
                    d = pool.f3at(PW_RD, s);
                    any = (entry & RAY_AO) != 0u;
                    best = Hit{any ? ao : INF, NONE, 0.0f, 0.0f, 0u};
                } else {
                    const uint32_t q = PW_Q + 7u * (kind - 1u);
                    o = pool.f3at(PW_SP, s);
                    d = pool.f3at(q, s);
                    any = true;
                    best = Hit{pool.f(q + 3u, s), NONE, 0.0f, 0.0f, 0u};
                }
                cnt.rays++;
                inv = safe_inv(d);
                rs = ray_space(d);
                sp = 0;
                nd = T.root;
                active = box_t(T.root_lo, T.root_hi, o, inv, best.t) < INF;
                if (!active && kind == 0u) pool.sh->stage[s] |= ST_MISS;
            }
            drained = __any_sync(0xffffffffu, !active && k >= total);
            continue;  // a ray that misses the root box leaves its lane free again
        }
        if (need == 0xffffffffu) break;
        bool pop = false, done = false;
        if (__popc(leaf) * POOL_LEAF >= __popc(inner)) {
            if (active && (nd & LEAF)) {
                const uint32_t id = nd & ~LEAF;
                const float4 A = __ldg(T.tris + 3 * (size_t)id);
                const float4 B = __ldg(T.tris + 3 * (size_t)id + 1);
                const float4 Cc = __ldg(T.tris + 3 * (size_t)id + 2);
                const uint32_t flags = __float_as_uint(Cc.w);
                if (STATS & MODE_STATS) cnt.tests++;
                float u, v;
                const float t = tri_t(xyz(A), xyz(B), xyz(Cc), o, rs, u, v);
                if (t < best.t) {
                    if (!any) {
                        best = Hit{t, id, u, v, 0u};
                    } else if (!(flags & FLAG_PASS)) {
                        best.tri = id;
                        done = true;
                    }
                }
                nd++;
                pop = (flags & FLAG_END) || id + 1u >= T.nslots;
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < POOL_STEPS && active && !(nd & LEAF); k++) {
                if (STATS & MODE_STATS) cnt.steps++;
                const float4* q = T.nodes + 4 * (size_t)nd;
                const float4 n0 = __ldg(q), n1 = __ldg(q + 1), n2 = __ldg(q + 2), n3 = __ldg(q + 3);
                const float tl = box_t(mk(n0.x, n0.y, n0.z), mk(n0.w, n1.x, n1.y), o, inv, best.t);
                const float tr = box_t(mk(n1.z, n1.w, n2.x), mk(n2.y, n2.z, n2.w), o, inv, best.t);
                const uint32_t l = __float_as_uint(n3.x), r = __float_as_uint(n3.y);
                const bool left = tl <= tr;  // the nearer; a child not hit is at INF
                if (fmaxf(tl, tr) < INF && sp < STACK) stack[sp++] = left ? r : l;
                nd = left ? l : r;
                if (fminf(tl, tr) >= INF) {
                    if (sp == 0) {
                        done = true;
                        break;
                    }
                    nd = stack[--sp];
                }
            }
        }
        if (pop && !done) {
            if (sp > 0) nd = stack[--sp];
            else done = true;
        }
        if (done) {
            active = false;
            const uint32_t s = entry & RAY_SLOT, kind = (entry >> RAY_KIND) & 3u;
            if (kind == 0u) {
                if (best.tri == NONE) {
                    pool.sh->stage[s] |= ST_MISS;
                } else {
                    pool.put(PW_HIT, s, best.t);
                    pool.w(PW_HIT + 1u, s) = best.tri;
                    pool.put(PW_HIT + 2u, s, best.u);
                    pool.put(PW_HIT + 3u, s, best.v);
                }
            } else if (best.tri != NONE) {
                atomicOr(&pool.sh->info[s], INFO_BLOCKED << (kind - 1u));
            }
        }
    }
}

// direct() up to its shadow rays: the light queries of s in the reference's
// order, those with light kept in the slot; their number.
template <int M, int P>
__device__ __noinline__ uint32_t pool_queries(const Scene& S, const Frame& F, const Surf& s, uint32_t& seed, f3 sun,
                                              const Pool<P>& pool, uint32_t slot) {
    if (uses_rig(F)) pool.put(PW_D0, slot, rig_fill(F, s));
    uint32_t nq = 0;
#pragma unroll 1
    for (uint32_t k = 0; k < 3u; k++) {
        const Query q = light_query<M>(S, F, k, s, seed, sun);
        if (!q.met) continue;
        const f3 c = brdf(s, q.l, q.e) * q.scale;
        if (maxc(c) > 0.0f) {
            const uint32_t at = PW_Q + 7u * nq;
            pool.put(at, slot, q.l);
            pool.put(at + 3u, slot, q.dist);
            pool.put(at + 4u, slot, c);
            nq++;
        }
    }
    if (nq) pool.put(PW_SP, slot, s.pos);
    return nq;
}

// direct()'s sum over the pending queries (integrate.wgsl:66-85).
template <int P>
__device__ __noinline__ f3 pool_light(const Frame& F, const Pool<P>& pool, uint32_t slot, uint32_t info) {
    f3 sum = uses_rig(F) ? pool.f3at(PW_D0, slot) : mk(0.0f);
#pragma unroll 1
    for (uint32_t k = 0; k < (info & 3u); k++) {
        const float vis = (info & (INFO_BLOCKED << k)) ? 0.0f : 1.0f;
        sum += pool.f3at(PW_Q + 7u * k + 4u, slot) * vis;
    }
    return sum;
}

// The background a camera ray of pixel i sees (shade.wgsl main).
__device__ __forceinline__ f3 sky_at(const Frame& F, uint32_t i) {
    const float across = dv((float)(i % F.w), fmaxf((float)F.w * 0.5f, 1.0f));
    const float lift = F.sky[3] * (1.0f - clampf(across, 0.0f, 1.0f));
    return mk(F.sky[0] + lift, F.sky[1] + lift, F.sky[2] + lift);
}

// Where a sample's terms go: word k of sample r at out[k * n + r].
struct PoolOut {
    uint32_t* out;
    uint64_t n;
    __device__ __forceinline__ void put(uint32_t k, uint32_t r, f3 v) const {
        out[k * n + r] = __float_as_uint(v.x);
        out[(k + 1) * n + r] = __float_as_uint(v.y);
        out[(k + 2) * n + r] = __float_as_uint(v.z);
    }
};
enum : uint32_t { PO_COL = 0, PO_ALB = 3, PO_NRM = 6, PO_DEP = 9, PO_WORDS = 10 };
constexpr float PO_MISSED = -1.0f;  // PO_DEP of a sample whose camera ray met nothing

// The end of a sample: the camera hit's light with its bounced light.
template <int P>
__device__ __noinline__ void pool_finish(const Frame& F, const Pool<P>& pool, const PoolOut& out, uint32_t slot, f3 c,
                                            f3 bounced) {
    c += clamp_light(bounced, F.limit_i);
    out.put(PO_COL, pool.w(PW_OUT, slot), pool.f3at(PW_COL, slot) + c);
    pool.sh->stage[slot] = ST_FREE;
}

template <int P>
__device__ __forceinline__ f3 pool_diffuse(const Pool<P>& pool, uint32_t slot, f3 aval) {
    return mk(0.0f) + dv(pool.f3at(PW_DW, slot) * aval, pool.f(PW_P, slot));
}

template <int P>
__device__ __forceinline__ f3 pool_glossy(const Pool<P>& pool, uint32_t slot, f3 rc) {
    return mk(0.0f) + dv(pool.f3at(PW_IACC, slot) * rc * pool.f(PW_IPB, slot) * 1.0f, 1.0f - pool.f(PW_P, slot));
}

// A camera ray that met nothing.
template <int P>
__device__ __noinline__ void pool_camera_miss(const Frame& F, const Pool<P>& pool, const PoolOut& out, uint32_t slot) {
    const uint32_t r = pool.w(PW_OUT, slot);
    if (((pool.sh->info[slot] / INFO_SEEN) & 255u) == 0u) {
        const f3 d = pool.f3at(PW_RD, slot);
        const uint32_t i = pool.w(PW_PIX, slot);
        const f3 sky = sky_at(F, i);
        out.put(PO_ALB, r, mk(srgb_to_linear1(sky.x), srgb_to_linear1(sky.y), srgb_to_linear1(sky.z)));
        out.put(PO_NRM, r, -d);
        out.out[PO_DEP * out.n + r] = __float_as_uint(PO_MISSED);
        out.put(PO_COL, r, mk(0.0f));
    } else {
        out.put(PO_COL, r, mk(0.0f) + mk(1.0f) * env_at(F));
    }
    pool.sh->stage[slot] = ST_FREE;
}

// A camera ray's hit (sample(), one bounce). True: the slot's ray is to be traced.
template <int M, int P>
__device__ __noinline__ bool pool_camera_hit(const Scene& S, const Frame& F, f3 sun, const Pool<P>& pool,
                                             const PoolOut& out, uint32_t slot) {
    const uint32_t info = pool.sh->info[slot];
    const uint32_t seen = (info / INFO_SEEN) & 255u;
    const f3 o = pool.f3at(PW_RO, slot), d = pool.f3at(PW_RD, slot);
    const uint32_t tri = pool.w(PW_HIT + 1u, slot), r = pool.w(PW_OUT, slot);
    uint32_t seed = pool.w(PW_SEED, slot);
    const float ht = pool.f(PW_HIT, slot), hu = pool.f(PW_HIT + 2u, slot), hv = pool.f(PW_HIT + 3u, slot);
    const Geo g = geo_at<M>(S, tri, 0u);
    const Mat t = mat_at(S, g.mat);
    const float w = 1.0f - hu - hv;
    const f3 hit = o + d * ht;
    const f3 ng0 = unit(cross(g.b - g.a, g.c - g.a));
    const bool front = dot(ng0, d) < 0.0f;
    const f3 ng = front ? ng0 : -ng0;
    f3 n = g.na * w + g.nb * hu + g.nc * hv;
    n = dot(n, n) > 1e-12f ? unit(n) * (front ? 1.0f : -1.0f) : ng;
    if (dot(n, -d) < 0.0f) n = ng;
    const f3 base = vmax(mk(t.color.x, t.color.y, t.color.z), mk(0.0f));
    if (seen == 0u) {
        out.put(PO_ALB, r, base);
        out.put(PO_NRM, r, n);
        out.out[PO_DEP * out.n + r] = __float_as_uint(ht);
    }
    if (rnd(seed) >= t.color.w) {
        if (seen + 1u > 8u) {  // see_through
            out.put(PO_COL, r, mk(0.0f));
            pool.sh->stage[slot] = ST_FREE;
            return false;
        }
        pool.put(PW_RO, slot, hit - ng * through_lift(F, hit, ht));
        pool.w(PW_SEED, slot) = seed;
        pool.sh->info[slot] = info + INFO_SEEN;
        return true;
    }
    const f3 pos = hit + ng * hit_lift(F, ht);
    pool.put(PW_COL, slot, mk(0.0f) + mk(1.0f) * t.emit);
    const float bleed = scatter_bleed(t.sss, t.sss_radius);
    const f3 fd = dielectric_f0(t.ior);
    f3 diffuse = base * (1.0f - t.metal);
    if (maxc(diffuse) > 0.0f)
        diffuse *= under_layer_real(t.ior, fmaxf(t.rough, 0.04f), fmaxf(dot(n, -d), 1e-4f));
    const Surf s{pos,   n,      -d,        diffuse,        vmix(fd, base, t.metal), fmaxf(t.rough, 0.04f),
                 bleed, scatter_tint(t.sss_radius), t.sheen, t.sheen_rough,    t.sheen_tint,
                 t.coat, t.coat_rough, t.ior, 1.0f - t.metal};
    uint32_t next = pool_queries<M, P>(S, F, s, seed, sun, pool, slot) | OWN_CAM * INFO_OWN;
    const f3 diffuse_weight = vmix(s.albedo, s.albedo * s.sss_tint, bleed);
    const f3 lw = mk(0.2126f, 0.7152f, 0.0722f);
    const float ndv = fmaxf(dot(n, -d), 1e-4f);
    const f3 gloss_guess = s.f0 + (mk(1.0f) - s.f0) * pow_of(1.0f - ndv, 5.0f);
    const float pd = dot(vmax(diffuse_weight, mk(0.0f)), lw);
    const float pg = dot(gloss_guess, lw);
    float p_diffuse = pd + pg > 0.0f ? dv(pd, pd + pg) : 1.0f;
    if (pd > 0.0f && pg > 0.0f) p_diffuse = clampf(p_diffuse, 0.15f, 0.85f);
    const bool take_diffuse = rnd(seed) < p_diffuse;
    uint32_t stage = ST_END;
    if (take_diffuse && pd > 0.0f) {
        pool.put(PW_DW, slot, diffuse_weight);
        pool.put(PW_P, slot, p_diffuse);
        pool.put(PW_IACC, slot, mk(0.0f));
        next |= INFO_DIFFUSE;
        if (S.lamp_count == 0u && !(dot(F.env, F.env) > 0.0f)) {
            const f3 dir = cosine_dir(n, seed);
            if (!(F.env.x == 0.0f && F.env.y == 0.0f && F.env.z == 0.0f)) {
                pool.put(PW_RO, slot, pos);
                pool.put(PW_RD, slot, dir);
                stage = ST_AO;
            }
        } else {
            const f3 dir = cosine_dir(n, seed);
            pool.put(PW_IPB, slot, dv(fmaxf(dot(n, dir), 0.0f), PI));
            pool.put(PW_ITHR, slot, mk(1.0f));
            pool.w(PW_IB, slot) = 0u;
            pool.put(PW_RO, slot, pos);
            pool.put(PW_RD, slot, dir);
            stage = ST_IND;
        }
    } else if (!take_diffuse) {
        const f3 v = -d;
        const f3 tx = unit(onb(n, 1.0f, 0.0f));
        const f3 ty = cross(n, tx);
        const float ggx_a = s.rough * s.rough;
        const f3 wi_local = mk(dot(v, tx), dot(v, ty), dot(v, n));
        const float r1 = rnd(seed);
        const float r2 = rnd(seed);
        const f3 h_local = ggx_sample_vndf(wi_local, ggx_a, r1, r2);
        const f3 hw = unit(tx * h_local.x + ty * h_local.y + n * h_local.z);
        const f3 refl = reflect(d, hw);
        const float cos_hi = fmaxf(dot(hw, v), 0.0f);
        const float cos_no = dot(n, refl);
        if (dot(refl, ng) > 0.0f && cos_hi > 0.0f && cos_no > 0.0f) {
            pool.put(PW_IACC, slot, fresnel_of(s, cos_hi));
            pool.put(PW_IPB, slot, ggx_weight(ggx_a * ggx_a, fmaxf(dot(n, v), 1e-4f), cos_no));
            pool.put(PW_P, slot, p_diffuse);
            pool.put(PW_RO, slot, pos);
            pool.put(PW_RD, slot, refl);
            stage = ST_GLS;
        }
    }
    pool.w(PW_SEED, slot) = seed;
    pool.sh->info[slot] = next;
    pool.sh->stage[slot] = (uint8_t)stage;
    return stage != ST_END;
}

// The light queries of a path's last surface resolved: the camera hit's
// light (kept in the slot from the first indirect ray on), and the indirect
// light so far.
template <int P>
__device__ __forceinline__ f3 pool_resolve(const Frame& F, const Pool<P>& pool, uint32_t slot, uint32_t info, f3& acc) {
    acc = pool.f3at(PW_IACC, slot);
    const f3 light = pool_light(F, pool, slot, info);
    if (((info / INFO_OWN) & 3u) == OWN_CAM) return clamp_light(light, F.limit_d);
    acc += pool.f3at(PW_ITP, slot) * light * ((info & INFO_NEAR) ? 0.25f : 1.0f);
    return pool.f3at(PW_C, slot);
}

// An indirect ray that met nothing.
template <int P>
__device__ __noinline__ void pool_indirect_miss(const Frame& F, const Pool<P>& pool, const PoolOut& out, uint32_t slot) {
    f3 acc;
    const f3 c = pool_resolve(F, pool, slot, pool.sh->info[slot], acc);
    acc += pool.f3at(PW_ITHR, slot) * env_at(F) * 1.0f;
    pool_finish(F, pool, out, slot, c, pool_diffuse(pool, slot, acc));
}

// One bounce of indirect() (integrate.wgsl:111-230) at a surface.
template <int M, int P>
__device__ __noinline__ bool pool_indirect_hit(const Scene& S, const Frame& F, f3 sun, const Pool<P>& pool,
                                               uint32_t slot) {
    const uint32_t info = pool.sh->info[slot];
    f3 acc;
    const f3 c = pool_resolve(F, pool, slot, info, acc);
    if (((info / INFO_OWN) & 3u) == OWN_CAM) pool.put(PW_C, slot, c);
    f3 thr = pool.f3at(PW_ITHR, slot);
    const uint32_t tri = pool.w(PW_HIT + 1u, slot);
    uint32_t seed = pool.w(PW_SEED, slot);
    const f3 org = pool.f3at(PW_RO, slot), dir = pool.f3at(PW_RD, slot);
    const float ht = pool.f(PW_HIT, slot);
    const bool lit = dot(F.env, F.env) > 0.0f;
    const Geo g = geo_at<M>(S, tri, 0u);
    const Mat t = mat_at(S, g.mat);
    const f3 ng0 = unit(cross(g.b - g.a, g.c - g.a));
    const f3 ng = dot(ng0, dir) < 0.0f ? ng0 : -ng0;
    const f3 hit = org + dir * ht + ng * (F.eps + ht * 1e-5f);
    const f3 base = vmax(mk(t.color.x, t.color.y, t.color.z), mk(0.0f));
    const float rough = fmaxf(t.rough, glossy_floor());
    const f3 fd = dielectric_f0(t.ior);
    f3 albedo = base * (1.0f - t.metal);
    if (maxc(albedo) > 0.0f) albedo *= under_layer(fd, rough, fmaxf(dot(ng, -dir), 1e-4f));
    {  // glow_mis (integrate.wgsl:15-23), the cosine pdf kept with the ray
        f3 e = t.emit;
        const float chance = lamp_chance<M>(S, tri, 0u);
        if (chance > 0.0f) {
            const f3 cr = cross(g.b - g.a, g.c - g.a);
            const float pl = dv(chance * ht * ht, fmaxf(0.5f * rt(dot(cr, cr)) * fabsf(dot(unit(cr), dir)), 1e-8f));
            const float pb = pool.f(PW_IPB, slot);
            e = dv(t.emit * pb * pb, fmaxf(pb * pb + pl * pl, 1e-12f));
        }
        acc += thr * e;
    }
    pool.put(PW_IACC, slot, acc);
    const Surf s = plain_surf(hit, ng, -dir, albedo, vmix(fd, base, t.metal), rough);
    uint32_t next = pool_queries<M, P>(S, F, s, seed, sun, pool, slot) | OWN_IND * INFO_OWN | INFO_DIFFUSE;
    if (!lit && ht <= F.ao) next |= INFO_NEAR;
    pool.put(PW_ITP, slot, thr);
    const uint32_t b = pool.w(PW_IB, slot);
    const uint32_t depth = F.bounces != 0u ? F.bounces : 1u;
    bool more = b + 1u < depth;
    thr *= albedo;
    if (more) {
        const float keep = clampf(maxc(thr), 0.0f, 0.95f);
        if (keep < 1e-4f || rnd(seed) > keep) {
            more = false;
        } else {
            thr = dv(thr, keep);
            const f3 nd = cosine_dir(ng, seed);
            pool.put(PW_IPB, slot, dv(fmaxf(dot(ng, nd), 0.0f), PI));
            pool.put(PW_ITHR, slot, thr);
            pool.w(PW_IB, slot) = b + 1u;
            pool.put(PW_RO, slot, hit);
            pool.put(PW_RD, slot, nd);
        }
    }
    pool.w(PW_SEED, slot) = seed;
    pool.sh->info[slot] = next;
    if (!more) pool.sh->stage[slot] = ST_END;
    return more;
}

// A glossy ray that met nothing.
template <int P>
__device__ __noinline__ void pool_glossy_miss(const Frame& F, const Pool<P>& pool, const PoolOut& out, uint32_t slot) {
    const f3 c = clamp_light(pool_light(F, pool, slot, pool.sh->info[slot]), F.limit_d);
    pool_finish(F, pool, out, slot, c, pool_glossy(pool, slot, env_at(F)));
}

// The glossy ray's hit: bounce_light (integrate.wgsl:236-250).
template <int M, int P>
__device__ __noinline__ void pool_glossy_hit(const Scene& S, const Frame& F, f3 sun, const Pool<P>& pool,
                                             uint32_t slot) {
    const f3 c = clamp_light(pool_light(F, pool, slot, pool.sh->info[slot]), F.limit_d);
    const uint32_t tri = pool.w(PW_HIT + 1u, slot);
    pool.put(PW_C, slot, c);
    uint32_t seed = pool.w(PW_SEED, slot);
    const f3 org = pool.f3at(PW_RO, slot), d = pool.f3at(PW_RD, slot);
    const float ht = pool.f(PW_HIT, slot);
    const Geo g = geo_at<M>(S, tri, 0u);
    const Mat t = mat_at(S, g.mat);
    const f3 ng0 = unit(cross(g.b - g.a, g.c - g.a));
    const f3 ng = dot(ng0, d) < 0.0f ? ng0 : -ng0;
    const f3 pos = org + d * ht + ng * (F.eps + ht * 1e-5f);
    const f3 base = vmax(mk(t.color.x, t.color.y, t.color.z), mk(0.0f));
    const float rough = fmaxf(t.rough, glossy_floor());
    const f3 fd = dielectric_f0(t.ior);
    f3 albedo = base * (1.0f - t.metal);
    if (maxc(albedo) > 0.0f) albedo *= under_layer(fd, rough, fmaxf(dot(ng, -d), 1e-4f));
    const Surf s = plain_surf(pos, ng, -d, albedo, vmix(fd, base, t.metal), rough);
    pool.put(PW_ITHR, slot, s.albedo);
    pool.put(PW_ITP, slot, t.emit);
    pool.sh->info[slot] = pool_queries<M, P>(S, F, s, seed, sun, pool, slot) | OWN_BL * INFO_OWN;
    pool.sh->stage[slot] = ST_END;
}

// The ambient-occlusion ray of a scene with neither emitters nor a lit world.
template <int P>
__device__ __forceinline__ void pool_ao(const Frame& F, const Pool<P>& pool, const PoolOut& out, uint32_t slot) {
    const f3 c = clamp_light(pool_light(F, pool, slot, pool.sh->info[slot]), F.limit_d);
    const float vis = (pool.sh->stage[slot] & ST_MISS) ? 1.0f : 0.0f;
    pool_finish(F, pool, out, slot, c, pool_diffuse(pool, slot, env_at(F) * mixf(0.25f, 1.0f, vis)));
}

// A path with no ray left but the shadow rays of its last surface.
template <int P>
__device__ __forceinline__ void pool_end(const Frame& F, const Pool<P>& pool, const PoolOut& out, uint32_t slot) {
    const uint32_t info = pool.sh->info[slot], own = (info / INFO_OWN) & 3u;
    const f3 light = pool_light(F, pool, slot, info);
    if (own == OWN_CAM) {
        const f3 bounced = (info & INFO_DIFFUSE) ? pool_diffuse(pool, slot, mk(0.0f)) : mk(0.0f);
        pool_finish(F, pool, out, slot, clamp_light(light, F.limit_d), bounced);
    } else if (own == OWN_IND) {
        const f3 acc = pool.f3at(PW_IACC, slot) +
                       pool.f3at(PW_ITP, slot) * light * ((info & INFO_NEAR) ? 0.25f : 1.0f);
        pool_finish(F, pool, out, slot, pool.f3at(PW_C, slot), pool_diffuse(pool, slot, acc));
    } else {
        const f3 rc = light + pool.f3at(PW_ITHR, slot) * env_at(F) * 0.8f + pool.f3at(PW_ITP, slot);
        pool_finish(F, pool, out, slot, pool.f3at(PW_C, slot), pool_glossy(pool, slot, rc));
    }
}

// One frame's samples, taken by the warps in units of a 32-pixel tile and
// one sample, the samples of a tile one after another.
struct PoolFrame {
    uint32_t first, count;  // pixels
    uint32_t spp;           // samples of this launch, from F.frame0 on
    PoolOut out;
};

// The block's slots listed by stage: each of the POOL_KINDS kinds (or, with
// `free`, the free slots) a run of sh->pick from a multiple of 32 on; the
// number of groups of 32. Every thread of the block calls.
template <int P, int T>
__device__ __forceinline__ uint32_t pool_list(const Pool<P>& pool, bool free) {
    PoolShared<P>& sh = *pool.sh;
    if (threadIdx.x < 16u) sh.count[threadIdx.x] = 0u;
    __syncthreads();
    uint32_t at[P / T];
#pragma unroll
    for (uint32_t j = 0; j < P / T; j++) {
        const uint32_t stage = sh.stage[j * T + threadIdx.x];
        const uint32_t m = __match_any_sync(0xffffffffu, stage);
        const uint32_t leader = __ffs(m) - 1u;
        uint32_t base = 0;
        if (pool.lane == leader) base = atomicAdd(&sh.count[stage], (uint32_t)__popc(m));
        at[j] = __shfl_sync(0xffffffffu, base, leader) + __popc(m & ((1u << pool.lane) - 1u));
    }
    __syncthreads();
    uint32_t groups = 0;
    if (free) {
        groups = sh.count[ST_FREE] / 32u;
#pragma unroll
        for (uint32_t j = 0; j < P / T; j++)
            if (sh.stage[j * T + threadIdx.x] == ST_FREE) sh.pick[at[j]] = (uint16_t)(j * T + threadIdx.x);
    } else {
#pragma unroll 1
        for (uint32_t k = 0; k < POOL_KINDS; k++) {
            const uint32_t stage = POOL_ORDER[k];
#pragma unroll
            for (uint32_t j = 0; j < P / T; j++)
                if (sh.stage[j * T + threadIdx.x] == stage)
                    sh.pick[groups * 32u + at[j]] = (uint16_t)(j * T + threadIdx.x);
            groups += (sh.count[stage] + 31u) / 32u;
        }
    }
    __syncthreads();
    return groups;
}

// New paths into the block's free slots, a unit for every 32; false when the
// frame has no unit left.
template <int P, int T>
__device__ __forceinline__ bool pool_fill(const Frame& F, const PoolFrame& J, const Pool<P>& pool, uint32_t* next) {
    PoolShared<P>& sh = *pool.sh;
    const uint32_t want = pool_list<P, T>(pool, true);
    const uint64_t units = (uint64_t)((J.count + 31u) / 32u) * J.spp;
    if (threadIdx.x == 0) sh.unit = want ? atomicAdd(next, want) : 0u;
    __syncthreads();
    const uint32_t first = sh.unit;
#pragma unroll 1
    for (uint32_t j = threadIdx.x / 32u; j < want && first + j < units; j += T / 32u) {
        const uint32_t tile = (first + j) / J.spp, smp = (first + j) - tile * J.spp;
        const uint32_t k = tile * 32u + pool.lane;
        const uint32_t slot = sh.pick[j * 32u + pool.lane];
        const bool on = k < J.count;
        if (on) {
            const uint32_t i = J.first + tile_px(F, k, J.first, J.count);
            uint32_t seed = hash(i * 9781u + (F.frame0 + smp) * 6271u + 1u);
            const CamRay cr = camera_ray(F, i, seed);
            pool.w(PW_SEED, slot) = seed;
            pool.w(PW_PIX, slot) = i;
            pool.w(PW_OUT, slot) = smp * J.count + k;
            pool.put(PW_RO, slot, cr.o);
            pool.put(PW_RD, slot, cr.d);
            sh.info[slot] = 0u;
            sh.stage[slot] = ST_CAM;
        }
        pool.push_ray(on, slot);
    }
    return want == 0u || first + want < units;
}

// The shading phase: each kind of slot, 32 at a time, the groups taken by
// the block's warps. The slots are listed before any is shaded, so a slot that
// changes stage here is not met again before its rays are traced.
template <int M, int P, int T>
__device__ __forceinline__ void pool_shade(const Scene& S, const Frame& F, f3 sun, const PoolOut& out,
                                           const Pool<P>& pool) {
    PoolShared<P>& sh = *pool.sh;
    const uint32_t groups = pool_list<P, T>(pool, false);
#pragma unroll 1
    for (;;) {
        uint32_t g = 0;
        if (pool.lane == 0) g = atomicAdd(&sh.group, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= groups) break;
        uint32_t kind = 0;
#pragma unroll 1
        while ((sh.count[POOL_ORDER[kind]] + 31u) / 32u <= g) {
            g -= (sh.count[POOL_ORDER[kind]] + 31u) / 32u;
            kind++;
        }
        // g is now the group within its kind; the run's start in sh.pick
        uint32_t start = 0;
#pragma unroll 1
        for (uint32_t k = 0; k < kind; k++) start += (sh.count[POOL_ORDER[k]] + 31u) / 32u;
        const uint32_t n = sh.count[POOL_ORDER[kind]];
        const bool on = g * 32u + pool.lane < n;
        const uint32_t slot = on ? sh.pick[(start + g) * 32u + pool.lane] : 0u;
        bool ray = false;
        if (on) {
            switch (kind) {
                case 0: ray = pool_camera_hit<M, P>(S, F, sun, pool, out, slot); break;
                case 1: ray = pool_indirect_hit<M, P>(S, F, sun, pool, slot); break;
                case 2: pool_glossy_hit<M, P>(S, F, sun, pool, slot); break;
                case 3: pool_end(F, pool, out, slot); break;
                case 4: pool_camera_miss(F, pool, out, slot); break;
                case 5: pool_indirect_miss(F, pool, out, slot); break;
                case 6: pool_glossy_miss(F, pool, out, slot); break;
                default: pool_ao(F, pool, out, slot); break;
            }
        }
        __syncwarp();
        if (kind < 3u) {
            const uint32_t stage = sh.stage[slot];
            pool.push_ray(ray, slot | (stage == ST_AO ? RAY_AO : 0u));
            // a path seen through a cut-out has no queries, one that ended no slot
            pool.push_shadows(on && stage != ST_FREE && stage != ST_CAM, slot);
        }
    }
}

template <int M, int MINB, int P, int T>
__global__ void __launch_bounds__(T, MINB) k_render_pool(const __grid_constant__ Scene scene,
                                                         const __grid_constant__ Frame frame, f3 sun, PoolFrame J,
                                                         uint32_t slots, uint32_t* pools, uint32_t* next,
                                                         unsigned long long* counters) {
    static_assert(P % T == 0 && P <= (int)RAY_SLOT + 1, "whole rounds of the block, a 12-bit slot");
    extern __shared__ __align__(16) uint8_t dyn[];
    PoolShared<P>& sh = *(PoolShared<P>*)dyn;
    // one copy of the records the shading reads, not one a thread in local memory
    if (threadIdx.x == 0) {
        sh.S = scene;
        sh.F = frame;
        setup(sh.S, sh.F);
        sh.nray = sh.nshadow = 0u;
    }
    const Scene& S = sh.S;
    const Frame& F = sh.F;
    const Pool<P> pool{pools + (size_t)blockIdx.x * PW_WORDS * slots, &sh, threadIdx.x & 31u};
    for (uint32_t s = threadIdx.x; s < P; s += T) sh.stage[s] = s < slots ? ST_FREE : ST_UNUSED;
    __syncthreads();
    Count cnt{0, 0, 0};
    bool more = true;
    for (;;) {
        if (more) more = pool_fill<P, T>(F, J, pool, next);
        __syncthreads();
        const uint32_t rays = sh.nray + sh.nshadow;
        if (threadIdx.x == 0) sh.head = 0u;
        __syncthreads();
        if (rays) pool_trace<M, P>(S, F, pool, cnt);
        __syncthreads();
        if (threadIdx.x == 0) sh.nray = sh.nshadow = sh.group = 0u;
        // pool_list's barriers come between this reset and the first push
        pool_shade<M, P, T>(S, F, sun, J.out, pool);
        __syncthreads();
        // every slot of the listing was free and nothing was traced: done
        if (rays == 0u && !more && sh.count[ST_FREE] == slots) break;
    }
    flush_counts<M>(cnt, counters);
}

// The samples' terms added to their pixels' sums in sample order, and the
// planes a launch's last sample leaves (render_px).
__global__ void __launch_bounds__(128) k_pool_resolve(Frame F, PoolFrame J, uint32_t* __restrict__ px) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= J.count) return;
    const uint32_t i = J.first + tile_px(F, k, J.first, J.count);
    Sums acc;
    load_sums(px, F.n, i, F.frame0 > 0u, acc);
    const uint64_t n = J.out.n;
    const f3 sky = sky_at(F, i);
    for (uint32_t s = 0; s < J.spp; s++) {
        const uint32_t r = s * J.count + k;
        auto at = [&](uint32_t w) {
            return mk(__uint_as_float(__ldcs(J.out.out + w * n + r)), __uint_as_float(__ldcs(J.out.out + (w + 1) * n + r)),
                      __uint_as_float(__ldcs(J.out.out + (w + 2) * n + r)));
        };
        const float dep = __uint_as_float(__ldcs(J.out.out + PO_DEP * n + r));
        acc.alb += at(PO_ALB);
        acc.nrm += at(PO_NRM);
        acc.dep += dep;
        acc.count += 1u;
        acc.film += 1.0f;
        acc.lin += at(PO_COL);
        if (dep == PO_MISSED) {
            acc.outline = 0u;
            acc.gone += 1.0f;
            acc.grid += sky * (1.0f - 0.0f) + mk(0.0f);
            acc.cov += 1.0f;
        } else {
            acc.outline = 1u;
            acc.gone += 0.0f;
        }
    }
    store_sums(px, F.n, i, F.frame0 == 0u, acc, F);
}

// The host's side of one form: its plan of a frame, and the frame's launches.
template <int M, int MINB, int P, int T>
struct PoolForm {
    static constexpr int SMEM = (int)sizeof(PoolShared<P>);

    int32_t plan(int sms, uint32_t count, uint32_t spp, PoolPlan& p) const {
        auto kernel = k_render_pool<M, MINB, P, T>;
        int per_sm = 0;
        PHX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        PHX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, T, SMEM));
        p = pool_plan(count, spp, (uint32_t)std::max(per_sm, 1) * (uint32_t)sms, P, PW_WORDS * 4, PO_WORDS * 4);
        return PHX_OK;
    }

    int32_t launch(const RenderLaunch& L, const PoolPlan& p, uint32_t* state, uint32_t* out) const {
        RenderLaunch R = L;
        uint32_t left = L.F.spp;
        while (left) {
            PoolFrame J{L.first, L.count, std::min(left, p.spp), PoolOut{out, (uint64_t)L.count * p.spp}};
            R.F.spp = J.spp;
            const uint32_t slots = launch_slots(p, L.count, J.spp, P);
            PHX_CUDA(cudaMemsetAsync(L.next, 0, 4, L.s));
            k_render_pool<M, MINB, P, T><<<p.blocks, T, SMEM, L.s>>>(L.S, R.F, L.sun, J, slots, state, L.next, L.counters);
            k_pool_resolve<<<(L.count + 127) / 128, 128, 0, L.s>>>(R.F, J, L.px);
            left -= J.spp;
            R.F.frame0 += J.spp;
        }
        return cuda_check(cudaGetLastError(), "pooled render");
    }
};

}  // namespace
}  // namespace phx
