// The host's decisions between paths, apart from the launches they decide on:
// plain C++, so that a host build can hold them to every case.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <numeric>
#include <vector>

#include "../../include/phiray_cuda.h"

namespace phx {

// Whether a kernel may read or write `p` by 16-byte words.
inline bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0u; }

// ---- which kernel traces a frame ----

// A tracer whose render kernel was neither set nor autotuned.
constexpr uint32_t KERNEL_UNSET = 0xFFFFFFFFu;

// Frames of so few samples trace in one fill of the pools (see POOL_FILLS).
constexpr uint64_t FEW_SAMPLES = 300000;

// What a frame asks of the kernel that traces it.
struct FrameForm {
    uint32_t kernel;  // the tracer's (set or autotuned, or KERNEL_UNSET)
    uint32_t mega;    // its megakernel form for frames that `kernel` cannot trace
    bool full;        // instances, or the floor grid
    bool adaptive;
    bool transmits;   // some material transmits light
    bool capturing;   // the launches are recorded into a graph
    uint32_t pixels, spp, faces;
};

inline bool pooled_id(uint32_t kernel) {
    return kernel >= PHX_KERNEL_STATE_MACHINE && kernel <= PHX_KERNEL_STATE_MACHINE_8;
}

// An autotuning's pick (of a frame that is not `full`), `fastest` by its times: of
// pooled forms within 6 % of one another the one of the largest blocks. At few
// samples the last paths' end decides between them, at many that form is ahead or
// even. (512 / 256 / 128 threads: the 1.3 M-face mesh at 1080p 2.71 / 2.67 / 2.83 ms
// at 1 spp, either of the first two fastest by chance; 7.54 / 7.70 / 8.40 at 4, 27.8
// / 28.6 / 31.5 at 16; a scene of 60,000 faces at 512 x 512 3.59 / 3.62 / 3.66 and
// 25.4 / 25.5 / 26.1.)
inline uint32_t autotuned(const float* ms, uint32_t fastest) {
    if (!pooled_id(fastest)) return fastest;
    uint32_t k = PHX_KERNEL_STATE_MACHINE;
    while (ms[k] > 1.06f * ms[fastest]) k++;
    return k;
}

// The fastest megakernel form by the times of an autotuning: what a tracer
// whose fastest kernel is another one traces adaptive frames, recorded ones and
// those without memory for the pools with. (The 1.3 M-face mesh at 1080p, 16
// spp: 46 ms in the 16-block form, 57 in the 4-block one.)
inline uint32_t fastest_megakernel(const float* ms) {
    uint32_t best = PHX_KERNEL_MEGAKERNEL;
    for (uint32_t k = 0; k < PHX_KERNEL_COUNT; k++)
        if (!pooled_id(k) && k != PHX_KERNEL_WAVEFRONT && ms[k] < ms[best]) best = k;
    return best;
}

// The kernel of a frame whose tracer names none, of those that compute the same
// image: the pooled render where it can run. On a 65,536-face cloud at 256 x 256,
// 16 spp, it took 4.9 ms against the 4-block megakernel's 27 ms, on the 1.3
// M-face mesh at 1080p, 16 spp, 28 ms against 57. Frames of few samples take the
// form of 256 threads (more and smaller pools end sooner): 256 x 256 at 1 spp,
// megakernel / 512 threads / 256 threads, cloud 2.06 / 1.59 / 1.49 ms, that mesh
// 0.76 / 0.84 / 0.73. One sample of few pixels of a small scene is a few walks
// one after another, which the megakernel does without phases (a scene of 1,600
// faces at 256 x 256, 1 spp 0.17 ms against 0.21; of two triangles 0.05 against
// 0.09; from 144,000 pixels on, or with two samples, the pools are even or ahead).
inline uint32_t default_kernel(const FrameForm& f) {
    if (f.full || (f.spp == 1 && f.pixels < 100000 && f.faces < 10000)) return f.mega;
    return (uint64_t)f.pixels * f.spp < FEW_SAMPLES ? PHX_KERNEL_STATE_MACHINE_6 : PHX_KERNEL_STATE_MACHINE;
}

// The id of the kernel that traces the frame. Adaptive Sampling runs on the
// megakernel forms (the others take pixels by index, not from the open list);
// the pooled render shades a path's one opaque camera hit, so it takes scenes
// whose materials transmit no light; the wavefront's host polls its queues
// between passes, which a recorded graph cannot.
inline uint32_t frame_kernel(const FrameForm& f) {
    uint32_t k = f.kernel;
    if (k == KERNEL_UNSET) k = default_kernel(f);
    if (k == PHX_KERNEL_WAVEFRONT && (f.adaptive || f.capturing)) return f.mega;
    if (pooled_id(k) && (f.adaptive || (f.transmits && !f.full))) return f.mega;
    return k;
}

// Whether that is the pooled render, which needs buffers (under the same ids a
// frame with `full` runs the state machine, which needs none).
inline bool frame_pooled(const FrameForm& f) { return !f.full && pooled_id(frame_kernel(f)); }

// ---- the pooled render's work and memory ----

// Fills of a pool a frame is cut into at least (fewer slots, so that a small
// frame's last paths do not leave most of a pool empty, against fewer and
// larger phases): the cloud above took 7.0, 4.9, 5.0, 5.3 and 6.3 ms at 1, 2,
// 3, 4 and 8 fills. Of few samples every phase is short, and one fill has the
// fewest: at 1 spp and 480 x 300 2.0 ms against 2.4, the 1.3 M-face mesh 0.95
// against 1.08; from 640 x 480 at 1 spp on two are even or ahead.
constexpr uint32_t POOL_FILLS = 2;

// Sample terms held at once; the rest of the samples run in further launches.
constexpr size_t POOL_OUT_BYTES = (size_t)1 << 30;

// Slots a block for `samples` paths over `blocks` blocks of at most `most`.
inline uint32_t pool_slots(uint64_t samples, uint32_t blocks, uint32_t most) {
    const uint64_t share = samples / blocks / (samples < FEW_SAMPLES ? 1u : POOL_FILLS) / 32u * 32u;
    return (uint32_t)std::min<uint64_t>(most, std::max<uint64_t>(share, 32u));
}

// A frame of `count` pixels and `spp` samples on `blocks` blocks of at most
// `most` slots: memory follows the frame up to what the chip and POOL_OUT_BYTES
// (or one sample of every pixel) ask for.
struct PoolPlan {
    uint32_t blocks, slots;
    uint32_t spp;       // samples a launch (the last may have fewer)
    size_t state, out;  // bytes
};

inline PoolPlan pool_plan(uint32_t count, uint32_t spp, uint32_t blocks, uint32_t most, size_t slot_bytes,
                          size_t sample_bytes) {
    const size_t sample = (size_t)count * sample_bytes;
    const uint32_t fit = (uint32_t)std::min<size_t>(std::max<size_t>(POOL_OUT_BYTES / sample, 1), spp);
    const uint32_t launches = (uint32_t)(((uint64_t)spp + fit - 1) / fit);
    PoolPlan p;
    p.spp = (uint32_t)(((uint64_t)spp + launches - 1) / launches);
    p.blocks = blocks;
    p.slots = pool_slots((uint64_t)count * p.spp, blocks, most);
    p.state = (size_t)blocks * p.slots * slot_bytes;
    p.out = sample * p.spp;
    return p;
}

// Slots a block of a launch of `spp` of the samples (the last may have few).
inline uint32_t launch_slots(const PoolPlan& p, uint32_t count, uint32_t spp, uint32_t most) {
    return std::min(p.slots, pool_slots((uint64_t)count * spp, p.blocks, most));
}

// ---- a batch's launches scene by scene, on side streams ----

struct LaneJob {
    uint64_t work;      // its samples
    bool pooled;        // it runs on the pooled render, whose buffers these are
    size_t state, out;  // bytes
};

struct LanePlan {
    std::vector<uint32_t> order, lane;  // jobs, the largest first; the lane of each job
    std::vector<uint8_t> buffers;       // job: the lane's buffers hold it (else it runs without)
};

// Jobs in order of their work, each on the lane with the least so far. A lane's
// buffers are reserved once, by reserve(lane, state, out), for the largest need
// of its pooled jobs; no buffer changes hands or size after that, since the
// memory is ordered on the context's stream and the jobs run beside it. The
// jobs of a lane without buffers run on a megakernel.
template <class Reserve>
LanePlan plan_lanes(const std::vector<LaneJob>& jobs, uint32_t lanes, const Reserve& reserve) {
    LanePlan p;
    p.order.resize(jobs.size());
    std::iota(p.order.begin(), p.order.end(), 0u);
    std::stable_sort(p.order.begin(), p.order.end(), [&](uint32_t x, uint32_t y) { return jobs[x].work > jobs[y].work; });
    p.lane.resize(jobs.size());
    p.buffers.assign(jobs.size(), 0);
    std::vector<uint64_t> load(lanes, 0);
    for (uint32_t j : p.order) {
        p.lane[j] = (uint32_t)(std::min_element(load.begin(), load.end()) - load.begin());
        load[p.lane[j]] += jobs[j].work;
    }
    for (uint32_t l = 0; l < lanes; l++) {
        size_t state = 0, out = 0;
        for (uint32_t j : p.order)
            if (p.lane[j] == l && jobs[j].pooled) {
                state = std::max(state, jobs[j].state);
                out = std::max(out, jobs[j].out);
            }
        if (!state || !reserve(l, state, out)) continue;
        for (uint32_t j : p.order)
            if (p.lane[j] == l) p.buffers[j] = jobs[j].pooled;
    }
    return p;
}

}  // namespace phx
