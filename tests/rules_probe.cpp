// A host build of the library's path decisions (phiray_b200/csrc/rules.cuh) and
// of a kernel's index arithmetic (conv_index.cuh).
#include "../phiray_b200/csrc/conv_index.cuh"
#include "../phiray_b200/csrc/rules.cuh"

extern "C" int probe_aligned16(const void* p) { return phx::aligned16(p) ? 1 : 0; }

extern "C" uint32_t probe_autotuned(const float* ms, uint32_t fastest) { return phx::autotuned(ms, fastest); }

extern "C" uint32_t probe_fastest_megakernel(const float* ms) { return phx::fastest_megakernel(ms); }

// The id of the kernel that traces a frame, and (bit 31) whether it needs the
// pooled render's buffers. flags: full, adaptive, transmits, capturing.
extern "C" uint32_t probe_frame_kernel(uint32_t kernel, uint32_t mega, uint32_t flags, uint32_t pixels, uint32_t spp,
                                       uint32_t faces) {
    const phx::FrameForm f{kernel, mega, (flags & 1u) != 0, (flags & 2u) != 0, (flags & 4u) != 0, (flags & 8u) != 0,
                           pixels, spp, faces};
    return phx::frame_kernel(f) | (phx::frame_pooled(f) ? 0x80000000u : 0u);
}

// plan_lanes over n jobs of (work, pooled, state, out); the reserve calls are
// written to calls as (lane, state, out), and call `fails` (from 0) fails.
// Returns the number of calls.
extern "C" uint32_t probe_lanes(const uint64_t* jobs, uint32_t n, uint32_t lanes, uint32_t fails, uint64_t* calls,
                                uint32_t* order, uint32_t* lane, uint8_t* buffers) {
    std::vector<phx::LaneJob> in;
    for (uint32_t j = 0; j < n; j++)
        in.push_back({jobs[4 * j], jobs[4 * j + 1] != 0, (size_t)jobs[4 * j + 2], (size_t)jobs[4 * j + 3]});
    uint32_t made = 0;
    const phx::LanePlan p = phx::plan_lanes(in, lanes, [&](uint32_t l, size_t state, size_t out) {
        calls[3 * made] = l;
        calls[3 * made + 1] = state;
        calls[3 * made + 2] = out;
        return made++ != fails;
    });
    std::copy(p.order.begin(), p.order.end(), order);
    std::copy(p.lane.begin(), p.lane.end(), lane);
    std::copy(p.buffers.begin(), p.buffers.end(), buffers);
    return made;
}

// pool_plan as (blocks, slots, spp, state, out), and the slots of its launch of
// `now` samples.
extern "C" uint32_t probe_pool_plan(uint32_t count, uint32_t spp, uint32_t blocks, uint32_t most, uint32_t now,
                                    uint64_t* plan) {
    const phx::PoolPlan p = phx::pool_plan(count, spp, blocks, most, 244, 40);
    plan[0] = p.blocks;
    plan[1] = p.slots;
    plan[2] = p.spp;
    plan[3] = p.state;
    plan[4] = p.out;
    return phx::launch_slots(p, count, now, most);
}

// A patch vector as (pixel, shared bytes, channel, row, column).
extern "C" void probe_patch_vec(int v, int groups, int px, int lbo, int width, int64_t* out) {
    const phx::PatchVec p(v, groups, px, lbo, width);
    out[0] = p.pixel;
    out[1] = p.shared_bytes();
    out[2] = p.channel();
    out[3] = p.row();
    out[4] = p.column();
}
