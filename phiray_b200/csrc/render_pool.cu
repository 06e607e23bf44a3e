// Single-instance render kernels, ids 1-3: the pooled render, blocks of 512,
// 256 and 128 threads (1,024 resident threads an SM, 64 registers each).
#include "render_pool.cuh"

namespace phx {
namespace {

// f(kernel form) of a kernel id.
template <class F>
int32_t with_form(uint32_t kernel, bool stats, const F& f) {
    switch (kernel) {
        case PHX_KERNEL_STATE_MACHINE_6: return stats ? f(PoolForm<MODE_STATS, 4, 2048, 256>{}) : f(PoolForm<0, 4, 2048, 256>{});
        case PHX_KERNEL_STATE_MACHINE_8: return stats ? f(PoolForm<MODE_STATS, 8, 1024, 128>{}) : f(PoolForm<0, 8, 1024, 128>{});
        default: return stats ? f(PoolForm<MODE_STATS, 2, 4096, 512>{}) : f(PoolForm<0, 2, 4096, 512>{});
    }
}

}  // namespace

int32_t plan_pooled(uint32_t kernel, bool stats, int sms, uint32_t count, uint32_t spp, PoolPlan& plan) {
    return with_form(kernel, stats, [&](auto form) { return form.plan(sms, count, spp, plan); });
}

int32_t render_pooled(uint32_t kernel, bool stats, const RenderLaunch& L, const PoolPlan& plan, void* state, void* out) {
    return with_form(kernel, stats, [&](auto form) { return form.launch(L, plan, (uint32_t*)state, (uint32_t*)out); });
}

}  // namespace phx
