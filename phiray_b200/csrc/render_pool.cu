// Single-instance render kernels, ids 1-3: the pooled render, blocks of 512,
// 256 and 128 threads (1,024 resident threads an SM, 64 registers each).
#include "render_pool.cuh"

namespace phx {

size_t pool_slot_bytes() { return (size_t)PW_WORDS * 4; }

uint32_t pool_out_words() { return PO_WORDS; }

int32_t render_pooled(uint32_t kernel, bool stats, const RenderLaunch& L, const PoolBuffers& B) {
    switch (kernel) {
        case PHX_KERNEL_STATE_MACHINE_6: return stats ? launch_pool<MODE_STATS, 4, 2048, 256>(L, B) : launch_pool<0, 4, 2048, 256>(L, B);
        case PHX_KERNEL_STATE_MACHINE_8: return stats ? launch_pool<MODE_STATS, 8, 1024, 128>(L, B) : launch_pool<0, 8, 1024, 128>(L, B);
        default: return stats ? launch_pool<MODE_STATS, 2, 4096, 512>(L, B) : launch_pool<0, 2, 4096, 512>(L, B);
    }
}

}  // namespace phx
