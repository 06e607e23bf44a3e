// Internal declarations shared by the phiray-b200 CUDA sources: the context,
// buffers, error reporting and the device helpers every kernel file uses.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstdarg>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/phiray_cuda.h"

namespace phx {

// Status word bits a kernel sets instead of trapping (read on the host at the
// next wait): a bounded spin ran out, or an input index was out of range.
enum : uint32_t {
    STATUS_SPIN_LIMIT = 1u << 0,
    STATUS_BAD_INDEX = 1u << 1,
    STATUS_STACK_OVERFLOW = 1u << 2,
};

struct Ctx;

// A growable device allocation. Reserved inside a context's call (after
// use()), it comes from the context's stream-ordered pool on the context's
// stream, and its release is a free ordered on that stream: the pool keeps
// the memory mapped, so the next object of the context reuses it without a
// cudaMalloc/cudaFree round trip through the driver. Otherwise cudaMalloc.
struct DevMem {
    void* ptr = nullptr;
    size_t bytes = 0;
    Ctx* owner = nullptr;          // the context whose pool holds ptr, or null
    int32_t reserve(size_t want);  // grows, discarding contents
    void release();
    ~DevMem() { release(); }
};

// The pooled render's path states and sample terms (render_pool.cuh).
struct PoolScratch {
    DevMem state, out;
};

struct Ctx {
    int device = 0;
    int sms = 148;
    cudaStream_t own = nullptr;     // created by phx_ctx_create
    cudaStream_t stream = nullptr;  // where work goes (own, or a caller's)
    cudaStream_t capture = nullptr; // private stream for graph capture
    uint32_t* status = nullptr;     // device status word
    cudaMemPool_t pool = nullptr;   // device memory of the context's objects
    DevMem denoise_scratch;         // guide and ping-pong planes of phx_denoise
    PoolScratch path_pool;          // the pooled render's buffers
    std::mutex path_pool_lock;      // from sizing them to the launches that use them (PathPoolHold)
    int live = 0;                   // buffers, passes, BVHs, tracers not yet freed
};

// The context's pooled buffers, held by this thread while it sizes them and
// launches what uses them. An allocation that finds no memory gives them back,
// but not those made under the hold.
class PathPoolHold {
    std::lock_guard<std::mutex> lock_;

public:
    explicit PathPoolHold(Ctx* c);
    ~PathPoolHold();
};

// Sets the thread's last error text and returns `code`.
int32_t fail(int32_t code, const char* fmt, ...);
// Maps a CUDA error to PHX_ERR_*, with context text; PHX_OK on success.
int32_t cuda_check(cudaError_t e, const char* what);
// Reads and clears the context's status word (synchronous), mapping set bits
// to PHX_ERR_KERNEL.
int32_t read_status(Ctx* c);
// Bounded drain of `stream` (polls an event with a deadline).
int32_t wait_stream(cudaStream_t s, uint32_t timeout_ms);
// Ensures ctx's device is current on this thread and makes ctx the one whose
// pool this thread's DevMem reservations draw on.
int32_t use(Ctx* c);
// Device allocation from the context's pool, ordered on its stream (cudaMalloc
// when the context has no pool); the matching free.
int32_t ctx_alloc(Ctx* c, void** p, size_t bytes);
void ctx_free(Ctx* c, void* p);

// Kernel launches the Pass layer replays (one per phx_kernel_id), defined in
// the kernel files. `params` is the step's params blob, `bufs` its buffers.
int32_t launch_skin_step(cudaStream_t s, const void* params, void* const* bufs, const uint64_t* sizes, uint32_t items,
                         uint32_t* status);
int32_t launch_denoise_step(cudaStream_t s, const void* params, void* const* bufs, uint32_t items);
int32_t launch_morton_step(cudaStream_t s, const void* params, void* const* bufs, uint32_t items);
int32_t launch_karras_step(cudaStream_t s, const void* params, void* const* bufs, uint32_t items);
int32_t launch_refit_step(cudaStream_t s, const void* params, void* const* bufs, uint32_t items);

// Face boxes (Aabb::of_tri) of vec4 vertices over uvec4 faces (skin.cu).
int32_t launch_face_boxes(cudaStream_t s, const float* verts, const uint32_t* faces, uint32_t nfaces, phx_aabb* boxes);

// Y = relu(conv3x3(X, W) + bias) (phx_nn_conv_fwd's arguments); with `below`,
// the input's first `up` channels are the nearest upsampling of that half-size
// tensor and X holds the others from xo on; with `pool`, the output's 2 x 2
// average goes there too (nn.cu).
int32_t nn_conv_relu(Ctx* c, const void* X, int xs, int xo, int cin, const void* W, int Kp, const float* bias, void* Y,
                     int ys, int yo, int cout, int B, int H, int Wd, const void* below, int up, void* pool);
// The weight and bias gradients of one 3x3 convolution, added to dWt
// ([9 cin][cout]) and db ([cout]) (nn.cu).
int32_t nn_conv_grads(Ctx* c, const void* X, int xs, int xo, int cin, const void* dY, int dys, int dyo, int cout,
                      float* dWt, float* db, int B, int H, int W);

// One layer of an Adam step over a whole network (nn.cu k_adam_net): weights
// [rows][Kp] with their moments, gradient [Kp][rows], bf16 copy and flipped
// copy (null: none), and the bias. rows and Kp are multiples of 32.
struct AdamLayer {
    float *w, *m, *v;
    const float* g;
    void *wb, *w2;
    float *b, *mb, *vb;
    const float* gb;
    int rows, Kp, K, cin, Kp2, block0;
};
struct AdamNet {
    AdamLayer l[20];
    int layers;
    float lr, b1, b2, eps, c1, c2;
};
int32_t nn_adam_net(Ctx* c, AdamNet& net);

inline uint32_t ceil_div(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

}  // namespace phx

struct phx_ctx_s {
    phx::Ctx c;
};

struct phx_buf_s {
    phx::Ctx* ctx = nullptr;
    void* ptr = nullptr;
    uint64_t bytes = 0;
    bool owned = false;
};

#define PHX_TRY(expr)                   \
    do {                                \
        int32_t _rc = (expr);           \
        if (_rc < 0) return _rc;        \
    } while (0)

#define PHX_CUDA(expr) PHX_TRY(phx::cuda_check((expr), #expr))

namespace phx {

// Raises a kernel's dynamic shared-memory limit (and carveout) once per device.
template <typename F>
int32_t smem_limit(F* kernel, int bytes, int device, std::atomic<uint64_t>& done) {
    const uint64_t bit = 1ull << (device & 63);
    if (done.load(std::memory_order_acquire) & bit) return PHX_OK;
    PHX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    // the largest shared-memory carveout, so that several blocks fit an SM
    PHX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    done.fetch_or(bit, std::memory_order_release);
    return PHX_OK;
}

}  // namespace phx
