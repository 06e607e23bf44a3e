// The SAH build's subtree kernels (phiray_b200/csrc/sah_subtree.cuh) over one
// seed, the whole tree, on the host: a warp's lanes as threads.
#include "warp_shim.h"

#include "../phiray_b200/csrc/sah_subtree.cuh"

extern "C" uint32_t warp_build_sah(const float* prims, uint32_t n, uint32_t leaf, uint32_t vec, float* nodes,
                                   uint32_t* order, uint32_t* depth) {
    using namespace phx;
    std::vector<float> centres(3 * (size_t)n);
    for (uint32_t i = 0; i < n; i++) {
        for (int k = 0; k < 3; k++) centres[3 * (size_t)i + k] = 0.5f * (prims[8 * (size_t)i + k] + prims[8 * (size_t)i + 4 + k]);
        order[i] = i;
    }
    const uint32_t seed = 0;
    const sah::TNode root{0, n, 0, sah::NONE, sah::NONE};
    std::vector<uint4> loc(2 * n);
    uint32_t count = 0, inner = 0, rank = 0, final_index = 0;
    sah::Box box;
    *depth = 0;
    run_warp([&] {
        k_sah_subtree(&seed, 1, &root, prims, centres.data(), order, leaf, loc.data(), &count, &inner, depth, vec != 0);
    });
    run_warp([&] {
        k_sah_subtree_emit(&seed, 1, &root, loc.data(), &count, &rank, &final_index, prims, order, &box, nodes, vec != 0);
    });
    return 2 * inner + 1;
}

extern "C" uint32_t warp_open_nodes(uint32_t n) { return phx::open_nodes(n); }
