// Grouped products on pairs of SMs (experts_sm100_pair.cu): what they read and write.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

struct omoe_handle;

namespace omoe {

enum class PairKind {
    kUpGate,      // o0 = silu(b * Wg^T) * (b * Wu^T)
    kUpGateKeep,  // the same, and o1 = b * Wg^T, o2 = b * Wu^T
    kPlain,       // o0 = b * W^T, W [n_out, K] per expert
    kSwigluBack,  // with dh = b * W, W [K, n_out] per expert, and g, u from s0, s1: o0 = (dh * u) * silu'(g), o1 = dh * silu(g)
    kPlainMN2,    // o0 = b0 * W0 + b1 * W1, both W [K, n_out] per expert
};

// Weights a*, rows b* (boxes of 128 and of 32 rows), results o* and rows s* that the epilogue
// reads (boxes of 32 rows); all bf16 with the 128-byte swizzle.
struct alignas(64) PairMaps {
    CUtensorMap a0, a1, b0, b0_32, b1, b1_32, o0, o1, o2, s0, s1;
};

// Rows [0, round_up(count, row_round)) of every local expert's segment are written, row_round 32 or 64: 64 where a
// product that reduces over the rows in blocks of 64 follows.
cudaError_t launch_pair(omoe_handle *h, cudaStream_t s, bool pdl, PairKind kind, const PairMaps &maps, int n_out, int K,
                        int row_round);

// bf16 (or, with f32, fp32) tensor map with the 128-byte swizzle: dims and box innermost first, strides of dims 1.. in
// elements.
bool encode_map_nd(CUtensorMap *m, void *ptr, int rank, const uint64_t *dims, const uint64_t *strides, const uint32_t *box,
                   bool f32 = false);

}  // namespace omoe
