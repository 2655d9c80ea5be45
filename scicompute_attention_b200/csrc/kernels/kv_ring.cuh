// The protocol of the K/V ring of the prefill kernel: the order of the loads and the barriers that say a tile has landed.
// Plain C++, so that the host tests run the same lines.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SCA_RING_FN __host__ __device__ __forceinline__
#else
#define SCA_RING_FN inline
#endif

namespace sca_b200 {

// The ring of a padded head dim: how many slots it has, whether the scores of a tile go out ahead of the products of the one
// before (see kOwnP in flash_kernel.cuh), how many slots a K or V tile takes, and how many warps rewrite V (bf16; none for fp16).
struct RingShape {
    int slots;
    bool scores_ahead;
    int parts;
    int converters;
};
constexpr RingShape RingOf(int padded_dim) {
    return padded_dim == 64 ? RingShape{8, true, 1, 2} : padded_dim == 128 ? RingShape{5, false, 1, 2} : RingShape{5, true, 2, 4};
}

struct RingLoad {
    bool is_v;
    int tile;
};
// The it-th of the 2 * n loads of an item of n KV tiles, in the order in which the products consume them:
// K_0 V_0 K_1 V_1 ..., or with the scores ahead K_0 K_1 V_0 K_2 V_1 K_3 ... (S(j+1) does not wait for P(j) V_j).
SCA_RING_FN RingLoad RingOrder(int it, int n, bool scores_ahead) {
    if (!scores_ahead) return {(it & 1) != 0, it >> 1};
    const int lead = n > 1 ? 2 : 1;
    if (it < lead) return {false, it};
    const int f = it - lead, rest = n - lead;  // `rest` K tiles still to come, one after each V
    if (f >= 2 * rest) return {true, f - rest};
    return (f & 1) == 0 ? RingLoad{true, f >> 1} : RingLoad{false, (f >> 1) + 2};
}

// Index of the barrier (of 2 * slots) that a load into `slot` completes. With an odd number of slots a slot holds K and V
// in turn, and a wait on an mbarrier tells two neighbouring phases apart, no more: a role that waits on a barrier has to
// see each of its phases. The warps that rewrite V see V tiles only and the products of a rewritten V wait for those
// warps, so K and V have barriers of their own. On a common one the wait for V in a slot returns at once while the K
// before it is still on its way, and waiting for the K tiles too does not help: the products free a K tile without those
// warps, V follows into its slot, and a warp that comes late waits for a phase that is already over.
SCA_RING_FN int RingFullBarrier(bool is_v, int slot, int slots) { return (is_v ? slots : 0) + slot; }

// Parity of the next phase of each slot's barrier, as seen by one role that waits for every phase in turn.
struct RingPhases {
    uint32_t bits = 0;
    SCA_RING_FN uint32_t Take(uint32_t slot) {
        const uint32_t parity = (bits >> slot) & 1u;
        bits ^= 1u << slot;
        return parity;
    }
};

}  // namespace sca_b200
