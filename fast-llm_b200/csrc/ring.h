// Walk through a ring of shared-memory stages that G consumer groups empty in turn (stage i is group i % G's).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define FLB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FLB_HOST_DEVICE inline
#endif

namespace flb {

// The next stage of the group whose last one lay in `slot`: group g has the slots g, g + G, .. below n for itself. A wait on a barrier's
// parity tells a use from the one before it only, so that whoever waits must have seen the one before: with slots that pass from
// group to group (n no multiple of G), a group whose stages all landed could come to a slot whose last stage, another group's,
// had not, pass the wait, and hand the slot back to a producer that then armed a barrier still pending.
template <int G>
FLB_HOST_DEVICE void ring_next(uint32_t &slot, uint32_t &par, uint32_t n) {
    static_assert((G & (G - 1)) == 0, "groups");
    slot += G;
    if (slot >= n) { slot &= G - 1; par ^= 1u; }
}

// The producer's walk: the groups' next slots in turn.
template <int G>
struct RingTurn {
    uint32_t slot[G], par[G];
    FLB_HOST_DEVICE RingTurn() {
        for (int g = 0; g < G; ++g) { slot[g] = g; par[g] = 1; }   // a fresh barrier passes a wait on parity 1
    }
    FLB_HOST_DEVICE void next(uint32_t n) {
        uint32_t s = slot[0], p = par[0];
        ring_next<G>(s, p, n);
        for (int g = 0; g + 1 < G; ++g) { slot[g] = slot[g + 1]; par[g] = par[g + 1]; }
        slot[G - 1] = s; par[G - 1] = p;
    }
};

} // namespace flb
