// Bookkeeping of the operator's stage ring: which slot the next stage goes to and
// which phase of the slot's barriers belongs to a stage.  Slot and round of the
// ring are counted side by side, not derived from the stage's number: the number
// of stages passes 2^32 in a long launch (an hour of a 12,813-patch network), and
// 2^32 is no multiple of kStages.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define QDFN_RING_HD __host__ __device__ __forceinline__
#else
#define QDFN_RING_HD inline
#endif

namespace qdfn {

constexpr int kStages = 5;
constexpr uint64_t kNoStage = ~0ull;

// a place in the ring; round wraps harmlessly, its lowest bit is the barriers' phase
struct RingPos {
    uint32_t slot = 0, round = 0;
    QDFN_RING_HD uint32_t phase() const { return round & 1u; }
    QDFN_RING_HD void next() {
        if (++slot == (uint32_t)kStages) { slot = 0; ++round; }
    }
    QDFN_RING_HD void back() {
        if (slot == 0) { slot = kStages; --round; }
        --slot;
    }
};

// the producer's side
struct RingFill {
    uint64_t filled = 0;                          // stages filled
    RingPos at;                                   // where the next one goes
    uint64_t last[2] = {kNoStage, kNoStage};      // last stage of the latest tile on each x buffer
    RingPos last_at[2];
    // the next stage's slot has held another one (with the phase before)
    QDFN_RING_HD bool reused() const { return filled >= (uint64_t)kStages; }
    // the x buffer's last stage may not be released yet: it was within kStages
    QDFN_RING_HD bool x_in_use(int xb) const { return last[xb] != kNoStage && last[xb] + kStages > filled; }
    QDFN_RING_HD void mark_last(int xb) { last[xb] = filled; last_at[xb] = at; }
    QDFN_RING_HD void advance() { ++filled; at.next(); }
};

}  // namespace qdfn
