// Whether a level runs inside the launch of small levels (fused_levels.cuh): the sizes the count stage
// found against what the launch has room for. Compiled for the host too (tests/native).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define HGX_RULE __host__ __device__ inline
#else
#define HGX_RULE inline
#endif

namespace hgx {

constexpr uint32_t kFusedEvents = 16384;    // most events of a level (a thread per event, 148 blocks)
// Most matches of a state that are enumerated one after another (a rule of more than four left-hand
// edges): a level that is left for having more has been counted in vain (0.8 us a match on states of
// 100 edges, 18 ms in front of the ordinary level's 107 when it was counted to the end).
constexpr uint32_t kFusedJoin = 512;
constexpr uint32_t kFusedEdges = 255;       // largest state record a level may produce
// Most branchial pairs to make room for ahead of a level. The launch has no count of them before it
// writes them, only the bound c (c - 1) / 2 of every state with c matches: 64 MB at this limit (one state
// of 4,096 matches), 1 GB for one of 16,384, of which the ordinary level, which counts first, needs a few
// percent. (At 8 MB a batch of 23 evolutions lost a level to the ordinary pipeline: 4.83 -> 5.04 ms.)
constexpr uint64_t kFusedPairs = 1u << 23;
constexpr uint64_t kIdLimit = 0xFFFFFFF0ull;   // 32-bit ids end here

// Why a level was left to the ordinary pipeline.
enum FusedStop : uint32_t {
    kStopDone = 0,          // no frontier left, or the level count asked for
    kStopRoom = 1,          // an array has no room: grow and come back
    kStopLevel = 2,         // too many events, items or pairs, a cap that can bind, ids that run out
    kStopTable = 3,         // a dedup table would pass half full
    kStopLayout = 4,        // a state's shared-memory region does not fit
};

// Events, consumed entries, edges, vertices, pairs (branchial; a bound) and record words (a bound):
// of the run so far, of the level at most, and what the arrays hold.
struct FusedSizes {
    uint64_t events, states, cons, edges, vertices, pairs, arena;
};

// Ids that run out come before room: an array may hold more than 2^32 elements (it grows by half), and
// the ordinary level reports them as an error.
HGX_RULE uint32_t fused_decide(const FusedSizes& have, const FusedSizes& level, const FusedSizes& room,
                               uint64_t room_front, uint64_t largest_record, bool branchial) {
    if (level.events > kFusedEvents || largest_record > kFusedEdges) return kStopLevel;
    if (branchial && level.pairs > kFusedPairs) return kStopLevel;
    if (have.events + level.events >= kIdLimit || have.states + level.events >= kIdLimit ||
        have.cons + level.cons >= kIdLimit || have.edges + level.edges >= kIdLimit ||
        have.vertices + level.vertices >= kIdLimit || (branchial && have.pairs + level.pairs >= kIdLimit))
        return kStopLevel;
    if (have.events + level.events > room.events || have.states + level.events > room.states ||
        have.cons + level.cons > room.cons || have.edges + level.edges > room.edges ||
        (branchial && have.pairs + level.pairs > room.pairs) || have.arena + level.arena > room.arena ||
        level.events > room_front)
        return kStopRoom;
    return kStopDone;
}

}  // namespace hgx
