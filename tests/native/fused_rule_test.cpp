// Which levels run inside the launch of small levels (csrc/fused_rule.cuh): ids and array room.
#include <cstdio>

#include "hypergraphrewritingengine_b200/csrc/fused_rule.cuh"

using namespace hgx;

static int bad = 0;
static void expect(const char* what, uint32_t got, uint32_t want) {
    if (got != want) { std::printf("%s: %u, not %u\n", what, got, want); ++bad; }
}

int main() {
    const uint64_t big = 1ull << 34;   // arrays of more than 2^32 elements
    const FusedSizes none{}, level{100, 100, 200, 300, 100, 1000, 5000}, room{big, big, big, big, big, big, big};
    auto decide = [&](const FusedSizes& have, const FusedSizes& lv, const FusedSizes& r, uint64_t front = 1 << 20,
                      uint64_t record = 10, bool branchial = true) {
        return fused_decide(have, lv, r, front, record, branchial);
    };
    expect("fits", decide(none, level, room), kStopDone);
    // every counter at the last id it may reach, and one past it, whatever the arrays hold
    uint64_t FusedSizes::* const ids[] = {&FusedSizes::events, &FusedSizes::states, &FusedSizes::cons,
                                          &FusedSizes::edges, &FusedSizes::vertices, &FusedSizes::pairs};
    for (auto f : ids) {
        FusedSizes have{};
        const uint64_t add = f == &FusedSizes::states ? level.events : level.*f;
        have.*f = 0xFFFFFFF0ull - add - 1;
        expect("last ids", decide(have, level, room), kStopDone);
        have.*f += 1;
        expect("ids out", decide(have, level, room), kStopLevel);
        have.*f = 0xFFFFFFF0ull;   // (past 2^32 with the level's own)
        expect("ids past 2^32", decide(have, level, room), kStopLevel);
        FusedSizes tight = room;   // ids before room: the arrays are not grown for such a level
        tight.*f = 10;
        expect("ids before room", decide(have, level, tight), kStopLevel);
    }
    // room
    uint64_t FusedSizes::* const arrays[] = {&FusedSizes::events, &FusedSizes::states, &FusedSizes::cons,
                                             &FusedSizes::edges, &FusedSizes::pairs, &FusedSizes::arena};
    for (auto f : arrays) {
        FusedSizes r = room;
        r.*f = f == &FusedSizes::states ? level.events : level.*f;
        expect("just room", decide(none, level, r), kStopDone);
        r.*f -= 1;
        expect("no room", decide(none, level, r), kStopRoom);
    }
    expect("no room for pairs that are not kept", decide(none, level, {big, big, big, big, big, 0, big}, 1 << 20, 10, false),
           kStopDone);
    expect("frontier", decide(none, level, room, 99), kStopRoom);
    // the level's own limits
    FusedSizes wide = level;
    wide.events = wide.states = kFusedEvents;
    expect("most events", decide(none, wide, room), kStopDone);
    wide.events = wide.states = kFusedEvents + 1;
    expect("too many events", decide(none, wide, room), kStopLevel);
    expect("largest record", decide(none, level, room, 1 << 20, kFusedEdges), kStopDone);
    expect("record too large", decide(none, level, room, 1 << 20, kFusedEdges + 1), kStopLevel);
    wide = level;
    wide.pairs = kFusedPairs;
    expect("most pairs", decide(none, wide, room), kStopDone);
    wide.pairs = kFusedPairs + 1;
    expect("too many pairs", decide(none, wide, room), kStopLevel);
    expect("too many pairs before room", decide(none, wide, {big, big, big, big, big, 10, big}), kStopLevel);
    expect("pairs that are not kept", decide(none, wide, room, 1 << 20, 10, false), kStopDone);
    std::printf("%d wrong\n", bad);
    return bad != 0;
}
