// Small levels of a run in one cooperative launch (included by engine.cu after make_layout).
//
// The level pipeline of engine.cu spends 20-25 launches and two host synchronisations on a level,
// which is 120-200 us however few events the level has. Here one block per SM keeps going from
// level to level on its own: the frontier, the id counters and every size stay on the device, the
// host is told about all levels at once when the launch ends. A level is five stages between four
// grid barriers:
//
//   count       warp per frontier state: matches and id-range sizes per (state, rule)
//   barrier 1   the last block to arrive scans the sizes and decides whether the level fits
//   expand      warp per run of consecutive events: child, WL hash, event record, table insert
//   barrier 2
//   select      thread per event: producers, first arrival, branchial partners; block totals
//   barrier 3
//   assign      thread per event: ids from the totals of the blocks before; pairs, records
//   barrier 4
//   output      thread per event: the class representative's id (then the next level's count)
//
// What bounds it is latency: dependent loads, first fetches of instructions and barriers (1.5-2 us each),
// not bytes or issue slots (5 % of them used; of 77 warps waiting per issue 61 stand at a barrier).
// So every stage spreads over the whole grid (one event per thread, children dealt to warps in equal
// runs whatever their parents), and children are hashed one per warp: a lane needs 30-50 us for its
// child, a warp 3-5 us. That stops paying once the children outnumber the warps several times;
// levels of more than kFusedEvents events, and anything the capacities at hand do not cover, leave
// the launch before their first write and are run by the ordinary pipeline.
//
// Same ids, same order, same arithmetic as the ordinary pipeline: results are identical.
//
// Measured per call (B200), ordinary pipeline -> this launch: C1 of two steps 358 -> 202 us, C1 (its
// last level, 20,739 events, is left to the ordinary pipeline) 1,011 -> 685 us, two rules with
// transitive reduction and signatures over five full levels 1,275 -> 539 us, C3 at six levels 5.43 ->
// 4.59 ms, 32 requests evolved one per call 19.2 -> 14.1 ms (the last two when it was introduced).
// Raising the event limit to 32,768 changed none of these.
#pragma once

constexpr uint32_t kFusedThreads = 512, kFusedWarps = kFusedThreads / 32;
constexpr uint32_t kFusedItems = 8192;      // most (state, rule) items of a level: one block scans them
constexpr uint32_t kFusedLevels = 16;       // most levels of a launch (records in mapped memory)
constexpr uint32_t kFusedSlice = kListMax;  // most events a warp builds in one run
static_assert(kFusedEvents <= kNumSMs * kFusedThreads, "one event per thread");
constexpr uint32_t kRangeWords = 10;        // per level and evolution: see k_levels
constexpr uint32_t kLevelWords = 8;         // per level: F, events, states, frontier, pairs, max ne / nocc

// Grid-wide words of the launch (zero between launches: the last block to leave clears them).
struct FusedState {
    uint32_t arrived, gen, abort, stop;
    uint32_t max_ne[2], max_no[2], max_nv[2];      // frontier maxima, by level parity
    unsigned long long pairs[2];                   // bound of the level's branchial pairs
    uint32_t n_ev, n_cons, n_prod, n_fresh;        // the level's totals (barrier 1)
};

struct FusedArgs {
    FusedState* fs;
    uint32_t* front[2];         // this level's and the next one's frontier
    uint32_t *cnt, *item_ev, *item_cons, *item_prod, *item_fresh;   // per item
    uint32_t* new_event;        // event of each new state of the level
    uint32_t* sums;             // [3][blocks] new states, next frontier, pairs
    uint32_t* bpairs;
    uint32_t* evo_last;         // per evolution: one past its last event of the level
    uint32_t* out;              // mapped: header, level records, ranges
    FusedSizes room;            // array sizes
    uint64_t arena_words;       // bound of the arena's bump pointer
    uint64_t n_pairs;
    uint32_t room_front;
    uint32_t n_states, n_events, n_edges, n_cons, next_vertex;      // totals so far
    uint32_t F, stride, nevo, levels, ne_bound, no_bound, smem;
    uint32_t ev_keys, tr, branchial, index;
    uint32_t hasty;             // barrier given up after one look, kNone: none
    RuleMax rm;
};

// Words of the mapped report: [0] stop, [1] levels done, [2] which frontier, [3] device errors,
// [4..5] classes, [6..7] states, [8] stopped (evolution 0), [9..13] what the level it stopped at
// needs, [14..15] consumed entries, [16] edges, [17] vertices used by the levels done.
constexpr uint32_t kReportWords = 32;

// Grid barrier of a cooperative launch; the last block to arrive runs `serial` before the others are
// released. gen counts the barriers passed. Returns false when a wait ran out: the waiter then closes
// the barrier for everyone -- release and closing are one compare-and-swap on the same word, so either
// all blocks pass it or all leave, the late ones included. The closed word keeps the count below it: a
// block still waiting at an earlier barrier sees that it was released, finishes its part of that level
// and leaves where the others do. Up to the end of the expansion nothing of a level counts yet (its
// table inserts repeat themselves with the same ids), so a level whose joins or hashes take one block
// longer than the wait is simply run again by the ordinary pipeline; later it is an error (`hard`).
// `hasty`: the barrier (of the launch, from 0) that is given up after one look (for tests).
constexpr uint32_t kBarrierClosed = 1u << 31;

template <class F>
__device__ bool fused_barrier(FusedState* fs, uint32_t& phase, uint32_t* err, bool hard, uint32_t hasty, F&& serial) {
    __shared__ uint32_t sh_last, sh_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        sh_last = atomicAdd(&fs->arrived, 1u) + 1 == (phase + 1) * gridDim.x ? 1u : 0u;
        sh_ok = 1;
    }
    __syncthreads();
    if (sh_last) {
        if (threadIdx.x == 0) __threadfence();
        __syncthreads();
        serial();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            sh_ok = atomicCAS(&fs->gen, phase, phase + 1) == phase ? 1u : 0u;
        }
    } else if (threadIdx.x == 0) {
        uint32_t g = phase;
        const uint32_t looks = phase == hasty ? 1u : 1u << 22;   // about two seconds
        for (uint32_t it = 0; g == phase && it < looks; ++it)
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(g) : "l"(&fs->gen) : "memory");
        if (g == phase) {
            g = atomicCAS(&fs->gen, phase, phase | kBarrierClosed);
            if (g == phase && hard) atomicOr(err, kErrBarrier);
        }
        sh_ok = (g & ~kBarrierClosed) > phase ? 1u : 0u;
        __threadfence();
    }
    __syncthreads();
    ++phase;
    return sh_ok != 0;
}

// Exclusive scan of n words in place by one block, the total at a[n].
__device__ void fused_scan(uint32_t* a, uint32_t n, uint32_t* sh) {
    constexpr uint32_t kPer = 4;
    uint32_t carry = 0;
    for (uint32_t b = 0; b < n; b += kFusedThreads * kPer) {
        uint32_t v[kPer], s = 0;
        const uint32_t i0 = b + threadIdx.x * kPer;
        for (uint32_t k = 0; k < kPer; ++k) {
            v[k] = i0 + k < n ? a[i0 + k] : 0u;
            s += v[k];
        }
        uint32_t total;
        uint32_t ex = carry + block_excl_scan(s, sh, total);
        carry += total;
        for (uint32_t k = 0; k < kPer; ++k) {
            if (i0 + k < n) a[i0 + k] = ex;
            ex += v[k];
        }
    }
    if (threadIdx.x == 0) a[n] = carry;
    __syncthreads();
}

// Event a of the level against its later siblings [a + 1, end): kept events all (no cut here).
// Returns the partners; writes them as (a, c) from out on when out is given.
__device__ uint32_t fused_pairs(const DevPtrs& P, uint32_t a, uint32_t end, uint32_t in, uint2* out) {
    const unsigned long long ma = P.ev_bmask[a];
    const bool exact = P.st_ne[in] <= 63;
    const uint32_t na = P.rules[P.ev_rule[a]].n_lhs, ca = P.ev_coff[a];
    uint32_t n = 0;
    for (uint32_t c = a + 1; c < end && P.ev_in[c] == in; ++c) {
        if ((ma & P.ev_bmask[c]) == 0ull || !(exact || share_edge(P, na, P.ev_cons + ca, c))) continue;
        if (out) out[n] = make_uint2(a, c);
        ++n;
    }
    return n;
}

__global__ void __launch_bounds__(kFusedThreads, 1) k_levels(DevPtrs P, FusedArgs G) {
    extern __shared__ __align__(16) char smem[];
    __shared__ Layout L;
    __shared__ SegTables tables;
    __shared__ uint32_t sh[33], pre[3], all[3];
    seg_tables_fill(tables);
    const uint32_t tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
    const uint32_t nb = gridDim.x, b = blockIdx.x;
    FusedState* fs = G.fs;
    uint32_t phase = 0, F = G.F, cur = 0, lv = 0;
    uint32_t ne_b = G.ne_bound, no_b = G.no_bound;
    uint32_t n_states = G.n_states, n_events = G.n_events, n_edges = G.n_edges, n_cons = G.n_cons,
             next_vertex = G.next_vertex;
    uint64_t n_pairs = G.n_pairs, arena_words = G.arena_words;
    uint64_t b_stage = 0, b_hbm = 0, n_child = 0, n_rounds = 0;
    uint32_t* level_out = G.out + kReportWords;
    uint32_t* range_out = level_out + kFusedLevels * kLevelWords;
    bool alive = true;
    for (; lv < G.levels && F; ++lv) {
        const uint32_t* frontier = G.front[cur];
        const uint32_t R = G.stride, NI = F * R, par = lv & 1;
        if (uint64_t(F) * R > kFusedItems) {
            if (b == 0 && tid == 0) fs->stop = kStopLevel;
            break;
        }
        // ---- count
        if (tid == 0) L = make_layout(ne_b, no_b, G.rm, LayoutKind::Count, false, kLaneJoinCap, G.index != 0);
        __syncthreads();
        uint32_t W = min(kFusedWarps, G.smem / L.bytes);   // warps that have a region
        if (w < W) {
            char* sm = smem + w * L.bytes;
            const DevRule& Rr = *smp<DevRule>(sm, L.o_rule);
            uint32_t mne = 0, mno = 0, mnv = 0;
            unsigned long long pairs = 0;
            // warps of different blocks first: a small frontier spreads over the SMs
            for (uint32_t f = w * nb + b; f < F; f += W * nb) {
                const uint32_t sid = frontier[f];
                const Parent pa = load_parent(P, L, sm, sid);
                build_join_index(L, sm, pa);
                const unsigned long long* vm = build_vmask(L, sm, pa);
                const DevEvo ev = P.evos[P.st_evo[sid]];
                unsigned long long c_all = 0;
                for (uint32_t r = 0; r < R; ++r) {
                    uint32_t cnt = 0;
                    if (r < ev.rule_count) {
                        load_rule(sm, L, &P.rules[ev.rule_begin + r]);
                        if (Rr.n_lhs <= kLaneJoinLhs) {
                            cnt = lane_join_count(L, sm, Rr, pa, vm, nullptr, 0, 1, kFusedEvents);
                        } else {
                            warp_join(L, sm, Rr, pa, Rr.sched, -1, [&](uint32_t) { ++cnt; }, kFusedJoin + 1,
                                      SkipCounter{&cnt, kFusedJoin});
                            if (cnt > kFusedJoin) cnt = kFusedEvents + 1;   // leave the level
                        }
                        cnt = min(cnt, kFusedEvents + 1);   // (the level's sum stays within 32 bits)
                    }
                    if (lane == 0) {
                        const uint32_t t = f * R + r;
                        G.cnt[t] = cnt;
                        G.item_ev[t] = cnt;
                        G.item_cons[t] = cnt ? cnt * Rr.n_lhs : 0u;
                        G.item_prod[t] = cnt ? cnt * Rr.n_rhs : 0u;
                        G.item_fresh[t] = cnt ? cnt * Rr.n_fresh : 0u;
                    }
                    c_all += cnt;
                    __syncwarp();
                }
                pairs += c_all * (c_all - (c_all ? 1 : 0)) / 2;
                mne = max(mne, pa.ne);
                mno = max(mno, pa.nocc);
                mnv = max(mnv, P.st_nv[sid]);
            }
            if (lane == 0 && mne) {
                atomicMax(&fs->max_ne[par], mne);
                atomicMax(&fs->max_no[par], mno);
                atomicMax(&fs->max_nv[par], mnv);
                if (pairs) atomicAdd(&fs->pairs[par], pairs);
            }
        }
        // ---- barrier 1: scans, per-evolution checks, the decision
        uint32_t* ranges = range_out + uint64_t(lv) * G.nevo * kRangeWords;
        alive = fused_barrier(fs, phase, P.err, false, G.hasty, [&] {
            fused_scan(G.item_ev, NI, sh);
            fused_scan(G.item_cons, NI, sh);
            fused_scan(G.item_prod, NI, sh);
            fused_scan(G.item_fresh, NI, sh);
            const uint32_t n_ev = G.item_ev[NI];
            if (tid == 0) {
                const uint64_t mne = uint64_t(fs->max_ne[par]) + G.rm.grow_e, mno = uint64_t(fs->max_no[par]) + G.rm.grow_o;
                const uint64_t rec = mne + (mne + 3) / 4 + mno;
                const FusedSizes have{n_events, n_states, n_cons, n_edges, next_vertex, n_pairs, arena_words};
                const FusedSizes level{n_ev, n_ev, G.item_cons[NI], G.item_prod[NI], G.item_fresh[NI], fs->pairs[par],
                                       n_ev * rec};
                uint32_t stop = W == 0 ? uint32_t(kStopLayout)
                                       : fused_decide(have, level, G.room, G.room_front, mne, G.branchial != 0);
                if (!stop) {
                    const Layout Lw = make_layout(max(fs->max_ne[par], 1u), max(fs->max_no[par], 1u), G.rm,
                                                  LayoutKind::Warp, false, kLaneJoinCap, G.index != 0,
                                                  fs->max_nv[par]);
                    const uint32_t Ww = min(kFusedWarps, G.smem / Lw.bytes);
                    if (!Ww || uint64_t(Ww) * nb * kFusedSlice < n_ev) stop = kStopLayout;
                }
                fs->stop = stop;
                fs->n_ev = n_ev;
                fs->n_cons = G.item_cons[NI];
                fs->n_prod = G.item_prod[NI];
                fs->n_fresh = G.item_fresh[NI];
                // what the level needs, for the host to make room
                volatile uint32_t* o = G.out;
                o[9] = n_ev;
                o[10] = G.item_cons[NI];
                o[11] = G.item_prod[NI];
                o[12] = static_cast<uint32_t>(min(fs->pairs[par], 0xFFFFFFF0ull));
                o[13] = static_cast<uint32_t>(min(uint64_t(n_ev) * rec, uint64_t(0xFFFFFFF0ull)));
            }
            __syncthreads();
            // per evolution of the level (its frontier states are consecutive): its table must
            // take every event at half load and its cap must not be within reach
            for (uint32_t f = tid; f < F; f += kFusedThreads) {
                const uint32_t evo = P.st_evo[frontier[f]];
                if (f == 0 || P.st_evo[frontier[f - 1]] != evo) P.evo_first_ev[evo] = G.item_ev[f * R];
                if (f + 1 == F || P.st_evo[frontier[f + 1]] != evo) G.evo_last[evo] = G.item_ev[(f + 1) * R];
            }
            __syncthreads();
            if (fs->stop == kStopDone)
                for (uint32_t f = tid; f < F; f += kFusedThreads) {
                    const uint32_t evo = P.st_evo[frontier[f]];
                    if (f && P.st_evo[frontier[f - 1]] == evo) continue;
                    const DevEvo& ev = P.evos[evo];
                    const uint64_t n = G.evo_last[evo] - P.evo_first_ev[evo];
                    if (2 * (P.evo_classes[evo] + n + 1) > ev.table_mask + 1) fs->stop = kStopTable;
                    if (G.ev_keys && (!ev.sig_mask || 2 * (P.evo_sigs[evo] + n + 1) > ev.sig_mask + 1))
                        fs->stop = kStopTable;
                    const uint64_t have = ev.quotient ? P.evo_classes[evo] : P.evo_states[evo];
                    if (ev.max_states && have + n > ev.max_states) fs->stop = kStopLevel;
                    uint32_t* q = ranges + uint64_t(evo) * kRangeWords;
                    q[8] = 1;   // takes part in the level
                }
            if (tid == 0) {   // the next level's slots
                fs->max_ne[par ^ 1] = fs->max_no[par ^ 1] = fs->max_nv[par ^ 1] = 0;
                fs->pairs[par ^ 1] = 0;
            }
        });
        if (!alive || fs->stop != kStopDone) break;
        const uint32_t n_ev = fs->n_ev, ev_base = n_events, ev_end = n_events + n_ev;
        const uint32_t mne = fs->max_ne[par], mno = fs->max_no[par];
        // ---- expand: warp k of the grid builds the events [k S, (k + 1) S)
        if (tid == 0) L = make_layout(max(mne, 1u), max(mno, 1u), G.rm, LayoutKind::Warp, false, kLaneJoinCap,
                                      G.index != 0, fs->max_nv[par]);
        // the record forwarding reads at a later level, should it be switched on between steps
        for (uint32_t f = b * kFusedThreads + tid; f < F; f += nb * kFusedThreads) {
            P.st_ev0[frontier[f]] = ev_base + G.item_ev[f * R];
            P.st_evn[frontier[f]] = G.item_ev[f * R + 1] - G.item_ev[f * R];
        }
        __syncthreads();
        W = min(kFusedWarps, G.smem / L.bytes);
        const uint32_t S = max(1u, (n_ev + W * nb - 1) / (W * nb));
        const uint32_t x0 = (w * nb + b) * S, x1 = min(n_ev, x0 + S);
        if (w < W && x0 < n_ev) {
            char* sm = smem + w * L.bytes;
            const DevRule& Rr = *smp<DevRule>(sm, L.o_rule);
            const uint32_t* peid = smp<uint32_t>(sm, L.o_peid);
            const uint16_t* match = smp<uint16_t>(sm, L.o_match);
            uint32_t lo_t = 0, hi_t = NI;   // the item holding event x0
            while (hi_t - lo_t > 1) {
                const uint32_t m = (lo_t + hi_t) >> 1;
                if (G.item_ev[m] <= x0) lo_t = m; else hi_t = m;
            }
            uint32_t staged = kNone;
            Parent pa{0, 0, 0};
            bool pconn = false;
            uint32_t ar = 0;   // the staged parent's one arity (2 or 3), or 0
            for (uint32_t t = lo_t, x = x0; x < x1; ++t) {
                const uint32_t t0 = G.item_ev[t], rn = G.cnt[t];
                if (x >= t0 + rn) continue;   // an item without events
                const uint32_t f = t / R, r = t - f * R, sid = frontier[f];
                const uint32_t evo = P.st_evo[sid];
                const DevEvo ev = P.evos[evo];
                if (f != staged) {
                    staged = f;
                    pa = load_parent(P, L, sm, sid);
                    pconn = parent_connected(L, sm, pa);
                    // one arity of 2 or 3, and the packed edges seg_wl reads
                    const uint8_t* pear = smp<uint8_t>(sm, L.o_pear);
                    const uint32_t a0 = pa.ne ? pear[0] : 0u;
                    bool one = (a0 == 2 || a0 == 3) && pa.ne <= kSegEMax && pa.nvp <= 32;
                    for (uint32_t k = lane; k < pa.ne; k += 32) one = one && pear[k] == a0;
                    ar = __all_sync(0xFFFFFFFFu, one) ? a0 : 0u;
                    if (ar)
                        for (uint32_t k = lane; k < pa.ne; k += 32) {
                            const uint16_t* v = smp<uint16_t>(sm, L.o_vloc) + smp<uint16_t>(sm, L.o_pevo)[k];
                            smp<uint32_t>(sm, L.o_ppk)[k] = v[0] | (uint32_t(v[1]) << 8) | (ar == 3 ? uint32_t(v[2]) << 16 : 0u);
                        }
                    __syncwarp();
                    if (lane == 0 && t0 == x) b_hbm += 4ull * (pa.ne + (pa.ne + 3) / 4 + pa.nocc) + 20;
                }
                load_rule(sm, L, &P.rules[ev.rule_begin + r]);
                const uint32_t cons0 = n_cons + G.item_cons[t], prod0 = n_edges + G.item_prod[t],
                               fresh0 = next_vertex + G.item_fresh[t];
                const uint32_t lo = x - t0, hi = min(rn, x1 - t0);
                // one child's event record and table insert
                auto record = [&](uint32_t idx, uint64_t h, const WlInfo& info, const uint16_t* pos, uint32_t nec) {
                    if (lane == 0) {
                        const uint32_t e = ev_base + t0 + idx, coff = cons0 + idx * Rr.n_lhs,
                                       pid = prod0 + idx * Rr.n_rhs;
                        P.ev_in[e] = sid;
                        P.ev_rule[e] = ev.rule_begin + r;
                        P.ev_coff[e] = coff;
                        P.ev_prod[e] = pid;
                        P.ev_fresh[e] = fresh0 + idx * Rr.n_fresh;
                        P.ev_hash[e] = h;
                        P.ev_nv[e] = info.nv;
                        for (uint32_t k = 0; k < Rr.n_lhs; ++k) P.ev_cons[coff + k] = peid[pos[k]];
                        P.ev_bmask[e] = branch_mask(Rr.n_lhs, pa.ne, pos);
                        for (uint32_t k = 0; k < Rr.n_rhs; ++k) P.edge_creator[pid + k] = e;
                        table_insert(P, ev, h, e);
                        const uint64_t k = Rr.n_lhs, rr = Rr.n_rhs;
                        b_stage += 4 * k + 8;
                        b_stage += 4ull * pa.ne + 4ull * nec + 4ull * Rr.rhs_total + 12 * rr + 16 + 4 * k + 4 * rr;
                        b_stage += 5ull * info.nocc + 8ull * info.nv +
                                   uint64_t(info.rounds) * (8ull * info.nbr + 5ull * info.nocc + 16ull * info.nv) +
                                   8ull * info.nv + 8ull * info.nocc;
                        b_stage += 16;
                        b_hbm += 20 + 8 + 8 * k + 4 * rr + 16;
                        n_child += 1;
                        n_rounds += info.rounds;
                    }
                    __syncwarp();
                };
                const bool joined = pconn && (Rr.flags & kRuleRhsJoinsLhs);
                // the run's matches listed, then one child after another
                const Fwd none{};
                const uint16_t* mpos = smp<uint16_t>(sm, L.o_mpos);
                if (!list_matches(P, L, sm, Rr, pa, none, lo, hi, rn)) {
                } else if (ar && (Rr.rhs_uni == ar || !Rr.n_rhs) && pa.nvp + Rr.n_fresh <= 32 &&
                           pa.ne + Rr.n_rhs <= kSegEMax + Rr.n_lhs) {
                    // small states of one arity: hashed from the staged edges, no child is built
                    const uint32_t* ppk = smp<uint32_t>(sm, L.o_ppk);
                    uint32_t* sprod = smp<uint32_t>(sm, L.o_sprod);
                    const uint16_t* pevo = smp<uint16_t>(sm, L.o_pevo);
                    const uint16_t* vloc = smp<uint16_t>(sm, L.o_vloc);
                    const uint32_t keep = pa.ne - Rr.n_lhs;
                    for (uint32_t i = lo; i < hi; ++i) {
                        const uint16_t* pos = mpos + (i - lo) * L.LH;
                        unsigned long long rm = 0;
                        for (uint32_t k = 0; k < Rr.n_lhs; ++k) rm |= 1ull << pos[k];
                        if (lane < Rr.n_rhs) {   // lane k packs produced edge k
                            uint32_t pk = 0;
                            for (uint32_t q = 0; q < ar; ++q) {
                                const uint32_t var = Rr.rhs_vars[Rr.rhs_off[lane] + q];
                                uint32_t x = pa.nvp + Rr.fresh_rank[var];
                                if (!((Rr.new_mask >> var) & 1u)) {   // its first place on the left
                                    uint32_t k = 0, p = 0;
                                    while (Rr.lhs_vars[Rr.lhs_off[k] + p] != var)
                                        if (++p == Rr.lhs_ar[k]) { ++k; p = 0; }
                                    x = vloc[pevo[pos[k]] + p];
                                }
                                pk |= x << (8 * q);
                            }
                            sprod[lane] = pk;
                        }
                        __syncwarp();
                        WlInfo info;
                        const uint64_t h = seg_wl<32>(keep + Rr.n_rhs, ar, joined, sm + L.o_seg, L.SEGE, L.SEGN,
                                                      tables, [&](uint32_t j) -> uint32_t {
                            if (j >= keep) return sprod[j - keep];
                            uint32_t p = j;   // the j-th kept edge: past every removed position at or before it
                            for (unsigned long long m = rm; m; m &= m - 1)
                                p += p >= static_cast<uint32_t>(__ffsll(static_cast<long long>(m)) - 1) ? 1u : 0u;
                            return ppk[p];
                        }, info);
                        record(i, h, info, pos, keep + Rr.n_rhs);
                    }
                } else {
                    uint32_t* taken = smp<uint32_t>(sm, L.o_taken);
                    for (uint32_t k = lane; k < L.W; k += 32) taken[k] = 0;
                    __syncwarp();
                    for (uint32_t i = lo; i < hi; ++i)
                        fwd_emit(L, sm, Rr, mpos + (i - lo) * L.LH, [&](uint32_t nm) {
                            const uint32_t nec = build_child(L, sm, Rr, pa, nm);
                            WlInfo info;
                            const uint64_t h = warp_wl(L, sm, nec, pa.nvp + Rr.n_fresh, info, joined);
                            record(i, h, info, match, nec);
                        });
                }
                if (lane == 0 && lo == 0) b_stage += 4ull * pa.ne + 4ull * pa.nocc;
                x = t0 + hi;
            }
        }
        alive = fused_barrier(fs, phase, P.err, false, G.hasty, [] {});
        if (!alive) break;
        // ---- select: this thread's event from here to the end of the level
        const uint32_t ec = (n_ev + nb - 1) / nb;
        const uint32_t t = b * ec + tid, e = ev_base + t;
        const bool mine = tid < ec && t < n_ev;
        uint32_t in = 0, evo = 0, win = 0, bc = 0, depth = 0, nc = 0;
        bool fresh = false, rep = false, front = false;
        DevEvo ev{};
        if (mine) {
            in = P.ev_in[e];
            evo = P.st_evo[in];
            ev = P.evos[evo];
            const uint32_t co = P.ev_coff[e], k = P.rules[P.ev_rule[e]].n_lhs;
            for (uint32_t i = 0; i < k; ++i) P.ev_cprod[co + i] = P.edge_creator[P.ev_cons[co + i]];
            if (G.tr) reduce_event(P, e);
            for (uint32_t i = 0; i < k; ++i) nc += P.ev_cprod[co + i] != kNone ? 1u : 0u;
            win = table_lookup(P, ev, P.ev_hash[e]);
            depth = P.st_depth[in];
            fresh = win == e;
            rep = ev.quotient ? fresh : true;
            front = rep && depth + 1 < ev.steps;
            P.ev_kept[e] = 1;
            if (win == kNone) atomicOr(P.err, kErrTableFull);
            if (G.branchial) bc = fused_pairs(P, e, ev_end, in, nullptr);
        }
        warp_count(P.evo_classes, evo, fresh);
        warp_count(P.evo_states, evo, rep);
        {   // causal triples per evolution, one atomic per warp and evolution
            const uint32_t act = __ballot_sync(0xFFFFFFFFu, nc != 0);
            if (nc) {
                const uint32_t peers = __match_any_sync(act, evo);
                const uint32_t sum = __reduce_add_sync(peers, nc);
                if (lane == static_cast<uint32_t>(__ffs(peers) - 1))
                    atomicAdd(&P.evo_causal[evo], static_cast<unsigned long long>(sum));
            }
        }
        uint32_t tot[3];
        const uint32_t r_at = block_excl_scan(rep ? 1u : 0u, sh, tot[0]);
        const uint32_t f_at = block_excl_scan(front ? 1u : 0u, sh, tot[1]);
        const uint32_t b_at = block_excl_scan(bc, sh, tot[2]);
        if (tid < 3) G.sums[tid * nb + b] = tot[tid];
        alive = fused_barrier(fs, phase, P.err, true, G.hasty, [] {});
        if (!alive) break;
        // ---- assign
        if (w < 3) {
            uint32_t p = 0, s = 0;
            for (uint32_t i = lane; i < nb; i += 32) {
                const uint32_t x = G.sums[w * nb + i];
                s += x;
                p += i < b ? x : 0u;
            }
            p = warp_sum32(p);
            s = warp_sum32(s);
            if (lane == 0) { pre[w] = p; all[w] = s; }
        }
        __syncthreads();
        const uint32_t j = pre[0] + r_at, jf = pre[1] + f_at;
        const uint64_t jb = n_pairs + pre[2] + b_at;
        if (mine) {
            if (rep) {
                const uint32_t sid = n_states + j;
                P.state_of_arrival[e] = sid;
                G.new_event[j] = e;
                P.st_event[sid] = e;
                P.st_evo[sid] = evo;
                P.st_depth[sid] = depth + 1;
                P.st_hash[sid] = P.ev_hash[e];
                if (front) G.front[cur ^ 1][jf] = sid;
            }
            if (bc) fused_pairs(P, e, ev_end, in, reinterpret_cast<uint2*>(G.bpairs) + jb);
            if (G.ev_keys) {
                const uint32_t fin = win == kNone ? kNone : P.ev_in[win];
                const uint32_t step = fin == kNone ? 0u : P.st_depth[fin] + 1;
                const uint64_t sig = event_signature(G.ev_keys, P.st_hash[in], P.ev_hash[e], step,
                                                     P.ev_rule[e] - ev.rule_begin);
                P.ev_sig[e] = sig;
                slot_insert(P, ev.sig_off, ev.sig_mask, sig, e);
            }
            // the evolution's runs of events, states, pairs and frontier states in this level
            uint32_t* q = ranges + uint64_t(evo) * kRangeWords;
            if (t == 0 || P.st_evo[P.ev_in[e - 1]] != evo) {
                q[0] = e;
                q[2] = n_states + j;
                q[4] = static_cast<uint32_t>(jb);
                q[6] = jf;
            }
            if (t + 1 == n_ev || P.st_evo[P.ev_in[e + 1]] != evo) {
                q[1] = e + 1;
                q[3] = n_states + j + (rep ? 1u : 0u);
                q[5] = static_cast<uint32_t>(jb + bc);
                q[7] = jf + (front ? 1u : 0u);
            }
        }
        __syncthreads();
        // records of this block's new states
        const uint32_t j0 = pre[0], j1 = pre[0] + tot[0];
        constexpr uint32_t kScratch = kMaxVars + kMaxPatternEdges;
        uint32_t* scratch = reinterpret_cast<uint32_t*>(smem) + w * kScratch * 4;
        if (mne <= 16) materialize_states<8>(P, G.new_event, n_states, j0, j1, w, kFusedWarps, scratch);
        else materialize_states<32>(P, G.new_event, n_states, j0, j1, w, kFusedWarps, scratch);
        if (b == 0 && tid == 0) {
            uint32_t* o = level_out + lv * kLevelWords;
            o[0] = F;
            o[1] = n_ev;
            o[2] = all[0];
            o[3] = all[1];
            o[4] = all[2];
            o[5] = mne + G.rm.grow_e;
            o[6] = mno + G.rm.grow_o;
        }
        const uint64_t rec = uint64_t(mne + G.rm.grow_e) + (mne + G.rm.grow_e + 3) / 4 + mno + G.rm.grow_o;
        n_states += all[0];
        n_pairs += all[2];
        F = all[1];
        arena_words += all[0] * rec;
        n_events += n_ev;
        n_cons += fs->n_cons;
        n_edges += fs->n_prod;
        next_vertex += fs->n_fresh;
        ne_b = mne + G.rm.grow_e;
        no_b = mno + G.rm.grow_o;
        cur ^= 1;
        alive = fused_barrier(fs, phase, P.err, true, G.hasty, [] {});
        if (!alive) break;
        // ---- output states (the next count reads none of it)
        bool swin = false;
        if (mine) {
            P.ev_out[e] = (rep || !ev.quotient) ? n_states - all[0] + j : (win == kNone ? kNone : P.state_of_arrival[win]);
            if (G.ev_keys) swin = slot_lookup(P, ev.sig_off, ev.sig_mask, P.ev_sig[e]) == e;
        }
        if (G.ev_keys) warp_count(P.evo_sigs, evo, swin);
    }
    // counters of the children hashed here (the warp-per-child figures)
    __shared__ unsigned long long st_sm[4];
    if (tid < 4) st_sm[tid] = 0;
    __syncthreads();
    if (n_child) {
        atomicAdd(&st_sm[0], static_cast<unsigned long long>(b_stage));
        atomicAdd(&st_sm[1], static_cast<unsigned long long>(b_hbm));
        atomicAdd(&st_sm[2], static_cast<unsigned long long>(n_child));
        atomicAdd(&st_sm[3], static_cast<unsigned long long>(n_rounds));
    }
    __syncthreads();
    if (tid < 4 && st_sm[tid]) atomicAdd(&P.stats[4 + tid], st_sm[tid]);
    // the last block to leave reports and clears the grid's words for the next launch
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        // (blocks that left at a closed barrier arrive here once, like the others)
        if (atomicAdd(&fs->abort, 1u) + 1 == nb) {
            __threadfence();
            volatile uint32_t* o = G.out;
            o[0] = (__ldcg(&fs->gen) & kBarrierClosed) ? uint32_t(kStopLevel) : __ldcg(&fs->stop);
            o[1] = lv;
            o[2] = cur;
            o[3] = __ldcg(P.err);
            const unsigned long long c = __ldcg(&P.evo_classes[0]), s = __ldcg(&P.evo_states[0]);
            o[4] = static_cast<uint32_t>(c);
            o[5] = static_cast<uint32_t>(c >> 32);
            o[6] = static_cast<uint32_t>(s);
            o[7] = static_cast<uint32_t>(s >> 32);
            o[8] = __ldcg(&P.evo_stopped[0]);
            o[14] = n_cons - G.n_cons;
            o[15] = 0;
            o[16] = n_edges - G.n_edges;
            o[17] = next_vertex - G.next_vertex;
            FusedState z{};
            *fs = z;
        }
    }
}
