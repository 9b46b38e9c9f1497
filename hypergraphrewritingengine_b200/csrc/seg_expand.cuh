// Expansion of small uniform-arity states: children hashed S lanes each (seg_wl.cuh). Included by
// step_kernels.cu after the lane kernels; single-rule evolutions without match forwarding.
//
// A warp takes slices of a parent's matches (at most A.slice of them, so a parent with thousands of
// matches is spread over many warps and a small level over the whole GPU), stages the parent, lists
// the slice's matches (lane walks; the warp join for rules of more than four left-hand edges) and
// goes through them in batches of up to 32: children hashed 32 / S at a time, then their events
// written and their hashes inserted one child per lane.
//
// Measured against the lane kernel (device time of the expand launches): the 1,024 random evolutions
// 67 -> 25 ms (35 launches, most of them small: one warp per parent left a launch waiting for the
// parent with the most matches), C3 2.35 -> 1.45 ms. Slices of at least 8 children instead of 1 on
// the small launches took 88 ms.
#pragma once

namespace hgx {

// Slices of the work indices [f_begin, f_begin + n) for the segment kernel.
__global__ void k_seg_slices(LevelArgs A, uint32_t n, uint32_t* cnt) {
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += gridDim.x * blockDim.x) {
        const uint32_t f = frontier_at(A, A.f_begin + w);
        const uint32_t c = children_of(A, f);
        cnt[w] = (A.fmode[f] & 4u) ? (c + A.slice - 1) / A.slice : 0u;
    }
}

template <int S, bool kWalk>
__global__ void __launch_bounds__(256, 3) k_expand_seg(DevPtrs P, LevelArgs A, Layout L) {
    constexpr uint32_t G = 32 / S;
    extern __shared__ __align__(16) char smem[];
    __shared__ SegTables tables;
    __shared__ uint32_t idx_sm[8][32], info_sm[8][32];
    __shared__ unsigned long long stats_sm[8][4];
    const uint32_t w = threadIdx.x >> 5, lane = lane_id(), seg = lane / S;
    char* const sm = smem + w * L.bytes;
    uint32_t* cidx = idx_sm[w];             // slot -> child index in its parent
    uint32_t* cinfo = info_sm[w];           // slot -> WL figures
    char* const batch = sm + L.o_batch;     // per child: removed positions (mask; then the hash), produced edges, positions
    char* const scr = sm + L.o_seg + seg * L.SEGB;
    const uint32_t o_pos = 8 + 4 * L.RHS;
    unsigned long long* wstats = stats_sm[w];
    if (lane < 4) wstats[lane] = 0;
    seg_tables_fill(tables);
    const DevRule& R = *smp<DevRule>(sm, L.o_rule);
    const uint32_t* ppk = smp<uint32_t>(sm, L.o_ppk);
    const uint32_t* peid = smp<uint32_t>(sm, L.o_peid);
    const uint16_t* pevo = smp<uint16_t>(sm, L.o_pevo);
    const uint16_t* vloc = smp<uint16_t>(sm, L.o_vloc);
    WarpWork q;
    const uint32_t units = A.soff ? A.soff[A.n_sw] : A.f_end - A.f_begin;
#pragma unroll 1
    while (true) {
        const uint32_t u = q.next(&A.work[1]);
        if (u >= units) break;
        uint32_t f, lo = 0;
        if (A.soff) {
            uint32_t a = 0, b = A.n_sw;   // the work index whose slices hold u
            while (b - a > 1) {
                const uint32_t m = (a + b) >> 1;
                if (A.soff[m] <= u) a = m; else b = m;
            }
            f = frontier_at(A, A.f_begin + a);
            lo = (u - A.soff[a]) * A.slice;
        } else {
            f = frontier_at(A, A.f_begin + u);
        }
        if (!(A.fmode[f] & 4u)) continue;
        const uint32_t rn = A.counts[f];              // single-rule evolutions: item = f
        const uint32_t hi = A.soff ? min(rn, lo + A.slice) : rn;
        const uint32_t sid = A.frontier[f];
        const DevEvo ev = P.evos[P.st_evo[sid]];
        if (rn == 0 || ev.rule_count == 0) {   // nothing to build: count what the join reads
            if (lane == 0) {
                const uint64_t ne = P.st_ne[sid], nocc = P.st_nocc[sid];
                wstats[1] += 4 * (ne + (ne + 3) / 4 + nocc) + 20;
                wstats[0] += 4 * ne + 4 * nocc;
            }
            continue;
        }
        const Parent pa = load_parent(P, L, sm, sid);
        load_rule(sm, L, &P.rules[ev.rule_begin]);
        const uint32_t ar = pa.ne ? smp<uint8_t>(sm, L.o_pear)[0] : 0u;   // every edge's (the host checked)
        bool conn;
        {   // packed edges, and whether the parent is one component
            uint32_t* pk_out = smp<uint32_t>(sm, L.o_ppk);
            uint32_t* adj = smp<uint32_t>(sm, L.o_first);   // load_parent's scratch
            if (lane < pa.nvp) adj[lane] = 0;
            __syncwarp();
            for (uint32_t e = lane; e < pa.ne; e += 32) {
                const uint32_t vo = pevo[e];
                uint32_t pk = 0, bits = 0;
                for (uint32_t k = 0; k < ar; ++k) {
                    const uint32_t v = vloc[vo + k];
                    pk |= v << (8 * k);
                    bits |= 1u << v;
                }
                pk_out[e] = pk;
                for (uint32_t m = bits; m; m &= m - 1) atomicOr(&adj[__ffs(m) - 1], bits);
            }
            __syncwarp();
            const uint32_t mine = lane < pa.nvp ? adj[lane] : 0u;
            uint32_t reach = pa.nvp ? 1u : 0u;
            for (uint32_t it = 0; it < pa.nvp; ++it) {
                const uint32_t nr = reach | __reduce_or_sync(0xFFFFFFFFu, ((reach >> lane) & 1u) ? mine : 0u);
                if (nr == reach) break;
                reach = nr;
            }
            conn = pa.nvp && reach == (pa.nvp >= 32 ? 0xFFFFFFFFu : (1u << pa.nvp) - 1u);
        }
        const bool joined = conn && (R.flags & kRuleRhsJoinsLhs);
        const uint32_t n_lhs = R.n_lhs, n_rhs = R.n_rhs, keep = pa.ne - n_lhs, nec = keep + n_rhs;
        const uint32_t ev0 = A.ev_base + A.item_ev[f], cons0 = A.cons_base + A.item_cons[f],
                       prod0 = A.prod_base + A.item_prod[f], fresh0 = A.fresh_base + A.item_fresh[f];
        if (lane == 0 && lo == 0) {
            wstats[1] += 4ull * (pa.ne + (pa.ne + 3) / 4 + pa.nocc) + 20;
            wstats[0] += 4ull * pa.ne + 4ull * pa.nocc;
        }
        // hash the nb children of the batch, then write their events
        auto flush = [&](uint32_t nb) {
#pragma unroll 1
            for (uint32_t c0 = 0; c0 < nb; c0 += G) {
                const uint32_t c = c0 + seg;
                const bool valid = c < nb;
                char* slot = batch + (valid ? c : 0u) * L.SB;
                const uint32_t* prod = reinterpret_cast<const uint32_t*>(slot + 8);
                const unsigned long long rm = *reinterpret_cast<const unsigned long long*>(slot);
                WlInfo x;
                const uint64_t h = seg_wl<S>(valid ? nec : 0u, ar, joined, scr, L.SEGE,
                                             L.SEGN, tables, [&](uint32_t i) -> uint32_t {
                    if (i >= keep) return prod[i - keep];
                    uint32_t p = i;   // the i-th kept edge: past every removed position at or before it
                    for (unsigned long long m = rm; m; m &= m - 1)
                        p += p >= static_cast<uint32_t>(__ffsll(static_cast<long long>(m)) - 1) ? 1u : 0u;
                    return ppk[p];
                }, x);
                __syncwarp();
                if (valid && (lane & (S - 1)) == 0) {
                    *reinterpret_cast<unsigned long long*>(slot) = h;
                    cinfo[c] = x.rounds | (x.nv << 8) | (x.nocc << 16);
                }
            }
            __syncwarp();
            uint32_t b_stage = 0, b_hbm = 0, n_rounds = 0;
            if (lane < nb) {
                const uint32_t idx = cidx[lane], info = cinfo[lane];
                const char* slot = batch + lane * L.SB;
                const uint64_t h = *reinterpret_cast<const unsigned long long*>(slot);
                const uint8_t* pos = reinterpret_cast<const uint8_t*>(slot + o_pos);
                const uint32_t e = ev0 + idx, coff = cons0 + idx * n_lhs, pid = prod0 + idx * n_rhs;
                P.ev_in[e] = sid;
                P.ev_rule[e] = ev.rule_begin;
                P.ev_coff[e] = coff;
                P.ev_prod[e] = pid;
                P.ev_fresh[e] = fresh0 + idx * R.n_fresh;
                P.ev_hash[e] = h;
                P.ev_nv[e] = (info >> 8) & 0xFFu;
                for (uint32_t k = 0; k < n_lhs; ++k) P.ev_cons[coff + k] = peid[pos[k]];
                P.ev_bmask[e] = branch_mask(n_lhs, pa.ne, pos);
                for (uint32_t k = 0; k < n_rhs; ++k) P.edge_creator[pid + k] = e;
                table_insert(P, ev, h, e);
                const uint32_t nv = (info >> 8) & 0xFFu, nocc = info >> 16, nbr = nocc * (ar - 1), rr = n_rhs;
                n_rounds = info & 0xFFu;
                b_stage = 8 * n_lhs + 8 + 4 * pa.ne + 4 * nec + 4 * R.rhs_total + 16 * rr + 16 + 5 * nocc + 8 * nv +
                          n_rounds * (8 * nbr + 5 * nocc + 16 * nv) + 8 * nv + 8 * nocc + 16;
                b_hbm = 44 + 8 * n_lhs + 4 * rr;
            }
            b_stage = warp_sum32(b_stage);
            b_hbm = warp_sum32(b_hbm);
            n_rounds = warp_sum32(n_rounds);
            if (lane == 0) {
                wstats[0] += b_stage;
                wstats[1] += b_hbm;
                wstats[2] += nb;
                wstats[3] += n_rounds;
            }
            __syncwarp();
        };
        if (kWalk && n_lhs <= kLaneJoinLhs && hi - lo <= L.MCAP) {
            const unsigned long long* vm = build_vmask(L, sm, pa);
            uint32_t* mlist = smp<uint32_t>(sm, L.o_mlist);
            uint32_t total = 0;
            for (uint32_t b = 0; b < pa.ne; b += 32) {
                const uint32_t e0 = b + lane;
                const uint32_t c = e0 < pa.ne ? lane_walk(L, sm, R, pa, e0, vm, [](uint32_t) {}) : 0u;
                const uint32_t inc = warp_incl_scan(c);
                uint32_t at = total + inc - c;
                if (c && at < hi && at + c > lo) lane_walk(L, sm, R, pa, e0, vm, [&](uint32_t pk) {
                    if (at >= lo && at < hi) mlist[at - lo] = pk;
                    ++at;
                });
                total += __shfl_sync(0xFFFFFFFFu, inc, 31);
            }
            __syncwarp();
            if (total != rn) {
                if (lane == 0) atomicOr(P.err, kErrJoinCount);
                continue;
            }
#pragma unroll 1
            for (uint32_t i0 = lo; i0 < hi; i0 += 32) {
                const uint32_t nb = min(hi - i0, 32u);
                if (lane < nb) {
                    char* slot = batch + lane * L.SB;
                    uint32_t* prod = reinterpret_cast<uint32_t*>(slot + 8);
                    uint8_t* pos = reinterpret_cast<uint8_t*>(slot + o_pos);
                    const uint32_t pk = mlist[i0 + lane - lo];
                    uint8_t bv[kMaxVars];
                    unsigned long long rm = 0;
                    for (uint32_t k = 0; k < n_lhs; ++k) {
                        const uint32_t p = (pk >> (8u * k)) & 0xFFu;
                        pos[k] = static_cast<uint8_t>(p);
                        rm |= 1ull << p;
                        const uint32_t pv = ppk[p];
                        for (uint32_t qq = 0; qq < ar; ++qq)
                            bv[R.lhs_vars[R.lhs_off[k] + qq]] = static_cast<uint8_t>(pv >> (8 * qq));
                    }
                    *reinterpret_cast<unsigned long long*>(slot) = rm;
                    for (uint32_t k = 0, t = 0; k < n_rhs; ++k) {
                        uint32_t v = 0;
                        for (uint32_t qq = 0; qq < ar; ++qq, ++t) {
                            const uint32_t var = R.rhs_vars[t];
                            v |= (((R.new_mask >> var) & 1u) ? pa.nvp + R.fresh_rank[var] : bv[var]) << (8 * qq);
                        }
                        prod[k] = v;
                    }
                    cidx[lane] = i0 + lane;
                }
                __syncwarp();
                flush(nb);
            }
        } else {
            const uint16_t* match = smp<uint16_t>(sm, L.o_match);
            const uint16_t* bind = smp<uint16_t>(sm, L.o_bind);
            uint32_t idx = 0, nb = 0;
            warp_join(L, sm, R, pa, R.sched, -1, [&](uint32_t nm) {
                if (idx >= lo && idx < hi) {
                    char* slot = batch + nb * L.SB;
                    if (lane < n_lhs) reinterpret_cast<uint8_t*>(slot + o_pos)[lane] = static_cast<uint8_t>(match[lane]);
                    if (lane == 0) {
                        unsigned long long rm = 0;
                        for (uint32_t k = 0; k < n_lhs; ++k) rm |= 1ull << match[k];
                        *reinterpret_cast<unsigned long long*>(slot) = rm;
                        cidx[nb] = idx;
                    }
                    for (uint32_t k = lane; k < n_rhs; k += 32) {
                        uint32_t v = 0;
                        for (uint32_t qq = 0; qq < ar; ++qq) {
                            const uint32_t var = R.rhs_vars[R.rhs_off[k] + qq];
                            v |= (((nm >> var) & 1u) ? bind[var] : pa.nvp + R.fresh_rank[var]) << (8 * qq);
                        }
                        reinterpret_cast<uint32_t*>(slot + 8)[k] = v;
                    }
                    __syncwarp();
                    if (++nb == 32 || idx + 1 == hi) {
                        flush(nb);
                        nb = 0;
                    }
                }
                ++idx;
            }, hi, SkipCounter{&idx, lo});
        }
    }
    __syncwarp();
    if (lane == 0 && wstats[1]) {
        atomicAdd(&P.stats[0], wstats[0]);
        atomicAdd(&P.stats[1], wstats[1]);
        atomicAdd(&P.stats[2], wstats[2]);
        atomicAdd(&P.stats[3], wstats[3]);
    }
}

}  // namespace hgx
