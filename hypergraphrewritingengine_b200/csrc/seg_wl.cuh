// WL canonical hash of small states, S lanes of a warp per state (S = 16: two states at once; 32).
//
// For states of at most S vertices and 64 edges whose edges share one arity A of 2 or 3. Lanes own
// vertices in the vertex steps and edges in the edge steps; colours, neighbour multisets and edge
// records live in a few hundred bytes of shared memory a state and in registers. Compared with one
// state per lane (lane_wl.cuh) nothing is kept in local memory, the lanes of a warp run the same
// step on equal work (a vertex's neighbour list in place of a whole state), and a state takes a
// few microseconds instead of tens, so a launch of few states finishes early. Bound by
// instruction fetch and issue slots (half of them used; stalls by count: no instruction, fixed latency,
// shared memory). Of the ways to sort a vertex's neighbour words, measured on states of
// 4-40 binary edges (200,003 of them) and on C2: insertion in shared memory 0.83 ms and 9.5 ms,
// registers for every length 0.94 and 9.5 ms, registers up to 8 words and ranks above 0.83 and 8.6 ms.
//
// The arithmetic is lane_wl.cuh's (the reference's common/include/hgcommon/wl_core.hpp:67-202), with
// the uniform-arity form of the initial colour: the sorted (arity, position) multiset is the
// positions in order with their multiplicities, and no truncation applies (A >= 2).
//
// Every lane of the warp calls it: control flow is warp-uniform (loops run to the warp's largest
// count, a segment that is finished keeps its values), so all shuffles and votes use the full mask.
#pragma once

namespace hgx {
namespace {

// Scratch bytes of one segment for states of at most ne edges with at most `list` neighbour entries
// (edges x arity x (arity - 1)).
HGX_HD uint32_t seg_scratch_bytes(uint32_t S, uint32_t ne, uint32_t list) {
    const uint32_t list8 = (list > 2 * S ? list : 2 * S) * 8;   // also two words a component
    return list8 + 8 * S /* colours */ + 8 * ne /* entry offsets */ + 4 * ne /* edges */ + 4 * S /* counts */ +
           (2 * list + 7) / 8 * 8 /* permutation */;
}

template <int S>
__device__ __forceinline__ uint64_t seg_sum64(uint64_t x) {
#pragma unroll
    for (int d = S / 2; d; d >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, d);
    return x;
}

// Batcher's odd-even merge sort of D keys in registers, every index a compile-time constant.
template <int D>
__device__ __forceinline__ void sort_keys(uint32_t (&k)[D]) {
#pragma unroll
    for (int p = 1; p < D; p <<= 1)
#pragma unroll
        for (int q = p; q >= 1; q >>= 1)
#pragma unroll
            for (int j = q % p; j + q < D; j += 2 * q)
#pragma unroll
                for (int i = 0; i < q; ++i)
                    if (i + j + q < D && (i + j) / (2 * p) == (i + j + q) / (2 * p)) {
                        const uint32_t lo = min(k[i + j], k[i + j + q]), hi = max(k[i + j], k[i + j + q]);
                        k[i + j] = lo;
                        k[i + j + q] = hi;
                    }
}

__device__ __noinline__ uint64_t fold_exact(uint64_t* l, uint32_t n, uint64_t f) {
#pragma unroll 1
    for (uint32_t i = 1; i < n; ++i) {
        const uint64_t k = l[i];
        uint32_t j = i;
        while (j > 0 && l[j - 1] > k) { l[j] = l[j - 1]; --j; }
        l[j] = k;
    }
#pragma unroll 1
    for (uint32_t j = 0; j < n; ++j) f = fnv(f, l[j]);
    return f;
}

// fnv fold of the n <= D words at l in ascending order, n <= n_max (warp-uniform). The sort runs on
// 32-bit keys -- a word's top 27 bits and its place, two instructions a compare-exchange in place of
// six -- and the fold checks that the words really ascend; words that agree in their top 27 bits and
// came out in the wrong order (one vertex in some ten million) are sorted exactly instead.
template <int D>
__device__ __forceinline__ uint64_t fold_sorted(uint64_t* l, uint32_t n, uint32_t n_max, uint64_t f0) {
    const uint32_t* hi = reinterpret_cast<const uint32_t*>(l) + 1;
    uint32_t k[D];
#pragma unroll
    for (uint32_t j = 0; j < D; ++j) k[j] = j < n ? (hi[2 * j] & ~31u) | j : 0xFFFFFFFFu;
    sort_keys<D>(k);
    uint64_t f = f0, last = 0;
    bool bad = false;
#pragma unroll
    for (uint32_t j = 0; j < D; ++j)
        if (D <= 8 || j < n_max) {
            if (j < n) {
                const uint64_t x = l[k[j] & 31u];
                bad |= x < last;
                last = x;
                f = fnv(f, x);
            }
        }
    return bad ? fold_exact(l, n, f0) : f;
}

// Initial colours by per-position occurrence counts: arity 2 with both counts below 16, arity 3 with
// all three below 8. Filled once per block.
struct SegTables {
    uint64_t c2[256], c3[512];
};
__device__ __forceinline__ uint64_t seg_initial(uint32_t c, uint32_t A) {
    uint64_t h = fnv(kFnvOffset, lane_bytesum(c));
#pragma unroll
    for (uint32_t q = 0; q < 3; ++q)
        if (q < A)
#pragma unroll 1
            for (uint32_t j = (c >> (8 * q)) & 0xFFu; j; --j) h = fnv(fnv(h, A), q);
    return h;
}
__device__ __forceinline__ void seg_tables_fill(SegTables& T) {
    for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) T.c2[i] = seg_initial((i >> 4) | ((i & 15u) << 8), 2);
    for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x)
        T.c3[i] = seg_initial((i >> 6) | (((i >> 3) & 7u) << 8) | ((i & 7u) << 16), 3);
    __syncthreads();
}

// Distinct colours among the alive lanes of each segment.
template <int S>
__device__ __forceinline__ uint32_t seg_distinct(uint64_t c, uint32_t alive_seg, uint32_t segmask, bool alive) {
    const uint32_t grp = __match_any_sync(0xFFFFFFFFu, static_cast<unsigned long long>(c)) & alive_seg;
    const bool lead = alive && lane_id() == static_cast<uint32_t>(__ffs(grp) - 1);
    return __popc(__ballot_sync(0xFFFFFFFFu, lead) & segmask);
}

// edge(i): the state's edge i < ne as its vertices' local ids (below S), position q in byte q. Per
// segment: ne (0: no state), A, connected (known to be one component). Returns the segment's hash on all
// its lanes. scr: the segment's scratch (seg_scratch_bytes, 8-byte aligned); ne_cap, listn the
// sizes it was made for.
template <int S, class EdgeAt>
__device__ __forceinline__ uint64_t seg_wl(uint32_t ne, uint32_t A, bool connected, char* scr,
                                           uint32_t ne_cap, uint32_t listn, const SegTables& T,
                                           EdgeAt&& edge, WlInfo& info) {
    constexpr uint32_t full = 0xFFFFFFFFu;
    const uint32_t lane = lane_id(), sl = lane & (S - 1);
    const uint32_t segmask = S == 32 ? full : (((1u << (S & 31)) - 1u) << (lane & ~(S - 1u)));
    uint64_t* list = reinterpret_cast<uint64_t*>(scr);
    uint64_t* cur = list + (listn > 2 * S ? listn : 2 * S);
    uint64_t* eoff = cur + S;                                  // entry offset of each position (16 bits)
    uint32_t* epk = reinterpret_cast<uint32_t*>(eoff + ne_cap);
    uint32_t* cnt = epk + ne_cap;
    uint16_t* perm = reinterpret_cast<uint16_t*>(cnt + S);     // long lists: entry by rank
    const uint32_t ne_max = __reduce_max_sync(full, ne);
    cnt[sl] = 0;
    __syncwarp();
    for (uint32_t i0 = 0; i0 < ne_max; i0 += S) {
        const uint32_t i = i0 + sl;
        if (i < ne) {
            const uint32_t pk = edge(i);
            epk[i] = pk;
            uint32_t slots = 0;   // earlier occurrences of each position's vertex
#pragma unroll
            for (uint32_t q = 0; q < 3; ++q)
                if (q < A) slots |= lane_bytesum(atomicAdd(&cnt[(pk >> (8 * q)) & 0xFFu], 1u << (8 * q))) << (8 * q);
            eoff[i] = slots;
        }
    }
    __syncwarp();
    const uint32_t c = cnt[sl];
    const uint32_t deg = lane_bytesum(c), n = deg * (A - 1);
    const bool alive = deg != 0;
    const uint32_t alive_seg = __ballot_sync(full, alive) & segmask;
    uint32_t base = n;   // exclusive scan of the neighbour counts over the segment
#pragma unroll
    for (uint32_t d = 1; d < S; d <<= 1) {
        const uint32_t y = __shfl_up_sync(full, base, d, S);
        if (sl >= d) base += y;
    }
    base -= n;
    const uint32_t n_max = __reduce_max_sync(full, n);
    // initial colours
    uint64_t h;
    if (A == 2 && (c & 0xF0F0u) == 0) h = T.c2[((c & 15u) << 4) | ((c >> 8) & 15u)];
    else if (A == 3 && (c & 0xF8F8F8u) == 0) h = T.c3[((c & 7u) << 6) | ((c >> 5) & 56u) | ((c >> 16) & 7u)];
    else h = seg_initial(c, A);
    uint64_t mine = alive ? h : 0;
    __syncwarp();
    cnt[sl] = base | (n << 16);
    cur[sl] = mine;
    __syncwarp();
    for (uint32_t i0 = 0; i0 < ne_max; i0 += S) {
        const uint32_t i = i0 + sl;
        if (i < ne) {
            const uint32_t pk = epk[i], slots = static_cast<uint32_t>(eoff[i]);
            uint64_t o = 0;
#pragma unroll
            for (uint32_t q = 0; q < 3; ++q)
                if (q < A)
                    o |= uint64_t((cnt[(pk >> (8 * q)) & 0xFFu] & 0xFFFFu) + ((slots >> (8 * q)) & 0xFFu) * (A - 1)) << (16 * q);
            eoff[i] = o;
        }
    }
    __syncwarp();
    uint32_t prev = seg_distinct<S>(mine, alive_seg, segmask, alive);
    bool done = ne == 0;
    uint32_t rounds = 0;
#pragma unroll 1
    for (uint32_t it = 0; it < kWlMaxRounds; ++it) {
        // edges: every position's neighbour entries, fnv(colour of the vertex at k, k), k != q
        for (uint32_t i0 = 0; i0 < ne_max; i0 += S) {
            const uint32_t i = i0 + sl;
            if (i < ne) {
                const uint32_t pk = epk[i];
                const uint64_t o = eoff[i];
                const uint64_t x0 = fnv(cur[pk & 0xFFu], 0), x1 = fnv(cur[(pk >> 8) & 0xFFu], 1);
                const uint32_t o0 = o & 0xFFFFu, o1 = (o >> 16) & 0xFFFFu;
                list[o0] = x1;
                list[o1] = x0;
                if (A == 3) {
                    const uint64_t x2 = fnv(cur[(pk >> 16) & 0xFFu], 2);
                    const uint32_t o2 = (o >> 32) & 0xFFFFu;
                    list[o0 + 1] = x2;
                    list[o1 + 1] = x2;
                    list[o2] = x0;
                    list[o2 + 1] = x1;
                }
            }
        }
        __syncwarp();
        // vertices: the sorted fold
        uint64_t f;
        if (n_max <= 4) f = fold_sorted<4>(list + base, n, n_max, mine);
        else if (n_max <= 8) f = fold_sorted<8>(list + base, n, n_max, mine);
        else {
            // a long list: the edge lanes rank their own entries within the vertex's list (equal
            // words by place), the vertex lane folds in rank order
            for (uint32_t i0 = 0; i0 < ne_max; i0 += S) {
                const uint32_t i = i0 + sl;
                if (i < ne) {
                    const uint32_t pk = epk[i];
                    const uint64_t o = eoff[i];
#pragma unroll 1
                    for (uint32_t q = 0; q < A; ++q) {
                        const uint32_t bn = cnt[(pk >> (8 * q)) & 0xFFu], b0 = bn & 0xFFFFu, m = bn >> 16;
                        const uint32_t at = (o >> (16 * q)) & 0xFFFFu;
                        const uint64_t x = list[at], y = list[at + A - 2];   // A - 1 entries: one or two
                        uint32_t rx = 0, ry = 0;
#pragma unroll 2
                        for (uint32_t j = 0; j < m; ++j) {
                            const uint64_t z = list[b0 + j];
                            rx += z < x || (z == x && b0 + j < at) ? 1u : 0u;
                            ry += z < y || (z == y && b0 + j < at + 1) ? 1u : 0u;
                        }
                        perm[b0 + rx] = static_cast<uint16_t>(at);
                        if (A == 3) perm[b0 + ry] = static_cast<uint16_t>(at + 1);
                    }
                }
            }
            __syncwarp();
            f = mine;
#pragma unroll 1
            for (uint32_t j = 0; j < n; ++j) f = fnv(f, list[perm[base + j]]);
        }
        if (alive && !done) mine = f;
        cur[sl] = mine;   // every edge step of this round has read the old colours
        const uint32_t d = seg_distinct<S>(mine, alive_seg, segmask, alive);
        if (!done) {
            ++rounds;
            done = d == prev;
            prev = d;
        }
        __syncwarp();
        if (__all_sync(full, done)) break;
    }
    // folds
    const uint64_t term = alive ? smix(mine) : 0;
    const uint64_t vs = seg_sum64<S>(term);
    uint64_t es = 0;
    for (uint32_t i0 = 0; i0 < ne_max; i0 += S) {
        const uint32_t i = i0 + sl;
        if (i < ne) {
            const uint32_t pk = epk[i];
            uint64_t x = fnv(kFnvOffset, A);
#pragma unroll
            for (uint32_t q = 0; q < 3; ++q)
                if (q < A) x = fnv(x, cur[(pk >> (8 * q)) & 0xFFu]);
            es += smix(x);
        }
    }
    es = seg_sum64<S>(es);
    const uint32_t nv = __popc(alive_seg);
    bool one = connected || ne == 0;
    uint64_t cs = 0;
    if (!__all_sync(full, one)) {
        // components: least label over the edges until nothing changes (at most V passes)
        __syncwarp();
        cnt[sl] = sl;
        __syncwarp();
#pragma unroll 1
        for (uint32_t it = 0; it < S; ++it) {
            bool moved = false;
            for (uint32_t i0 = 0; i0 < ne_max; i0 += S) {
                const uint32_t i = i0 + sl;
                if (i >= ne) continue;
                const uint32_t pk = epk[i];
                uint32_t lo = 0xFFu, hi = 0;
#pragma unroll
                for (uint32_t q = 0; q < 3; ++q)
                    if (q < A) {
                        const uint32_t x = *reinterpret_cast<volatile uint32_t*>(&cnt[(pk >> (8 * q)) & 0xFFu]);
                        lo = min(lo, x);
                        hi = max(hi, x);
                    }
                if (lo == hi) continue;
                moved = true;
#pragma unroll
                for (uint32_t q = 0; q < 3; ++q)
                    if (q < A) atomicMin(&cnt[(pk >> (8 * q)) & 0xFFu], lo);
            }
            __syncwarp();
            if (!__any_sync(full, moved)) break;
        }
        const uint32_t r = cnt[sl];
        const bool root = alive && r == sl;
        one = __popc(__ballot_sync(full, root) & segmask) <= 1;
        // per component: its colour terms, and edges << 32 | vertices
        unsigned long long* csum = reinterpret_cast<unsigned long long*>(list);
        unsigned long long* ccnt = csum + S;
        csum[sl] = 0;
        ccnt[sl] = 0;
        __syncwarp();
        if (alive) {
            atomicAdd(&csum[r], static_cast<unsigned long long>(term));
            atomicAdd(&ccnt[r], 1ull);
        }
        for (uint32_t i0 = 0; i0 < ne_max; i0 += S) {
            const uint32_t i = i0 + sl;
            if (i < ne) atomicAdd(&ccnt[cnt[epk[i] & 0xFFu]], 1ull << 32);
        }
        __syncwarp();
        cs = seg_sum64<S>(root ? smix(fnv(fnv(kFnvOffset, ccnt[sl]), csum[sl])) : 0ull);
        __syncwarp();
    }
    if (one) cs = lane_one_component(ne, nv, vs);
    info.rounds = rounds;
    info.nv = nv;
    info.nocc = A * ne;
    info.nbr = A * ne * (A - 1);
    if (ne == 0) return kEmptyStateHash;
    uint64_t r = kFnvOffset;
    r = fnv(r, nv);
    r = fnv(r, ne);
    r = fnv(r, vs);
    r = fnv(r, es);
    r = fnv(r, cs);
    return r;
}

}  // namespace
}  // namespace hgx
