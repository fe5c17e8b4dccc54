// Orientation: degrees, (degree, id) orientation with order-preserving compaction of every
// adjacency list to its out-neighbours, and the per-vertex out-list descriptors.
//
// Restates on the device what DistributedGraph::orient (distributed_graph.h:538-566) with
// node_ordering::degree_outward (distributed_graph.h:148-163) computes: u is kept in the
// out-list of v iff (deg(v), v) < (deg(u), u).  The reference partitions each list in place;
// here the input CSR is read-only and the out-lists are written to a separate gapped array.
// A list that one merge-path tile holds entirely keeps its input order.  A list that spans
// tiles is assembled from per-tile pieces; the id sort (sort_neighborhoods,
// distributed_graph.h:578-593) runs only where a strategy needs sorted lists.
#include "ktri_device.cuh"
#include "ktri_kernels.h"

namespace ktri {

constexpr u32 TILE_BUCKETS = 4096;  // keys of a tile order

// deg[v] = first_out[v+1] - first_out[v]; zero the out-degrees and the per-vertex counts.
// Also tabulates the merge-path tile boundaries: vertex v covers the diagonals
// [first_out[v] + v, first_out[v+1] + v] (its slots and its end event), so every boundary
// k * TILE_BASE in that range crosses the path at vertex v.
// HUB: also a histogram of the degrees from HUB_MIN_DEGREE on (hub_bins[0, HUB_BINS), zeroed by the
// caller).  The block that finishes last turns it into the hub choice: the hubs are the vertices
// of the highest bins that together hold fewer than HUB_H; hub_bins[HUB_BINS + b] receives the number
// of hubs above bin b (the scatter's cursor) and hub_bins[2 * HUB_BINS + b] the same for the ranking.
constexpr int PREP_BLOCK = 256;
template <bool HUB>
__global__ void __launch_bounds__(PREP_BLOCK) k_prep(const u64* __restrict__ fo, u64 n, u64 nnz, u32* __restrict__ deg,
                                                     u32* __restrict__ dplus, u64* __restrict__ cnt,
                                                     u32* __restrict__ tile_i0, u32* __restrict__ hub_bins,
                                                     Control* ctl) {
    chain_begin();
    __shared__ u32 s_bins[HUB ? HUB_BINS : 1];
    if constexpr (HUB) {
        for (u32 b = threadIdx.x; b < HUB_BINS; b += PREP_BLOCK) s_bins[b] = 0;
        __syncthreads();
    }
    const u64 stride = (u64)gridDim.x * blockDim.x;
    const u64 nt = (n + nnz + TILE_BASE - 1) / TILE_BASE;
    u32 err = 0;
    for (u64 v = (u64)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
        u64 a = fo[v], b = fo[v + 1];
        u32 d = 0;
        if (b < a || b - a > 0xFFFFFFFFull || b > nnz) {
            err |= DEV_ERR_DEGREE;
        } else {
            d = (u32)(b - a);
            const u64 k0 = (a + v + TILE_BASE - 1) / TILE_BASE, k1 = (b + v) / TILE_BASE;
            for (u64 k = k0; k <= k1 && k < nt; ++k) tile_i0[k] = (u32)v;
        }
        deg[v] = d;
        dplus[v] = 0;
        if (cnt) cnt[v] = 0;
        if constexpr (HUB) {
            if (d >= HUB_MIN_DEGREE) atomicAdd(&s_bins[degree_bin(d)], 1u);
            // n is below HUB_MAX_N, so such a list repeats a neighbour; the orientation counts on shorter
            // ones (keys below HUB_FLAG, list starts at most 2^31 entries before a tile)
            if (d >= HUB_MAX_N) err |= DEV_ERR_DUPLICATE;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        tile_i0[nt] = (u32)n;
        if (fo[0] != 0 || fo[n] != nnz) err |= DEV_ERR_DEGREE;
    }
    if (err) atomicOr(&ctl->err, err);
    if constexpr (HUB) {
        __shared__ u32 s_last;
        __shared__ u32 s_warp[PREP_BLOCK / 32];
        __shared__ u32 s_bin, s_hubs, s_crowd;
        __syncthreads();
        for (u32 b = threadIdx.x; b < HUB_BINS; b += PREP_BLOCK)
            if (s_bins[b]) atomicAdd(&hub_bins[b], s_bins[b]);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(&ctl->prep_blocks, 1u) + 1 == gridDim.x;
        __syncthreads();
        if (!s_last) return;
        // vertices above each bin, from the highest bin down (thread t holds PER bins)
        constexpr int PER = HUB_BINS / PREP_BLOCK;
        if (threadIdx.x == 0) {
            s_bin = HUB_BINS;
            s_hubs = s_crowd = 0;
        }
        u32 c[PER];
        unsigned long long sum = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            c[k] = __ldcg(&hub_bins[HUB_BINS - 1 - (threadIdx.x * PER + k)]);
            sum += c[k];
        }
        // counts above 2 HUB_H do not matter: saturate, so that 32 bits hold every prefix
        u32 total;
        u32 run = block_exclusive_scan<PREP_BLOCK>(sum > 2 * HUB_H ? 2 * HUB_H : (u32)sum, s_warp, &total);
        u32 bin = HUB_BINS, upto = 0, crowd = 0;  // of this thread's bins: the last hub bin, hubs down to it, largest
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const u32 b = HUB_BINS - 1 - (threadIdx.x * PER + k);
            hub_bins[HUB_BINS + b] = run;
            hub_bins[2 * HUB_BINS + b] = run;
            const u32 next = run + (c[k] > 2 * HUB_H ? 2 * HUB_H : c[k]);
            if (next < HUB_H) {
                bin = b;
                upto = next;
                crowd = c[k] > crowd ? c[k] : crowd;
            }
            run = next < 4 * HUB_H ? next : 4 * HUB_H;
        }
        bin = __reduce_min_sync(0xFFFFFFFFu, bin);
        upto = __reduce_max_sync(0xFFFFFFFFu, upto);
        crowd = __reduce_max_sync(0xFFFFFFFFu, crowd);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&s_bin, bin);
            atomicMax(&s_hubs, upto);
            atomicMax(&s_crowd, crowd);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            ctl->hub_bin = s_bin;
            ctl->hubs = s_hubs;
            ctl->hub_crowd = s_crowd;
        }
    }
}

// The hubs' vertices by bin, unordered inside a bin (with their degrees: the ranking below
// overwrites deg).
__global__ void k_hub_place(u64 n, const u32* __restrict__ deg, u32* __restrict__ hub_bins, uint2* __restrict__ hub_tmp,
                            const Control* ctl) {
    chain_begin();
    if (ctl->hubs == 0 || (ctl->err & DEV_ERR_MASK)) return;
    const u32 low = ctl->hub_bin;
    const u64 stride = (u64)gridDim.x * blockDim.x;
    for (u64 v = (u64)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
        const u32 d = deg[v];
        if (d < HUB_MIN_DEGREE) continue;
        const u32 b = degree_bin(d);
        if (b >= low) hub_tmp[atomicAdd(&hub_bins[HUB_BINS + b], 1u)] = make_uint2((u32)v, d);
    }
}

// Where a bin holds more than HUB_CROWD hubs: the hubs by (degree, id), highest first, inside each chunk
// of HUB_CHUNK places (a bitonic network in shared memory; the places are in bin order already, so no
// hub leaves its bin).
constexpr u32 HUB_CHUNK = HUB_H / 32;  // k_hub_rank: a chunk per lane
constexpr u32 HUB_CROWD = 4096;        // reading a bin of this many takes 7 us, the sort of all chunks 9 us
__global__ void __launch_bounds__(HUB_CHUNK / 2) k_hub_sort(u64* hub_tmp, const Control* ctl) {
    chain_begin();
    __shared__ u64 s[HUB_CHUNK];  // degree << 32 | id, as hub_tmp holds them
    const u32 hubs = ctl->hubs, base = blockIdx.x * HUB_CHUNK;
    if (base >= hubs || ctl->hub_crowd <= HUB_CROWD || (ctl->err & DEV_ERR_MASK)) return;
    const u32 len = hubs - base < HUB_CHUNK ? hubs - base : HUB_CHUNK;
    for (u32 i = threadIdx.x; i < HUB_CHUNK; i += HUB_CHUNK / 2) s[i] = i < len ? hub_tmp[base + i] : 0ull;
    for (u32 k = 2; k <= HUB_CHUNK; k <<= 1) {
        for (u32 j = k >> 1; j > 0; j >>= 1) {
            __syncthreads();
            const u32 i = 2 * threadIdx.x - (threadIdx.x & (j - 1));
            const u64 a = s[i], b = s[i + j];
            if ((a < b) == ((i & k) == 0)) {
                s[i] = b;
                s[i + j] = a;
            }
        }
    }
    __syncthreads();
    for (u32 i = threadIdx.x; i < len; i += HUB_CHUNK / 2) hub_tmp[base + i] = s[i];
}

// Hub index = rank by (degree, id) from the top: the hubs above the bin plus those of the bin that
// order higher.  key[v] (the degree of every other vertex) becomes the hub's orientation key, so
// one gather gives a neighbour's place in the order and its hub index.
// A warp per hub, which reads its bin whole, or, where the bin is crowded, searches the sorted chunks the
// bin reaches into, one per lane.  With 31 000 vertices of one degree, reading the bin
// took 430 us (by blocks of 128 hubs that share their reads 260 us), sort and search take 45 us.
__global__ void k_hub_rank(const u32* __restrict__ hub_bins, const u64* hub_tmp, u32* __restrict__ hub_ids,
                           u32* __restrict__ key, const Control* ctl) {
    chain_begin();
    const u32 p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (p >= ctl->hubs || (ctl->err & DEV_ERR_MASK)) return;
    const u64 me = hub_tmp[p];
    const u32 b = degree_bin((u32)(me >> 32));
    const u32 first = hub_bins[2 * HUB_BINS + b], count = hub_bins[b], end = first + count;
    u32 higher = 0;
    if (count <= HUB_CROWD) {
        for (u32 q = first + lane; q < end; q += 32) higher += hub_tmp[q] > me ? 1u : 0u;
    } else {
        const u32 at = lane * HUB_CHUNK;  // the chunk's part of the bin, highest first
        const u32 from = at > first ? at : first, to = at + HUB_CHUNK < end ? at + HUB_CHUNK : end;
        u32 lo = from, hi = to > from ? to : from;
        while (lo < hi) {
            const u32 mid = (lo + hi) >> 1;
            if (hub_tmp[mid] > me) lo = mid + 1;
            else hi = mid;
        }
        higher = lo - from;
    }
    const u32 r = first + __reduce_add_sync(0xFFFFFFFFu, higher);
    if (lane == 0) {
        hub_ids[r] = (u32)me;
        key[(u32)me] = HUB_FLAG | (HUB_H - 1 - r);
    }
}

// Orientation of one merge-path tile of W = 32 * IPT diagonals per warp.  The tile holds the
// window vertices i0..i1 and the adjacency slots [j0, j1); every list with slots in the tile
// has one piece there, numbered in slot order.  Slots are taken 32 at a time, one per lane: the
// gathers, and the writes of what is kept, then touch the fewest lines.  All per-list work is done
// once per piece by the window's lanes, and a slot finds its piece by one population count over
// the bits of the pieces' first slots.
// Inside the tile all arithmetic is 32-bit (ids are below 2^32, slots relative to j0).
//   vertex pass  per window vertex with slots here: its piece's first slot as a bit of s_start, the
//                slot before it as a bit of s_stop, (key, id) of its vertex in s_piece
//   pass 1       per slot: its piece, the (key, id) decision, input checks; per row of 32 the kept
//                slots' mask and the kept slots before the row
//   piece pass   per window vertex: the tile ranks at the piece's ends (from the rows' masks), its
//                out-degree share (a plain store, or an atomic reservation for a piece of a split
//                list) and the gapped-array index of tile rank 0 for its entries
//   pass 2       kept entries written from registers, in slot order
// A list held by one tile keeps its input order.  A split list's pieces reserve their ranges
// with one atomic each; which lists are split follows from the tiles' bounds (SplitLists): a list
// of them kept with one counter took an atomic of one address per tile (130 k of them on RGG
// n = 2^20), which bounded the kernel: orientation of RGG-24 3.2 -> 2.4 ms without it.
// HUB: deg holds orientation keys (the degree, or a hub's key above every degree), a kept entry that
// is a hub goes to the hub array as its index and the others to headp, so a piece has two ranks
// and two shares of its out-list's length word (hubs << 16 | others, as everywhere with hubs).
// What bounds it: latency (a tile's offset, its slots, their keys, one after the other, with 32
// warps per SM of 64 registers) and instruction issue: 112 instructions per row of 32 slots, 172 when
// every slot carried its piece's ends and rank.  Measured (orientation phase, RGG-24 / RMAT n = 10^6
// / 512-graph batch): 3.7 / 0.42 / 3.5 ms in that form, 2.44 / 0.31 / 2.2 ms now.  Five blocks per SM
// spill: 2.29 / 0.33 / 2.25 ms.  Copying the next tile's slots to shared memory while one is at work
// (a persistent grid) takes the L1 cache that the keys' gathers use: 2.50 / 0.31 / 3.0 ms.
template <int IPT>
struct OrientWarp {
    static constexpr int W = 32 * IPT;
    union {
        uint2 piece[W];  // until the piece pass: key and id of the piece's vertex
        // then: the headp index of tile rank 0 for its entries (HUB: the indices in both arrays
        // relative to where the tile's first vertex would start, 32 bits each)
        u64 base[W];
    };
    uint4 row[IPT + 1];  // kept slots (others, hubs) of the row and the tile rank before it
    u32 start[IPT];      // a piece starts at this slot
    u32 stop[IPT];       // the next slot is another piece's or past the tile
};

template <int IPT, bool HUB>
__device__ __forceinline__ void orient_tile(OrientWarp<IPT>& sw, const u64* __restrict__ fo,
                                            const u32* __restrict__ head, u64 n, u64 nnz,
                                            const u32* __restrict__ deg, const u32* __restrict__ tile_i0,
                                            u32* __restrict__ headp, u16* __restrict__ hubp, u32* __restrict__ dplus,
                                            Control* ctl, u64 tile) {
    constexpr int W = 32 * IPT;
    constexpr u32 FULL = 0xFFFFFFFFu;
    static_assert(W <= 256 && IPT % 4 == 0, "piece numbers in bytes");
    const u32 lane = threadIdx.x & 31;
    const u64 total = n + nnz;
    const u64 d0 = tile * W;
    if (d0 >= total) return;
    const u64 d1 = d0 + W < total ? d0 + W : total;
    // tile_i0 holds base_tiles + 1 entries (the last is n), and tile + 1 <= base_tiles here
    const u64 i0 = tile_i0[tile], i1 = tile_i0[tile + 1];
    const u64 j0 = d0 - i0, j1 = d1 - i1;
    const u32 ns = (u32)(j1 - j0);
    if (ns == 0) return;  // only vertex ends: those lists have no slots here (out-degrees start at 0)
    const u32 n32 = (u32)n;  // n < 2^32: every id fits
    // every slot's neighbour and its key, all in flight before the window is read
    u32 y_r[IPT], dy_r[IPT];
    const u32* hl = head + j0 + lane;
#pragma unroll
    for (int it = 0; it < IPT; ++it) y_r[it] = (u32)it * 32 + lane < ns ? __ldcs(hl + it * 32) : 0u;
    u32 y_max = 0;
#pragma unroll
    for (int it = 0; it < IPT; ++it) {
        y_max = y_r[it] > y_max ? y_r[it] : y_max;
        // 0 past the tile and for an id out of range: below every owner's key, so never kept
        dy_r[it] = ((u32)it * 32 + lane < ns && y_r[it] < n32) ? __ldg(deg + y_r[it]) : 0u;
    }
    if (lane < IPT) {
        sw.start[lane] = 0;
        const u32 used = ns - 1;  // slots with a next one in the tile
        sw.stop[lane] = used >= (lane + 1) * 32 ? 0u : used <= lane * 32 ? FULL : FULL << (used - lane * 32);
    }
    __syncwarp();
    const u64 last_v = i1 < n ? i1 : n - 1;
    const u32 nwin = (u32)(last_v - i0) + 1;  // window vertices (at most W + 1)
    const u32 lt = (1u << lane) - 1u, le = lt | (1u << lane);
    u32 end_y = 0, end_nx = 1;  // the neighbours on both sides of the tile's end, when one list has both
    // the window vertex' piece starts at slot s0 and has the number q
    auto enter = [&](u64 v, u32 s0, u32 q, u32 key, u64 b) {
        if (b > j1) {
            end_y = head[j1 - 1];
            end_nx = head[j1];
        }
        atomicOr(&sw.start[s0 >> 5], 1u << (s0 & 31u));
        if (s0) atomicOr(&sw.stop[(s0 - 1) >> 5], 1u << ((s0 - 1) & 31u));
        sw.piece[q] = make_uint2(key, (u32)v);
    };
    // the first 32 window vertices with every lane present (lane 0's list may begin before the
    // tile); their bounds stay in registers for the piece pass
    const bool have0 = lane < nwin;
    const u64 a0 = have0 ? fo[i0 + lane] : 0, b0 = have0 ? fo[i0 + lane + 1] : 0;
    const bool in0 = have0 && b0 > a0 && a0 < j1 && b0 > j0;
    const u32 ball0 = __ballot_sync(FULL, in0);
    if (in0)
        enter(i0 + lane, a0 > j0 ? (u32)(a0 - j0) : 0u, __popc(ball0 & lt),
              HUB ? __ldg(deg + i0 + lane) : (u32)(b0 - a0), b0);
    for (u32 k0 = 32, q0 = __popc(ball0); k0 < nwin; k0 += 32) {
        const u64 v = i0 + k0 + lane;
        const bool have = k0 + lane < nwin;
        const u64 a = have ? fo[v] : 0, b = have ? fo[v + 1] : 0;
        const bool in = b > a && a < j1 && b > j0;
        const u32 ball = __ballot_sync(FULL, in);
        if (in) enter(v, (u32)(a - j0), q0 + __popc(ball & lt), HUB ? __ldg(deg + v) : (u32)(b - a), b);
        q0 += __popc(ball);
    }
    __syncwarp();
    bool dup = false, unsorted = false, self_loop = false;
    u32 q_r[IPT / 4];        // the slots' pieces, a byte each
    u32 rank = 0;            // kept entries of the tile before this row (HUB: hubs << 16 | others)
    u32 q_row = 0u - 1u;     // the last piece that starts before this row
#pragma unroll
    for (int it = 0; it < IPT; ++it) {
        if (it % 4 == 0) q_r[it / 4] = 0;
        if ((u32)it * 32 >= ns) continue;
        const u32 starts = sw.start[it], stop = sw.stop[it];
        const u32 q = q_row + __popc(starts & le);
        q_row += __popc(starts);
        q_r[it / 4] |= q << (8 * (it % 4));
        const uint2 px = sw.piece[q];
        const u32 y = y_r[it], dy = dy_r[it];
        const bool tie = dy == px.x;
        const bool kept = dy > px.x || (tie && y > px.y);
        self_loop |= tie && y == px.y;  // a slot past the tile has the key 0: no tie
        u32 km = __ballot_sync(FULL, kept), hm = 0;
        if constexpr (HUB) {
            hm = __ballot_sync(FULL, kept && dy >= HUB_FLAG);
            km &= ~hm;
        }
        // the next slot's neighbour (the next lane's, or lane 0's of the next row) when it belongs
        // to the same list: adjacent duplicates and order
        const u32 nx = __shfl_sync(FULL, (lane == 0 && it + 1 < IPT) ? y_r[it + 1 < IPT ? it + 1 : it] : y, lane + 1);
        if (!(stop & (le ^ lt))) {
            unsorted |= nx < y;
            dup |= nx == y;
        }
        if (lane == 0) sw.row[it] = make_uint4(km, hm, rank, 0);
        rank += __popc(km) + (HUB ? __popc(hm) << 16 : 0u);
    }
    // the row after the last slot: where a piece that fills the tile ends
    if (lane == 0 && (ns & 31u) == 0) sw.row[ns >> 5] = make_uint4(0, 0, rank, 0);
    dup |= end_nx == end_y;
    unsorted |= end_nx < end_y;
    const u32 err = (y_max >= n32 ? DEV_ERR_ID_RANGE : 0u) | (self_loop ? DEV_ERR_SELF_LOOP : 0u) |
                    (dup ? DEV_ERR_DUPLICATE : 0u) | (unsorted ? DEV_FLAG_UNSORTED : 0u);
    if (err & ~*(volatile u32*)&ctl->err) atomicOr(&ctl->err, err);
    __syncwarp();
    // piece pass: out-degree shares and where each piece's kept entries go
    const u64 ref = oriented_start(j0, i0), href = hub_start(ref, i0);  // HUB: origins of the 32-bit indices
    {
        auto rank_at = [&](u32 s) {
            const uint4 r = sw.row[s >> 5];
            const u32 m = (1u << (s & 31u)) - 1u;
            return r.z + __popc(r.x & m) + (HUB ? __popc(r.y & m) << 16 : 0u);
        };
        auto settle = [&](u64 v, u64 a, u64 b, u32 q) {
            const u32 first = rank_at(a > j0 ? (u32)(a - j0) : 0u);
            const u32 cnt = rank_at(b < j1 ? (u32)(b - j0) : ns) - first;
            u32 carry = 0;
            if (a < j0 || b > j1) {
                if (cnt) carry = atomicAdd(&dplus[v], cnt);
                if constexpr (HUB) {
                    // a half of the length word that overflows counts some neighbour twice (HUB_MAX_NNZ)
                    if ((carry & 0xFFFFu) + (cnt & 0xFFFFu) > 0xFFFFu || (carry >> 16) + (cnt >> 16) > 0xFFFFu)
                        atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
                }
            } else {
                dplus[v] = cnt;
            }
            const u64 start = oriented_start(a, v);
            if constexpr (HUB) {
                // differences stay below 2^31: a list begins at most its degree before the tile
                const u32 to = (u32)(start - ref) + (carry & 0xFFFFu) - (first & 0xFFFFu);
                const u32 hto = (u32)(hub_start(start, v) - href) + (carry >> 16) - (first >> 16);
                sw.base[q] = (u64)to | ((u64)hto << 32);
            } else {
                sw.base[q] = start + carry - first;
            }
        };
        if (in0) settle(i0 + lane, a0, b0, __popc(ball0 & lt));
        for (u32 k0 = 32, q0 = __popc(ball0); k0 < nwin; k0 += 32) {
            const u64 v = i0 + k0 + lane;
            const bool have = k0 + lane < nwin;
            const u64 a = have ? fo[v] : 0, b = have ? fo[v + 1] : 0;
            const bool in = b > a && a < j1 && b > j0;
            const u32 ball = __ballot_sync(FULL, in);
            if (in) settle(v, a, b, q0 + __popc(ball & lt));
            q0 += __popc(ball);
        }
    }
    __syncwarp();
#pragma unroll
    for (int it = 0; it < IPT; ++it) {
        if ((u32)it * 32 >= ns) continue;
        const uint4 r = sw.row[it];
        const u32 q = (q_r[it / 4] >> (8 * (it % 4))) & 0xFFu;
        if constexpr (HUB) {
            if (((r.x | r.y) >> lane) & 1u) {
                const u64 base = sw.base[q];
                if ((r.x >> lane) & 1u) {
                    const u32 at = (u32)base + (r.z & 0xFFFFu) + __popc(r.x & lt);
                    __stcs(headp + ref + (long long)(int)at, y_r[it]);
                } else {
                    const u32 at = (u32)(base >> 32) + (r.z >> 16) + __popc(r.y & lt);
                    __stcs(hubp + href + (long long)(int)at, (u16)(HUB_H - 1 - (dy_r[it] & ~HUB_FLAG)));
                }
            }
        } else {
            if ((r.x >> lane) & 1u) __stcs(headp + sw.base[q] + (r.z + __popc(r.x & lt)), y_r[it]);
        }
    }
}

// One tile per warp.  HUB: a graph without hubs (hubs = 0) runs the plain body, whose lists and
// length words are then the same.
template <int BLOCK, int IPT, bool HUB>
__global__ void __launch_bounds__(BLOCK, ORIENT_BLOCKS)
    k_orient(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n, u64 nnz, const u32* __restrict__ deg,
             const u32* __restrict__ tile_i0, u32* __restrict__ headp, u16* __restrict__ hubp, u32* __restrict__ dplus,
             Control* ctl, u64 tile_begin) {
    chain_begin();
    __shared__ OrientWarp<IPT> s_warp[BLOCK / 32];
    if (ctl->err & DEV_ERR_MASK) return;
    const int wid = threadIdx.x >> 5;
    const u64 tile = (tile_begin + blockIdx.x) * (BLOCK / 32) + wid;
    if (HUB && ctl->hubs)
        orient_tile<IPT, true>(s_warp[wid], fo, head, n, nnz, deg, tile_i0, headp, hubp, dplus, ctl, tile);
    else
        orient_tile<IPT, false>(s_warp[wid], fo, head, n, nnz, deg, tile_i0, headp, nullptr, dplus, ctl, tile);
}

// Out-list descriptors, and the (owner, segment) tiles of owners above the small
// out-degree threshold.  The slots in the tile lists and in the list of long hub lists are reserved
// once per block and 256 vertices: with an atomic per warp the counters' L2 slice was 70 % busy (RMAT
// n = 2^24: 470 us, 338 us so).  order_hist: the tile orders' histograms, zeroed here.
constexpr int DESC_BLOCK = 256;
template <typename OffT, bool HUB>
__global__ void __launch_bounds__(DESC_BLOCK) k_desc(const u64* __restrict__ fo, u64 n, const u32* __restrict__ dplus,
                                                     Desc<OffT>* __restrict__ vdesc, u16* __restrict__ hubp,
                                                     u32* __restrict__ top_info, u32* __restrict__ top_long,
                                                     uint2* __restrict__ mtiles, uint2* __restrict__ ltiles,
                                                     u32 small_d, u32 medium_d, u32 seg, u32* __restrict__ order_hist,
                                                     Control* ctl) {
    chain_begin();
    constexpr int WARPS = DESC_BLOCK / 32;
    __shared__ u32 s_sum[3][WARPS];  // of each warp: medium tiles, large tiles, long hub lists
    __shared__ u64 s_at[3][WARPS];   // where its entries go
    if (ctl->err & DEV_ERR_MASK) return;
    const bool plain = HUB && ctl->hubs == 0;
    const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const u64 stride = (u64)gridDim.x * DESC_BLOCK;
    if (order_hist)
        for (u64 k = (u64)blockIdx.x * DESC_BLOCK + threadIdx.x; k < 2 * TILE_BUCKETS; k += stride) order_hist[k] = 0;
    for (u64 base = (u64)blockIdx.x * DESC_BLOCK; base < n; base += stride) {
        const u64 v = base + threadIdx.x;
        u32 nt = 0;
        bool large = false, is_long = false;
        if (v < n) {
            const u64 a = fo[v], b = fo[v + 1];
            const u32 d = dplus[v];
            Desc<OffT> ds;
            set_list_start(ds, oriented_start(a, v));
            ds.d = d;
            if constexpr (sizeof(OffT) == 8) ds.pad = 0;
            vdesc[v] = ds;
            if constexpr (HUB) {
                // oriented without hubs: a count past the low half is of a list with duplicates, too
                if (plain && d > 0xFFFFu) atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
                const u64 hs = hub_start(list_start(ds), v);
                for (u32 k = hub_len<HUB>(d); k & 7u; ++k) hubp[hs + k] = (u16)HUB_PAD;
                top_info[v] = 0;
                is_long = hub_len<HUB>(d) > HUB_TOP_LIST;
            }
            // no tiles at all without tile arrays (the reference strategies pass none)
            if (mtiles && ltiles && list_len<HUB>(d) > small_d) nt = (u32)((b - a + seg - 1) / seg);
            large = list_len<HUB>(d) > medium_d;
        }
        if (!__syncthreads_or(nt || is_long)) continue;
        u32 before[2], mine[2] = {large ? 0 : nt, large ? nt : 0};
#pragma unroll
        for (int cls = 0; cls < 2; ++cls) {
            u32 incl = mine[cls];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) s_sum[cls][wid] = incl;
            before[cls] = incl - mine[cls];
        }
        const u32 longs = __ballot_sync(0xFFFFFFFFu, is_long);
        if (lane == 0) s_sum[2][wid] = __popc(longs);
        __syncthreads();
        if (threadIdx.x < 3) {
            u64 total = 0;
            for (int w = 0; w < WARPS; ++w) {
                s_at[threadIdx.x][w] = total;
                total += s_sum[threadIdx.x][w];
            }
            u64 at = 0;
            if (total)
                at = threadIdx.x == 0   ? atomicAdd(&ctl->medium_tiles, total)
                     : threadIdx.x == 1 ? atomicAdd(&ctl->large_tiles, total)
                                        : atomicAdd(&ctl->hub_long, (u32)total);
            for (int w = 0; w < WARPS; ++w) s_at[threadIdx.x][w] += at;
        }
        __syncthreads();
        if (HUB && is_long) top_long[s_at[2][wid] + __popc(longs & ((1u << lane) - 1))] = (u32)v;
        const u64 my = s_at[large][wid] + (large ? before[1] : before[0]);
        uint2* out = large ? ltiles : mtiles;
        for (u32 s = 0; s < nt; ++s) out[tile_at(large, my + s)] = make_uint2((u32)v, s);
    }
}

// Top bitmaps of the long hub lists, one warp per list: the entries below HUB_TOP move to a bitmap,
// the others close up at the front of the list in their order (a row is read before anything is
// written at or past its start).
constexpr int TOPS_BLOCK = 256;
__global__ void __launch_bounds__(TOPS_BLOCK) k_hub_tops(const Desc<u32>* __restrict__ vdesc, u16* __restrict__ hubp,
                                                         const u32* __restrict__ top_long, u32* __restrict__ top_info,
                                                         uint2* __restrict__ top_bits, u32 cap, Control* ctl) {
    chain_begin();
    __shared__ __align__(8) u32 s_bits[TOPS_BLOCK / 32][HUB_TOP / 32];
    static_assert(HUB_TOP / 32 == 64, "two words per lane");
    if (ctl->err & DEV_ERR_MASK) return;
    const u32 lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    u32* bits = s_bits[threadIdx.x >> 5];
    if (blockIdx.x == 0 && threadIdx.x < 32) top_bits[threadIdx.x] = make_uint2(0, 0);  // the empty bitmap
    const u32 count = ctl->hub_long;
    const u32 nwarps = gridDim.x * (TOPS_BLOCK / 32);
    u32 dup = 0;
    for (u32 i = (blockIdx.x * TOPS_BLOCK + threadIdx.x) >> 5; i < count; i += nwarps) {
        const u32 v = top_long[i];
        const Desc<u32> d = load_desc(vdesc + v);
        const u32 len = hub_len<true>(d.d);
        u16* lst = hubp + hub_start(list_start(d), v);
        u32 tops = 0;
        for (u32 k = lane; k < len; k += 32) tops += lst[k] < HUB_TOP ? 1u : 0u;
        tops = __reduce_add_sync(0xFFFFFFFFu, tops);
        if (tops < HUB_TOP_MIN) continue;
        u32 slot = 0;
        if (lane == 0) slot = atomicAdd(&ctl->hub_tops, 1u) + 1;
        slot = __shfl_sync(0xFFFFFFFFu, slot, 0);
        if (slot >= cap) continue;
        bits[lane] = 0;
        bits[lane + 32] = 0;
        __syncwarp();
        u32 out = 0;
        for (u32 k0 = 0; k0 < len; k0 += 32) {
            const u32 h = k0 + lane < len ? lst[k0 + lane] : HUB_PAD;
            const bool other = k0 + lane < len && h >= HUB_TOP;
            if (h < HUB_TOP && (atomicOr(&bits[h >> 5], 1u << (h & 31u)) & (1u << (h & 31u)))) dup = 1;
            const u32 ball = __ballot_sync(0xFFFFFFFFu, other);
            if (other) lst[out + __popc(ball & lt)] = (u16)h;
            out += __popc(ball);
        }
        if (lane < ((8u - out) & 7u)) lst[out + lane] = (u16)HUB_PAD;
        __syncwarp();
        top_bits[(u64)slot * 32 + lane] = reinterpret_cast<const uint2*>(bits)[lane];
        if (lane == 0) top_info[v] = (slot << 12) | tops;
        __syncwarp();
    }
    if (dup) atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
}

// Large-owner tiles in the order of the first vertex each segment streams (a counting sort
// on the top id bits).  Input adjacency lists are mostly in id order, so tiles that run at the
// same time then stream out-lists from the same region of the list array, and the L2 cache
// serves the repeats.  Counts do not depend on the order.

// Sort key of a tile (TILE_BY_VERTEX): the top id bits of the first vertex its segment
// streams; (TILE_BY_DEGREE): the owner's out-degree, largest first (longest tiles first);
// (TILE_BY_COST): the key k_tile_cost left.
__device__ __forceinline__ u32 tile_key(const u64* fo, const u32* head, const u32* dplus, uint2 tl, u32 seg,
                                        u32 shift, u32 mode, bool hub, u32 cost_key) {
    u32 key;
    if (mode == TILE_BY_COST) {
        key = cost_key;
    } else if (mode == TILE_BY_DEGREE) {
        const u32 d = hub ? list_len<true>(dplus[tl.x]) : dplus[tl.x];
        key = d >= TILE_BUCKETS ? 0u : TILE_BUCKETS - 1 - d;
    } else {
        key = __ldg(head + fo[tl.x] + (u64)tl.y * seg) >> shift;
    }
    return key < TILE_BUCKETS ? key : TILE_BUCKETS - 1;
}

// The work of each tile, for TILE_BY_COST: the entries its owner x streams over the tile's
// segment, sum of d+(y) over the neighbours y below x in (out-degree, id) -- the edge cost of
// the reference's DPD cost function (cost_function.h:287-376, cetric_edge_iterator.h:584-593)
// restated for owner-side tiles.  One warp per tile; the key orders heaviest first on a
// log scale (7 fractional bits).
__global__ void k_tile_cost(const u64* __restrict__ fo, const u32* __restrict__ head, const u32* __restrict__ dplus,
                            TileOrders orders, u32 seg, bool hub, Control* ctl) {
    chain_begin();
    if (ctl->err & DEV_ERR_MASK) return;
    const TileOrder& o = orders.of[blockIdx.y];
    const u64 nt = *(volatile const unsigned long long*)o.count;
    const int lane = threadIdx.x & 31;
    const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
    for (u64 t = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += nwarps) {
        const uint2 tl = o.tiles[tile_at(o.back, t)];
        const u64 x = tl.x;
        const u32 dx = hub ? list_len<true>(dplus[x]) : dplus[x];
        const u64 a = fo[x] + (u64)tl.y * seg, e1 = fo[x + 1], b = a + seg < e1 ? a + seg : e1;
        u64 cost = 0;
        for (u64 e = a + lane; e < b; e += 32) {
            const u32 y = __ldg(head + e);
            const u32 word = __ldg(dplus + y), dy = hub ? list_len<true>(word) : word;
            if (dy > 0 && key_less(dy, y, dx, x)) cost += dy;
        }
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) cost += __shfl_down_sync(0xFFFFFFFFu, cost, k);
        if (lane == 0) {
            const u32 c = cost > 0xFFFFFFFFull ? 0xFFFFFFFFu : (u32)cost;
            const u32 lg = 31 - __clz(c | 1u);
            const u32 frac = lg >= 7 ? (c >> (lg - 7)) & 0x7Fu : (c << (7 - lg)) & 0x7Fu;
            const u32 bucket = lg * 128 + frac;  // < 32 * 128 = TILE_BUCKETS
            o.keys[tile_at(o.back, t)] = TILE_BUCKETS - 1 - bucket;
        }
    }
}

// Tiles [t0, t1) of block b when the tiles are cut into gridDim.x contiguous chunks.
__device__ __forceinline__ void tile_chunk(u64 nt, u64& t0, u64& t1) {
    const u64 per = (nt + gridDim.x - 1) / gridDim.x;
    t0 = (u64)blockIdx.x * per;
    t1 = t0 + per < nt ? t0 + per : nt;
    if (t0 > t1) t0 = t1;
}

// Histogram of the tiles' keys.  Each block counts its contiguous chunk in shared memory and
// adds the non-zero counts to the global histogram (one atomic per key present in the chunk,
// not per tile: the medium tiles' degree keys crowd onto a few hundred values).  The keys are
// left in keys[t] for the scatter (TILE_BY_COST finds them there already).
constexpr int TILE_ORDER_BLOCK = 256;
__global__ void __launch_bounds__(TILE_ORDER_BLOCK) k_tile_hist(const u64* __restrict__ fo,
                                                                const u32* __restrict__ head,
                                                                const u32* __restrict__ dplus, TileOrders orders,
                                                                u32 seg, u32 shift, bool hub, u32* hist,
                                                                Control* ctl) {
    chain_begin();
    __shared__ u32 s_cnt[TILE_BUCKETS];
    if (ctl->err & DEV_ERR_MASK) return;
    const TileOrder& o = orders.of[blockIdx.y];
    hist += blockIdx.y * TILE_BUCKETS;
    const u64 nt = *(volatile const unsigned long long*)o.count;
    u64 t0, t1;
    tile_chunk(nt, t0, t1);
    if (t0 == t1) return;
    for (u32 k = threadIdx.x; k < TILE_BUCKETS; k += TILE_ORDER_BLOCK) s_cnt[k] = 0;
    __syncthreads();
    for (u64 t = t0 + threadIdx.x; t < t1; t += TILE_ORDER_BLOCK) {
        const long long at = tile_at(o.back, t);
        const u32 key = tile_key(fo, head, dplus, o.tiles[at], seg, shift, o.mode, hub, o.keys[at]);
        if (o.mode != TILE_BY_COST) o.keys[at] = key;
        atomicAdd(&s_cnt[key], 1u);
    }
    __syncthreads();
    for (u32 k = threadIdx.x; k < TILE_BUCKETS; k += TILE_ORDER_BLOCK)
        if (s_cnt[k]) atomicAdd(&hist[k], s_cnt[k]);
}

// 256 threads: a block this small also fits beside the serving engine's resident blocks.
constexpr int TILE_SCAN_BLOCK = 256;
__global__ void __launch_bounds__(TILE_SCAN_BLOCK) k_tile_scan(u32* hist, Control* ctl) {
    chain_begin();
    constexpr int PER = TILE_BUCKETS / TILE_SCAN_BLOCK;
    __shared__ u32 s_warp[TILE_SCAN_BLOCK / 32];
    if (ctl->err & DEV_ERR_MASK) return;
    hist += blockIdx.x * TILE_BUCKETS;
    u32 v[PER], t = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        v[k] = hist[threadIdx.x * PER + k];
        t += v[k];
    }
    u32 total;
    u32 run = block_exclusive_scan<TILE_SCAN_BLOCK>(t, s_warp, &total);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        hist[threadIdx.x * PER + k] = run;
        run += v[k];
    }
}

// Scatter of the tiles into key order (cursor = the scanned histogram).  Each block counts its
// chunk's keys again, reserves one range per key present with one atomic, and hands out the
// positions inside its ranges with shared-memory atomics.
__global__ void __launch_bounds__(TILE_ORDER_BLOCK) k_tile_scatter(TileOrders orders, u32* cursor, Control* ctl) {
    chain_begin();
    __shared__ u32 s_pos[TILE_BUCKETS];
    if (ctl->err & DEV_ERR_MASK) return;
    const TileOrder& o = orders.of[blockIdx.y];
    cursor += blockIdx.y * TILE_BUCKETS;
    const u64 nt = *(volatile const unsigned long long*)o.count;
    u64 t0, t1;
    tile_chunk(nt, t0, t1);
    if (t0 == t1) return;
    for (u32 k = threadIdx.x; k < TILE_BUCKETS; k += TILE_ORDER_BLOCK) s_pos[k] = 0;
    __syncthreads();
    for (u64 t = t0 + threadIdx.x; t < t1; t += TILE_ORDER_BLOCK) atomicAdd(&s_pos[o.keys[tile_at(o.back, t)]], 1u);
    __syncthreads();
    for (u32 k = threadIdx.x; k < TILE_BUCKETS; k += TILE_ORDER_BLOCK) {
        const u32 c = s_pos[k];
        if (c) s_pos[k] = atomicAdd(&cursor[k], c);
    }
    __syncthreads();
    for (u64 t = t0 + threadIdx.x; t < t1; t += TILE_ORDER_BLOCK) {
        const long long at = tile_at(o.back, t);
        o.sorted[tile_at(o.back, atomicAdd(&s_pos[o.keys[at]], 1u))] = o.tiles[at];
    }
}

// ---- launchers ------------------------------------------------------------------------

u64 tile_order_scratch_words() { return 2ull * TILE_BUCKETS; }

void launch_order_tiles(const u64* fo, const u32* head, const u32* dplus, u64 n, const TileOrders& orders, u32 seg,
                        bool hub, u32* hist, Control* ctl, int num_sms, LaunchStream st) {
    if (n == 0) return;
    u32 bits = 0;
    while ((1ull << bits) < n) ++bits;
    const u32 shift = bits > 12 ? bits - 12 : 0;
    if (orders.of[0].mode == TILE_BY_COST)
        launch_chained(k_tile_cost, dim3(num_sms * 8, 2), 256, 0, st, fo, head, dplus, orders, seg, hub, ctl);
    launch_chained(k_tile_hist, dim3(num_sms * 4, 2), TILE_ORDER_BLOCK, 0, st, fo, head, dplus, orders, seg, shift,
                   hub, hist, ctl);
    launch_chained(k_tile_scan, 2, TILE_SCAN_BLOCK, 0, st, hist, ctl);
    launch_chained(k_tile_scatter, dim3(num_sms * 4, 2), TILE_ORDER_BLOCK, 0, st, orders, hist, ctl);
}

void launch_prep(const u64* fo, u64 n, u64 nnz, u32* deg, u32* dplus, u64* cnt, u32* tile_i0, const HubState& hub,
                 Control* ctl, int num_sms, LaunchStream st) {
    if (n == 0) return;
    const u64 blocks = (n + PREP_BLOCK - 1) / PREP_BLOCK;
    const u64 cap = (u64)num_sms * 8;
    const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
    if (!hub) {
        launch_chained(k_prep<false>, grid, PREP_BLOCK, 0, st, fo, n, nnz, deg, dplus, cnt, tile_i0, nullptr, ctl);
        return;
    }
    launch_chained(k_prep<true>, grid, PREP_BLOCK, 0, st, fo, n, nnz, deg, dplus, cnt, tile_i0, hub.bins, ctl);
    launch_chained(k_hub_place, grid, 256, 0, st, n, deg, hub.bins, hub.tmp, ctl);
    auto* tmp = reinterpret_cast<u64*>(hub.tmp);  // {id, degree} as one number
    launch_chained(k_hub_sort, HUB_H / HUB_CHUNK, HUB_CHUNK / 2, 0, st, tmp, ctl);
    launch_chained(k_hub_rank, HUB_H / 8, 256, 0, st, hub.bins, tmp, hub.ids, deg, ctl);
}

void launch_hub_tops(const void* vdesc, const HubState& hub, Control* ctl, int num_sms, LaunchStream st) {
    launch_chained(k_hub_tops, num_sms * 8, TOPS_BLOCK, 0, st, reinterpret_cast<const Desc<u32>*>(vdesc), hub.lists,
                   hub.top_long, hub.top_info, hub.top_bits, hub.top_cap, ctl);
}

u64 hub_bins_words() { return 3ull * HUB_BINS; }
size_t hub_bins_zeroed() { return sizeof(u32) * HUB_BINS; }

u64 orient_tiles(u64 n, u64 nnz) { return (n + nnz + ORIENT_TILE - 1) / ORIENT_TILE; }

void launch_orient(const u64* fo, const u32* head, u64 n, u64 nnz, const u32* deg, const u32* tile_i0, u32* headp,
                   const HubState& hub, u32* dplus, Control* ctl, LaunchStream st, u64 tile_begin,
                   u64 tile_end) {
    constexpr int BLOCK = ORIENT_BLOCK, IPT = ORIENT_IPT;
    const u64 tiles = orient_tiles(n, nnz);
    if (tile_end > tiles) tile_end = tiles;
    if (tile_begin >= tile_end) return;
    const unsigned grid = (unsigned)(tile_end - tile_begin);
    if (hub)
        launch_chained(k_orient<BLOCK, IPT, true>, grid, BLOCK, 0, st, fo, head, n, nnz, deg, tile_i0, headp, hub.lists,
                       dplus, ctl, tile_begin);
    else
        launch_chained(k_orient<BLOCK, IPT, false>, grid, BLOCK, 0, st, fo, head, n, nnz, deg, tile_i0, headp, nullptr,
                       dplus, ctl, tile_begin);
}

template <typename OffT, bool HUB>
void launch_desc(const u64* fo, u64 n, const u32* dplus, void* vdesc, const HubState& hub, uint2* mtiles,
                 uint2* ltiles, u32 small_d, u32 medium_d, u32 seg, u32* order_hist, Control* ctl, int num_sms,
                 LaunchStream st) {
    if (n == 0) return;
    u64 blocks = (n + DESC_BLOCK - 1) / DESC_BLOCK;
    u64 cap = (u64)num_sms * 8;
    launch_chained(k_desc<OffT, HUB>, (unsigned)(blocks < cap ? blocks : cap), DESC_BLOCK, 0, st, fo, n, dplus,
                   reinterpret_cast<Desc<OffT>*>(vdesc), hub.lists, hub.top_info, hub.top_long, mtiles, ltiles, small_d,
                   medium_d, seg, order_hist, ctl);
}

#define KTRI_INST(OffT, HUB)                                                                                     \
    template void launch_desc<OffT, HUB>(const u64*, u64, const u32*, void*, const HubState&, uint2*, uint2*,    \
                                         u32, u32, u32, u32*, Control*, int, LaunchStream);
KTRI_INST(u32, false)
KTRI_INST(u32, true)
KTRI_INST(u64, false)
#undef KTRI_INST

}  // namespace ktri
