// Owner-side hash counting (KTRI_METHOD_AUTO): the GPU form of CetricEdgeIterator::run_local
// (cetric_edge_iterator.h:889-1066) with intersection() (intersection.h:41-79).
//
// Every undirected edge {x,y} contributes |N+(x) ∩ N+(y)| triangles, where N+ is the
// out-list after orientation by (degree, id); the sum over all edges is the triangle total,
// exactly as the reference's sum over oriented edges (v,u) of |N+(v) ∩ N+(u)|.  Each edge is
// evaluated once: one endpoint's out-list sits in a shared-memory hash table and the other's is
// streamed through it.  Edges between two out-degrees of at most small_outdegree are evaluated
// at their tail; the others at their "owner", the endpoint whose (out-degree, id) is larger, so
// that their work is min(|N+(x)|, |N+(y)|) probes.
//
// Per-vertex counts: a hit w of edge {x,y} is the triangle {x,y,w}.  w is a key of the
// table: its hits accumulate in a shared-memory counter next to the key and are flushed once per
// table.  The streamed endpoint gets its list's hits, the other one its table's total.
//
// The kernels (the bounds are runtime options, at most SMALL_D and MEDIUM_D):
//   k_count_small: the edges between out-degrees of at most small_outdegree, groups of tails per
//     warp, one streamed list per pair of lanes.  No block barrier.
//   k_count_medium: owners up to medium_outdegree, one warp per (owner, segment) tile with the
//     warp's own table, so tiles need no block barrier.
//   k_count_large: larger owners, one (owner, segment) tile per block iteration.  Short
//     streamed lists are handled one per thread while the segment is scanned; longer ones are
//     queued and taken one at a time by whole warps (one entry per lane, eight loads in
//     flight), so no block-wide barrier separates the lists.  Every streamed entry is tested
//     against a one-hash filter of the owner's keys first, and only the survivors are looked up,
//     packed 32 at a time.
// Graphs with split lists (hubs) have k_count_hub for the hub part of all owner tiles, and
// k_count_medium takes the other entries of all of them.
#include "ktri_device.cuh"
#include "ktri_kernels.h"

namespace ktri {

constexpr size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// Bulk (TMA) copies into shared memory, completed on an mbarrier.  The copy engine moves a
// 16-byte-aligned run of bytes (a multiple of 16) from global to shared memory and counts the
// bytes against the barrier's expected transaction count.
__device__ __forceinline__ u32 smem_u32(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, u32 count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, u32 bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, u32 bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, u32 parity) {
    u32 ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the barrier's phase of the given parity; gives up after `polls` polls (each poll
// itself blocks for a short hardware-defined time) and reports false.  polls = 0 gives up at
// once without looking.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, u32 parity, u32 polls) {
    for (u32 it = 0; it < polls; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Loads of the counting bodies.  The standalone kernels read through the read-only path
// (CG = false): their inputs do not change while they run.  The serving engine (CG = true) runs
// across many batches whose buffers other kernels rewrite meanwhile, so it reads at L2 only,
// where those writes are visible, never from lines an SM cached earlier.
template <bool CG, typename T>
__device__ __forceinline__ T ld_in(const T* p) {
    if constexpr (CG) return __ldcg(p);
    else return __ldg(p);
}
template <bool CG, typename OffT>
__device__ __forceinline__ Desc<OffT> ld_desc(const Desc<OffT>* p) {
    if constexpr (!CG) {
        return load_desc(p);
    } else if constexpr (sizeof(OffT) == 4) {
        const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
        return Desc<OffT>{v.x, v.y};
    } else {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p));
        return Desc<OffT>{(u64)v.x | ((u64)v.y << 32), v.z, 0};
    }
}

// Hit counters of the owners' tables are 16-bit, two per word: a key gets at most one hit per
// streamed list, and a tile streams at most LARGE_SEG (block and warp kernels) or one tile's
// slots (small-owner kernel) lists, so they cannot overflow.
__device__ __forceinline__ void hit16(u32* hits32, u32 slot) { atomicAdd(&hits32[slot >> 1], 1u << ((slot & 1u) << 4)); }
__device__ __forceinline__ u32 read16(const u32* hits32, u32 slot) { return (hits32[slot >> 1] >> ((slot & 1u) << 4)) & 0xFFFFu; }

// Count a lookup of w in a table of buckets of four: on a hit, add one to the slot's 16-bit counter and
// return 1.
__device__ __forceinline__ u32 bucket_probe16(const u32* keys, u32* hits32, u32 lg, u32 w) {
    const u32 nb_mask = (1u << (lg - 2)) - 1;
    u32 b = bucket_home(w, lg);
    for (u32 it = 0; it <= nb_mask; ++it) {
        const uint4 q = *reinterpret_cast<const uint4*>(keys + 4 * b);
        const bool m0 = q.x == w, m1 = q.y == w, m2 = q.z == w, m3 = q.w == w;
        if (m0 | m1 | m2 | m3) {
            hit16(hits32, 4 * b + (m0 ? 0u : (m1 ? 1u : (m2 ? 2u : 3u))));
            return 1u;
        }
        if (q.w == EMPTY_KEY) return 0u;
        b = (b + 1) & nb_mask;
    }
    return 0u;
}

// Index of the segment holding item base + lane, for segments that start at strictly increasing
// positions: before = segments started at or below base (at least one), starts = bit p set when
// a segment starts at base + p (p in 1..31).
__device__ __forceinline__ u32 segment_of(u32 before, u32 starts, u32 le_mask) {
    return before - 1 + __popc(starts & le_mask);
}
// Bit (s - base) for a segment start s inside (base, base + 32), else 0.
__device__ __forceinline__ u32 start_bit(bool have, u32 s, u32 base) {
    return (have && s > base && s < base + 32) ? 1u << (s - base) : 0u;
}

// The same lookup without early exits: one bucket read, a walk along full buckets only when
// the home bucket is full and holds no w (rare at the tables' load factors), and a predicated
// hit count, so the lanes of a warp that look up 32 packed filter survivors stay together.
__device__ __forceinline__ u32 bucket_probe16_flat(const u32* keys, u32* hits32, u32 lg, u32 w) {
    const u32 nb_mask = (1u << (lg - 2)) - 1;
    u32 b = bucket_home(w, lg);
    uint4 q = *reinterpret_cast<const uint4*>(keys + 4 * b);
    for (u32 it = 0; it < nb_mask && q.w != EMPTY_KEY && q.x != w && q.y != w && q.z != w && q.w != w; ++it) {
        b = (b + 1) & nb_mask;
        q = *reinterpret_cast<const uint4*>(keys + 4 * b);
    }
    const u32 slot = q.x == w ? 0u : (q.y == w ? 1u : (q.z == w ? 2u : (q.w == w ? 3u : 4u)));
    if (slot < 4u) hit16(hits32, 4 * b + slot);
    return slot < 4u ? 1u : 0u;
}

// Small edges (k_count_small), warp-granular: the edges (v, u) whose endpoints both have an
// out-degree of at most small_outdegree, each counted at its tail v.  A warp takes a few
// consecutive vertices and counts their out-lists in groups of up to GROUP tails that hold up to
// QCAP keys together.  A key is both an entry of its tail's table and an edge whose head's list
// is streamed through that table, so one pass over the keys builds the tables and the queue, and
// neither the input adjacency nor the lower neighbours are read.  The queue is counting-sorted
// by list length and streamed longest first, a list per pair of lanes.  Only __syncwarp orders the
// phases: the warps of a block never wait for one another.
//
// What bounds it: the shared-memory pipe (89 % busy on RGG n = 2^20, where half of the lookups hit;
// issue 68 %).  A lookup reads one bucket of two keys (8 bytes, about six wavefronts per 32 random
// buckets) and never walks: a table of 3 d buckets for d keys is rebuilt with another multiplier
// until no bucket holds more than two (about 0.013 d overfull buckets expected, so most tables of
// d <= 32 succeed at once), and a table that never does is searched entry by entry.
// Measured (this kernel, RGG 2^20 / RGG-24 / G(n,m) n = 10^6 of degree 60): one table per owner in
// buckets of four with early exits, streamed over the whole adjacency 0.915 / 13.2 ms / -; tails
// with a list per lane 0.514 / 7.55 / 3.22 ms; with keys placed by stores instead of
// compare-and-swap, the queue sorted by ballots and a list per pair of lanes 0.508 / 7.43 / 2.21 ms.
// The head's list is streamed instead of the shorter one: 1.0x to 1.05x the entries on uniform and
// geometric graphs.
template <typename OffT, bool HUB>
struct SmallWarpLayout {
    static constexpr int GROUP = 16;             // tails per group
    static constexpr int QCAP = 128;             // keys (and queued lists) of a group
    static constexpr int ROWS = QCAP / 32;       // keys per lane
    static constexpr int NB = 3 * QCAP;          // buckets: three per key
    static constexpr int MAX_TRIES = 16;         // multipliers tried per table
    // u32 words per warp
    static constexpr int W_KEYS = 0;                                    // two keys per bucket
    static constexpr int W_HITS = W_KEYS + 2 * NB;                      // two 16-bit counters per bucket
    static constexpr int W_REC = W_HITS + NB;                           // tail records (uint4)
    static constexpr int W_QS = W_REC + 4 * GROUP;                      // list starts (OffT), by key
    static constexpr int W_OS = W_QS + QCAP * (int)(sizeof(OffT) / 4);  // tails' list starts (OffT)
    // by key: slot << 16 | tail << 12 | hubs << 6 | others
    static constexpr int W_QM = W_OS + GROUP * (int)(sizeof(OffT) / 4);
    static constexpr int W_QH = W_QM + QCAP;                            // HUB: hub list starts (16-byte groups), by key
    static constexpr int W_TOT = W_QH + (HUB ? QCAP : 0);               // tails' hit totals
    static constexpr int W_VTX = W_TOT + GROUP;                         // tails' vertices
    static constexpr int W_BIN = W_VTX + GROUP;                         // lists by length in 16-byte groups
    static constexpr int W_ORD = W_BIN + 32;                            // queue order (u16)
    static constexpr int PER_WARP = (W_ORD + QCAP / 2 + 3) & ~3;
    static constexpr size_t bytes(int warps) { return sizeof(u32) * PER_WARP * warps; }
};

constexpr u32 NO_SLOT = 1023;  // a key without a table slot (its tail's table could not be built)

// A warp's tables are empty between groups: keys and counters are cleared as they are flushed.
template <typename OffT, bool HUB>
__device__ __forceinline__ void small_init(u32* base) {
    using L = SmallWarpLayout<OffT, HUB>;
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < 2 * L::NB; i += 32) base[L::W_KEYS + i] = EMPTY_KEY;
    for (int i = lane; i < L::NB; i += 32) base[L::W_HITS + i] = 0;
    __syncwarp();
}

// One batch: the tails among the vertices [bi * vb, (bi + 1) * vb), vb <= 32, counted by one warp in
// its slice of shared memory.  distinct: no list holds an entry twice (the input lists ascend), so
// the tables need no compare-and-swap to find duplicates.  HUB: lists are split, and hub i is the
// key n + i of a table.
template <typename OffT, bool HUB, bool CG = false>
__device__ __forceinline__ void small_batch(u32* base, u64 bi, u32 vb, u64 n, const Desc<OffT>* __restrict__ vdesc,
                                            const u32* __restrict__ headp, const u16* __restrict__ hubp,
                                            const u32* __restrict__ hub_ids, u32 sd, bool distinct,
                                            u64* __restrict__ cnt, u64& local_total, u32& dup) {
    using L = SmallWarpLayout<OffT, HUB>;
    constexpr u32 FULL = 0xFFFFFFFFu;
    static_assert(SMALL_D < 64 && SMALL_D <= L::QCAP && L::GROUP <= 16, "field widths of the queue entries");
    static_assert(2 * L::NB <= (int)NO_SLOT && (SMALL_D + 3) / 4 + 1 < 16, "slots and length bins");
    const u32 lane = threadIdx.x & 31;
    const u32 lt_mask = (1u << lane) - 1, le_mask = lt_mask | (1u << lane);
    u32* keys = base + L::W_KEYS;
    u32* hits = base + L::W_HITS;
    unsigned short* hits16 = reinterpret_cast<unsigned short*>(hits);
    uint4* rec = reinterpret_cast<uint4*>(base + L::W_REC);  // x: first key, y: out-degree, z: multiplier
    OffT* q_s = reinterpret_cast<OffT*>(base + L::W_QS);
    OffT* o_s = reinterpret_cast<OffT*>(base + L::W_OS);
    u32* q_m = base + L::W_QM;
    u32* q_h = base + L::W_QH;
    u32* tot = base + L::W_TOT;
    u32* vtx = base + L::W_VTX;
    u32* bins = base + L::W_BIN;
    unsigned short* q_ord = reinterpret_cast<unsigned short*>(base + L::W_ORD);
    const uint4* headp4 = reinterpret_cast<const uint4*>(headp);
    const uint4* hubp8 = reinterpret_cast<const uint4*>(hubp);
    const u32 n32 = (u32)n;
    auto vertex_of = [&](u32 key) { return HUB && key >= n32 ? ld_in<CG>(hub_ids + (key - n32)) : key; };
    const u64 v = bi * vb + lane;
    Desc<OffT> dv;
    dv.start = 0;
    dv.d = 0;
    if (lane < vb && v < n) dv = ld_desc<CG>(vdesc + v);
    const u32 len_v = list_len<HUB>(dv.d);
    u32 todo = __ballot_sync(FULL, len_v >= 2 && len_v <= sd);  // a tail needs two out-neighbours
    while (todo) {
        // the group: the next tails in lane order while their keys fit
        const bool cand = (todo >> lane) & 1u;
        u32 pk = cand ? len_v : 0u;  // inclusive prefix of the tails' out-degrees
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(FULL, pk, o);
            if (lane >= (u32)o) pk += y;
        }
        const u32 rank = __popc(todo & lt_mask);
        const bool in = cand && pk <= (u32)L::QCAP && rank < (u32)L::GROUP;
        const u32 gmask = __ballot_sync(FULL, in);
        todo &= ~gmask;
        const u32 G = __popc(gmask);
        const u32 K = __shfl_sync(FULL, pk, 31 - __clz(gmask));
        if (in) {
            rec[rank] = make_uint4(pk - len_v, len_v, 0x9E3779B1u, rest_len<HUB>(dv.d));
            o_s[rank] = (OffT)list_group(dv);
            tot[rank] = 0;
            vtx[rank] = (u32)v;
        }
        bins[lane] = 0;
        __syncwarp();
        // this lane's keys (one per row): the tail by start masks, the key, its out-list
        const bool mem = lane < G;
        const u32 kst = mem ? rec[lane].x : 0u;
        u32 w[L::ROWS], gi[L::ROWS], slot[L::ROWS];
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) {
            w[r] = EMPTY_KEY;
            gi[r] = 0;
            slot[r] = NO_SLOT;
            const u32 q0 = 32 * r;
            if (q0 >= K) continue;
            const u32 before = __popc(__ballot_sync(FULL, mem && kst <= q0));
            const u32 starts = __reduce_or_sync(FULL, start_bit(mem, kst, q0));
            if (q0 + lane < K) {
                gi[r] = segment_of(before, starts, le_mask);
                const uint4 t = rec[gi[r]];
                const u64 s = 4 * (u64)o_s[gi[r]];
                const u32 k = q0 + lane - t.x;
                if (!HUB || k < t.w) w[r] = ld_in<CG>(headp + s + k);
                else w[r] = n32 + ld_in<CG>(hubp + hub_start(s, vtx[gi[r]]) + (k - t.w));
            }
        }
        Desc<OffT> dw[L::ROWS];
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) {
            dw[r].start = 0;
            dw[r].d = 0;
            if (w[r] != EMPTY_KEY) dw[r] = ld_desc<CG>(vdesc + vertex_of(w[r]));
        }
        // the tables: a tail whose keys overfill a bucket starts over with another multiplier
        u32 brute = 0;  // tails without a table
        {
            u32 need = 0;
#pragma unroll
            for (int r = 0; r < L::ROWS; ++r) need |= (w[r] != EMPTY_KEY ? 1u : 0u) << r;
            for (int attempt = 0;; ++attempt) {
                u32 failed = 0;
                if (distinct) {
                    // all keys are written to their bucket's first slot and read back; who lost tries the
                    // second slot the same way (a third of a compare-and-swap's wavefronts)
                    u32 lost = 0;
#pragma unroll
                    for (int r = 0; r < L::ROWS; ++r) {
                        if (!((need >> r) & 1u)) continue;
                        const uint4 t = rec[gi[r]];
                        slot[r] = 2 * (3 * t.x + __umulhi(w[r] * t.z, 3 * t.y));
                        keys[slot[r]] = w[r];
                    }
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < L::ROWS; ++r)
                        if (((need >> r) & 1u) && keys[slot[r]] != w[r]) lost |= 1u << r;
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < L::ROWS; ++r)
                        if ((lost >> r) & 1u) keys[++slot[r]] = w[r];
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < L::ROWS; ++r)
                        if (((lost >> r) & 1u) && keys[slot[r]] != w[r]) {
                            slot[r] = NO_SLOT;
                            failed |= 1u << gi[r];
                        }
                    need = 0;
                }
#pragma unroll
                for (int r = 0; r < L::ROWS; ++r) {
                    if (!((need >> r) & 1u)) continue;
                    const uint4 t = rec[gi[r]];
                    const u32 at = 2 * (3 * t.x + __umulhi(w[r] * t.z, 3 * t.y));
                    u32 prev = atomicCAS(&keys[at], EMPTY_KEY, w[r]);
                    slot[r] = at;
                    if (prev != EMPTY_KEY && prev != w[r]) {
                        prev = atomicCAS(&keys[at + 1], EMPTY_KEY, w[r]);
                        slot[r] = at + 1;
                        if (prev != EMPTY_KEY && prev != w[r]) {
                            slot[r] = NO_SLOT;
                            failed |= 1u << gi[r];
                        }
                    }
                    if (prev == w[r]) dup = 1;
                }
                const u32 fmask = __reduce_or_sync(FULL, failed);
                if (!fmask) break;
                need = 0;
#pragma unroll
                for (int r = 0; r < L::ROWS; ++r) {
                    if (w[r] == EMPTY_KEY || !((fmask >> gi[r]) & 1u)) continue;
                    if (slot[r] != NO_SLOT) keys[slot[r]] = EMPTY_KEY;
                    slot[r] = NO_SLOT;
                    need |= 1u << r;
                }
                if (attempt + 1 == L::MAX_TRIES) {
                    brute = fmask;
                    break;
                }
                if ((fmask >> lane) & 1u) rec[lane].z = rec[lane].z * 0x2C1B3C6Du + 2u;  // stays odd
                __syncwarp();
            }
        }
        // the queue: heads with a small out-list, binned by length
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) {
            const u32 d = list_len<HUB>(dw[r].d);
            if (d == 0 || d > sd) continue;
            const u32 q = 32 * r + lane, dr = rest_len<HUB>(dw[r].d), dh = hub_len<HUB>(dw[r].d);
            q_s[q] = (OffT)list_group(dw[r]);
            if constexpr (HUB) q_h[q] = (u32)(hub_start(list_start(dw[r]), vertex_of(w[r])) >> 3);
            q_m[q] = (slot[r] << 16) | (gi[r] << 12) | (dh << 6) | dr;
        }
        // counting sort by length in 16-byte groups: lanes of a row with the same length are found by
        // ballots, and their first lane adds for all of them
        u32 same[L::ROWS], len[L::ROWS];
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) {
            const u32 d = list_len<HUB>(dw[r].d);
            const bool sel = d != 0 && d <= sd;
            len[r] = sel ? (rest_len<HUB>(dw[r].d) + 3) / 4 + (hub_len<HUB>(dw[r].d) + 7) / 8 : 0u;
            same[r] = 0;
            if (32u * r >= K) continue;
            same[r] = __ballot_sync(FULL, sel);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const u32 set = __ballot_sync(FULL, (len[r] >> b) & 1u);
                same[r] &= (len[r] >> b) & 1u ? set : ~set;
            }
            if (sel && !(same[r] & lt_mask)) atomicAdd(&bins[len[r]], (u32)__popc(same[r]));
        }
        __syncwarp();
        u32 qn;
        {
            // exclusive sums from the longest bin down
            const u32 c = bins[31 - lane];
            u32 x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 y = __shfl_up_sync(FULL, x, o);
                if (lane >= (u32)o) x += y;
            }
            bins[31 - lane] = x - c;
            qn = __shfl_sync(FULL, x, 31);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) {
            if (32u * r >= K) continue;
            const u32 first = same[r] & lt_mask;
            u32 at = 0;
            if (len[r] && !first) at = atomicAdd(&bins[len[r]], (u32)__popc(same[r]));
            at = __shfl_sync(FULL, at, __ffs(same[r] | (1u << lane)) - 1);
            if (len[r]) q_ord[at + __popc(first)] = (unsigned short)(32 * r + lane);
        }
        __syncwarp();
        // stream the queued lists, longest first, one per pair of lanes that take turns at its 16-byte
        // groups (a pair's reads share a 32-byte sector: half the wavefronts of one list per lane); the
        // next group is in flight while the current one is looked up (groups are padded, so the load
        // stays inside the list's slots)
        const u32 half = lane & 1u;
        for (u32 i0 = 0; i0 < qn; i0 += 16) {
            const u32 i = i0 + (lane >> 1);
            const bool have = i < qn;
            const u32 q = have ? q_ord[i] : 0u;
            const u32 m = have ? q_m[q] : 0u;
            const u32 g = (m >> 12) & 15u;
            const uint4* lp = headp4 + (have ? (u64)q_s[q] : 0ull);
            const uint4 t = rec[g];
            int rem = (int)(m & 63u), hrem = HUB ? (int)((m >> 6) & 63u) : 0;
            u32 found = 0;
            if ((brute >> g) & 1u) {
                const u64 own = 4 * (u64)o_s[g], hown = hub_start(own, vtx[g]);
                auto own_key = [&](u32 k) {
                    return !HUB || k < t.w ? ld_in<CG>(headp + own + k) : n32 + ld_in<CG>(hubp + hown + (k - t.w));
                };
                for (int e = (int)half; e < rem + hrem; e += 2) {
                    const u32 z = e < rem ? ld_in<CG>(reinterpret_cast<const u32*>(lp) + e)
                                          : n32 + ld_in<CG>(reinterpret_cast<const u16*>(hubp8 + q_h[q]) + (e - rem));
                    for (u32 k = 0; k < t.y; ++k)
                        if (own_key(k) == z) {
                            atomicAdd(&cnt[vertex_of(z)], 1ull);
                            ++found;
                        }
                }
                if (found) atomicAdd(&cnt[vertex_of(own_key(q - t.x))], (u64)found);
                if (found) atomicAdd(&tot[g], found);
                found = 0;
            } else {
                const u32 nb = 3 * t.y, mult = t.z;
                const uint2* tk = reinterpret_cast<const uint2*>(keys) + 3 * t.x;
                u32* th = hits + 3 * t.x;
                auto look4 = [&](u32 z0, u32 z1, u32 z2, u32 z3, int r) {
                    const u32 z[4] = {z0, z1, z2, z3};
                    u32 b[4];
                    uint2 kk[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        b[k] = __umulhi(z[k] * mult, nb);
                        kk[k] = tk[b[k]];
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const bool h0 = kk[k].x == z[k], h1 = kk[k].y == z[k];
                        if ((h0 | h1) & (k < r)) {
                            atomicAdd(&th[b[k]], h1 ? 0x10000u : 1u);
                            ++found;
                        }
                    }
                };
                rem -= 4 * (int)half;
                if (rem > 0) {
                    lp += half;
                    uint4 cur = ld_in<CG>(lp);
                    while (true) {
                        uint4 nxt = cur;
                        if (rem > 8) nxt = ld_in<CG>(lp += 2);
                        look4(cur.x, cur.y, cur.z, cur.w, rem);
                        rem -= 8;
                        if (rem <= 0) break;
                        cur = nxt;
                    }
                }
                if constexpr (HUB) {
                    const uint4* hp = hubp8 + (have ? q_h[q] : 0u) + half;
                    for (hrem -= 8 * (int)half; hrem > 0; hrem -= 16, hp += 2) {
                        const uint4 cur = ld_in<CG>(hp);
                        look4(n32 + (cur.x & 0xFFFFu), n32 + (cur.x >> 16), n32 + (cur.y & 0xFFFFu),
                              n32 + (cur.y >> 16), hrem);
                        if (hrem > 4)
                            look4(n32 + (cur.z & 0xFFFFu), n32 + (cur.z >> 16), n32 + (cur.w & 0xFFFFu),
                                  n32 + (cur.w >> 16), hrem - 4);
                    }
                }
            }
            __syncwarp();
            found += __shfl_xor_sync(FULL, found, 1);
            if (found && !half) {
                const u32 s = m >> 16;
                atomicAdd(&hits[s >> 1], found << ((s & 1u) << 4));  // the edge's head
                atomicAdd(&tot[g], found);
            }
        }
        __syncwarp();
        // flush and clear: every key's hits (as the third corner and as the head of its edge), then
        // the tails' totals
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) {
            if (slot[r] == NO_SLOT) continue;
            const u32 h = hits16[slot[r]];
            keys[slot[r]] = EMPTY_KEY;
            hits16[slot[r]] = 0;
            if (h) atomicAdd(&cnt[vertex_of(w[r])], (u64)h);
        }
        if (mem) {
            const u32 t = tot[lane];
            if (t) {
                atomicAdd(&cnt[vtx[lane]], (u64)t);
                local_total += t;
            }
        }
        __syncwarp();  // the next group reuses the slice only after every lane has flushed
    }
}

template <int BLOCK, typename OffT, bool HUB>
__global__ void __launch_bounds__(BLOCK, 4) k_count_small(u64 n, u32 vb, const Desc<OffT>* __restrict__ vdesc,
                                                          const u32* __restrict__ headp, const u16* __restrict__ hubp,
                                                          const u32* __restrict__ hub_ids, u32 sd,
                                                          u64* __restrict__ cnt, u64* __restrict__ partials,
                                                          Control* ctl) {
    chain_begin();
    using L = SmallWarpLayout<OffT, HUB>;
    constexpr int NW = BLOCK / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ u64 s_red[NW];
    if (ctl->err & DEV_ERR_MASK) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u32* base = reinterpret_cast<u32*>(smem) + warp * L::PER_WARP;
    small_init<OffT, HUB>(base);
    const bool distinct = !(ctl->err & DEV_FLAG_UNSORTED);
    const bool split = HUB && ctl->hubs != 0;  // without hubs the plain body reads the same lists
    const u64 nbatch = (n + vb - 1) / vb;
    u64 local_total = 0;
    u32 dup = 0;
    while (true) {
        unsigned long long bi = 0;
        if (lane == 0) bi = atomicAdd(&ctl->small_next, 1ull);
        bi = __shfl_sync(0xFFFFFFFFu, bi, 0);
        if (bi >= nbatch) break;
        if (split)
            small_batch<OffT, HUB>(base, bi, vb, n, vdesc, headp, hubp, hub_ids, sd, distinct, cnt, local_total, dup);
        else
            small_batch<OffT, false>(base, bi, vb, n, vdesc, headp, nullptr, nullptr, sd, distinct, cnt, local_total,
                                     dup);
    }
    if (dup) atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
    const u64 bt = block_sum_u64<BLOCK>(local_total, s_red);
    if (threadIdx.x == 0) partials[blockIdx.x] = bt;
}

template <int BLOCK, int CAP, typename OffT>
struct LargeLayout {
    static constexpr int TS = 2 * CAP;       // table slots (at most half full)
    static constexpr int FWORDS = CAP / 2;   // filter words: 16 bits per key at CAP keys
    static constexpr int WBUF = 64;          // per-warp buffer of filter survivors
    static constexpr size_t off_keys = 0;
    static constexpr size_t off_hits = align16(off_keys + sizeof(u32) * TS);         // two u16 counters per word
    static constexpr size_t off_filt = align16(off_hits + sizeof(u32) * (TS / 2));
    static constexpr size_t off_wbuf = align16(off_filt + sizeof(u32) * FWORDS);
    static constexpr size_t off_qy = align16(off_wbuf + sizeof(u32) * WBUF * (BLOCK / 32));
    static constexpr size_t off_qd = align16(off_qy + sizeof(u32) * LARGE_SEG);
    // block scalars: reduction slots, queue length and cursor, the bulk copy's mbarrier
    static constexpr size_t off_red = align16(off_qd + sizeof(Desc<OffT>) * LARGE_SEG);
    static constexpr size_t off_qn = off_red + sizeof(u64) * (BLOCK / 32);
    static constexpr size_t off_next = off_qn + sizeof(u32);
    static constexpr size_t off_bar = align16(off_next + sizeof(u32));
    static constexpr size_t bytes = align16(off_bar + sizeof(unsigned long long));
};

// One-hash membership filter of the owner's keys (2^fl bits): a clear bit is a sure miss.
__device__ __forceinline__ u32 filter_bit(u32 w, u32 fl) { return (w * 0x85EBCA6Bu) >> (32 - fl); }
__device__ __forceinline__ bool filter_test(const u32* filt, u32 fl, u32 w) {
    const u32 h = filter_bit(w, fl);
    return (filt[h >> 5] >> (h & 31u)) & 1u;
}

// A whole warp streams one list (d entries at lst) through the owner's filter and table.
// Entries that pass the filter are packed into the warp's buffer (64 entries) and looked up
// 32 at a time.  Returns this lane's share of the hits.
template <int U, bool CG = false>
__device__ __forceinline__ u32 warp_stream_list(const u32* __restrict__ lst, u32 d, const u32* keys, u32* hitc, u32 lg,
                                                const u32* filt, u32 fl, u32* wbuf, int lane, u32 lt_mask) {
    u32 hits = 0, nbuf = 0;
    // a running pointer and a running count of the entries left from this lane's position,
    // so each load is one instruction with an immediate offset and one compare
    const u32* lp = lst + lane;
    int rem = (int)d - lane;
    for (u32 p0 = 0; p0 < d; p0 += 32 * U, lp += 32 * U, rem -= 32 * U) {
        u32 w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = rem > 32 * u ? ld_in<CG>(lp + 32 * u) : EMPTY_KEY;
        const int left = (int)(d - p0);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (left <= 32 * u) break;
            // both tests evaluated (no branch): past the list's end w[u] is EMPTY_KEY, a harmless
            // filter read whose result the range test masks
            const bool maybe = (rem > 32 * u) & filter_test(filt, fl, w[u]);
            const u32 ball = __ballot_sync(0xFFFFFFFFu, maybe);
            if (maybe) wbuf[nbuf + __popc(ball & lt_mask)] = w[u];
            nbuf += __popc(ball);
            if (nbuf >= 32) {
                __syncwarp();
                hits += bucket_probe16_flat(keys, hitc, lg, wbuf[lane]);
                const u32 rest = nbuf - 32;
                const u32 carry = lane < rest ? wbuf[32 + lane] : 0u;
                __syncwarp();
                if (lane < rest) wbuf[lane] = carry;
                __syncwarp();
                nbuf = rest;
            }
        }
    }
    __syncwarp();
    if (lane < nbuf) hits += bucket_probe16_flat(keys, hitc, lg, wbuf[lane]);
    __syncwarp();
    return hits;
}

// A lane streams one short list (d <= LONG_LIST entries, 16-byte aligned) through the owner's
// filter and table.
template <typename OffT, bool CG = false>
__device__ __forceinline__ u32 lane_stream_short(const uint4* __restrict__ headp4, const Desc<OffT>& vy,
                                                 const u32* keys, u32* hitc, u32 lg, const u32* filt, u32 fl) {
    const u32 dy = vy.d;
    const u64 q0 = list_group(vy);
    uint4 qv[LONG_LIST / 4];
#pragma unroll
    for (int c = 0; c < LONG_LIST / 4; ++c)
        qv[c] = 4 * c < (int)dy ? ld_in<CG>(headp4 + q0 + c) : make_uint4(EMPTY_KEY, EMPTY_KEY, EMPTY_KEY, EMPTY_KEY);
    u32 hits = 0;
#pragma unroll
    for (int c = 0; c < LONG_LIST / 4; ++c) {
        if (4 * c < (int)dy) {
            const u32 wv[4] = {qv[c].x, qv[c].y, qv[c].z, qv[c].w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if ((4 * c + k < (int)dy) & filter_test(filt, fl, wv[k])) hits += bucket_probe16(keys, hitc, lg, wv[k]);
        }
    }
    return hits;
}

// Table and filter sizes of an owner chunk of klen keys: a quarter-full table (at most
// max_lg) and 16 filter bits per key (at most max_fl).
__device__ __forceinline__ void chunk_sizes(u32 klen, u32 max_lg, u32 max_fl, u32* lg, u32* fl) {
    u32 a = ceil_log2(4 * klen);
    if (a > max_lg) a = max_lg;
    if (a < 2) a = 2;
    u32 f = ceil_log2(16 * klen);
    if (f > max_fl) f = max_fl;
    if (f < 5) f = 5;
    *lg = a;
    *fl = f;
}

// One (owner, segment) tile of a large owner, counted by the whole block.  bar is the block's
// bulk-copy mbarrier, initialised once and kept where no other use of shared memory reaches.
// Returns true when a bounded wait for a bulk copy ran out (inflight: the second wait ran out too).
template <int BLOCK, int CAP, typename OffT, bool CG = false>
__device__ __forceinline__ bool large_tile(unsigned char* smem, unsigned long long* bar, uint2 tl,
                                           const u64* __restrict__ fo,
                                           const u32* __restrict__ head, u64 n, const Desc<OffT>* __restrict__ vdesc,
                                           const u32* __restrict__ headp, u32 seg, u64* __restrict__ cnt,
                                           u32 first_wait_polls, u32& phase, bool& inflight, u64& local_total,
                                           u32& dup) {
    using L = LargeLayout<BLOCK, CAP, OffT>;
    constexpr int NW = BLOCK / 32;
    constexpr int U = 8;  // loads in flight per lane and list
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 lt_mask = (1u << lane) - 1;
    const uint4* headp4 = reinterpret_cast<const uint4*>(headp);
    u32* keys = reinterpret_cast<u32*>(smem + L::off_keys);
    u32* hitc = reinterpret_cast<u32*>(smem + L::off_hits);
    u32* filt = reinterpret_cast<u32*>(smem + L::off_filt);
    u32* qy = reinterpret_cast<u32*>(smem + L::off_qy);
    Desc<OffT>* qd = reinterpret_cast<Desc<OffT>*>(smem + L::off_qd);
    // the owner's keys are staged in the queue's descriptor region, which is free until the scan
    u32* stage = reinterpret_cast<u32*>(smem + L::off_qd);
    static_assert(sizeof(Desc<OffT>) * LARGE_SEG >= sizeof(u32) * CAP, "staging fits the queue region");
    u32* wbuf = reinterpret_cast<u32*>(smem + L::off_wbuf) + warp * L::WBUF;
    u64* s_red = reinterpret_cast<u64*>(smem + L::off_red);
    u32& s_qn = *reinterpret_cast<u32*>(smem + L::off_qn);
    u32& s_next = *reinterpret_cast<u32*>(smem + L::off_next);
    unsigned long long& s_bar = *bar;  // the block's bulk-copy barrier (its phase persists across tiles)
    bool timed_out = false;
    const u64 x = tl.x;
    const Desc<OffT> dxd = ld_desc<CG>(vdesc + x);
    const u32 dx = dxd.d;
    const u64 fx1 = ld_in<CG>(fo + x + 1);
    const u64 a = ld_in<CG>(fo + x) + (u64)tl.y * seg;
    const u64 b = a + seg < fx1 ? a + seg : fx1;
    u64 T = 0;
    for (u32 c0 = 0; c0 < dx; c0 += CAP) {
        const u32 klen = dx - c0 < (u32)CAP ? dx - c0 : (u32)CAP;
        u32 lg, fl;
        chunk_sizes(klen, 31 - __clz((u32)L::TS), 31 - __clz((u32)(L::FWORDS * 32)), &lg, &fl);
        const u32 size = 1u << lg, fwords = (1u << fl) >> 5;
        for (u32 s = threadIdx.x; s < size; s += BLOCK) keys[s] = EMPTY_KEY;
        for (u32 s = threadIdx.x; s < size / 2; s += BLOCK) hitc[s] = 0;
        for (u32 s = threadIdx.x; s < fwords; s += BLOCK) filt[s] = 0;
        if (threadIdx.x == 0) {
            s_qn = 0;
            s_next = 0;
        }
        fence_proxy_async_smem();  // earlier generic accesses of the staging region come first
        __syncthreads();
        // one bulk copy of the chunk's keys (list starts are 16-byte aligned, and the gapped
        // layout leaves room to round the length up to whole 16-byte groups)
        if (threadIdx.x == 0) {
            const u32 bytes = ((klen + 3u) & ~3u) * (u32)sizeof(u32);
            mbar_expect_tx(&s_bar, bytes);
            bulk_copy_g2s(stage, headp + list_start(dxd) + c0, bytes, &s_bar);
        }
        const bool arrived = mbar_wait_bounded(&s_bar, phase, first_wait_polls);
        if (__syncthreads_or(!arrived)) {  // the same decision in every thread
            // give the copy in flight a second bounded wait, so that it does not land in
            // shared memory after the block has left; then report the timeout (and, if the
            // copy still has not landed, that it may be in flight as the block leaves)
            if (!__syncthreads_or(!mbar_wait_bounded(&s_bar, phase, COPY_WAIT_POLLS))) {
                timed_out = true;
                phase ^= 1u;  // the copy landed: the barrier's phase completed (a block that goes on
                              // taking tiles, as the engine's do, waits on the next one)
            } else {
                timed_out = inflight = true;
            }
            break;
        }
        phase ^= 1u;
        for (u32 q = threadIdx.x; q < klen; q += BLOCK) {
            const u32 w = stage[q];
            if (!bucket_insert(keys, lg, w)) dup = 1;
            const u32 h = filter_bit(w, fl);
            atomicOr(&filt[h >> 5], 1u << (h & 31u));
        }
        __syncthreads();
        // scan the segment: short lists now, long lists into the queue
        for (u64 e0 = a + (u64)warp * 32; e0 < b; e0 += (u64)NW * 32) {
            const u64 e = e0 + lane;
            bool queue = false;
            u32 y = 0;
            Desc<OffT> vy;
            vy.start = 0;
            vy.d = 0;
            if (e < b) {
                y = ld_in<CG>(head + e);
                if (y < n) vy = ld_desc<CG>(vdesc + y);
                const u32 dy = vy.d;
                if (dy > 0 && key_less(dy, y, dx, x)) {
                    if (dy <= (u32)LONG_LIST) {
                        const u32 hits = lane_stream_short<OffT, CG>(headp4, vy, keys, hitc, lg, filt, fl);
                        if (hits) {
                            atomicAdd(&cnt[y], (u64)hits);
                            T += hits;
                        }
                    } else {
                        queue = true;
                    }
                }
            }
            const u32 ball = __ballot_sync(0xFFFFFFFFu, queue);
            u32 base = 0;
            if (lane == 0 && ball) base = atomicAdd(&s_qn, (u32)__popc(ball));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (queue) {
                const u32 qi = base + __popc(ball & lt_mask);
                qy[qi] = y;
                qd[qi] = vy;
            }
        }
        __syncthreads();
        // long lists: one warp per list, taken from the queue.  Every entry is tested against
        // the filter; the survivors are packed into the warp's buffer and looked up in the
        // table 32 at a time, so the lookups run with full warps.
        const u32 qn = s_qn;
        while (true) {
            u32 qi = 0;
            if (lane == 0) qi = atomicAdd(&s_next, 1u);
            qi = __shfl_sync(0xFFFFFFFFu, qi, 0);
            if (qi >= qn) break;
            const Desc<OffT> vy = qd[qi];
            u32 hits = warp_stream_list<U, CG>(headp + list_start(vy), vy.d, keys, hitc, lg, filt, fl, wbuf, lane,
                                           lt_mask);
            hits = __reduce_add_sync(0xFFFFFFFFu, hits);
            if (lane == 0 && hits) {
                atomicAdd(&cnt[qy[qi]], (u64)hits);
                T += hits;
            }
        }
        __syncthreads();
        // flush the hits of every key
        for (u32 s = threadIdx.x; s < size; s += BLOCK) {
            const u32 h = read16(hitc, s);
            if (h) atomicAdd(&cnt[keys[s]], (u64)h);
        }
        __syncthreads();
    }
    const u64 bt = block_sum_u64<BLOCK>(T, s_red);
    if (threadIdx.x == 0 && bt) {
        atomicAdd(&cnt[x], bt);
        local_total += bt;
    }
    return timed_out;
}

template <int BLOCK, int CAP, typename OffT>
__global__ void __launch_bounds__(BLOCK) k_count_large(const u64* __restrict__ fo, const u32* __restrict__ head,
                                                       u64 n, const Desc<OffT>* __restrict__ vdesc,
                                                       const u32* __restrict__ headp,
                                                       const uint2* __restrict__ ltiles, u32 seg,
                                                       u64* __restrict__ cnt, u64* __restrict__ partials,
                                                       Control* ctl, u32 first_wait_polls) {
    chain_begin();
    using L = LargeLayout<BLOCK, CAP, OffT>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ u64 s_t;
    unsigned long long* s_bar = reinterpret_cast<unsigned long long*>(smem + L::off_bar);  // the bulk copy's barrier

    if (ctl->err & DEV_ERR_MASK) return;
    const u64 ntiles = *(volatile unsigned long long*)&ctl->large_tiles;
    if (ntiles == 0) {
        if (threadIdx.x == 0) partials[blockIdx.x] = 0;
        return;
    }
    if (threadIdx.x == 0) mbar_init(s_bar, 1);
    fence_proxy_async_smem();
    __syncthreads();
    u32 phase = 0;
    bool timed_out = false, inflight = false;
    u64 local_total = 0;
    u32 dup = 0;
    while (true) {
        if (threadIdx.x == 0) s_t = atomicAdd(&ctl->large_next, 1ull);
        __syncthreads();
        const u64 t = s_t;
        if (t >= ntiles) break;
        timed_out = large_tile<BLOCK, CAP, OffT>(smem, s_bar, ltiles[tile_at(true, t)], fo, head, n, vdesc, headp, seg,
                                                 cnt, first_wait_polls, phase, inflight, local_total, dup);
        if (timed_out) break;
    }
    if (dup) atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
    if (timed_out) atomicOr(&ctl->err, DEV_ERR_TIMEOUT | (inflight ? DEV_ERR_COPY_INFLIGHT : 0u));
    if (threadIdx.x == 0) partials[blockIdx.x] = local_total;
}

// Owner tiles counted by single warps (k_count_medium): owners of small_outdegree < out-degree <=
// medium_outdegree, and with hubs every owner's other entries.  A warp's table holds up to CAP of
// the owner's keys (owners with more are counted in chunks) in buckets of two; a bucket that
// overflowed is marked by a cleared top bit of its second key, so a lookup reads one bucket and
// walks on only past a marked one (about 1.5 % of them at CAP keys), and a miss in a full bucket ends
// there.  Streamed lists are cut into units of 32 entries, eight lanes to a unit and four units of
// any lists to a row; lists of up to four entries go one per lane.
// What bounds it: instruction issue (71 to 73 %) beside the lookups' shared-memory wavefronts
// (53 to 62 % of the pipe).  It replaced a one-hash filter with packed survivors and one list per warp
// iteration, which left most lanes idle on lists below 100 entries: RMAT n = 8191 0.182 -> 0.061 ms
// (medium + large), 512-graph batch 6.2 -> 5.0 ms, the other entries of RMAT-24 27.6 -> 18 ms.
// Measured against NB = 768 (24 warps per SM: RMAT-24 +0.8 %, batch +1 %, small graphs -10 %) and
// fewer keys per chunk (more owners in two chunks: RMAT-24 66.3 ms, CAP = 192 68.0, CAP = 128 +7 %; a
// lattice of out-degree 200 without hubs 1.41 ms, CAP = 192 2.49).  All of a medium owner's keys fit one chunk.
template <typename OffT>
struct TileLayout {
    static constexpr u32 NB = 512;   // buckets
    static constexpr u32 CAP = MEDIUM_D;  // keys per chunk
    static constexpr int W_KEYS = 0;
    static constexpr int W_HITS = W_KEYS + 2 * NB;  // two 16-bit counters per bucket, a spare word per lane
    static constexpr int PER_WARP = W_HITS + NB + 32;
    static constexpr size_t bytes(int warps) { return sizeof(u32) * PER_WARP * warps; }
};
constexpr u32 TILE_MULT = 0x9E3779B1u;

// A warp's table is empty between chunks.
template <typename OffT>
__device__ __forceinline__ void tile_init(u32* base) {
    using L = TileLayout<OffT>;
    const u32 lane = threadIdx.x & 31;
    for (u32 i = lane; i < 2 * L::NB; i += 32) base[L::W_KEYS + i] = EMPTY_KEY;
    for (u32 i = lane; i < L::NB + 32; i += 32) base[L::W_HITS + i] = 0;
    __syncwarp();
}

// One (owner, segment) tile of an owner's out-list (HUB: of its entries that are not hubs), counted by
// one warp in its slice of shared memory.  top: the bit that marks keys, 0 where ids need all bits
// (a full bucket is then walked past, marked or not).  Where some input list does not ascend, the
// tables are the only check for entries that a list holds twice, so the owner's first tile also looks
// the keys of later chunks up in each chunk's table (its conditions are read again there: kept in
// registers they made the kernel spill).
template <typename OffT, bool HUB, bool CG = false>
__device__ __forceinline__ void medium_tile(u32* base, u32 top, uint2 tl, const u64* __restrict__ fo,
                                            const u32* __restrict__ head, const Desc<OffT>* __restrict__ vdesc,
                                            const u32* __restrict__ headp, u32 seg, u64* __restrict__ cnt,
                                            const Control* ctl, u64& local_total, u32& dup) {
    using L = TileLayout<OffT>;
    constexpr u32 FULL = 0xFFFFFFFFu;
    const u32 lane = threadIdx.x & 31;
    u32* keys = base + L::W_KEYS;
    u32* hits = base + L::W_HITS;
    const uint2* buckets = reinterpret_cast<const uint2*>(keys);
    const uint4* headp4 = reinterpret_cast<const uint4*>(headp);
    const u32 x = tl.x;
    const Desc<OffT> dx = ld_desc<CG>(vdesc + x);
    const u32 xr = rest_len<HUB>(dx.d), xt = list_len<HUB>(dx.d);
    if (xr == 0) return;
    const u64 a = ld_in<CG>(fo + x) + (u64)tl.y * seg, fx1 = ld_in<CG>(fo + x + 1);
    const u32 ns = (u32)(a + seg < fx1 ? (u64)seg : fx1 - a);
    // the first `rem` of four streamed entries: counts their hits at their keys.  One branch for the
    // four (a lane's misses then count at its spare word), and one for the rare walk.
    auto look4 = [&](const uint4& w, u32 rem) -> u32 {
        const u32 z[4] = {w.x, w.y, w.z, w.w};
        u32 at[4], found = 0;
        uint2 kk[4];
#pragma unroll
        for (u32 k = 0; k < 4; ++k) {
            at[k] = __umulhi(z[k] * TILE_MULT, L::NB);
            kk[k] = buckets[at[k]];
        }
        u32 walk = 0;
        u32 one[4];
#pragma unroll
        for (u32 k = 0; k < 4; ++k) {
            const u32 zt = z[k] | top;
            const bool h0 = kk[k].x == zt, h1 = (kk[k].y | top) == zt;
            const bool hit = (h0 | h1) & (k < rem);
            if ((k < rem) & !(h0 | h1) & !(kk[k].y & top)) walk |= 1u << k;
            one[k] = h0 ? 1u : 0x10000u;
            at[k] = hit ? at[k] : L::NB + lane;
            found += hit ? 1u : 0u;
        }
        if (found) {
#pragma unroll
            for (u32 k = 0; k < 4; ++k) atomicAdd(&hits[at[k]], one[k]);
        }
        if (walk) {
#pragma unroll
            for (u32 k = 0; k < 4; ++k) {
                if (!((walk >> k) & 1u)) continue;
                const u32 zt = z[k] | top;
                u32 b = __umulhi(z[k] * TILE_MULT, L::NB);
                uint2 q = buckets[b];
                while (q.y != EMPTY_KEY && !(q.y & top)) {  // marked (or, without marks, full): the next bucket too
                    b = b + 1 < L::NB ? b + 1 : 0;
                    q = buckets[b];
                    const bool h0 = q.x == zt, h1 = (q.y | top) == zt;
                    if (h0 | h1) {
                        atomicAdd(&hits[b], h0 ? 1u : 0x10000u);
                        ++found;
                        break;
                    }
                }
            }
        }
        return found;
    };
    u64 T = 0;
    for (u32 c0 = 0; c0 < xr; c0 += L::CAP) {
        const u32 klen = xr - c0 < L::CAP ? xr - c0 : L::CAP;
        for (u32 k = lane; k < klen; k += 32) {
            const u32 w = ld_in<CG>(headp + list_start(dx) + c0 + k), wt = w | top;
            u32 b = __umulhi(w * TILE_MULT, L::NB);
            while (true) {  // ends: at most CAP of the 2 NB slots are taken
                const u32 p0 = atomicCAS(&keys[2 * b], EMPTY_KEY, wt);
                if (p0 == EMPTY_KEY) break;
                const u32 p1 = p0 == wt ? wt : atomicCAS(&keys[2 * b + 1], EMPTY_KEY, wt);
                if (p1 == EMPTY_KEY) break;
                if (p0 == wt || (p1 | top) == wt) {
                    dup = 1;
                    break;
                }
                if (top) atomicAnd(&keys[2 * b + 1], ~top);
                b = b + 1 < L::NB ? b + 1 : 0;
            }
        }
        __syncwarp();
        if (c0 + L::CAP < xr && a == ld_in<CG>(fo + x) && (__ldcg(&ctl->err) & DEV_FLAG_UNSORTED)) {
            for (u32 k = c0 + L::CAP + lane; k < xr; k += 32) {
                const u32 wt = ld_in<CG>(headp + list_start(dx) + k) | top;
                u32 b = __umulhi((wt & ~top) * TILE_MULT, L::NB);
                while (true) {  // ends: a bucket without a second key, or without a mark
                    const uint2 q = buckets[b];
                    if (q.x == wt || (q.y | top) == wt) dup = 1;
                    if (q.y == EMPTY_KEY || (q.y & top)) break;
                    b = b + 1 < L::NB ? b + 1 : 0;
                }
            }
        }
        u32 Tc = 0;
        // two chunks of slots ahead the neighbours, one ahead their descriptors are in flight
        auto neighbour = [&](u32 e) { return e + lane < ns ? ld_in<CG>(head + a + e + lane) : x; };
        u32 y0 = neighbour(0), y1 = neighbour(32);
        Desc<OffT> v0 = ld_desc<CG>(vdesc + y0);
        for (u32 e0 = 0; e0 < ns; e0 += 32) {
            const u32 y = y0;
            const Desc<OffT> vy = v0;
            const bool have = e0 + lane < ns;
            y0 = y1;
            v0 = ld_desc<CG>(vdesc + y0);
            y1 = neighbour(e0 + 64);
            const u32 yr = rest_len<HUB>(vy.d), yt = list_len<HUB>(vy.d);
            const bool sel = have && yr > 0 && (yt < xt || (yt == xt && y < x));
            const OffT ys = (OffT)list_group(vy);
            u32 f = 0;
            if (sel && yr <= 4) {
                const uint4 w = ld_in<CG>(headp4 + ys);
                f = look4(w, yr);
            }
            __syncwarp();
            const u32 units = sel && yr > 4 ? (yr + 31) / 32 : 0u;
            u32 P = units;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 z = __shfl_up_sync(FULL, P, o);
                if (lane >= (u32)o) P += z;
            }
            const u32 U = __shfl_sync(FULL, P, 31);
            P = units ? P - units : 0xFFFFFFFFu;  // the list's first unit
            uint4 nw = make_uint4(0, 0, 0, 0);
            u32 nrem = 0;                         // entries from this lane's first on
            int n0 = 0, n1 = 0, n2 = 0, n3 = 0;   // the lanes whose lists the row's units belong to
            auto fetch = [&](u32 u) {
                n0 = 31 - __clz(__ballot_sync(FULL, P <= u));
                n1 = 31 - __clz(__ballot_sync(FULL, P <= u + 1));
                n2 = 31 - __clz(__ballot_sync(FULL, P <= u + 2));
                n3 = 31 - __clz(__ballot_sync(FULL, P <= u + 3));
                const int k = lane < 16 ? (lane < 8 ? n0 : n1) : (lane < 24 ? n2 : n3);
                const u32 o = (u + (lane >> 3) - __shfl_sync(FULL, P, k)) * 8 + (lane & 7u);
                const u32 len = __shfl_sync(FULL, yr, k);
                const uint4* lp = headp4 + (u64)__shfl_sync(FULL, ys, k);
                nrem = 4 * o < len ? len - 4 * o : 0u;
                if (nrem) nw = ld_in<CG>(lp + o);
            };
            if (U) fetch(0);
            for (u32 u = 0; u < U; u += 4) {
                const uint4 w = nw;
                const u32 rem = nrem;
                const int k0 = n0, k1 = n1, k2 = n2, k3 = n3;
                if (u + 4 < U) fetch(u + 4);
                const u32 g = look4(w, rem);
                // the four units' hits (at most 32 each) side by side in one sum
                const u32 s4 = __reduce_add_sync(FULL, g << (lane & 24u));
                if ((int)lane == k0) f += s4 & 0xFFu;
                if ((int)lane == k1) f += (s4 >> 8) & 0xFFu;
                if ((int)lane == k2) f += (s4 >> 16) & 0xFFu;
                if ((int)lane == k3) f += s4 >> 24;
            }
            if (f) {
                atomicAdd(&cnt[y], (u64)f);
                Tc += f;
            }
        }
        __syncwarp();
        // flush and clear
        for (u32 b = lane; b < L::NB; b += 32) {
            const u32 h = hits[b];
            if (h) {
                const uint2 kk = buckets[b];
                if (h & 0xFFFFu) atomicAdd(&cnt[kk.x & ~top], (u64)(h & 0xFFFFu));
                if (h >> 16) atomicAdd(&cnt[kk.y & ~top], (u64)(h >> 16));
                hits[b] = 0;
            }
            reinterpret_cast<uint2*>(keys)[b] = make_uint2(EMPTY_KEY, EMPTY_KEY);
        }
        T += __reduce_add_sync(FULL, Tc);
        __syncwarp();
    }
    if (lane == 0 && T) {
        atomicAdd(&cnt[x], T);
        local_total += T;
    }
}

// HUB: the large owners' tiles come first.
template <int BLOCK, typename OffT, bool HUB>
__global__ void __launch_bounds__(BLOCK, 4)
    k_count_medium(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n,
                   const Desc<OffT>* __restrict__ vdesc, const u32* __restrict__ headp,
                   const uint2* __restrict__ mtiles, const uint2* __restrict__ ltiles, u32 seg,
                   u64* __restrict__ cnt, u64* __restrict__ partials, Control* ctl) {
    chain_begin();
    using L = TileLayout<OffT>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ u64 s_red[BLOCK / 32];
    if (ctl->err & DEV_ERR_MASK) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u32* base = reinterpret_cast<u32*>(smem) + warp * L::PER_WARP;
    const u64 nl = HUB ? *(volatile unsigned long long*)&ctl->large_tiles : 0;
    const u64 ntiles = nl + *(volatile unsigned long long*)&ctl->medium_tiles;
    if (ntiles == 0) {
        if (threadIdx.x == 0) partials[blockIdx.x] = 0;
        return;
    }
    tile_init<OffT>(base);
    const u32 top = n < 0x7FFFFFFFu ? 0x80000000u : 0u;
    u64 local_total = 0;
    u32 dup = 0;
    while (true) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(&ctl->medium_next, 1ull);
        t = __shfl_sync(0xFFFFFFFFu, t, 0);
        if (t >= ntiles) break;
        const uint2 tl = HUB && t < nl ? ltiles[tile_at(true, t)] : mtiles[t - nl];
        medium_tile<OffT, HUB>(base, top, tl, fo, head, vdesc, headp, seg, cnt, ctl, local_total, dup);
    }
    if (dup) atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
    const u64 bt = block_sum_u64<BLOCK>(local_total, s_red);
    if (threadIdx.x == 0) partials[blockIdx.x] = bt;
}

// The hub part of the owner tiles (k_count_hub): for every edge {x, y} of an owner x, the hubs that
// both out-lists hold.  Hubs are the few thousand vertices of highest degree, which most entries of
// a skewed graph's out-lists name (80 % of the entries RMAT-24 streams are among its first 2^15,
// 98 % of RMAT-20's), and a hub list holds 16-bit indices.  So an owner's table is a bitmap of HUB_H
// bits: a lookup is one 4-byte shared-memory read without hash, filter or walk, and a streamed
// entry costs two bytes of L2 traffic instead of four.
// A block holds one counter per hub for its whole life and flushes them once, so a tile clears
// nothing but its bitmap.  Each warp takes its own (owner, segment) tiles and has its own bitmap.
// Lists above HUB_LANE entries are streamed in units of 64 entries by eight lanes each, eight
// consecutive entries per lane, the shorter ones one per lane.  The densest part of the lists, the
// first HUB_TOP hubs, does not go through the lists where that pays: half of the streamed lists of
// RMAT-24 keep 45 % of the streamed hub entries in bitmaps of 256 bytes (81 MB in all), and one
// AND, a population count and 3.5 additions per word count 32 of them (TopCounters).
// Measured (medium and large tiles, RMAT n = 10^6 / RMAT-24): ids through filters and hash tables
// 4.31 / 119.4 ms; hub lists, one list per warp 1.90 / 74.7 ms; with the top bitmaps and units
// 1.50 / 71.6 ms, of which this kernel takes 1.4 / 44 ms.  What is left: on RMAT-24 the lists'
// reads (2.9 TB/s from L2 at a 70 % hit rate, 22 warps per SM beside 128 KB of counters), on
// smaller graphs instruction issue.
struct HubLayout {
    static constexpr u32 BITS = HUB_H / 32;  // bitmap words of a warp
    static constexpr u32 off_bits = 0;       // the warps' bitmaps, each aligned to its own size
    static constexpr u32 off_cnt = sizeof(u32) * BITS * HUB_WARPS;  // u32 counter per hub
    static constexpr u32 off_queue = off_cnt + sizeof(u32) * HUB_H;  // the warps' top bitmaps of a chunk
    static constexpr u32 align = sizeof(u32) * BITS;
    static constexpr size_t bytes = off_queue + sizeof(u32) * 32 * HUB_WARPS;
};
constexpr size_t HUB_SMEM = HubLayout::bytes + HubLayout::align;  // room to align the bitmaps
constexpr u32 HUB_LANE = 8;                        // hub lists up to this length are streamed by one lane
constexpr u32 HUB_PAD2 = HUB_PAD | (HUB_PAD << 16);  // two entries that hit nothing

// Eight entries of a hub list looked up in the bitmap at shared address `bits` (aligned to its
// size): counts the hits at the hubs' counters (shared address spare + base4) and returns their
// number.  A miss counts at the spare word: a predicated reduction becomes a branch around it (four
// more instructions per entry, and with a hit in almost every row it skips nothing; 2.12 against
// 1.90 ms on RMAT n = 10^6), and the address comes from a multiplication by the bit, since the
// logic units are the busiest (72 % with compares and selects).  All reads go out before the
// first test.
__device__ __forceinline__ u32 hub_probe8(const uint4& w, u32 bits, u32 base4, u32 spare) {
    const u32 pair[4] = {w.x, w.y, w.z, w.w};
    u32 h[8], v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[2 * i] = pair[i] & 0xFFFFu;
        h[2 * i + 1] = pair[i] >> 16;
        const u32 a0 = ((pair[i] >> 3) & (HUB_H / 8 - 4)) | bits;
        const u32 a1 = ((pair[i] >> 19) & (HUB_H / 8 - 4)) | bits;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[2 * i]) : "r"(a0) : "memory");
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[2 * i + 1]) : "r"(a1) : "memory");
    }
    u32 found = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const u32 hit = __funnelshift_r(v[i], v[i], h[i]) & 1u;
        const u32 at = (h[i] * 4 + base4) * hit + spare;
        asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(at) : "memory");
        found += hit;
    }
    return found;
}

// A warp's hit counts of the first HUB_TOP hubs, bit-sliced: lane l holds the words 2 l and 2 l + 1,
// plane p the bits of weight 2^p of 64 counters.  Four masks are added by carry-save adders, so a
// mask costs about 3.5 logic instructions per word instead of one atomic per hit.
struct TopCounters {
    static constexpr int PLANES = 11;
    u32 c[PLANES][2];
    u32 pend[2];     // a carry of weight 4 not yet added
    u32 added, odd;  // masks since the last flush; whether pend holds one
    static __device__ __forceinline__ u32 csa(u32& a, u32 b, u32 d) {  // a + b + d: sum bit to a, carry returned
        const u32 carry = (a & b) | (a & d) | (b & d);
        a = a ^ b ^ d;
        return carry;
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int p = 0; p < PLANES; ++p) c[p][0] = c[p][1] = 0;
        pend[0] = pend[1] = 0;
        added = odd = 0;
    }
    __device__ __forceinline__ void add4(const uint2 (&m)[4], u32* hcnt, u32 lane) {
        u32 four[2];
        four[0] = csa(c[1][0], csa(c[0][0], m[0].x, m[1].x), csa(c[0][0], m[2].x, m[3].x));
        four[1] = csa(c[1][1], csa(c[0][1], m[0].y, m[1].y), csa(c[0][1], m[2].y, m[3].y));
        if (odd) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                u32 carry = csa(c[2][k], pend[k], four[k]);
#pragma unroll
                for (int p = 3; p < PLANES; ++p) {
                    const u32 next = c[p][k] & carry;
                    c[p][k] ^= carry;
                    carry = next;
                }
            }
            odd = 0;
        } else {
            pend[0] = four[0];
            pend[1] = four[1];
            odd = 1;
        }
        added += 4;
        if (added + 4 >= (1u << PLANES)) flush(hcnt, lane);
    }
    // Adds the counters to the block's (lanes start at different bits: no two in one bank).
    __device__ __forceinline__ void flush(u32* hcnt, u32 lane) {
        for (u32 i = 0; i < 64; ++i) {
            const u32 k = i >> 5, b = (i + lane) & 31u;
            u32 v = odd ? ((k ? pend[1] : pend[0]) >> b & 1u) << 2 : 0u;
#pragma unroll
            for (int p = 0; p < PLANES; ++p) v += ((k ? c[p][1] : c[p][0]) >> b & 1u) << p;
            if (v) atomicAdd(&hcnt[(2 * lane + k) * 32 + b], v);
        }
        clear();
    }
};

__global__ void __launch_bounds__(32 * HUB_WARPS, 1)
    k_count_hub(const u64* __restrict__ fo, const u32* __restrict__ head, const Desc<u32>* __restrict__ vdesc,
                const u16* __restrict__ hubp, const u32* __restrict__ hub_ids, const u32* __restrict__ top_info,
                const uint2* __restrict__ top_bits, const uint2* __restrict__ mtiles,
                const uint2* __restrict__ ltiles, u32 seg, u64* __restrict__ cnt, u64* __restrict__ partials,
                Control* ctl) {
    chain_begin();
    using L = HubLayout;
    constexpr u32 FULL = 0xFFFFFFFFu;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ u64 s_red[HUB_WARPS];
    if (ctl->err & DEV_ERR_MASK) return;
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 nh = ctl->hubs;
    const u64 nl = *(volatile unsigned long long*)&ctl->large_tiles;
    const u64 nt = nh ? nl + *(volatile unsigned long long*)&ctl->medium_tiles : 0;
    if (nt == 0) {
        if (threadIdx.x == 0) partials[blockIdx.x] = 0;
        return;
    }
    unsigned char* sbase = smem + ((L::align - (smem_u32(smem) & (L::align - 1))) & (L::align - 1));
    u32* hcnt = reinterpret_cast<u32*>(sbase + L::off_cnt);
    u32* bits = reinterpret_cast<u32*>(sbase + L::off_bits) + warp * L::BITS;
    const u32 bits_at = smem_u32(bits);
    u32* queue = reinterpret_cast<u32*>(sbase + L::off_queue) + warp * 32;
    const u32 spare_at = smem_u32(hcnt + HUB_PAD);  // no hub's counter
    const u32 base4 = 0u - (u32)sizeof(u32) * HUB_PAD;  // the counters from there
    for (u32 i = threadIdx.x; i < HUB_H; i += 32 * HUB_WARPS) hcnt[i] = 0;
    for (u32 i = lane; i < L::BITS; i += 32) bits[i] = 0;
    __syncthreads();
    u64 total = 0;
    u32 dup = 0;
    TopCounters tops;
    tops.clear();
    while (true) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(&ctl->hub_next, 1ull);
        t = __shfl_sync(FULL, t, 0);
        if (t >= nt) break;
        const uint2 tl = t < nl ? ltiles[tile_at(true, t)] : mtiles[t - nl];
        const u32 x = tl.x;
        const Desc<u32> dx = load_desc(vdesc + x);
        const u32 xh = hub_len<true>(dx.d), xt = list_len<true>(dx.d);
        if (xh == 0) continue;
        const u16* own = hubp + hub_start(list_start(dx), x);
        const u32 xinfo = __ldg(top_info + x), xo = xh - (xinfo & 0xFFFu);
        uint2* top_words = reinterpret_cast<uint2*>(bits) + lane;  // this lane's two words of the top bits
        if (xinfo) *top_words = __ldg(top_bits + (u64)(xinfo >> 12) * 32 + lane);
        __syncwarp();
        for (u32 k = lane; k < xo; k += 32) {
            const u32 h = __ldg(own + k), bit = 1u << (h & 31u);
            if (atomicOr(&bits[h >> 5], bit) & bit) dup = 1;
        }
        const u64 a = fo[x] + (u64)tl.y * seg, fx1 = fo[x + 1];
        const u32 ns = (u32)(a + seg < fx1 ? (u64)seg : fx1 - a);
        __syncwarp();
        const uint2 xtop = *top_words;
        u32 T = 0;
        // two chunks ahead the neighbours, one chunk ahead their descriptors are in flight
        auto neighbour = [&](u32 e) { return e + lane < ns ? __ldg(head + a + e + lane) : x; };
        u32 y0 = neighbour(0), y1 = neighbour(32);
        Desc<u32> v0 = load_desc(vdesc + y0);
        u32 i0 = __ldg(top_info + y0);
        for (u32 e0 = 0; e0 < ns; e0 += 32) {
            const u32 yc = y0, info0 = i0;
            const Desc<u32> vy = v0;
            const bool have = e0 + lane < ns;
            y0 = y1;
            v0 = load_desc(vdesc + y0);
            i0 = __ldg(top_info + y0);
            y1 = neighbour(e0 + 64);
            const u32 yh = hub_len<true>(vy.d);
            const bool sel = have && yh > 0 && key_less(list_len<true>(vy.d), yc, xt, x);
            const u32 ys = (u32)(hub_start(list_start(vy), yc) >> 3);  // in 16-byte groups
            const u32 info = sel ? info0 : 0u;
            const u32 yo = yh - (info & 0xFFFu);  // entries left in the list
            u32 hits = 0;
            // top bitmaps, four at a time: one AND for 32 entries, counted per bit position
            const u32 with_top = __ballot_sync(FULL, info != 0);
            if (with_top) {
                const u32 rank = __popc(with_top & ((1u << lane) - 1));
                queue[lane] = 0;
                __syncwarp();
                if (info) queue[rank] = info >> 12;
                __syncwarp();
                u32 v = 0;  // lane r: the hits of the chunk's r-th bitmap
                const u32 nb = __popc(with_top);
                for (u32 r = 0; r < nb; r += 4) {
                    const uint4 at = *reinterpret_cast<const uint4*>(queue + r);
                    uint2 m[4];
                    m[0] = __ldg(top_bits + (u64)at.x * 32 + lane);
                    m[1] = __ldg(top_bits + (u64)at.y * 32 + lane);
                    m[2] = __ldg(top_bits + (u64)at.z * 32 + lane);
                    m[3] = __ldg(top_bits + (u64)at.w * 32 + lane);
                    u32 p[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        m[j].x &= xtop.x;
                        m[j].y &= xtop.y;
                        p[j] = __popc(m[j].x) + __popc(m[j].y);
                    }
                    const u32 r01 = __reduce_add_sync(FULL, p[0] | (p[1] << 16));
                    const u32 r23 = __reduce_add_sync(FULL, p[2] | (p[3] << 16));
                    const u32 mine = lane - r;  // 0..3: one of these four is this lane's
                    if (mine < 4) v = ((mine & 2u ? r23 : r01) >> (16 * (mine & 1u))) & 0xFFFFu;
                    tops.add4(m, hcnt, lane);
                }
                v = __shfl_sync(FULL, v, rank & 31);
                if (info) hits = v;
            }
            if (sel && yo > 0 && yo <= HUB_LANE) {
                const uint4* lp = reinterpret_cast<const uint4*>(hubp) + ys;
                const uint4 g0 = __ldg(lp);
                hits += hub_probe8(g0, bits_at, base4, spare_at);
            }
            __syncwarp();
            // the longer lists, cut into units of 64 entries: eight lanes take a unit, four units
            // (of one list or of several) a row.  The next row is in flight while the current one
            // is looked up.
            const u32 yq = (yo + 7) / 8;  // 16-byte groups
            const u32 units = sel && yo > HUB_LANE ? (yq + 7) / 8 : 0u;
            u32 P = units;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 z = __shfl_up_sync(FULL, P, o);
                if (lane >= (u32)o) P += z;
            }
            const u32 U = __shfl_sync(FULL, P, 31);
            P = units ? P - units : 0xFFFFFFFFu;  // the list's first unit
            uint4 nw = make_uint4(HUB_PAD2, HUB_PAD2, HUB_PAD2, HUB_PAD2);
            int n0 = 0, n1 = 0, n2 = 0, n3 = 0;  // the lanes whose lists the row's units belong to
            auto fetch = [&](u32 u) {
                n0 = 31 - __clz(__ballot_sync(FULL, P <= u));
                n1 = 31 - __clz(__ballot_sync(FULL, P <= u + 1));
                n2 = 31 - __clz(__ballot_sync(FULL, P <= u + 2));
                n3 = 31 - __clz(__ballot_sync(FULL, P <= u + 3));
                const int k = lane < 16 ? (lane < 8 ? n0 : n1) : (lane < 24 ? n2 : n3);
                const u32 o = (u + (lane >> 3) - __shfl_sync(FULL, P, k)) * 8 + (lane & 7u);
                const bool in = o < __shfl_sync(FULL, yq, k);
                const uint4* lp = reinterpret_cast<const uint4*>(hubp) + __shfl_sync(FULL, ys, k);
                nw = make_uint4(HUB_PAD2, HUB_PAD2, HUB_PAD2, HUB_PAD2);
                if (in) nw = __ldg(lp + o);
            };
            if (U) fetch(0);
            for (u32 u = 0; u < U; u += 4) {
                const uint4 w = nw;
                const int k0 = n0, k1 = n1, k2 = n2, k3 = n3;
                if (u + 4 < U) fetch(u + 4);
                const u32 f = hub_probe8(w, bits_at, base4, spare_at);
                // the four units' hits (at most 64 each) side by side in one sum
                const u32 s4 = __reduce_add_sync(FULL, f << (lane & 24u));
                if ((int)lane == k0) hits += s4 & 0xFFu;
                if ((int)lane == k1) hits += (s4 >> 8) & 0xFFu;
                if ((int)lane == k2) hits += (s4 >> 16) & 0xFFu;
                if ((int)lane == k3) hits += s4 >> 24;
            }
            if (hits) {
                atomicAdd(&cnt[yc], (u64)hits);
                T += hits;
            }
        }
        const u32 wt = __reduce_add_sync(FULL, T);
        if (lane == 0 && wt) {
            atomicAdd(&cnt[x], (u64)wt);
            total += wt;
        }
        __syncwarp();
        *top_words = make_uint2(0, 0);
        for (u32 k = lane; k < xo; k += 32) bits[__ldg(own + k) >> 5] = 0;
        __syncwarp();
    }
    tops.flush(hcnt, lane);
    if (dup) atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
    const u64 bt = block_sum_u64<32 * HUB_WARPS>(total, s_red);  // also orders the counters' last hits
    if (threadIdx.x == 0) partials[blockIdx.x] = bt;
    for (u32 i = threadIdx.x; i < nh; i += 32 * HUB_WARPS) {
        const u32 c = hcnt[i];
        if (c) atomicAdd(&cnt[hub_ids[i]], (u64)c);
    }
}

// Sum of the per-block partial totals (a u64 tree reduction in one block), without the slots
// [skip0, skip1) of blocks that were not launched.  After a device error (invalid input, a
// bounded wait that ran out) the partials are incomplete or stale, so the total is written as 0.
__global__ void __launch_bounds__(1024) k_final(const u64* __restrict__ partials, u32 np, u32 skip0, u32 skip1,
                                                u64* total, const Control* ctl) {
    chain_begin();
    __shared__ u64 s_red[32];
    if (*(volatile const u32*)&ctl->err & DEV_ERR_MASK) {
        if (threadIdx.x == 0) *total = 0;
        return;
    }
    u64 s = 0;
    for (u32 i = threadIdx.x; i < np; i += 1024)
        if (i < skip0 || i >= skip1) s += partials[i];
    const u64 t = block_sum_u64<1024>(s, s_red);
    if (threadIdx.x == 0) *total = t;
}

// Batched counting: per-graph totals of a disjoint union (graph g owns the vertices
// [graph_first[g], graph_first[g+1])).  Every triangle adds one to each of its three corners,
// all inside one graph, so a graph's total is the sum of its per-vertex counts over three.
// `parts` blocks share a graph (totals are zeroed by the caller when there are several): few graphs
// would otherwise leave the largest to one block (11 graphs with one of 2.7 M vertices: 711 us by
// one block each, 21 us by 64 with eight loads in flight per thread; 512 graphs 57 -> 46 us).  A part's
// sum need not be a multiple of three, so the parts add up their sums, and the last to arrive (the top
// bits of totals[g] count them: the sum of all per-vertex counts of 2^36 entries is below 2^57) divides.
constexpr int GRAPH_PARTS = 64;  // most blocks of a graph
__global__ void __launch_bounds__(256) k_graph_totals(const u64* __restrict__ cnt, const u64* __restrict__ graph_first,
                                                      u64 num_graphs, u64 n, u64* __restrict__ totals, u32 parts,
                                                      Control* ctl) {
    chain_begin();
    __shared__ u64 s_red[8];
    if (ctl->err & DEV_ERR_MASK) return;
    const u32 per = gridDim.x / parts;  // blocks of one part
    const u32 part = blockIdx.x / per;
    for (u64 g = blockIdx.x % per; g < num_graphs; g += per) {
        const u64 a = graph_first[g], b = graph_first[g + 1];
        const bool ok = a <= b && b <= n;
        u64 s = 0;
        if (ok) {
            // eight loads in flight per thread
            const u64 step = 256 * (u64)parts;
            for (u64 v = a + part * 256 + threadIdx.x; v < b; v += 8 * step) {
                u64 c[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) c[k] = v + k * step < b ? cnt[v + k * step] : 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) s += c[k];
            }
        }
        s = block_sum_u64<256>(s, s_red);
        if (threadIdx.x == 0) {
            if (parts == 1) {
                totals[g] = s / 3;
            } else if (ok) {
                constexpr u64 ARRIVED = 1ull << 57;
                static_assert(GRAPH_PARTS < (1 << 7), "arrivals fit above the sum");
                const u64 before = atomicAdd(&totals[g], s + ARRIVED);
                if (before / ARRIVED + 1 == parts) totals[g] = (before + s) % ARRIVED / 3;
            }
            if (!ok) atomicOr(&ctl->err, DEV_ERR_DEGREE);
        }
    }
}

// collect_stats: wedge_checks = sum over oriented (v,u) of |N+(u)|, the reference's counter
// (cetric_edge_iterator.h:279-281), plus the entries streamed by the AUTO kernels, also counted
// once per table chunk of their owner: LARGE_CAP keys for owners above medium_d, TileLayout's CAP for the
// others and, with hubs, for what no owner's hubs take.  medium_d = 0: a strategy without tables.
template <typename OffT, bool HUB>
__global__ void k_stats(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n,
                        const Desc<OffT>* __restrict__ vdesc, const u32* __restrict__ headp,
                        const u16* __restrict__ hubp, const u32* __restrict__ hub_ids, u32 small_d, u32 medium_d,
                        Control* ctl) {
    chain_begin();
    if (ctl->err & DEV_ERR_MASK) return;
    const int lane = threadIdx.x & 31;
    const u64 gw = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
    u64 wedge = 0, isz = 0, streamed = 0, oriented = 0, chunked = 0;
    for (u64 v = gw; v < n; v += nwarps) {
        const Desc<OffT> dv = load_desc(vdesc + v);
        const u32 lv = list_len<HUB>(dv.d), rv = rest_len<HUB>(dv.d);
        const u32 keys = medium_d == 0 ? ~0u : !HUB && lv > medium_d ? (u32)LARGE_CAP : TileLayout<OffT>::CAP;
        const u64 chunks = rv > keys ? ((u64)rv + keys - 1) / keys : 1;
        if (lane == 0) oriented += lv;
        for (u32 k = lane; k < lv; k += 32) {
            const u32 u = k < rv ? headp[list_start(dv) + k]
                                 : hub_ids[hubp[hub_start(list_start(dv), v) + (k - rv)]];
            const u32 du = list_len<HUB>(load_desc(vdesc + u).d);
            wedge += du;
            isz += (u64)lv + du;
            if (lv >= 2 && lv <= small_d && du <= small_d) {  // counted at the tail
                streamed += du;
                chunked += du;
            }
        }
        if (lv <= small_d) continue;  // no owner
        for (u64 e = fo[v] + lane; e < fo[v + 1]; e += 32) {
            const u32 y = head[e];
            const u32 word = load_desc(vdesc + y).d, dy = list_len<HUB>(word);
            if (dy > 0 && key_less(dy, y, lv, v)) {
                streamed += dy;
                chunked += hub_len<HUB>(word) + rest_len<HUB>(word) * chunks;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        wedge += __shfl_down_sync(0xFFFFFFFFu, wedge, o);
        isz += __shfl_down_sync(0xFFFFFFFFu, isz, o);
        streamed += __shfl_down_sync(0xFFFFFFFFu, streamed, o);
        oriented += __shfl_down_sync(0xFFFFFFFFu, oriented, o);
        chunked += __shfl_down_sync(0xFFFFFFFFu, chunked, o);
    }
    if (lane == 0) {
        atomicAdd(&ctl->stat_wedge, wedge);
        atomicAdd(&ctl->stat_isz, isz);
        atomicAdd(&ctl->stat_streamed, streamed);
        atomicAdd(&ctl->stat_oriented, oriented);
        atomicAdd(&ctl->stat_chunked, chunked);
    }
}

// ---- the serving engine ----------------------------------------------------------------

using EngineSmallL = SmallWarpLayout<u32, false>;
using EngineMediumL = TileLayout<u32>;
using EngineLargeL = LargeLayout<ENGINE_BLOCK, LARGE_CAP, u32>;
constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }
constexpr size_t ENGINE_SMEM =
    cmax(cmax(EngineSmallL::bytes(ENGINE_BLOCK / 32), EngineMediumL::bytes(ENGINE_BLOCK / 32)), EngineLargeL::bytes);
static_assert(SMALL_BLOCK == ENGINE_BLOCK && MEDIUM_BLOCK == ENGINE_BLOCK && LARGE_BLOCK == ENGINE_BLOCK,
              "the engine runs every kind of unit with one block shape");

// The claim cursor of a job holds the publication's tag (low 24 bits of its sequence number) in
// its top 24 bits and the next unit in its low 40 bits.  Units are claimed by compare-and-swap
// against a cursor whose tag matches the sequence number read before and after it, so a block
// can never take a unit of a later publication of the same slot, nor read a half-written record.
constexpr int ENGINE_TAG_SHIFT = 40;
constexpr unsigned long long ENGINE_COUNT_MASK = (1ull << ENGINE_TAG_SHIFT) - 1;
__device__ __forceinline__ unsigned long long engine_tag(unsigned long long seq) { return seq & 0xFFFFFFull; }

__global__ void k_publish(EngineJob* job, unsigned long long seq, const u64* fo, const u32* head, u64 n,
                          const void* vdesc, const u32* headp, const uint2* mtiles, const uint2* ltiles, u64* cnt,
                          Control* ctl, u32 small_d, u32 seg, unsigned long long* done_word) {
    if (threadIdx.x != 0) return;
    volatile EngineJob* vj = job;
    vj->seq = 0;  // unpublished while the record changes
    __threadfence();
    const bool bad = (*(volatile u32*)&ctl->err & DEV_ERR_MASK) != 0;
    const unsigned long long nbatch = (n + 31) / 32;
    const unsigned long long us = bad ? 0 : (nbatch + ENGINE_UNIT_ITEMS - 1) / ENGINE_UNIT_ITEMS;
    const unsigned long long um =
        bad ? 0 : (*(volatile unsigned long long*)&ctl->medium_tiles + ENGINE_UNIT_ITEMS - 1) / ENGINE_UNIT_ITEMS;
    const unsigned long long ul = bad ? 0 : *(volatile unsigned long long*)&ctl->large_tiles;
    if (us + um + ul == 0) {  // nothing for the engine: done at once
        __threadfence_system();
        *(volatile unsigned long long*)done_word = seq;
        return;
    }
    vj->fo = fo;
    vj->head = head;
    vj->n = n;
    vj->vdesc = vdesc;
    vj->headp = headp;
    vj->mtiles = mtiles;
    vj->ltiles = ltiles;
    vj->cnt = cnt;
    vj->ctl = ctl;
    vj->small_d = small_d;
    vj->seg = seg;
    vj->units_small = us;
    vj->units_medium = um;
    vj->units = us + um + ul;
    vj->done = 0;
    __threadfence();
    vj->next = engine_tag(seq) << ENGINE_TAG_SHIFT;
    __threadfence();
    vj->seq = seq;
}

__global__ void __launch_bounds__(ENGINE_BLOCK, 4) k_engine(EngineJob* jobs, u32 njobs, unsigned long long* done_words,
                                                         unsigned* stop, u32 idle_polls) {
    constexpr int BLOCK = ENGINE_BLOCK;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_job;
    __shared__ unsigned long long s_unit;
    __shared__ EngineJob s_jb;  // the claimed job's record, read at L2 by thread 0
    __shared__ u32 s_jb_slot;
    __shared__ unsigned s_stop;
    __shared__ int s_work;  // some published job was unfinished in the last scan
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    (void)lane;
    // the large-owner tiles' bulk-copy barrier: outside the dynamic region, which the small- and
    // medium-owner units overwrite between large tiles, since its phase persists across units
    __shared__ __align__(8) unsigned long long s_bar_engine;
    unsigned long long* s_bar = &s_bar_engine;
    if (threadIdx.x == 0) {
        mbar_init(s_bar, 1);
        s_jb.seq = 0;
        s_jb_slot = 0xFFFFFFFFu;
    }
    fence_proxy_async_smem();
    __syncthreads();
    u32 phase = 0;
    bool inflight = false;
    u32 idle = 0, start = blockIdx.x % (njobs ? njobs : 1);
    while (true) {
        if (threadIdx.x == 0) {
            s_job = -1;
            s_work = 0;
            // a launch leaves as a whole: once any block has set the stop word (or the host has),
            // no block claims another unit
            s_stop = *(volatile const unsigned*)stop;
            for (u32 k = 0; k < njobs && s_job < 0 && !s_stop; ++k) {
                const u32 j = (start + k) % njobs;
                volatile EngineJob* vj = jobs + j;
                for (int attempt = 0; attempt < 4; ++attempt) {
                    const unsigned long long s1 = vj->seq;
                    if (s1 == 0) break;
                    s_work = 1;  // a published job is not finished
                    __threadfence();
                    const unsigned long long cur = vj->next;
                    const unsigned long long units = vj->units;
                    __threadfence();
                    if (vj->seq != s1 || (cur >> ENGINE_TAG_SHIFT) != engine_tag(s1)) break;
                    if ((cur & ENGINE_COUNT_MASK) >= units) break;
                    if (atomicCAS(const_cast<unsigned long long*>(&vj->next), cur, cur + 1) != cur) continue;
                    // unit (cur & mask) of publication s1: its record stays as it is until the job
                    // is done, which needs this unit
                    s_job = (int)j;
                    s_unit = cur & ENGINE_COUNT_MASK;
                    start = j + 1;  // the next scan begins at the following job: no job is favoured
                    if (s_jb.seq == s1 && s_jb_slot == j) break;  // this block holds the record already
                    s_jb_slot = j;
                    s_jb.fo = vj->fo;
                    s_jb.head = vj->head;
                    s_jb.n = vj->n;
                    s_jb.vdesc = vj->vdesc;
                    s_jb.headp = vj->headp;
                    s_jb.mtiles = vj->mtiles;
                    s_jb.ltiles = vj->ltiles;
                    s_jb.cnt = vj->cnt;
                    s_jb.ctl = vj->ctl;
                    s_jb.small_d = vj->small_d;
                    s_jb.seg = vj->seg;
                    s_jb.units_small = vj->units_small;
                    s_jb.units_medium = vj->units_medium;
                    s_jb.units = units;
                    s_jb.seq = s1;
                    break;
                }
            }
        }
        __syncthreads();
        const int j = s_job;
        if (j < 0) {
            // Only scans that found every published job finished count towards leaving: while a
            // job's last units run on other blocks, this block stays for the jobs published next.
            // The first block to leave sets the stop word, and the others follow at their next
            // scan: a launch that shrank to a few blocks would serve a job published meanwhile at
            // a trickle, and the host relaunches the engine only once the launch has ended.
            if (s_work) idle = 0;
            if (s_stop) break;  // the same decision in every thread
            if (++idle > idle_polls) {
                if (threadIdx.x == 0) {
                    *(volatile unsigned*)stop = 1u;
                    __threadfence();
                }
                break;
            }
            __nanosleep(2000);
            __syncthreads();  // every thread has read s_job before thread 0 writes it again
            continue;
        }
        idle = 0;
        const EngineJob* jb = &s_jb;
        const unsigned long long u = s_unit;
        Control* ctl = jb->ctl;
        const auto* vd = reinterpret_cast<const Desc<u32>*>(jb->vdesc);
        u64 unused_total = 0;
        u32 dup = 0;
        bool timed_out = false;
        if (u < jb->units_small) {
            const u64 nb = (jb->n + 31) / 32;
            u32* slice = reinterpret_cast<u32*>(smem) + warp * EngineSmallL::PER_WARP;
            const bool distinct = !(*(volatile u32*)&ctl->err & DEV_FLAG_UNSORTED);
            small_init<u32, false>(slice);  // other kinds of unit use the same shared memory
            for (u32 r = 0; r < ENGINE_REPS; ++r) {
                const u64 bi = (u * (ENGINE_BLOCK / 32) + warp) * ENGINE_REPS + r;
                if (bi < nb)
                    small_batch<u32, false, true>(slice, bi, 32, jb->n, vd, jb->headp, nullptr, nullptr, jb->small_d,
                                                  distinct, jb->cnt, unused_total, dup);
            }
        } else if (u < jb->units_small + jb->units_medium) {
            const u64 nt = *(volatile unsigned long long*)&ctl->medium_tiles;
            u32* slice = reinterpret_cast<u32*>(smem) + warp * EngineMediumL::PER_WARP;
            tile_init<u32>(slice);
            const u32 top = jb->n < 0x7FFFFFFFu ? 0x80000000u : 0u;
            for (u32 r = 0; r < ENGINE_REPS; ++r) {
                const u64 t = ((u - jb->units_small) * (ENGINE_BLOCK / 32) + warp) * ENGINE_REPS + r;
                if (t < nt)
                    medium_tile<u32, false, true>(slice, top, __ldcg(jb->mtiles + t), jb->fo, jb->head, vd, jb->headp,
                                                  jb->seg, jb->cnt, ctl, unused_total, dup);
            }
        } else {
            const u64 t = u - jb->units_small - jb->units_medium;
            timed_out = large_tile<BLOCK, LARGE_CAP, u32, true>(smem, s_bar, __ldcg(jb->ltiles + tile_at(true, t)), jb->fo,
                                                                jb->head, jb->n, vd, jb->headp, jb->seg, jb->cnt,
                                                                COPY_WAIT_POLLS, phase, inflight, unused_total, dup);
        }
        if (dup) atomicOr(&ctl->err, DEV_ERR_DUPLICATE);
        if (timed_out && threadIdx.x == 0)
            atomicOr(&ctl->err, DEV_ERR_TIMEOUT | (inflight ? DEV_ERR_COPY_INFLIGHT : 0u));
        __syncthreads();  // the unit's counts are all issued
        if (threadIdx.x == 0) {
            __threadfence();
            const unsigned long long d = atomicAdd(&jobs[j].done, 1ull) + 1;
            if (d == jb->units) {
                *(volatile unsigned long long*)&jobs[j].seq = 0;
                __threadfence_system();
                *(volatile unsigned long long*)(done_words + j) = jb->seq;
            }
        }
        // a copy that may still be landing in shared memory: this block stops taking units
        if (inflight) break;
    }
}

void launch_publish(EngineJob* job, unsigned long long seq, const u64* fo, const u32* head, u64 n,
                    const void* vdesc, const u32* headp, const uint2* mtiles, const uint2* ltiles, u64* cnt,
                    Control* ctl, u32 small_d, u32 seg, unsigned long long* done_word, cudaStream_t st) {
    k_publish<<<1, 32, 0, st>>>(job, seq, fo, head, n, vdesc, headp, mtiles, ltiles, cnt, ctl, small_d, seg, done_word);
}

size_t engine_smem_bytes() { return ENGINE_SMEM; }

int engine_grid(int num_sms) {
    static int occ = -1;
    if (occ < 0) {
        cudaFuncSetAttribute(k_engine, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ENGINE_SMEM);
        int o = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_engine, ENGINE_BLOCK, ENGINE_SMEM);
        occ = o > 0 ? o : 1;
    }
    // leave room on every SM for the preparation kernels of the batches being published: the
    // engine's blocks stay resident while any published job is unfinished, so with one block
    // slot per SM left the next batches' orientation starved (6.4K against 0.6-2.5K graphs/s at
    // saturation with two slots left against one)
    return num_sms * (occ > 2 ? occ - 2 : 1);
}

void launch_engine(EngineJob* jobs, u32 njobs, unsigned long long* done_words, unsigned* stop, u32 idle_polls,
                   int grid, cudaStream_t st) {
    k_engine<<<grid, ENGINE_BLOCK, ENGINE_SMEM, st>>>(jobs, njobs, done_words, stop, idle_polls);
}

// ---- launchers ------------------------------------------------------------------------

namespace {
template <typename OffT>
using LargeL = LargeLayout<LARGE_BLOCK, LARGE_CAP, OffT>;

// Resident blocks per SM of a kernel, looked up once; also allows it its dynamic shared memory.
template <typename Kernel>
int occupancy_of(Kernel kern, int block, size_t bytes) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    int o = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, block, bytes);
    return o > 0 ? o : 1;
}
}  // namespace

template <typename OffT, bool HUB>
int count_grid_small(int num_sms) {
    static const int occ = occupancy_of(k_count_small<SMALL_BLOCK, OffT, HUB>, SMALL_BLOCK,
                                        SmallWarpLayout<OffT, HUB>::bytes(SMALL_BLOCK / 32));
    return num_sms * occ;
}
template <typename OffT, bool HUB>
int count_grid_medium(int num_sms) {
    static const int occ = occupancy_of(k_count_medium<MEDIUM_BLOCK, OffT, HUB>, MEDIUM_BLOCK,
                                        TileLayout<OffT>::bytes(MEDIUM_BLOCK / 32));
    return num_sms * occ;
}
template <typename OffT, bool HUB>
int count_grid_large(int num_sms) {
    if constexpr (HUB) return 0;  // the hub and medium kernels take every tile
    static const int occ = occupancy_of(k_count_large<LARGE_BLOCK, LARGE_CAP, OffT>, LARGE_BLOCK, LargeL<OffT>::bytes);
    return num_sms * occ;
}
template <bool HUB>
int count_grid_hub(int num_sms) {
    if constexpr (!HUB) return 0;
    static const int occ = occupancy_of(k_count_hub, 32 * HUB_WARPS, HUB_SMEM);
    return num_sms * occ;
}
// Vertices per batch of the small kernel: 32, or fewer where the graph does not hold a batch of 32
// for every resident warp (a power of two, at least 4: a warp's serial chain is then shorter).
static u32 small_batch_vertices(u64 n, int cap) {
    u32 vb = 32;
    while (vb > 4 && n < (u64)cap * (SMALL_BLOCK / 32) * vb) vb >>= 1;
    return vb;
}
// Blocks the small kernel is launched with: enough for one vertex batch per warp, at most its
// resident grid (a small graph does not start hundreds of warps that find no batch).
int small_grid_launched(u64 n, int cap) {
    const u32 vb = small_batch_vertices(n, cap);
    const u64 need = ((n + vb - 1) / vb + SMALL_BLOCK / 32 - 1) / (SMALL_BLOCK / 32);
    return (int)(need < 1 ? 1 : (need < (u64)cap ? need : (u64)cap));
}

template <typename OffT, bool HUB>
int count_grid_auto(int num_sms) {
    return count_grid_small<OffT, HUB>(num_sms) + count_grid_medium<OffT, HUB>(num_sms) +
           count_grid_large<OffT, HUB>(num_sms) + count_grid_hub<HUB>(num_sms);
}

template <typename OffT, bool HUB>
cudaError_t launch_count_auto(const u64* fo, const u32* head, u64 n, const void* vdesc, const u32* headp,
                              const HubState& hub, const uint2* mtiles, const uint2* ltiles, u32 small_d, u32 seg,
                              u64* cnt, u64* partials, Control* ctl, int num_sms, LaunchStream st,
                              cudaEvent_t after_small, cudaEvent_t after_large, u32 copy_wait_polls) {
    const int cap = count_grid_small<OffT, HUB>(num_sms);
    const int gs = small_grid_launched(n, cap);
    const int gm = count_grid_medium<OffT, HUB>(num_sms);
    const int gl = count_grid_large<OffT, HUB>(num_sms);
    const auto* vd = reinterpret_cast<const Desc<OffT>*>(vdesc);
    launch_chained(k_count_small<SMALL_BLOCK, OffT, HUB>, gs, SMALL_BLOCK,
                   SmallWarpLayout<OffT, HUB>::bytes(SMALL_BLOCK / 32), st, n, small_batch_vertices(n, cap), vd, headp,
                   hub.lists, hub.ids, small_d, cnt, partials, ctl);
    if (after_small) cudaEventRecord(after_small, st);
    if constexpr (HUB)
        launch_chained(k_count_hub, count_grid_hub<HUB>(num_sms), 32 * HUB_WARPS, HUB_SMEM, st, fo, head, vd,
                       hub.lists, hub.ids, hub.top_info, hub.top_bits, mtiles, ltiles, seg, cnt,
                       partials + cap + gm + gl, ctl);
    launch_chained(k_count_medium<MEDIUM_BLOCK, OffT, HUB>, gm, MEDIUM_BLOCK,
                   TileLayout<OffT>::bytes(MEDIUM_BLOCK / 32), st, fo, head, n, vd, headp, mtiles, ltiles, seg, cnt,
                   partials + cap, ctl);
    if constexpr (!HUB)
        launch_chained(k_count_large<LARGE_BLOCK, LARGE_CAP, OffT>, gl, LARGE_BLOCK, LargeL<OffT>::bytes, st, fo, head,
                       n, vd, headp, ltiles, seg, cnt, partials + cap + gm, ctl, copy_wait_polls);
    if (after_large) cudaEventRecord(after_large, st);
    return cudaGetLastError();
}

void launch_graph_totals(const u64* cnt, const u64* graph_first, u64 num_graphs, u64 n, u64* totals, Control* ctl,
                         int num_sms, LaunchStream st) {
    if (num_graphs == 0) return;
    const u64 cap = (u64)num_sms * 8;
    const u64 blocks = num_graphs < cap ? num_graphs : cap;
    // as many parts as fill the chip, none smaller than 4096 vertices if one graph has them all
    const u64 fill = cap / blocks < n / 4096 ? cap / blocks : n / 4096;
    const u64 parts = fill < 1 ? 1 : fill < GRAPH_PARTS ? fill : GRAPH_PARTS;
    if (parts > 1) cudaMemsetAsync(totals, 0, sizeof(u64) * num_graphs, st.st);
    launch_chained(k_graph_totals, (unsigned)(blocks * parts), 256, 0, st, cnt, graph_first, num_graphs, n, totals,
                   (u32)parts, ctl);
}

void launch_final(const u64* partials, u32 np, u64* total, Control* ctl, LaunchStream st) {
    launch_chained(k_final, 1, 1024, 0, st, partials, np, 0, 0, total, ctl);
}

template <typename OffT, bool HUB>
void launch_final_auto(const u64* partials, u64 n, int num_sms, u64* total, Control* ctl, LaunchStream st) {
    const int cap = count_grid_small<OffT, HUB>(num_sms);
    launch_chained(k_final, 1, 1024, 0, st, partials, (u32)count_grid_auto<OffT, HUB>(num_sms),
                   (u32)small_grid_launched(n, cap), (u32)cap, total, ctl);
}

template <typename OffT, bool HUB>
void launch_stats(const u64* fo, const u32* head, u64 n, const void* vdesc, const u32* headp, const HubState& hub,
                  u32 small_d, u32 medium_d, Control* ctl, int num_sms, LaunchStream st) {
    if (n == 0) return;
    launch_chained(k_stats<OffT, HUB>, num_sms * 8, 256, 0, st, fo, head, n,
                   reinterpret_cast<const Desc<OffT>*>(vdesc), headp, hub.lists, hub.ids, small_d, medium_d, ctl);
}

#define KTRI_INST(OffT, HUB)                                                                                        \
    template void launch_final_auto<OffT, HUB>(const u64*, u64, int, u64*, Control*, LaunchStream);                 \
    template int count_grid_auto<OffT, HUB>(int);                                                                   \
    template cudaError_t launch_count_auto<OffT, HUB>(const u64*, const u32*, u64, const void*, const u32*,         \
                                                      const HubState&, const uint2*, const uint2*, u32, u32, u64*,  \
                                                      u64*, Control*, int, LaunchStream, cudaEvent_t, cudaEvent_t,  \
                                                      u32);                                                         \
    template void launch_stats<OffT, HUB>(const u64*, const u32*, u64, const void*, const u32*, const HubState&,    \
                                          u32, u32, Control*, int, LaunchStream);
KTRI_INST(u32, false)
KTRI_INST(u32, true)
KTRI_INST(u64, false)
#undef KTRI_INST

}  // namespace ktri
