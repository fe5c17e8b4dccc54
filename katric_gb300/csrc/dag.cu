// Symmetrisation of oriented out-lists into the undirected CSR of their edges.
//
// KaTric's local phase (CetricEdgeIterator::run_local, cetric_edge_iterator.h:230-298, and
// the variant with ghosts, :301-388) walks out-lists the caller has already oriented: out_adj
// of the rank's vertices and ghost_adj of its ghosts.  The triangles it finds are the
// triangles whose three edges appear in those lists.  That set does not depend on the
// orientation, so the lists are turned back into an undirected CSR here and counted by the
// ordinary pipeline, under its own (degree, id) orientation.
//
// Vertex v's undirected list is its out-list (in the given order) followed by its in-list
// (in arrival order).  Entries that are out of range or self-loops are copied into the out part as
// they are, so the pipeline's validation reports them (out of range: without an in-list entry).
// Offsets that do not hold m entries read none: their lists come out too long, which it reports.
#include <algorithm>

#include "ktri.h"
#include "ktri_device.cuh"
#include "ktri_kernels.h"

namespace ktri {

namespace {

constexpr int SCAN_BLOCK = 256;
constexpr int SCAN_IPT = 8;
constexpr u64 SCAN_CHUNK = (u64)SCAN_BLOCK * SCAN_IPT;

// Where vertex u is counted: a permutation of [0, 2^k) that puts neighbouring ids on lines apart.
// Graphs with neighbouring hubs (RMAT: ids below 32 are named by 3 % of all entries) otherwise queue
// their atomics at one line of the L2 cache: the arrivals of 8.6 M entries took 230 us, 117 us so.
// (Counting a block's entries in a table in shared memory first: 144 us, and 5 to 9 % more for the
// whole count of a uniform graph.)
__device__ __forceinline__ u32 count_slot(u32 u, u32 mask) { return (u * 0x9E3779B1u) & mask; }

// Do the offsets hold m entries?  (Any first offset: the lists may lie inside a larger buffer.)
__device__ __forceinline__ bool holds(const u64* fo, u64 n, u64 m) { return fo[n] - fo[0] == m; }

// Arrivals: pos[e] = the place of entry e among the entries that name the same vertex, in_deg[slot of
// u] = the number of entries that name u (zeroed by the caller).  The only atomics of the symmetrisation; an
// entry needs no owner here (a self-loop gets a place like any other and is reported as what it is).
__global__ void k_dag_arrive(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n, u64 m,
                             u32* __restrict__ in_deg, u32 mask, u32* __restrict__ pos) {
    if (!holds(fo, n, m)) return;
    const u32* h = head + fo[0];
    const u64 stride = (u64)gridDim.x * blockDim.x;
    for (u64 e = (u64)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += 4 * stride) {
        u32 u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = e + k * stride < m ? __ldcs(h + e + k * stride) : 0xFFFFFFFFu;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (u[k] < n) pos[e + k * stride] = atomicAdd(&in_deg[count_slot(u[k], mask)], 1u);
    }
}

// |out(v)|; descending offsets, and vertex 0 of offsets that do not hold m entries, give a length that
// no graph of m edges has.
__device__ __forceinline__ u64 out_length(const u64* fo, u64 v, u64 n, u64 m) {
    const u64 a = fo[v], b = fo[v + 1];
    return b >= a && (v || holds(fo, n, m)) ? b - a : 2 * m + 1;
}

// In-place exclusive scan of x[0..len), pass 1: every chunk scanned locally, its sum to sums.
// DAG: of the undirected lists' lengths, |out(v)| + the entries that name v, instead of x.
template <bool DAG>
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_chunks(u64* x, u64 len, u64* sums, const u64* __restrict__ fo,
                                                            const u32* __restrict__ in_deg, u32 mask, u64 m) {
    __shared__ u64 s_warp[SCAN_BLOCK / 32];
    const u64 c0 = (u64)blockIdx.x * SCAN_CHUNK + (u64)threadIdx.x * SCAN_IPT;
    u64 v[SCAN_IPT], t = 0;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        if constexpr (DAG) {
            v[k] = 0;
            if (c0 + k + 1 < len) v[k] = out_length(fo, c0 + k, len - 1, m) + in_deg[count_slot((u32)(c0 + k), mask)];
        } else {
            v[k] = c0 + k < len ? x[c0 + k] : 0ull;
        }
        t += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    u64 wbase = 0, total = 0;
#pragma unroll
    for (int w = 0; w < SCAN_BLOCK / 32; ++w) {
        if (w < warp) wbase += s_warp[w];
        total += s_warp[w];
    }
    u64 run = wbase + incl - t;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        if (c0 + k < len) x[c0 + k] = run;
        run += v[k];
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Pass 2: exclusive scan of the chunk sums in one block (any number of chunks).
__global__ void __launch_bounds__(1024) k_scan_sums(u64* sums, u64 nchunks) {
    __shared__ u64 s_warp[32];
    __shared__ u64 s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (u64 base = 0; base < nchunks; base += 1024) {
        const u64 i = base + threadIdx.x;
        const u64 t = i < nchunks ? sums[i] : 0ull;
        u64 incl = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        u64 wbase = 0, total = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) wbase += s_warp[w];
            total += s_warp[w];
        }
        const u64 carry = s_carry;
        if (i < nchunks) sums[i] = carry + wbase + incl - t;
        __syncthreads();
        if (threadIdx.x == 0) s_carry = carry + total;
        __syncthreads();
    }
}

// Pass 3: add each chunk's offset.  DAG: also where each vertex' in-list starts.
template <bool DAG>
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_add(u64* x, u64 len, const u64* sums, const u64* __restrict__ fo,
                                                         u64* __restrict__ in_start, u64 m) {
    const u64 off = sums[blockIdx.x];
    const u64 c0 = (u64)blockIdx.x * SCAN_CHUNK;
    for (u64 k = c0 + threadIdx.x; k < c0 + SCAN_CHUNK && k < len; k += SCAN_BLOCK) {
        const u64 s = x[k] + off;
        x[k] = s;
        if constexpr (DAG)
            if (k + 1 < len) in_start[k] = s + out_length(fo, k, len - 1, m);
    }
}

// The last vertex whose list starts at or before entry e (its owner, where the offsets ascend), by
// the whole warp: 32 probes a step.
__device__ __forceinline__ u64 owner_of(const u64* __restrict__ fo, u64 n, u64 e, u32 lane) {
    u64 lo = 0, hi = n;
    while (hi - lo > 1) {
        const u64 step = (hi - lo + 32) / 33, p = lo + (lane + 1) * step;
        lo += __popc(__ballot_sync(0xFFFFFFFFu, p < hi && fo[p] <= e)) * step;
        hi = lo + step < hi ? lo + step : hi;
    }
    return lo;
}

// Undirected lists: v's out-list copied to the front of its range, v put at the entry's place in
// the in part of every valid out-neighbour.  A warp takes DAG_TILE entries whatever lists they are
// of, so long lists are shared by many warps.  Offsets that do not give 2 m entries write nothing
// (the count reports them).
// What bounds it: the scattered 4-byte writes and the gather of in_start.  Measured (8.6 M entries of
// an RMAT rank, n = 7 10^5): 352 us with a warp per list, an atomic and three gathers per entry,
// 141 us so.
constexpr u32 DAG_TILE = 128;
__global__ void k_dag_scatter(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n, u64 m,
                              const u64* __restrict__ fs, const u64* __restrict__ in_start,
                              const u32* __restrict__ pos, u32* __restrict__ hs) {
    if (fs[n] != 2 * m || !holds(fo, n, m)) return;
    const u32 lane = threadIdx.x & 31;
    const u64 warp = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
    const u64 first = fo[0];
    for (u64 t0 = warp * DAG_TILE; t0 < m; t0 += nwarps * DAG_TILE) {
        u64 vb = owner_of(fo, n, first + t0, lane);     // the window's first vertex
        u64 end = fo[vb + 1 + lane < n ? vb + 1 + lane : n];  // where each of its lists ends
        for (u32 r = 0; r < DAG_TILE && t0 + r < m; r += 32) {
            const u64 i = t0 + r + lane, e = first + i;
            const bool valid = i < m;
            const u32 u = valid ? __ldcs(head + e) : 0u;
            const u32 at = valid ? __ldcs(pos + i) : 0u;
            const u64 to = valid && u < n ? in_start[u] : 0;
            u64 v = n;
            for (;;) {
                u32 idx = 0;  // the window's lists that end at or before e
#pragma unroll
                for (int s = 16; s > 0; s >>= 1)
                    if (__shfl_sync(0xFFFFFFFFu, end, idx + s - 1) <= e) idx += s;
                if (__shfl_sync(0xFFFFFFFFu, end, idx) <= e) ++idx;
                if (v == n && valid && idx < 32) v = vb + idx;
                const u32 open = __ballot_sync(0xFFFFFFFFu, v == n && valid);
                if (!open) break;
                // the first entry past the window has a list of its own further on
                const int f = __ffs(open) - 1;
                vb = owner_of(fo, n, __shfl_sync(0xFFFFFFFFu, e, f), lane);
                end = fo[vb + 1 + lane < n ? vb + 1 + lane : n];
                if ((int)lane == f) v = vb;
            }
            if (!valid || v >= n) continue;
            const u64 a = fo[v];
            if (e >= a && e < fo[v + 1]) hs[fs[v] + (e - a)] = u;
            if (u < n) hs[to + at] = (u32)v;
        }
    }
}

// Contraction, pass 1: per local vertex the number of ghosts in its out-list (the edges that
// survive), whether it survives, and the longest surviving list.
__global__ void k_contract_count(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n, u64 n_local,
                                 u64* __restrict__ cnt, u64* __restrict__ keep, unsigned long long* maxlen) {
    const int lane = threadIdx.x & 31;
    const u64 warp = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
    for (u64 v = warp; v < n_local; v += nwarps) {
        u64 c = 0;
        for (u64 e = fo[v] + lane; e < fo[v + 1]; e += 32) {
            const u32 u = head[e];
            c += (u >= n_local && u < n) ? 1u : 0u;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
        if (lane == 0) {
            cnt[v] = c;
            keep[v] = c ? 1ull : 0ull;
            if (c) atomicMax(maxlen, c);
        }
    }
}

// Contraction, pass 2: the surviving vertices renumbered in order, their ghost lists copied
// in list order, and one descriptor per surviving list (for the id sort).
__global__ void k_contract_scatter(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n, u64 n_local,
                                   const u64* __restrict__ cnt_scan, const u64* __restrict__ keep_scan,
                                   u32* __restrict__ kept, u64* __restrict__ out_fo, u32* __restrict__ out_head,
                                   Desc<u64>* __restrict__ desc) {
    const int lane = threadIdx.x & 31;
    const u64 warp = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
    if (warp == 0 && lane == 0) out_fo[keep_scan[n_local]] = cnt_scan[n_local];
    for (u64 v = warp; v < n_local; v += nwarps) {
        const u64 base = cnt_scan[v], c = cnt_scan[v + 1] - base;
        if (c == 0) continue;
        const u64 k = keep_scan[v];
        if (lane == 0) {
            kept[k] = (u32)v;
            out_fo[k] = base;
            Desc<u64> d;
            d.start = base;
            d.d = (u32)c;
            d.pad = 0;
            desc[k] = d;
        }
        u64 at = base;
        for (u64 e0 = fo[v]; e0 < fo[v + 1]; e0 += 32) {
            const u64 e = e0 + lane;
            const u32 u = e < fo[v + 1] ? head[e] : 0xFFFFFFFFu;
            const bool g = u >= n_local && u < n;
            const u32 ball = __ballot_sync(0xFFFFFFFFu, g);
            if (g) out_head[at + __popc(ball & ((1u << lane) - 1))] = u;
            at += __popc(ball);
        }
    }
}

// Per-vertex cost of the reference's load-balancing cost functions (cost_function.h:287-345),
// one warp per vertex; deg = undirected degree, dplus = out-degree in (degree, id) order.
__global__ void k_vertex_cost(const u64* __restrict__ fo, const u32* __restrict__ head, u64 n,
                              const u32* __restrict__ deg, const u32* __restrict__ dplus, int fn, u64* __restrict__ cost) {
    const int lane = threadIdx.x & 31;
    const u64 warp = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
    for (u64 v = warp; v < n; v += nwarps) {
        const u64 dv = deg[v], ov = dplus[v];
        u64 c = 0;
        if (fn == KTRI_COST_DPD || fn == KTRI_COST_IDPD) {
            const bool higher = fn == KTRI_COST_DPD;
            for (u64 e = fo[v] + lane; e < fo[v + 1]; e += 32) {
                const u32 u = head[e];
                if (u >= n) continue;
                const bool above = key_less(dv, v, deg[u], u);  // (deg u, u) > (deg v, v)
                if (above == higher) c += ov + dplus[u];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
        } else {
            c = fn == KTRI_COST_N ? 1 : fn == KTRI_COST_D ? dv : fn == KTRI_COST_DH ? ov : fn == KTRI_COST_DDH ? dv * ov : ov * ov;
        }
        if (lane == 0) cost[v] = c;
    }
}

// boundaries[i] = first vertex whose cost prefix reaches i / parts of the total (prefix holds
// the exclusive prefix sums, prefix[n] = total); boundaries[parts] = n.
__global__ void k_cost_boundaries(const u64* __restrict__ prefix, u64 n, u32 parts, u64* __restrict__ boundaries) {
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > parts) return;
    if (i == parts) {
        boundaries[i] = n;
        return;
    }
    const u64 total = prefix[n];
    const u64 target = (u64)(((unsigned __int128)total * i + parts - 1) / parts);
    u64 lo = 0, hi = n;  // smallest v with prefix[v] >= target
    while (lo < hi) {
        const u64 mid = (lo + hi) >> 1;
        if (prefix[mid] >= target) hi = mid;
        else lo = mid + 1;
    }
    boundaries[i] = lo;
}

}  // namespace

u64 dag_scan_chunks(u64 n) { return (n + 1 + SCAN_CHUNK - 1) / SCAN_CHUNK; }

void launch_cost_partition(const u64* fo, const u32* head, u64 n, const u32* deg, const u32* dplus, int fn, u32 parts,
                           u64* cost, u64* sums, u64* boundaries, int num_sms, cudaStream_t st) {
    if (n == 0) return;
    u64 blocks = (n * 32 + 255) / 256;
    const u64 cap = (u64)num_sms * 16;
    if (blocks > cap) blocks = cap;
    cudaMemsetAsync(cost + n, 0, sizeof(u64), st);
    k_vertex_cost<<<(unsigned)blocks, 256, 0, st>>>(fo, head, n, deg, dplus, fn, cost);
    launch_scan_u64(cost, n + 1, sums, st);
    k_cost_boundaries<<<(unsigned)((parts + 1 + 255) / 256), 256, 0, st>>>(cost, n, parts, boundaries);
}

void launch_scan_u64(u64* x, u64 len, u64* sums, cudaStream_t st) {
    if (len == 0) return;
    const u64 nch = (len + SCAN_CHUNK - 1) / SCAN_CHUNK;
    k_scan_chunks<false><<<(unsigned)nch, SCAN_BLOCK, 0, st>>>(x, len, sums, nullptr, nullptr, 0, 0);
    k_scan_sums<<<1, 1024, 0, st>>>(sums, nch);
    k_scan_add<false><<<(unsigned)nch, SCAN_BLOCK, 0, st>>>(x, len, sums, nullptr, nullptr, 0);
}

void launch_contract(const u64* fo, const u32* head, u64 n, u64 n_local, u64* cnt, u64* keep, u64* sums,
                     unsigned long long* maxlen, u32* kept, u64* out_fo, u32* out_head, void* desc, int num_sms,
                     cudaStream_t st) {
    if (n_local == 0) return;
    u64 blocks = (n_local * 32 + 255) / 256;
    const u64 cap = (u64)num_sms * 16;
    if (blocks > cap) blocks = cap;
    cudaMemsetAsync(cnt + n_local, 0, sizeof(u64), st);
    cudaMemsetAsync(keep + n_local, 0, sizeof(u64), st);
    cudaMemsetAsync(maxlen, 0, sizeof(u64), st);
    k_contract_count<<<(unsigned)blocks, 256, 0, st>>>(fo, head, n, n_local, cnt, keep, maxlen);
    launch_scan_u64(cnt, n_local + 1, sums, st);
    launch_scan_u64(keep, n_local + 1, sums, st);
    k_contract_scatter<<<(unsigned)blocks, 256, 0, st>>>(fo, head, n, n_local, cnt, keep, kept, out_fo, out_head,
                                                       reinterpret_cast<Desc<u64>*>(desc));
}

void launch_dag_symmetrize(const u64* fo, const u32* head, u64 n, u64 m, u64* fs, u32* hs, u32* in_deg,
                           u64* in_start, u32* pos, u64* sums, int num_sms, cudaStream_t st) {
    if (n == 0) return;
    u64 slots = 1;  // at most 2 n
    while (slots < n) slots <<= 1;
    const u32 mask = (u32)(slots - 1);
    cudaMemsetAsync(in_deg, 0, sizeof(u32) * slots, st);
    const u64 cap = (u64)num_sms * 8;
    auto grid = [&](u64 threads) { return (unsigned)std::max<u64>(1, std::min(cap, (threads + 255) / 256)); };
    if (m) k_dag_arrive<<<grid(m / 4), 256, 0, st>>>(fo, head, n, m, in_deg, mask, pos);
    const u64 nch = dag_scan_chunks(n);
    k_scan_chunks<true><<<(unsigned)nch, SCAN_BLOCK, 0, st>>>(fs, n + 1, sums, fo, in_deg, mask, m);
    k_scan_sums<<<1, 1024, 0, st>>>(sums, nch);
    k_scan_add<true><<<(unsigned)nch, SCAN_BLOCK, 0, st>>>(fs, n + 1, sums, fo, in_start, m);
    if (m) k_dag_scatter<<<grid((m + DAG_TILE - 1) / DAG_TILE * 32), 256, 0, st>>>(fo, head, n, m, fs, in_start, pos, hs);
}

}  // namespace ktri
