// Triangle counting by degree order, and of small graphs in one kernel.
//
// Reference: triangle_counting_masked_sandia (src/main.cpp:69-90), the sum of
// C<L> = L·L.  For a strict lower triangle L of an undirected graph that sum is
// the graph's triangle count whatever the order of the vertices, so the order
// is chosen here: descending degree, every edge (i, k) in the row of its
// higher rank i.  A triangle i > k > j is then found at its middle vertex k, by
// reading the columns of row i below k (i an in-edge of k) against the columns
// of row k: sum_i d_i^2 / 2 columns read over the rows' lengths d_i, where the
// product over the given order reads sum over the entries (i, k) of nnz(L_k)
// (RMAT-20: 1.2e9 against 8.1e9; RMAT-24: 4.3e10 against 4.0e11).
//
//  orientation  k_tri_col_counts, k_tri_vertex_keys, radix sort, k_tri_degrees:
//               the order; k_tri_scatter: every edge to its row; k_tri_row_sizes,
//               scans: the sizes; k_tri_rows, k_tri_long_rows: the rows, sorted, in
//               16-byte units; k_tri_entries: for every k the entries {where, how
//               much} of the rows i it is a column of
//  count        k_tri_count, a warp per (k, up to `chunk` in-edges)
//
// Flat graphs (little work per entry) and small ones keep the given order, in
// kernels without a plan: k_tri_walk and k_tri_small.
//
// RMAT-24 (260 M edges): 274 ms with the engine's product (spgemm.cu), 42 ms
// here: 23 ms count, 19 ms orientation; RMAT-20: 8.8 -> 1.9 ms; batches of 409
// uneven graphs: 34 to 45 -> 12 to 15 ms.
#include <cub/cub.cuh>

#include <algorithm>
#include "gk_device.cuh"
#include "gk_sched.cuh"
#include "gk_tri.cuh"

namespace gk {

constexpr uint32_t TRI_NONE = 0xFFFFFFFFu;  // padding of the 32-bit columns

// ---------------------------------------------------------------------------
// degrees and the vertex order
// ---------------------------------------------------------------------------
// In-degree of every vertex.  A CTA counts the first column it sees of every slot of
// a table in shared memory, which the frequent columns mostly are, and adds those to
// memory at the end: their counters share cache lines, and an L2 line takes an
// atomic every 0.8 ns (RMAT-18 85 -> 59 us, RMAT-20 250 -> 144, RMAT-24 3080 -> 2370;
// 2^10 slots 153 and 2430; 2^12, which fewer CTAs an SM can have, 206 and 5510).  Its
// entries are consecutive and 2^15 at most, so that those of a batch are of few graphs
// (409 uneven graphs, entries dealt out by grid strides 1.13 ms, so 0.54).
constexpr int TRI_CACHE = 11;  // log2 slots
__global__ void __launch_bounds__(256) k_tri_col_counts(DevCsr L, int64_t ebase, int64_t vbase, uint32_t *cnt) {
    __shared__ uint32_t s_col[1 << TRI_CACHE], s_cnt[1 << TRI_CACHE];
    for (int t = threadIdx.x; t < 1 << TRI_CACHE; t += blockDim.x) {
        s_col[t] = TRI_NONE;
        s_cnt[t] = 0;
    }
    __syncthreads();
    const int64_t part = (L.nnz + gridDim.x - 1) / gridDim.x, end = min(part * (blockIdx.x + 1), L.nnz);
    for (int64_t p = part * blockIdx.x + threadIdx.x; p < end; p += blockDim.x) {
        const uint32_t c = static_cast<uint32_t>(L.col[ebase + p] - vbase);
        const uint32_t h = (c * 0x9E3779B1u) >> (32 - TRI_CACHE);
        uint32_t owner = *static_cast<volatile uint32_t *>(s_col + h);
        if (owner == TRI_NONE) {
            owner = atomicCAS(s_col + h, TRI_NONE, c);
            if (owner == TRI_NONE) owner = c;
        }
        if (owner == c) atomicAdd(s_cnt + h, 1u);
        else atomicAdd(cnt + c, 1u);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 1 << TRI_CACHE; t += blockDim.x)
        if (s_cnt[t]) atomicAdd(cnt + s_col[t], s_cnt[t]);
}

// Sort key of every vertex: its graph, then descending degree.
template <class KeyT>
__global__ void __launch_bounds__(256) k_tri_vertex_keys(DevCsr L, int64_t vbase, const int32_t *key, int dbits,
                                                         const uint32_t *cnt, KeyT *vkey, uint32_t *iota) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < L.m; r += stride) {
        const uint32_t d = cnt[r] + static_cast<uint32_t>(L.rp[r + 1] - L.rp[r]);
        KeyT k = (KeyT(1) << dbits) - 1 - d;
        if (key) k |= static_cast<KeyT>(key[vbase + r]) << dbits;
        vkey[r] = k;
        iota[r] = static_cast<uint32_t>(r);
    }
}

// nnz(L_k) of the columns k of TRI_SAMPLE entries, evenly spaced, added up.
__global__ void __launch_bounds__(256) k_tri_sample(DevCsr L, int64_t ebase, int64_t vbase, int n,
                                                    const CsrCheckOut *chk, unsigned long long *sum) {
    __shared__ unsigned long long red[8];
    if (chk && !chk->sound()) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long w = 0;
    if (t < n) {
        const int64_t k = L.col[ebase + L.nnz * t / n] - vbase;
        w = static_cast<unsigned long long>(L.rp[k + 1] - L.rp[k]);
    }
    w = block_sum(w, red);
    if (threadIdx.x == 0 && w) atomicAdd(sum, w);
}

// ---------------------------------------------------------------------------
// rows in rank order
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long tri_pack(uint32_t n, uint32_t hub, uint32_t high) {
    return n | (static_cast<unsigned long long>(hub) << 16) | (static_cast<unsigned long long>(high) << 32);
}

struct TriBase {  // column origin of a row: its graph's first rank
    const int32_t *key;
    const int64_t *gvbase;
    int64_t vbase;
    __device__ __forceinline__ uint32_t of(uint32_t rank) const {
        return key ? static_cast<uint32_t>(__ldg(gvbase + __ldg(key + vbase + rank)) - vbase) : 0u;
    }
};

// Degree of every rank, whose sum over the ranks below is where its row starts: a
// row has room for all of the vertex's edges, so that the edges can be moved
// without counting the rows first (a pass of its own over all edges, 2.8 ms of
// RMAT-24's 48).
__global__ void __launch_bounds__(256) k_tri_degrees(int64_t m, const uint32_t *perm, const uint32_t *cnt, DevCsr L,
                                                     uint32_t *rank, uint32_t *deg) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += stride) {
        const uint32_t v = perm[r];
        rank[v] = static_cast<uint32_t>(r);
        deg[r] = cnt[v] + static_cast<uint32_t>(L.rp[v + 1] - L.rp[v]);
    }
}

// Every edge to the row of its higher rank, its lower rank to the next free
// slot there (in any order; k_tri_rows sorts the rows).  A row's cursor counts its
// columns, the hub columns among them and the high ones, 16 bits each (the d
// columns of a row have at least its degree each, so d^2 <= 2 E < 2^32).  The
// entries of a row of L that stay in it are counted once per warp step, those
// that move one by one.
__global__ void __launch_bounds__(256) k_tri_scatter(DevCsr L, int64_t ebase, int64_t vbase, int walk, TriBase tb,
                                                     uint32_t hub_lim, uint32_t low_lim,
                                                     const uint32_t *__restrict__ rank,
                                                     const uint32_t *__restrict__ start, unsigned long long *cur,
                                                     uint32_t *cols) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int64_t p0 = ebase + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * walk;
    const int64_t p1 = min(p0 + walk, ebase + L.nnz);
    if (p0 >= p1) return;
    walk_entries(L.rp, L.m, p0, p1, lane, [&](int64_t p, int64_t row, int leader, unsigned peers, bool on) {
        uint32_t ri = 0, rj = 0;
        if (on) {
            ri = __ldg(rank + row);
            rj = __ldg(rank + (__ldg(L.col + p) - vbase));
        }
        const bool stays = on && rj < ri;
        const uint32_t hi = stays ? ri : rj, lo = stays ? rj : ri;
        const uint32_t x = on ? lo - tb.of(ri) : hub_lim;
        const unsigned sm = __ballot_sync(FULL, stays) & peers;
        const unsigned am = __ballot_sync(FULL, x < hub_lim) & sm;
        const unsigned hm = __ballot_sync(FULL, x >= low_lim) & sm;
        const uint32_t to = on ? __ldg(start + hi) : 0;
        uint32_t at = 0;
        if (on && lane == leader && sm)
            at = static_cast<uint32_t>(atomicAdd(cur + ri, tri_pack(__popc(sm), __popc(am), __popc(hm))) & 0xFFFFu);
        at = __shfl_sync(FULL, at, leader) + __popc(sm & ((1u << lane) - 1u));
        if (on) {
            if (!stays)
                at = static_cast<uint32_t>(atomicAdd(cur + rj, tri_pack(1, x < hub_lim, x >= low_lim)) & 0xFFFFu);
            cols[to + at] = lo;
        }
    });
}

// Bands (k_tri_items) of the in-edge lists of rows with at least TRI_BAND_MIN
// entries, in graphs of TRI_BAND_EDGES edges: where the rows' storage (two to eight
// bytes an edge) is several times L2, a list entry's row has left it before the
// next k names it.  RMAT-24 (260M edges) read 57 of the 78 GB it asks for from
// DRAM: 24.7 ms, in 16 or 32 bands 23.0, in 64 23.4.  RMAT-22 (64M) reads 4.6 of
// 14.4 GB and gains nothing (3.31 against 3.29).
constexpr uint32_t TRI_BANDS = 32, TRI_BAND_MIN = 4096;
constexpr int64_t TRI_BAND_EDGES = int64_t(1) << 27;
__device__ __forceinline__ uint32_t tri_band(uint32_t in) { return (in + TRI_BANDS - 1) / TRI_BANDS; }

// Columns, units, in-edge entries and work items of every row.
__global__ void __launch_bounds__(256) k_tri_row_sizes(int64_t m, const uint32_t *deg, uint32_t chunk,
                                                       const unsigned long long *counts, uint32_t *len,
                                                       uint2 *shape, uint32_t *nunits, uint32_t *nin, uint32_t *nitems,
                                                       uint32_t *banded) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= m; r += stride) {
        uint32_t n = 0, u = 0, in = 0, it = 0, bd = 0;
        if (r < m) {
            const unsigned long long c = counts[r];
            n = static_cast<uint32_t>(c & 0xFFFFu);
            const uint32_t a = static_cast<uint32_t>((c >> 16) & 0xFFFFu), h = static_cast<uint32_t>(c >> 32);
            const TriShape sh{a, n - h, n};
            shape[r] = make_uint2(a | ((n - h) << 16), n);
            u = sh.units();
            in = deg[r] - n;
            bd = banded && n && in >= TRI_BAND_MIN;
            it = n && !bd ? (in + chunk - 1) / chunk : 0;
        }
        len[r] = n;
        nunits[r] = u;
        nin[r] = in;
        nitems[r] = it;
        if (banded) banded[r] = bd;
    }
}

struct TriRowArgs {
    int64_t m, E;
    const uint32_t *lrp;    // [m + 1] columns of the rows before
    const uint32_t *start;  // first column of every row in cols
    const uint32_t *cols;   // the rows' columns in any order
    TriBase tb;
    uint32_t low_lim;      // columns below it are low; also the padding of the low units
    const uint2 *shape;    // {hubs | lows << 16, n} of every row
    const uint32_t *vstart;
    uint4 *units;
    uint32_t *ucur;        // next free in-edge entry of every row
    uint2 *uent;
    uint32_t *longrows;    // rows beyond the warp sort
    unsigned int *nlong;
};

__device__ __forceinline__ TriShape tri_shape(const TriRowArgs &a, uint32_t i) {
    const uint2 w = __ldg(a.shape + i);
    return TriShape{w.x & 0xFFFFu, w.x >> 16, w.y};
}

// The q-th column of a row (x) to its place.
__device__ __forceinline__ void tri_put(const TriRowArgs &a, uint32_t v0, const TriShape &sh, uint32_t q, uint32_t x) {
    if (q < sh.lows) {
        const bool hub = q < sh.hubs;
        uint16_t *w = reinterpret_cast<uint16_t *>(a.units + v0 + (hub ? 0 : sh.hub_units() + sh.map_units()));
        const uint32_t h = hub ? q : q - sh.hubs, n = hub ? sh.hubs : sh.lows - sh.hubs;
        w[h] = static_cast<uint16_t>(x ^ 31u);
        if (h == n - 1)
            for (uint32_t z = n; z & 7u; ++z) w[z] = static_cast<uint16_t>(a.low_lim ^ 31u);
    } else {
        uint32_t *w =
            reinterpret_cast<uint32_t *>(a.units + v0 + sh.hub_units() + sh.map_units() + sh.mid_units());
        const uint32_t h = q - sh.lows, n = sh.n - sh.lows;
        w[h] = x;
        if (h == n - 1)
            for (uint32_t z = n; z & 3u; ++z) w[z] = TRI_NONE;
    }
}

// The q-th column of a row from its place: one load, whichever class it is in.
__device__ __forceinline__ uint32_t tri_get(const TriRowArgs &a, uint32_t v0, const TriShape &sh, uint32_t q) {
    const uint32_t mid = 16 * (sh.hub_units() + sh.map_units());
    const uint32_t b = q < sh.hubs   ? 2 * q
                       : q < sh.lows ? mid + 2 * (q - sh.hubs)
                                     : mid + 16 * sh.mid_units() + 4 * (q - sh.lows);
    const uint32_t w = reinterpret_cast<const uint32_t *>(a.units + v0)[b >> 2];
    return q < sh.lows ? ((w >> (8 * (b & 2u))) & 0xFFFFu) ^ 31u : w;
}

// Sorts the K consecutive values of every lane (lane-major) of the warp
// ascending: a bitonic network, its distances below K inside the lane.
template <int K>
__device__ __forceinline__ void warp_sort(uint32_t (&x)[K], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * K; size <<= 1) {
#pragma unroll
        for (int d = size >> 1; d > 0; d >>= 1) {
            if (d >= K) {
                const int ld = d / K;
                const bool upper = lane & ld;
                const bool asc = size >= 32 * K || !((lane * K) & size);
#pragma unroll
                for (int t = 0; t < K; ++t) {
                    const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x[t], ld);
                    x[t] = (upper == asc) ? max(x[t], y) : min(x[t], y);
                }
            } else {
#pragma unroll
                for (int t = 0; t < K; ++t)
                    if (!(t & d)) {
                        const bool asc = size >= 32 * K || !((lane * K + t) & size);
                        const uint32_t a = min(x[t], x[t | d]), b = max(x[t], x[t | d]);
                        x[t] = asc ? a : b;
                        x[t | d] = asc ? b : a;
                    }
            }
        }
    }
}

template <int K>
__device__ __forceinline__ void tri_sort_row(const TriRowArgs &a, uint32_t i, uint32_t n, uint32_t base, int lane,
                                             uint32_t *map) {
    const uint32_t r0 = __ldg(a.start + i);
    uint32_t x[K];
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const uint32_t q = t * 32 + lane;
        x[t] = q < n ? __ldg(a.cols + r0 + q) - base : TRI_NONE;
    }
    warp_sort<K>(x, lane);
    const TriShape sh = tri_shape(a, i);
    const uint32_t v0 = __ldg(a.vstart + i);
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const uint32_t q = lane * K + t;
        if (q < n) tri_put(a, v0, sh, q, x[t]);
    }
    if (sh.map_units()) {  // the hub columns' bitmap, built in the warp's shared-memory words
        if (lane < TRI_MAP) reinterpret_cast<uint4 *>(map)[lane] = make_uint4(0, 0, 0, 0);
        __syncwarp();
#pragma unroll
        for (int t = 0; t < K; ++t)
            if (x[t] < TRI_HUB) atomicOr(map + (x[t] >> 5), 1u << (x[t] & 31));
        __syncwarp();
        if (lane < TRI_MAP) a.units[v0 + sh.hub_units() + lane] = reinterpret_cast<const uint4 *>(map)[lane];
        __syncwarp();
    }
}

// Sorts the rows of more than TRI_SHORT_ROW columns, a warp each, and writes
// their columns' units.
constexpr uint32_t TRI_WARP_ROW = 1024;
constexpr uint32_t TRI_SHORT_ROW = 32;
__global__ void __launch_bounds__(256, 4) k_tri_rows(TriRowArgs a) {
    __shared__ __align__(16) uint32_t s_map[8][TRI_HUB / 32];
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    // 32 rows per warp step, `warps` apart (neighbours in rank have like
    // lengths): their lengths, then the longer ones one by one
    for (int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < a.m; b += 32 * warps) {
        const int64_t mine = b + lane * warps;
        const uint32_t len = mine < a.m ? __ldg(a.shape + mine).y : 0;
        if (len > TRI_WARP_ROW) a.longrows[atomicAdd(a.nlong, 1u)] = static_cast<uint32_t>(mine);
        for (unsigned todo = __ballot_sync(0xFFFFFFFFu, len > TRI_SHORT_ROW && len <= TRI_WARP_ROW); todo;
             todo &= todo - 1) {
            const int j = __ffs(todo) - 1;
            const uint32_t ii = static_cast<uint32_t>(b + j * warps);
            const uint32_t n = __shfl_sync(0xFFFFFFFFu, len, j), base = a.tb.of(ii);
            uint32_t *map = s_map[threadIdx.x >> 5];
            if (n <= 64) tri_sort_row<2>(a, ii, n, base, lane, map);
            else if (n <= 128) tri_sort_row<4>(a, ii, n, base, lane, map);
            else if (n <= 256) tri_sort_row<8>(a, ii, n, base, lane, map);
            else if (n <= 512) tri_sort_row<16>(a, ii, n, base, lane, map);
            else tri_sort_row<32>(a, ii, n, base, lane, map);
        }
    }
}

// The column at position p of the rows laid end to end: unsorted in a short row,
// sorted in a longer one.
__device__ __forceinline__ uint32_t tri_column(const TriRowArgs &a, uint32_t i, uint32_t p) {
    const uint32_t q = p - __ldg(a.lrp + i);
    const TriShape sh = tri_shape(a, i);
    return sh.n <= TRI_SHORT_ROW ? __ldg(a.cols + __ldg(a.start + i) + q) - a.tb.of(i)
                                 : tri_get(a, __ldg(a.vstart + i), sh, q);
}

// The entry of every edge (row i, column k) at the next free slot of k's list:
// what of row i lies below k.  Where that includes a mapped row's hub columns
// (or many of them), the entry starts at the bitmap.  A short row's columns
// are still in any order: a column's place is the number of smaller ones (the
// row's reads hit L1), and its unit is written here.  With PLACE the entry is the
// edge's row and position instead.
// Bound by the cursors' atomics: nearly every row holds the first few ranks, whose
// cursors share a few cache lines, and an L2 line takes an atomic every 0.8 ns.  With
// HOT a CTA walks its 4,096 entries twice: it counts the columns below TRI_HOT in
// shared memory, takes its part of each of their lists at once, then places all
// (RMAT-18 0.26 -> 0.12 ms, RMAT-20 0.81 -> 0.38, RMAT-22 2.04 -> 1.42; 512 hot
// columns 0.41 on RMAT-20).
// (As a part of k_tri_rows, whose registers allow half the warps: RMAT-24 12.8 ms
// against 3.1 and 5.7 for the two.)
constexpr uint32_t TRI_HOT = 2048;
constexpr int TRI_WALK = 512;  // most entries a warp walks with HOT
template <bool PLACE, bool HOT>
__global__ void __launch_bounds__(256) k_tri_entries(TriRowArgs a, int walk) {
    __shared__ uint32_t s_x[HOT ? 8 : 1][HOT ? TRI_WALK : 1], s_hot[HOT ? TRI_HOT : 1];
    const int lane = threadIdx.x & 31;
    uint32_t *xs = s_x[HOT ? threadIdx.x >> 5 : 0];
    const int64_t p0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * walk;
    const int64_t p1 = min(p0 + walk, a.E);
    if (HOT) {
        for (uint32_t t = threadIdx.x; t < TRI_HOT; t += blockDim.x) s_hot[t] = 0;
        __syncthreads();
        if (p0 < p1)
            walk_entries(a.lrp, a.m, p0, p1, lane, [&](int64_t p, int64_t row, int, unsigned, bool on) {
                if (!on) return;
                uint32_t x = tri_column(a, static_cast<uint32_t>(row), static_cast<uint32_t>(p));
                if (x < TRI_HOT) x = 0x80000000u | (x << 16) | atomicAdd(s_hot + x, 1u);
                xs[p - p0] = x;
            });
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < TRI_HOT; t += blockDim.x)
            if (s_hot[t]) s_hot[t] = atomicAdd(a.ucur + t, s_hot[t]);
        __syncthreads();
    }
    if (p0 >= p1) return;
    walk_entries(a.lrp, a.m, p0, p1, lane, [&](int64_t p, int64_t row, int, unsigned, bool on) {
        if (!on) return;
        const uint32_t i = static_cast<uint32_t>(row), base = HOT ? 0 : a.tb.of(i);
        const TriShape sh = tri_shape(a, i);
        uint32_t q = static_cast<uint32_t>(p) - __ldg(a.lrp + i), v0 = __ldg(a.vstart + i);
        uint32_t x = HOT ? xs[p - p0] : tri_column(a, i, static_cast<uint32_t>(p)), part = TRI_NONE;
        if (HOT && x >> 31) {
            part = x & 0xFFFFu;
            x = (x >> 16) & 0x7FFFu;
        }
        if (sh.n <= TRI_SHORT_ROW) {
            const uint32_t *c = a.cols + __ldg(a.start + i);
            q = 0;
            for (uint32_t t = 0; t < sh.n; ++t) q += __ldg(c + t) < base + x;
            tri_put(a, v0, sh, q, x);
        }
        const uint32_t slot = HOT && part != TRI_NONE ? s_hot[x] + part : atomicAdd(a.ucur + base + x, 1u);
        if (PLACE) {
            a.uent[slot] = make_uint2(i, q);
            return;
        }
        uint32_t nlist, nhigh = 0, map = 0;
        if (q <= sh.hubs) {
            nlist = (q + 7) / 8;
            if (nlist >= TRI_MAP_MIN) {
                map = 1;
                v0 += sh.hub_units();
                nlist = 0;
            }
        } else {
            map = sh.map_units() ? 1 : 0;
            if (map) v0 += sh.hub_units();
            nlist = (map ? 0 : sh.hub_units()) + (min(q, sh.lows) - sh.hubs + 7) / 8;
            if (q > sh.lows) nhigh = (q - sh.lows + 3) / 4;
        }
        a.uent[slot] = make_uint2(v0, nlist | (map << 14) | (nhigh << 15));
    });
}

// The rows beyond the warp sort, a CTA each: windows of 2^17 columns in
// ascending order, a bitmap of the window's columns, whose set bits in order
// are the sorted columns.
constexpr int TRI_WIN = 17;
__global__ void __launch_bounds__(512) k_tri_long_rows(TriRowArgs a) {
    constexpr int NW = 1 << (TRI_WIN - 5), NT = 512, PER = NW / NT;
    __shared__ __align__(16) uint32_t bits[NW];
    __shared__ uint32_t s_scan[NT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (unsigned int t = blockIdx.x; t < *a.nlong; t += gridDim.x) {
        const uint32_t i = a.longrows[t];
        const uint32_t r0 = a.start[i], base = a.tb.of(i);
        const TriShape sh = tri_shape(a, i);
        const uint32_t v0 = a.vstart[i], n = sh.n;
        uint32_t done = 0;
        for (uint32_t w0 = 0; done < n; w0 += 1u << TRI_WIN) {
            for (int z = threadIdx.x; z < NW; z += NT) bits[z] = 0;
            __syncthreads();
            for (uint32_t q = threadIdx.x; q < n; q += NT) {
                const uint32_t x = a.cols[r0 + q] - base - w0;
                if (x < (1u << TRI_WIN)) atomicOr(bits + (x >> 5), 1u << (x & 31));
            }
            __syncthreads();
            uint32_t mine = 0;
#pragma unroll
            for (int z = 0; z < PER; ++z) mine += __popc(bits[threadIdx.x * PER + z]);
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) s_scan[warp] = incl;
            __syncthreads();
            uint32_t before = 0, all = 0;
            for (int z = 0; z < NT / 32; ++z) {
                if (z < warp) before += s_scan[z];
                all += s_scan[z];
            }
            if (w0 == 0 && sh.map_units() && threadIdx.x < TRI_MAP)
                a.units[v0 + sh.hub_units() + threadIdx.x] = reinterpret_cast<const uint4 *>(bits)[threadIdx.x];
            uint32_t q = done + before + incl - mine;
            for (int z = 0; z < PER; ++z)
                for (uint32_t b = bits[threadIdx.x * PER + z]; b; b &= b - 1, ++q) {
                    const uint32_t x = w0 + 32 * (threadIdx.x * PER + z) + (__ffs(b) - 1);
                    tri_put(a, v0, sh, q, x);
                }
            done += all;
            __syncthreads();
        }
    }
}

// Work items {k, first entry}.  With bands (bpre: their rows' scan), the items of
// the rows with many in-edges come first, band by band: the lists are in about
// the order of the rows they name, so the items of one band read about the same
// rows, whichever their k.
__global__ void __launch_bounds__(256) k_tri_items(int64_t m, const uint32_t *ipre, const uint32_t *bpre,
                                                   const uint32_t *urp, uint32_t chunk, uint2 *items) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const uint32_t nb = bpre ? bpre[m] : 0;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m; r += stride) {
        const uint32_t u0 = urp[r];
        if (bpre && bpre[r + 1] != bpre[r]) {
            const uint32_t step = tri_band(urp[r + 1] - u0);
            for (uint32_t b = 0; b < TRI_BANDS; ++b)
                items[b * nb + bpre[r]] = make_uint2(static_cast<uint32_t>(r), min(u0 + b * step, urp[r + 1]));
        }
        for (uint32_t t = ipre[r], c = 0; t < ipre[r + 1]; ++t, ++c)
            items[TRI_BANDS * nb + t] = make_uint2(static_cast<uint32_t>(r), u0 + c * chunk);
    }
}

// ---------------------------------------------------------------------------
// count
// ---------------------------------------------------------------------------
struct TriArgs {
    TriGraph g;
    const uint2 *items;
    const uint32_t *nitems;  // in chunks, and in bands (null: none)
    const uint32_t *nbanded;
    unsigned int *fetch;
    uint32_t chunk;
    unsigned long long *sums;
    const int32_t *key;  // with the group's first vertex already added
};

constexpr int TRI_FB = 13;  // log2 bits of the high columns' filter
__device__ __forceinline__ uint32_t tri_hash(uint32_t x) { return (x * 0x9E3779B1u) >> (32 - TRI_FB); }

// Bits of the two 16-bit columns of w in the bitmap, added to cnt.  The columns
// are stored with their low five bits inverted, so that a left shift by the
// stored value brings the column's bit to the top.
__device__ __forceinline__ void tri_test2(uint32_t w, const uint32_t *bm, uint32_t &cnt) {
    const uint32_t a = bm[(w >> 5) & 0x7FFu], b = bm[w >> 21];
    cnt += (a << (w & 31)) >> 31;
    cnt += (b << ((w >> 16) & 31)) >> 31;
}

__device__ __forceinline__ bool tri_in_high(const uint32_t *h, uint32_t n, uint32_t x) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t md = (lo + hi) >> 1;
        if (__ldg(h + md) < x) lo = md + 1;
        else hi = md;
    }
    return lo < n && __ldg(h + lo) == x;
}

// The columns of `units` 16-bit units into the warp's bitmap.
template <uint32_t PAD>
__device__ __forceinline__ void tri_set_bits(uint32_t *bm, const uint4 *list, uint32_t units, int lane) {
    for (uint32_t u = lane; u < 4 * units; u += 32) {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(list) + u);
        const uint32_t a = (w & 0xFFFFu) ^ 31u, b = (w >> 16) ^ 31u;
        if (a != PAD) atomicOr(bm + (a >> 5), 1u << (a & 31));
        if (b != PAD) atomicOr(bm + (b >> 5), 1u << (b & 31));
    }
}

__device__ __forceinline__ uint32_t warp_incl_sum(uint32_t x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// First lane whose inclusive count exceeds u (31 when none does).
__device__ __forceinline__ int warp_find(uint32_t incl, uint32_t u) {
    int j = 0;
#pragma unroll
    for (int st = 16; st > 0; st >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, incl, j + st - 1) <= u) j += st;
    return j;
}

constexpr int TRI_WARPS = 4;  // warps per CTA, each with its own item and bitmap

template <int LB>
constexpr size_t tri_smem() {
    return TRI_WARPS * ((size_t(1) << LB) / 8 + (size_t(1) << TRI_FB) / 8);
}

// A warp per item: row k's columns as a bitmap of its own in shared memory (low
// ones), a filter (high ones) and four words per lane (hubs); then its in-edges
// 32 at a time.  What row i holds below k needs no cut at k: k's bitmap is empty
// from k on, so whole units are read.
//  * hub bitmaps: two entries per step, half a warp each, AND and popcount with
//    the registers (2,048 columns for 256 bytes and 8 operations a lane: from 6
//    units of hub columns on that is the cheaper reading);
//  * lists: the units of the 32 entries are packed onto the lanes (a scan, a
//    five-step search), eight bitmap tests each.
// Bound by the L1 data pipe (bitmap loads' bank conflicts, shuffles and 16-byte
// loads: 74% of its wavefronts on RMAT-22, ALU 61%, DRAM 1.3 TB/s).  A CTA of two
// warps per item instead spent its time in barriers (RMAT-20: 0.73 against
// 0.57 ms).  48 registers, ten CTAs an SM; the 2^16-bit bitmaps leave room for five
// CTAs only, whose lanes then keep four list units in flight instead of two (RMAT-24
// 26.1 -> 24.7 ms; eight bitmap loads 25.0).
template <int LB, bool KEYED>
__global__ void __launch_bounds__(32 * TRI_WARPS, LB == 16 ? 5 : 10) k_tri_count(TriArgs p) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr int UM = 4, UL = LB == 16 ? 4 : 2;  // loads in flight per lane: bitmaps, list units
    constexpr int BW = 1 << (LB - 5), FW = 1 << (TRI_FB - 5);
    constexpr uint32_t PAD = (1u << LB) - 1;
    extern __shared__ uint4 smem4[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *bm = reinterpret_cast<uint32_t *>(smem4) + warp * (BW + FW);
    uint32_t *flt = bm + BW;
    for (int i = lane; i < BW + FW; i += 32) bm[i] = 0;
    __syncwarp();
    const uint32_t banded = p.nbanded ? *p.nbanded * TRI_BANDS : 0, nitems = *p.nitems + banded;
    unsigned long long local = 0;
    uint32_t next = 0;
    if (lane == 0) next = atomicAdd(p.fetch, 1u);
    for (;;) {
        const uint32_t it = __shfl_sync(FULL, next, 0);
        if (it >= nitems) break;
        if (lane == 0) next = atomicAdd(p.fetch, 1u);  // the next item's number arrives behind this one's work
        const uint2 im = __ldg(p.items + it);
        const uint32_t k = im.x, u0 = im.y;
        const uint32_t uend = __ldg(p.g.urp + k + 1);
        const uint32_t u1 = min(u0 + (it < banded ? tri_band(uend - __ldg(p.g.urp + k)) : p.chunk), uend);
        const uint2 shw = __ldg(p.g.shape + k);
        const TriShape sh{shw.x & 0xFFFFu, shw.x >> 16, shw.y};
        const uint4 *row = p.g.units + __ldg(p.g.vstart + k);
        const uint4 *mid = row + sh.hub_units() + sh.map_units();
        const uint32_t *hcol = reinterpret_cast<const uint32_t *>(mid + sh.mid_units());
        const uint32_t nh = sh.n - sh.lows;
        uint2 e = make_uint2(0, 0);
        if (u0 + lane < u1) e = __ldg(p.g.uent + u0 + lane);
        if (sh.map_units()) {
            if (lane < TRI_MAP) reinterpret_cast<uint4 *>(bm)[lane] = __ldg(row + sh.hub_units() + lane);
            __syncwarp();
        } else {
            tri_set_bits<PAD>(bm, row, sh.hub_units(), lane);
        }
        tri_set_bits<PAD>(bm, mid, sh.mid_units(), lane);
        for (uint32_t u = lane; u < nh; u += 32) {
            const uint32_t h = tri_hash(__ldg(hcol + u));
            atomicOr(flt + (h >> 5), 1u << (h & 31));
        }
        __syncwarp();
        uint32_t cnt = 0;
        const uint4 km = reinterpret_cast<const uint4 *>(bm)[lane & 15];  // k's hub columns
        for (uint32_t eb = u0; eb < u1; eb += 32) {
            uint2 en = make_uint2(0, 0);
            if (eb + 32 + lane < u1) en = __ldg(p.g.uent + eb + 32 + lane);
            // the bitmaps: two at a time, half a warp each, four loads in flight per lane
            for (unsigned mm = __ballot_sync(FULL, (e.y >> 14) & 1u); mm;) {
                uint4 v[UM];
#pragma unroll
                for (int h = 0; h < UM; ++h) {
                    const int a = __ffs(mm) - 1;
                    mm &= mm - 1;
                    const int b = __ffs(mm) - 1;
                    mm &= mm - 1;
                    const int j = lane < 16 ? a : b;
                    const uint32_t o = __shfl_sync(FULL, e.x, j & 31);
                    v[h] = make_uint4(0, 0, 0, 0);
                    if (j >= 0) v[h] = __ldg(p.g.units + o + (lane & 15));
                }
#pragma unroll
                for (int h = 0; h < UM; ++h)
                    cnt += __popc(v[h].x & km.x) + __popc(v[h].y & km.y) + __popc(v[h].z & km.z) +
                           __popc(v[h].w & km.w);
            }
            const uint32_t el = e.y & 0x3FFFu, eh = e.y >> 15;
            const uint32_t start = e.x + ((e.y >> 14) & 1u ? TRI_MAP : 0u);
            uint32_t incl = warp_incl_sum(el, lane);
            const uint32_t total = __shfl_sync(FULL, incl, 31);
            const uint32_t off = start - (incl - el);  // unit address minus position in the batch
            for (uint32_t b = 0; b < total; b += 32 * UL) {
                uint4 v[UL];
                bool ok[UL];
#pragma unroll
                for (int h = 0; h < UL; ++h) {
                    const uint32_t u = b + 32 * h + lane;
                    const uint32_t o = __shfl_sync(FULL, off, warp_find(incl, u) & 31);
                    ok[h] = u < total;
                    if (ok[h]) v[h] = __ldg(p.g.units + (o + u));
                }
#pragma unroll
                for (int h = 0; h < UL; ++h)
                    if (ok[h]) {
                        tri_test2(v[h].x, bm, cnt);
                        tri_test2(v[h].y, bm, cnt);
                        tri_test2(v[h].z, bm, cnt);
                        tri_test2(v[h].w, bm, cnt);
                    }
            }
            // high columns (a row's lie behind all of its low ones)
            if (nh && __any_sync(FULL, eh)) {
                incl = warp_incl_sum(eh, lane);
                const uint32_t htot = __shfl_sync(FULL, incl, 31);
                const uint32_t hoff = start + el - (incl - eh);
                for (uint32_t b = 0; b < htot; b += 32) {
                    const uint32_t u = b + lane;
                    const uint32_t o = __shfl_sync(FULL, hoff, warp_find(incl, u) & 31);
                    if (u < htot) {
                        const uint4 v = __ldg(p.g.units + (o + u));
                        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t h = tri_hash(x[c]);
                            if ((flt[h >> 5] >> (h & 31)) & 1u) cnt += tri_in_high(hcol, nh, x[c]);
                        }
                    }
                }
            }
            e = en;
        }
        if (KEYED) {
            const unsigned long long tot = __reduce_add_sync(FULL, cnt);
            if (lane == 0 && tot) atomicAdd(p.sums + p.key[k], tot);
        } else {
            local += cnt;
        }
        __syncwarp();
        if (sh.hubs && lane < TRI_MAP) reinterpret_cast<uint4 *>(bm)[lane] = make_uint4(0, 0, 0, 0);
        for (uint32_t u = lane; u < 4 * sh.mid_units(); u += 32) {
            const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(mid) + u);
            bm[(w & PAD) >> 5] = 0;
            bm[(w >> 16) >> 5] = 0;
        }
        for (uint32_t u = lane; u < nh; u += 32) flt[tri_hash(__ldg(hcol + u)) >> 5] = 0;
        __syncwarp();
    }
    if (!KEYED) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(FULL, local, o);
        if (lane == 0 && local) atomicAdd(p.sums, local);
    }
}

// ---------------------------------------------------------------------------
// support of every edge
// ---------------------------------------------------------------------------
struct TriSupArgs {
    TriArgs t;
    int32_t *sup;
};

// The count's walk with a hit's three edges credited: (i, j) by an atomic on
// its number, which is where the hit was read; (i, k) once per entry and step with
// the lanes' hits; (k, j) in shared memory, at j's place in row k (the bitmap word's
// prefix count and the bits below j), written out once per item.  Bound by the
// atomics: two neighbouring columns' counters are one 64-bit add (a support lies
// below 2^31, so the lower one never carries), and the lanes of one entry add
// their hits first (RMAT-20, 424M triangles: an add per column and per unit 7.15 ms,
// so 3.75).  Two warps share an item, since its shared memory would leave half as
// many warps an SM otherwise; the sums in shared memory are 16-bit for the same
// reason (11 -> 9 KB an item, 3.75 -> 3.3 ms).
constexpr int TRI_SUP_ACC = 1024;  // places kept in shared memory; the others take an atomic per hit
constexpr int TRI_SUP_LB = 15;     // log2 bits of the bitmap
__global__ void __launch_bounds__(64) k_tri_support(TriSupArgs sa) {
    const TriArgs &p = sa.t;
    int32_t *sup = sa.sup;
    constexpr unsigned FULL = 0xFFFFFFFFu;
    constexpr int NT = 64, BW = 1 << (TRI_SUP_LB - 5), FW = 1 << (TRI_FB - 5), PER = BW / NT;
    constexpr uint32_t PAD = (1u << TRI_SUP_LB) - 1;
    __shared__ __align__(16) uint32_t bm[BW];
    __shared__ __align__(16) uint16_t pre[BW];  // columns of row k in the words before
    // acc: two 16-bit sums a word (an item's entries, at most `chunk` = 2,048, hit a place once each)
    __shared__ uint32_t flt[FW], acc[TRI_SUP_ACC / 2];
    __shared__ uint32_t s_item, s_half;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < BW; i += NT) bm[i] = 0;
    for (int i = threadIdx.x; i < FW; i += NT) flt[i] = 0;
    for (int i = threadIdx.x; i < TRI_SUP_ACC / 2; i += NT) acc[i] = 0;
    const uint32_t nitems = *p.nitems;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(p.fetch, 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= nitems) break;
        const uint2 im = __ldg(p.items + it);
        const uint32_t k = im.x, u0 = im.y;
        const uint32_t u1 = min(u0 + p.chunk, __ldg(p.g.urp + k + 1));
        const uint2 shw = __ldg(p.g.shape + k);
        const uint32_t lows = shw.x >> 16, nh = shw.y - lows, lu = (lows + 7) / 8, vk = __ldg(p.g.vstart + k);
        const uint4 *row = p.g.units + vk;
        const uint32_t *hcol = reinterpret_cast<const uint32_t *>(row + lu);
        for (uint32_t u = threadIdx.x; u < 4 * lu; u += NT) {
            const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(row) + u);
            const uint32_t a = (w & 0xFFFFu) ^ 31u, b = (w >> 16) ^ 31u;
            if (a != PAD) atomicOr(bm + (a >> 5), 1u << (a & 31));
            if (b != PAD) atomicOr(bm + (b >> 5), 1u << (b & 31));
        }
        for (uint32_t u = threadIdx.x; u < nh; u += NT) {
            const uint32_t h = tri_hash(__ldg(hcol + u));
            atomicOr(flt + (h >> 5), 1u << (h & 31));
        }
        __syncthreads();
        {  // prefix counts, PER words a thread
            uint32_t w[PER], n = 0;
#pragma unroll
            for (int z = 0; z < PER; z += 4) {
                const uint4 v = reinterpret_cast<const uint4 *>(bm)[(threadIdx.x * PER + z) / 4];
                w[z] = __popc(v.x);
                w[z + 1] = __popc(v.y);
                w[z + 2] = __popc(v.z);
                w[z + 3] = __popc(v.w);
                n += w[z] + w[z + 1] + w[z + 2] + w[z + 3];
            }
            const uint32_t incl = warp_incl_sum(n, lane);
            if (threadIdx.x == 31) s_half = incl;
            __syncthreads();
            uint32_t at = incl - n + (warp ? s_half : 0);
#pragma unroll
            for (int z = 0; z < PER; z += 2) {  // two 16-bit counts a word
                const uint32_t a = at, b = a + w[z];
                at = b + w[z + 1];
                reinterpret_cast<uint32_t *>(pre)[(threadIdx.x * PER + z) / 2] = a | (b << 16);
            }
        }
        __syncthreads();
        // a hit at place `at` of row k
        auto credit = [&](uint32_t at) {
            if (at < TRI_SUP_ACC) atomicAdd(acc + (at >> 1), 1u << (16 * (at & 1u)));
            else atomicAdd(sup + (at < lows ? 8 * vk + at : 8 * (vk + lu + ((at - lows) >> 2)) + ((at - lows) & 3u)), 1);
        };
        for (uint32_t eb = u0 + 32 * warp; eb < u1; eb += NT) {
            uint32_t v0 = 0, el = 0, eh = 0, num = 0, hs = 0;
            if (eb + lane < u1) {
                const uint2 e = __ldg(p.g.uent + eb + lane);
                const uint32_t q = e.y, rl = __ldg(p.g.shape + e.x).x >> 16;
                v0 = __ldg(p.g.vstart + e.x);
                hs = v0 + (rl + 7) / 8;
                if (q < rl) {
                    el = (q + 7) / 8;
                    num = 8 * v0 + q;
                } else {
                    el = (rl + 7) / 8;
                    eh = (q - rl + 3) / 4;
                    num = 8 * (hs + ((q - rl) >> 2)) + ((q - rl) & 3u);
                }
            }
            uint32_t incl = warp_incl_sum(el, lane);
            const uint32_t total = __shfl_sync(FULL, incl, 31);
            const uint32_t off = v0 - (incl - el);
            for (uint32_t b = 0; b < total; b += 32) {
                const uint32_t u = b + lane;
                const int j = warp_find(incl, u) & 31;
                const uint32_t o = __shfl_sync(FULL, off, j) + u, nj = __shfl_sync(FULL, num, j);
                int hits = 0;
                if (u < total) {
                    const uint4 v = __ldg(p.g.units + o);
                    const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
                    auto *sup2 = reinterpret_cast<unsigned long long *>(sup + 8 * static_cast<size_t>(o));
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t x0 = (w4[c] & 0xFFFFu) ^ 31u, x1 = (w4[c] >> 16) ^ 31u;
                        const uint32_t b0 = bm[x0 >> 5], b1 = bm[x1 >> 5];
                        const uint32_t h0 = (b0 >> (x0 & 31)) & 1u, h1 = (b1 >> (x1 & 31)) & 1u;
                        if (h0 | h1) {
                            hits += h0 + h1;
                            atomicAdd(sup2 + c, h0 | (static_cast<unsigned long long>(h1) << 32));
                            if (h0) credit(pre[x0 >> 5] + __popc(b0 & ((1u << (x0 & 31)) - 1u)));
                            if (h1) credit(pre[x1 >> 5] + __popc(b1 & ((1u << (x1 & 31)) - 1u)));
                        }
                    }
                }
                const unsigned peers = __match_any_sync(FULL, j);
                hits = __reduce_add_sync(peers, hits);
                if (hits && lane == __ffs(peers) - 1) atomicAdd(sup + nj, hits);
            }
            if (nh && __any_sync(FULL, eh)) {
                incl = warp_incl_sum(eh, lane);
                const uint32_t htot = __shfl_sync(FULL, incl, 31);
                const uint32_t hoff = hs - (incl - eh);
                for (uint32_t b = 0; b < htot; b += 32) {
                    const uint32_t u = b + lane;
                    const int j = warp_find(incl, u) & 31;
                    const uint32_t o = __shfl_sync(FULL, hoff, j) + u, nj = __shfl_sync(FULL, num, j);
                    if (u < htot) {
                        const uint4 v = __ldg(p.g.units + o);
                        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
                        int hits = 0;
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t h = tri_hash(x[c]);
                            if (!((flt[h >> 5] >> (h & 31)) & 1u)) continue;
                            uint32_t lo = 0, hi = nh;
                            while (lo < hi) {
                                const uint32_t md = (lo + hi) >> 1;
                                if (__ldg(hcol + md) < x[c]) lo = md + 1;
                                else hi = md;
                            }
                            if (lo < nh && __ldg(hcol + lo) == x[c]) {
                                ++hits;
                                atomicAdd(sup + 8 * static_cast<size_t>(o) + c, 1);
                                credit(lows + lo);
                            }
                        }
                        if (hits) atomicAdd(sup + nj, hits);
                    }
                }
            }
        }
        __syncthreads();
        for (uint32_t t = threadIdx.x; 2 * t < min(shw.y, static_cast<uint32_t>(TRI_SUP_ACC)); t += NT) {
            const uint32_t w = acc[t];
            if (!w) continue;
            acc[t] = 0;
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t at = 2 * t + h, n = h ? w >> 16 : w & 0xFFFFu;
                if (n)
                    atomicAdd(sup + (at < lows ? 8 * vk + at : 8 * (vk + lu + ((at - lows) >> 2)) + ((at - lows) & 3u)),
                              static_cast<int>(n));
            }
        }
        for (uint32_t u = threadIdx.x; u < 4 * lu; u += NT) {
            const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(row) + u);
            bm[(w & PAD) >> 5] = 0;
            bm[(w >> 16) >> 5] = 0;
        }
        for (uint32_t u = threadIdx.x; u < nh; u += NT) flt[tri_hash(__ldg(hcol + u)) >> 5] = 0;
    }
}

// ---------------------------------------------------------------------------
// small graphs: the product over the given order in one kernel
// ---------------------------------------------------------------------------
// What a kernel queued before the host has read the facts depends on: a sound
// matrix (chk null: not checked), and the sampled work in [lo, hi).
struct TriGate {
    const CsrCheckOut *chk = nullptr;
    const unsigned long long *sample = nullptr;
    unsigned long long lo = 0, hi = 0;
    __device__ __forceinline__ bool open() const {
        return (!chk || chk->sound()) && (!sample || (*sample >= lo && *sample < hi));
    }
};

constexpr int64_t TRI_SMALL_M = 65536;  // vertices: a bitmap of a row's columns fits the warp's shared memory
constexpr int TRI_SMALL_WARPS = 4;

// Whether x is among the n ascending columns of c.
__device__ __forceinline__ bool tri_small_has(const int32_t *__restrict__ c, uint32_t n, int x) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t md = (lo + hi) >> 1;
        if (__ldg(c + md) < x) lo = md + 1;
        else hi = md;
    }
    return lo < n && __ldg(c + lo) == x;
}

// Hits of a row L_i (ri, len columns) in the rows L_k of up to 32 entries (one per
// lane: n columns from col + b0) without its bitmap: an L_k far longer than L_i is
// searched for L_i's columns, the others' columns are searched for in L_i.
constexpr uint32_t TRI_SMALL_UNEVEN = 32;
__device__ __forceinline__ bool tri_small_longer(uint32_t n, uint32_t len) { return n > TRI_SMALL_UNEVEN * (len + 32); }

__device__ __forceinline__ uint32_t tri_small_search(const int32_t *__restrict__ col, const int32_t *__restrict__ ri,
                                                  uint32_t len, int64_t b0, uint32_t n) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const bool longer = tri_small_longer(n, len);
    uint32_t cnt = 0;
    for (unsigned todo = __ballot_sync(FULL, longer); todo; todo &= todo - 1) {
        const int j = __ffs(todo) - 1;
        const int64_t bj = __shfl_sync(FULL, b0, j);
        const uint32_t nj = __shfl_sync(FULL, n, j);
        for (uint32_t q = lane; q < len; q += 32) cnt += tri_small_has(col + bj, nj, __ldg(ri + q));
    }
    const uint32_t m = longer ? 0 : n, incl = warp_incl_sum(m, lane), total = __shfl_sync(FULL, incl, 31);
    for (uint32_t b = 0; b < total; b += 32) {
        const uint32_t at = b + lane;
        const int j = warp_find(incl, at) & 31;
        const int64_t q = __shfl_sync(FULL, b0, j) + (at - __shfl_sync(FULL, incl - m, j));
        if (at < total) cnt += tri_small_has(ri, len, __ldg(col + q));
    }
    return cnt;
}

// Sum of C<L> = L·L.  A warp takes 32 entries of L at a time; for each row i
// among them the columns of L_i go to a bitmap in shared memory, and the rows
// L_k of the entries k are read four columns per lane and tested.  No plan: the
// entries, not the rows, are dealt out, so a hub row is spread over warps.
// Very uneven pairs take the search above, since a warp would read a whole long row
// for a few columns: the bitmap of a long L_i whose L_k hold little (16,384
// vertices, 32 rows of all columns: 1.20 -> 0.05 ms), or an L_k far longer than L_i
// (65,536 vertices, one row of 32,768 columns named by as many rows: 3.35 -> 0.10
// ms).  The ordinary rows' loads are left as they were, the bitmap's in flight with
// those of the L_k (bitmap only once the L_k's columns are counted: RMAT-16 340 ->
// 490 us; the search out of line: RMAT-8 45 -> 48 us, in line 43).
constexpr uint32_t TRI_SMALL_MAP = 1024;  // columns of an L_i that is mapped in any case
__global__ void __launch_bounds__(32 * TRI_SMALL_WARPS) k_tri_small(DevCsr L, int words, TriGate gate,
                                                                    unsigned long long *sum) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    extern __shared__ uint32_t smem[];
    if (!gate.open()) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *bm = smem + warp * words;
    for (int i = lane; i < words; i += 32) bm[i] = 0;
    __syncwarp();
    unsigned long long local = 0;
    const int64_t step = (int64_t)gridDim.x * TRI_SMALL_WARPS * 32;
    for (int64_t p0 = ((int64_t)blockIdx.x * TRI_SMALL_WARPS + warp) * 32; p0 < L.nnz; p0 += step) {
        const int64_t p1 = min(p0 + 32, L.nnz);
        uint32_t cnt = 0;
        // the ends of 32 rows, one per lane, and where the first of them starts
        int64_t r = warp_row_of(L.rp, 0, L.m - 1, p0, lane), first = __ldg(L.rp + r);
        int64_t end = r + lane < L.m ? __ldg(L.rp + r + lane + 1) : L.nnz;
        for (int64_t p = p0; p < p1;) {
            const int past = __popc(__ballot_sync(FULL, end <= p));  // rows that p has passed
            if (past == 32) {
                // on to the row of p; behind more than 32 empty rows by a search (63
                // edges on 10,856 vertices, row by row 661 us, so 62)
                first = __shfl_sync(FULL, end, 31);
                r += 32;
                end = r + lane < L.m ? __ldg(L.rp + r + lane + 1) : L.nnz;
                if (__shfl_sync(FULL, end, 31) <= p) {
                    r = warp_row_of(L.rp, r + 32, L.m - 1, p, lane);
                    first = __ldg(L.rp + r);
                    end = r + lane < L.m ? __ldg(L.rp + r + lane + 1) : L.nnz;
                }
                continue;
            }
            const int64_t r1 = __shfl_sync(FULL, end, past), before = __shfl_sync(FULL, end, (past - 1) & 31);
            const int64_t r0 = past ? before : first, e = min(r1, p1);
            // the rows of the entries p .. e - 1, one per lane
            const int64_t t = p + lane;
            int64_t b0 = 0;
            uint32_t n = 0;
            if (t < e) {
                const int k = __ldg(L.col + t);
                b0 = __ldg(L.rp + k);
                n = static_cast<uint32_t>(__ldg(L.rp + k + 1) - b0);
            }
            const uint32_t len = static_cast<uint32_t>(r1 - r0);
            p = e;
            if (len > TRI_SMALL_MAP && 8 * __reduce_add_sync(FULL, min(n, 1u << 16)) < len) {
                cnt += tri_small_search(L.col, L.col + r0, len, b0, n);
                continue;
            }
            for (int64_t q = r0 + lane; q < r1; q += 32) {
                const int x = __ldg(L.col + q);
                atomicOr(bm + (x >> 5), 1u << (x & 31));
            }
            __syncwarp();
            const bool longer = tri_small_longer(n, len);
            if (__any_sync(FULL, longer)) {
                cnt += tri_small_search(L.col, L.col + r0, len, b0, longer ? n : 0);
                if (longer) n = 0;
            }
            const uint32_t u = (n + 3) / 4, incl = warp_incl_sum(u, lane);
            const uint32_t total = __shfl_sync(FULL, incl, 31);
            for (uint32_t b = 0; b < total; b += 32) {
                const uint32_t at = b + lane;
                const int j = warp_find(incl, at) & 31;
                const uint32_t z = 4 * (at - __shfl_sync(FULL, incl - u, j));
                const uint32_t nj = __shfl_sync(FULL, n, j);
                const int64_t bj = __shfl_sync(FULL, b0, j);
                if (at < total) {
#pragma unroll
                    for (uint32_t c = 0; c < 4; ++c)
                        if (z + c < nj) {
                            const uint32_t x = static_cast<uint32_t>(__ldg(L.col + bj + z + c));
                            cnt += (bm[x >> 5] >> (x & 31)) & 1u;
                        }
                }
            }
            __syncwarp();
            for (int64_t q = r0 + lane; q < r1; q += 32) bm[__ldg(L.col + q) >> 5] = 0;
            __syncwarp();
        }
        local += cnt;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(FULL, local, o);
    if (lane == 0 && local) atomicAdd(sum, local);
}

// ---------------------------------------------------------------------------
// little work per entry: the product over the given order, entry by entry
// ---------------------------------------------------------------------------
// Sum of C<L> = L·L for rows [0, L.m) (per graph with keys).  A warp walks
// the entries (i, k) 32 at a time, whatever their rows; for each the shorter of
// the rows L_i and L_k is read, its elements packed onto the lanes, four to a
// lane, and looked up in the other by binary search.  Rows of a few columns are a
// few steps in L1, and there is no plan.  Where L is a strict lower triangle, only
// the columns of L_i before k count.  In front of the searches in the rows L_i of
// a step's entries stands a filter of their columns, unless they are too many or
// the elements too few (Erdos-Renyi 400,000 x 64: 1.13 ms with searches alone,
// bound by the ALU at seven steps an element; 0.80 with the filter).
constexpr int TRI_WF = 13;           // log2 bits of a warp's filter
constexpr uint32_t TRI_WF_ROWS = 512;  // columns it takes at most
__device__ __forceinline__ uint32_t tri_walk_hash(uint32_t x, uint32_t row) {
    return (x * 0x9E3779B1u + row * 0x85EBCA77u) >> (32 - TRI_WF);
}

template <bool KEYED>
__global__ void __launch_bounds__(256, 5) k_tri_walk(DevCsr L, DevCsr B, int64_t ebase, int walk, const int32_t *key,
                                                  TriGate gate, int lower, unsigned long long *sums) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    if (!gate.open()) return;
    const bool prefix = lower >= 0 ? lower != 0 : (gate.chk && !gate.chk->not_lower);
    const int lane = threadIdx.x & 31;
    __shared__ uint32_t s_filt[8][(1 << TRI_WF) / 32];
    uint32_t *filt = s_filt[threadIdx.x >> 5];
    const int64_t p0 = ebase + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * walk;
    const int64_t p1 = min(p0 + walk, ebase + L.nnz);
    if (p0 >= p1) return;
    unsigned long long local = 0;
    walk_entries(L.rp, L.m, p0, p1, lane, [&](int64_t p, int64_t row, int leader, unsigned peers_of_row, bool on) {
        uint32_t n = 0, len = 0;  // elements read, and those they are looked up in
        int64_t b0 = 0, s0 = 0;
        bool direct = false;
        if (on) {
            const int k = __ldg(L.col + p);
            b0 = __ldg(B.rp + k);
            n = static_cast<uint32_t>(__ldg(B.rp + k + 1) - b0);
            s0 = __ldg(L.rp + row);
            len = static_cast<uint32_t>((prefix ? p : __ldg(L.rp + row + 1)) - s0);
            direct = 2 * len < n;
            if (direct) {
                const uint32_t x = n;
                n = len;
                len = x;
                const int64_t y = b0;
                b0 = s0;
                s0 = y;
            }
        }
        const uint32_t u = (n + 3) / 4, incl = warp_incl_sum(u, lane);
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        // a filter of the rows' columns in front of the searches, where it pays
        // for being built: a row's last entry here has the longest part of it
        const bool last = on && !direct && (peers_of_row >> lane) == 1u;
        const unsigned lasts = __ballot_sync(FULL, last);
        const uint32_t rows = __reduce_add_sync(FULL, last ? len : 0u);
        const bool use = rows > 0 && rows <= TRI_WF_ROWS && 2 * total > rows;
        if (use) {
#pragma unroll
            for (int z = 0; z < (1 << TRI_WF) / 32; z += 32) filt[z + lane] = 0;
            __syncwarp();
            for (unsigned todo = lasts; todo; todo &= todo - 1) {
                const int src = __ffs(todo) - 1;
                const int64_t q0 = __shfl_sync(FULL, s0, src);
                const uint32_t m = __shfl_sync(FULL, len, src), r = __shfl_sync(FULL, static_cast<uint32_t>(row), src);
                for (uint32_t q = lane; q < m; q += 32) {
                    const uint32_t h = tri_walk_hash(static_cast<uint32_t>(__ldg(L.col + q0 + q)), r);
                    atomicOr(filt + (h >> 5), 1u << (h & 31));
                }
            }
            __syncwarp();
        }
        // (a row whose last entry here is direct is not in the filter)
        const unsigned filtered = __ballot_sync(FULL, use && on && !direct && (lasts & peers_of_row));
        for (uint32_t b = 0; b < total; b += 32) {
            const uint32_t at = b + lane;
            const int j = warp_find(incl, at) & 31;
            const uint32_t z = 4 * (at - __shfl_sync(FULL, incl - u, j));
            const uint32_t nj = __shfl_sync(FULL, n, j), lj = __shfl_sync(FULL, len, j);
            const uint32_t rj = __shfl_sync(FULL, static_cast<uint32_t>(row), j);
            const int64_t bj = __shfl_sync(FULL, b0, j) + z;
            const int32_t *__restrict__ ri = L.col + __shfl_sync(FULL, s0, j);
            uint32_t hits = 0;
            if (at < total) {
                int x[4];
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) x[c] = z + c < nj ? __ldg(L.col + bj + c) : -1;
                if ((filtered >> j) & 1u) {
                    uint32_t cand = 0;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t h = tri_walk_hash(static_cast<uint32_t>(x[c]), rj);
                        cand |= ((filt[h >> 5] >> (h & 31)) & 1u) << c;
                    }
                    for (; cand; cand &= cand - 1) {  // rare: one search at a time
                        const int y = (cand & 1) ? x[0] : (cand & 2) ? x[1] : (cand & 4) ? x[2] : x[3];
                        uint32_t lo = 0;
                        for (uint32_t m = lj; m > 1;) {
                            const uint32_t half = m >> 1;
                            if (__ldg(ri + lo + half) <= y) lo += half;
                            m -= half;
                        }
                        hits += __ldg(ri + lo) == y;
                    }
                } else {
                    // four searches side by side: last position with ri <= x
                    uint32_t lo[4] = {0, 0, 0, 0};
                    for (uint32_t m = lj; m > 1;) {
                        const uint32_t half = m >> 1;
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (__ldg(ri + lo[c] + half) <= x[c]) lo[c] += half;
                        m -= half;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) hits += __ldg(ri + lo[c]) == x[c];
                }
            }
            if (KEYED) {
                if (!__any_sync(FULL, hits)) continue;
                // hits of entry j's graph
                const int kj = key[__shfl_sync(FULL, static_cast<int>(on ? row : 0), j)];
                const unsigned peers = __match_any_sync(FULL, kj);
                const uint32_t sum = __reduce_add_sync(peers, hits);
                if (sum && lane == __ffs(peers) - 1) atomicAdd(sums + kj, static_cast<unsigned long long>(sum));
            } else {
                local += hits;
            }
        }
    });
    if (!KEYED) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(FULL, local, o);
        if (lane == 0 && local) atomicAdd(sums, local);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int bits_for(int64_t n) {  // bits that hold 0 .. n - 1
    int b = 1;
    while ((int64_t(1) << b) < n) ++b;
    return b;
}

__global__ void __launch_bounds__(256) k_tri_unit_sum(int64_t E, const uint2 *uent, unsigned long long *sum) {
    __shared__ unsigned long long red[8];
    unsigned long long n = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < E; t += stride) {
        const uint32_t y = uent[t].y;
        n += (y & 0x3FFFu) + (y >> 15) + ((y >> 14) & 1u ? TRI_MAP : 0u);
    }
    n = block_sum(n, red);
    if (threadIdx.x == 0 && n) atomicAdd(sum, n);
}

// Units of m rows with E columns at most: a quarter of the columns, a partly
// filled unit of each class per row, and a bitmap for at least every
// 8 * (TRI_MAP_MIN - 1) columns.
static int64_t unit_bound(int64_t m, int64_t E) {
    return E / 4 + 3 * std::min(m, E) + TRI_MAP * (E / (8 * (TRI_MAP_MIN - 1)) + 1);
}

template <int LB, bool KEYED>
static int launch_count(const TriArgs &a, cudaStream_t s) {
    constexpr int NT = 32 * TRI_WARPS;
    int per_sm = 0;
    GK_CUDA(cudaFuncSetAttribute(k_tri_count<LB, KEYED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(tri_smem<LB>())));
    GK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tri_count<LB, KEYED>, NT, tri_smem<LB>()));
    ProfWindow prof(s, NV + 1);
    prof.begin(NV, s);
    k_tri_count<LB, KEYED><<<ctx().num_sms * std::max(per_sm, 1), NT, tri_smem<LB>(), s>>>(a);
    prof.end(NV, s);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    if (!prof.active()) return GK_OK;
    // the record's work: the 16-byte units that the entries name
    Scratch scr(s);
    unsigned long long *units, h = 0;
    GK_CHECK(scr.alloc(&units, 1));
    GK_CUDA(cudaMemsetAsync(units, 0, sizeof(*units), s));
    k_tri_unit_sum<<<ctx().num_sms * 8, 256, 0, s>>>(a.g.E, a.g.uent, units);
    GK_CUDA(cudaMemcpyAsync(&h, units, sizeof(h), cudaMemcpyDeviceToHost, s));
    GK_CUDA(cudaStreamSynchronize(s));
    ProfTotals tot[NV + 1] = {};
    tot[NV] = ProfTotals{static_cast<unsigned long long>(a.g.m), static_cast<unsigned long long>(a.g.E),
                         static_cast<unsigned long long>(a.g.E), h};
    return prof.finish(tot);
}

// The graph in rank order and its work items; `place`: for the support, with
// no hub class and with places as entries.
static int orient(const TriInput &in, const uint32_t *deg, const uint32_t *rank, int lb, bool place, TriArgs *out,
                  cudaStream_t s, Scratch &scr) {
    const DevCsr &L = in.L;
    const int64_t m = L.m, E = L.nnz, ebase = in.ebase;
    const int sms = ctx().num_sms;
    const uint32_t low_lim = (1u << lb) - 1;
    // in-edges per work item: small graphs need many items to fill the GPU
    // (RMAT-18 count: 128 of them 0.13 ms, 512 0.16, 2048 0.22), large ones pay
    // for every item's bitmap (RMAT-24: 2048 26.2 ms, 512 27.1)
    const uint32_t chunk = static_cast<uint32_t>(std::min<int64_t>(std::max<int64_t>(E >> 15, 128), 2048));
    const bool bands = !place && E >= TRI_BAND_EDGES;
    uint32_t *start, *len, *nun, *nin, *nit, *lrp, *vstart, *urp, *ipre, *ucur, *cols, *longrows;
    uint32_t *bnd = nullptr, *bpre = nullptr;
    unsigned long long *counts;
    uint2 *shape, *uent;
    unsigned int *ctr;
    GK_CHECK(scr.alloc(&start, m + 1));
    GK_CHECK(scr.alloc(&len, m + 1));
    GK_CHECK(scr.alloc(&lrp, m + 1));
    GK_CHECK(scr.alloc(&nun, 3 * (m + 1)));
    nin = nun + (m + 1);
    nit = nin + (m + 1);
    if (bands) {
        GK_CHECK(scr.alloc(&bnd, m + 1));
        GK_CHECK(scr.alloc(&bpre, m + 1));
    }
    GK_CHECK(scr.alloc(&vstart, m + 1));
    GK_CHECK(scr.alloc(&shape, m + 1));
    GK_CHECK(scr.alloc(&counts, m));
    GK_CHECK(scr.alloc(&urp, m + 1));
    GK_CHECK(scr.alloc(&ipre, m + 1));
    GK_CHECK(scr.alloc(&ucur, m + 1));
    GK_CHECK(scr.alloc(&cols, 2 * E));
    GK_CHECK(scr.alloc(&uent, E));
    GK_CHECK(scr.alloc(&longrows, E / TRI_WARP_ROW + 1));
    GK_CHECK(scr.alloc(&ctr, 2));
    GK_CUDA(cudaMemsetAsync(ctr, 0, sizeof(unsigned int) * 2, s));
    GK_CUDA(cudaMemsetAsync(counts, 0, sizeof(unsigned long long) * m, s));
    size_t sb = 0;
    GK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, sb, nun, vstart, m + 1, s));
    void *tmp;
    GK_CHECK(scr.alloc(reinterpret_cast<char **>(&tmp), sb));
    GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, sb, deg, start, m, s));
    // entries a warp walks: enough warps to fill the GPU on a small graph
    const int walk = static_cast<int>(std::min<int64_t>(std::max<int64_t>(E / (sms * 64) & ~int64_t(31), 32), 1024));
    const int walkers = ceil_div(E, walk * 8);
    const TriBase tb{in.key, in.gvbase, in.vbase};
    k_tri_scatter<<<walkers, 256, 0, s>>>(L, ebase, in.vbase, walk, tb, place ? 0 : TRI_HUB, low_lim, rank, start,
                                          counts, cols);
    k_tri_row_sizes<<<sms * 8, 256, 0, s>>>(m, deg, chunk, counts, len, shape, nun, nin, nit, bnd);
    GK_CUDA(cudaGetLastError());
    GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, sb, len, lrp, m + 1, s));
    GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, sb, nun, vstart, m + 1, s));
    GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, sb, nin, urp, m + 1, s));
    GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, sb, nit, ipre, m + 1, s));
    if (bands) GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, sb, bnd, bpre, m + 1, s));
    GK_CUDA(cudaMemcpyAsync(ucur, urp, sizeof(uint32_t) * m, cudaMemcpyDeviceToDevice, s));
    uint4 *units;
    GK_CHECK(scr.alloc(&units, unit_bound(m, E)));
    uint2 *items;
    GK_CHECK(scr.alloc(&items, std::min(m, E) + E / chunk + 1 + (bands ? TRI_BANDS * (E / TRI_BAND_MIN) : 0)));
    const TriRowArgs ra{m, E, lrp, start, cols, tb, low_lim, shape, vstart, units, ucur, uent, longrows, ctr};
    k_tri_rows<<<sms * 8, 256, 0, s>>>(ra);
    k_tri_long_rows<<<sms * 2, 512, 0, s>>>(ra);
    // not for a batch, whose graphs have hubs of their own (409 graphs 2.83 ms, 3.34
    // with HOT for the graph that a CTA starts in), nor for a very large graph, whose
    // hubs are a smaller share of its entries (RMAT-24 5.7 ms, 6.1)
    const bool hot = !in.key && E < TRI_BAND_EDGES;
    const int ewalk = hot ? std::min(walk, TRI_WALK) : walk, eblocks = ceil_div(E, ewalk * 8);
    auto *entries = place ? (hot ? k_tri_entries<true, true> : k_tri_entries<true, false>)
                          : (hot ? k_tri_entries<false, true> : k_tri_entries<false, false>);
    entries<<<eblocks, 256, 0, s>>>(ra, ewalk);
    k_tri_items<<<sms * 8, 256, 0, s>>>(m, ipre, bpre, urp, chunk, items);
    GK_CUDA(cudaGetLastError());
    note_launches(6);
    unsigned int *fetch;
    GK_CHECK(scr.alloc(&fetch, 1));
    GK_CUDA(cudaMemsetAsync(fetch, 0, sizeof(unsigned int), s));
    TriArgs &a = *out;
    a.g.m = m;
    a.g.E = E;
    a.g.units = units;
    a.g.vstart = vstart;
    a.g.shape = shape;
    a.g.urp = urp;
    a.g.uent = uent;
    a.items = items;
    a.nitems = ipre + m;
    a.nbanded = bands ? bpre + m : nullptr;
    a.fetch = fetch;
    a.chunk = chunk;
    return GK_OK;
}

// The vertex order (perm: vertex of every rank).
template <class KeyT>
static int vertex_order(const TriInput &in, int dbits, int gbits, const uint32_t *cnt, uint32_t *iota, uint32_t *perm,
                        cudaStream_t s, Scratch &scr) {
    const int64_t m = in.L.m;
    KeyT *vkey, *vkey2;
    GK_CHECK(scr.alloc(&vkey, m));
    GK_CHECK(scr.alloc(&vkey2, m));
    k_tri_vertex_keys<KeyT><<<ctx().num_sms * 8, 256, 0, s>>>(in.L, in.vbase, in.key, dbits, cnt, vkey, iota);
    note_launches(2);
    GK_CUDA(cudaGetLastError());
    size_t vb = 0;
    GK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, vb, vkey, vkey2, iota, perm, m, 0, dbits + gbits, s));
    void *tmp;
    GK_CHECK(scr.alloc(reinterpret_cast<char **>(&tmp), vb));
    GK_CUDA(cub::DeviceRadixSort::SortPairs(tmp, vb, vkey, vkey2, iota, perm, m, 0, dbits + gbits, s));
    return GK_OK;
}

// Vertices up to which the small kernel runs without a look at the work, and the
// columns an entry's row holds on average below which a larger graph is walked.
constexpr int64_t TRI_SMALL_SURE = 16384;
constexpr unsigned long long TRI_SMALL_FLAT = 30;

// The small kernel reads the given order's work, about nnz * (nnz / m) columns
// times the graph's skew (RMAT-14: 7), and has no other passes; the orientation's
// some twenty launches cost 0.15 ms before the first column is read.  RMAT-14: 91
// us against 254, RMAT-16 340 against 390.
bool tri_small_fits(int64_t m, int64_t nnz) {
    return m >= 1 && nnz >= 1 && m <= TRI_SMALL_M && nnz <= (int64_t(1) << 24) && nnz * nnz / m <= (int64_t(1) << 24);
}

// lower: whether in.L is a strict lower triangle (-1: gate.chk knows).
static int launch_walk(const TriInput &in, const TriGate &gate, int lower, unsigned long long *sums, cudaStream_t s) {
    const int64_t E = in.L.nnz;
    if (E < 1) return GK_OK;
    const int sms = ctx().num_sms;
    const int walk = static_cast<int>(std::min<int64_t>(std::max<int64_t>(E / (sms * 128) & ~int64_t(31), 32), 512));
    const int blocks = ceil_div(E, walk * 8);
    // row pointers of the columns: the group's rows are all the columns name
    DevCsr B = in.L;
    B.rp -= in.vbase;
    ProfWindow prof(s, NV + 2);
    prof.begin(NV + 1, s);
    if (in.key)
        k_tri_walk<true><<<blocks, 256, 0, s>>>(in.L, B, in.ebase, walk, in.key + in.vbase, gate, lower, sums);
    else
        k_tri_walk<false><<<blocks, 256, 0, s>>>(in.L, B, in.ebase, walk, nullptr, gate, lower, sums);
    prof.end(NV + 1, s);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    if (!prof.active()) return GK_OK;
    ProfTotals tot[NV + 2] = {};
    tot[NV + 1].rows = static_cast<unsigned long long>(in.L.m);
    tot[NV + 1].sum_a = tot[NV + 1].sum_m = static_cast<unsigned long long>(E);
    return prof.finish(tot);
}

int tri_count_small(const DevCsr &L, const CsrCheckOut *chk, unsigned long long *sample, unsigned long long *sum,
                    cudaStream_t s) {
    TriGate gate;
    gate.chk = chk;
    if (L.m > TRI_SMALL_SURE) {
        // flat graphs are better walked (Erdos-Renyi 60,000 x 27: 142 against 96
        // us), skewed ones have longer rows to search (RMAT-16: 340 against 450):
        // both kernels are queued, and the sampled work lets one of them run
        TriInput in;
        in.L = L;
        GK_CHECK(tri_sample(in, chk, sample, s));
        TriGate wg = gate;
        wg.sample = gate.sample = sample;
        wg.hi = gate.lo = TRI_SMALL_FLAT * static_cast<unsigned long long>(std::min<int64_t>(L.nnz, TRI_SAMPLE));
        gate.hi = ~0ull;
        GK_CHECK(launch_walk(in, wg, -1, sum, s));
    }
    const int words = static_cast<int>((L.m + 31) / 32);
    const size_t smem = size_t(TRI_SMALL_WARPS) * words * 4;  // at most 32 KB
    const int64_t ctas = (L.nnz + 32 * TRI_SMALL_WARPS - 1) / (32 * TRI_SMALL_WARPS);
    const int resident = static_cast<int>(std::min<size_t>(16, (200u << 10) / (smem + 1024)));
    ProfWindow prof(s, NV + 2);
    prof.begin(NV + 1, s);
    k_tri_small<<<static_cast<int>(std::min<int64_t>(ctas, int64_t(ctx().num_sms) * resident)), 32 * TRI_SMALL_WARPS,
                  smem, s>>>(L, words, gate, sum);
    prof.end(NV + 1, s);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    if (!prof.active()) return GK_OK;
    ProfTotals tot[NV + 2] = {};
    tot[NV + 1].rows = static_cast<unsigned long long>(L.m);
    tot[NV + 1].sum_a = tot[NV + 1].sum_m = static_cast<unsigned long long>(L.nnz);
    return prof.finish(tot);
}

// Device bytes of one count: eighteen arrays of a word per row (one of them
// twice as wide, the keys up to twice), the columns, entries and units, and
// the sort's and the scans' temporary storage.
static int64_t tri_bytes(int64_t m, int64_t E) {
    return 26 * 4 * (m + 64) + 16 * (E + 64) + 16 * (unit_bound(m, E) + 64) + 8 * (std::min(m, E) + E / 64) +
           (E / TRI_WARP_ROW + 64) * 4 + (m / 2 + (int64_t(1) << 20));
}

// Order of the vertices: rank of every vertex, degree of every rank.
static int order_vertices(const TriInput &in, uint32_t **deg, uint32_t **rank, cudaStream_t s, Scratch &scr) {
    const int64_t m = in.L.m;
    const int sms = ctx().num_sms;
    uint32_t *cnt, *iota, *perm;
    GK_CHECK(scr.alloc(&cnt, m));
    GK_CHECK(scr.alloc(&iota, m));
    GK_CHECK(scr.alloc(&perm, m));
    GK_CHECK(scr.alloc(rank, m));
    GK_CHECK(scr.alloc(deg, m));
    GK_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * m, s));
    const int cc = static_cast<int>(std::max<int64_t>(sms * 8, (in.L.nnz + (1 << 15) - 1) >> 15));
    k_tri_col_counts<<<cc, 256, 0, s>>>(in.L, in.ebase, in.vbase, cnt);
    const int dbits = bits_for(in.key ? in.max_m : m), gbits = in.key ? bits_for(in.nkeys) : 0;
    if (dbits + gbits <= 32) GK_CHECK(vertex_order<uint32_t>(in, dbits, gbits, cnt, iota, perm, s, scr));
    else GK_CHECK(vertex_order<unsigned long long>(in, dbits, gbits, cnt, iota, perm, s, scr));
    k_tri_degrees<<<sms * 8, 256, 0, s>>>(m, perm, cnt, in.L, *rank, *deg);
    note_launches(2);
    GK_CUDA(cudaGetLastError());
    return GK_OK;
}

// Sampled work per entry of every graph of a batch not yet checked: whatever the
// arrays hold, nothing is read outside them.
__global__ void __launch_bounds__(64) k_tri_sample_graphs(const TriGraphRef *g, float *per_entry) {
    __shared__ unsigned long long red[2];
    const TriGraphRef r = g[blockIdx.x];
    const int n = static_cast<int>(min(r.nnz, int64_t(256)));
    unsigned long long w = 0;
    for (int t = threadIdx.x; t < n; t += 64) {
        const int64_t k = r.col[r.nnz * t / n];
        if (k >= 0 && k < r.m) {
            const int64_t len = r.rp[k + 1] - r.rp[k];
            if (len > 0) w += static_cast<unsigned long long>(min(len, r.m));
        }
    }
    w = block_sum(w, red);
    if (threadIdx.x == 0) per_entry[blockIdx.x] = n ? static_cast<float>(w) / n : 0.f;
}

int tri_sample_graphs(const TriGraphRef *graphs, int n, float *per_entry, cudaStream_t s) {
    k_tri_sample_graphs<<<n, 64, 0, s>>>(graphs, per_entry);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    return GK_OK;
}

int tri_sample(const TriInput &in, const CsrCheckOut *chk, unsigned long long *sum, cudaStream_t s) {
    if (in.L.nnz < 1) return GK_OK;
    const int n = static_cast<int>(std::min<int64_t>(in.L.nnz, TRI_SAMPLE));
    k_tri_sample<<<ceil_div(n, 256), 256, 0, s>>>(in.L, in.ebase, in.vbase, n, chk, sum);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    return GK_OK;
}

int tri_support(const DevCsr &L, TriSupport *out, cudaStream_t s, Scratch &scr, bool *done) {
    *done = false;
    const int64_t m = L.m, E = L.nnz;
    out->numbers = 8 * (E / 4 + 2 * std::min(m, E) + 2);
    if (m < 2 || E < 1 || out->numbers >= (int64_t(1) << 32)) return GK_OK;
    GK_CHECK(scr.reserve(static_cast<size_t>(tri_bytes(m, E) + 4 * out->numbers)));
    TriInput in;
    in.L = L;
    uint32_t *deg, *rank;
    GK_CHECK(order_vertices(in, &deg, &rank, s, scr));
    GK_CHECK(scr.alloc(&out->sup, out->numbers));
    GK_CUDA(cudaMemsetAsync(out->sup, 0, sizeof(int32_t) * out->numbers, s));
    TriSupArgs a;
    GK_CHECK(orient(in, deg, rank, TRI_SUP_LB, true, &a.t, s, scr));
    a.sup = out->sup;
    int per_sm = 0;
    GK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tri_support, 64, 0));
    k_tri_support<<<ctx().num_sms * std::max(per_sm, 1), 64, 0, s>>>(a);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    out->g = a.t.g;
    out->rank = rank;
    *done = true;
    return GK_OK;
}

// The graph in degree order, ready to be counted (nothing is added to the sums yet).
static int degree_order(const TriInput &in, unsigned long long *sums, TriArgs *a, int *lb, cudaStream_t s,
                        Scratch &scr) {
    GK_CHECK(scr.reserve(static_cast<size_t>(tri_bytes(in.L.m, in.L.nnz))));
    uint32_t *deg, *rank;
    GK_CHECK(order_vertices(in, &deg, &rank, s, scr));
    // Columns below the low limit are tested in the warp's bitmap, the others
    // by filter and search.  2^15 keeps 40 warps an SM (2^16: 20, with 8 KB
    // bitmaps): RMAT-22 count 3.3 against 3.9 ms; on RMAT-24, where more of the
    // columns read lie beyond 2^15, 28.5 against 26.2 ms.
    *lb = (in.key ? in.max_m : in.L.m) > (int64_t(1) << 23) ? 16 : 15;
    GK_CHECK(orient(in, deg, rank, *lb, false, a, s, scr));
    a->sums = sums;
    a->key = in.key ? in.key + in.vbase : nullptr;
    return GK_OK;
}

int tri_count(const TriInput &in, const CsrCheckOut &facts, unsigned long long sample, unsigned long long *sums,
              cudaStream_t s, bool *done) {
    *done = false;
    const DevCsr &L = in.L;
    const int64_t m = L.m, E = L.nnz;
    if (m < 2 || E < 1 || E >= (int64_t(1) << 31) || unit_bound(m, E) >= (int64_t(1) << 32)) return GK_OK;
    // Where an entry's row holds only a few columns, the walk over the given order
    // is done before the orientation's passes over the edges are (columns an entry:
    // us walked / in degree order): Erdos-Renyi 1.5 M vertices 6.7: 626 / 2811,
    // 21: 2898 / 6791; RMAT-17 74: 199 / 305; RMAT-19 69: 256 / 442, 126: 682 / 539;
    // RMAT-21 115: 1044 / 1282; RMAT-18 171: 941 / 485.
    const unsigned long long limit = in.key ? TRI_WALK_WORK_BATCH : TRI_WALK_WORK;
    if (sample < limit * std::min<int64_t>(E, TRI_SAMPLE)) {
        *done = true;
        return launch_walk(in, TriGate{}, facts.not_lower ? 0 : 1, sums, s);
    }
    if (facts.not_lower) return GK_OK;  // not a triangle: the sum depends on the order
    // scratch beyond what the product needs: where there is no room, that runs
    Scratch scr(s);
    TriArgs a;
    int lb = 0;
    const int status = degree_order(in, sums, &a, &lb, s, scr);
    if (status == GK_ERR_OOM) {
        scr.release();
        scratch_reclaim(s);
        return GK_OK;
    }
    GK_CHECK(status);
    if (lb == 16) GK_CHECK((in.key ? launch_count<16, true>(a, s) : launch_count<16, false>(a, s)));
    else GK_CHECK((in.key ? launch_count<15, true>(a, s) : launch_count<15, false>(a, s)));
    *done = true;
    return GK_OK;
}

}  // namespace gk
