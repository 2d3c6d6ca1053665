// Internal interface of the degree-ordered triangle kernels (tri.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gk_common.cuh"

namespace gk {

// A graph's edges, its vertices renamed by descending degree (rank 0: the
// largest degree), each edge kept once, in the row of its higher rank.  Row i's
// columns (ascending ranks below i) are stored in 16-byte units: first the hub
// columns (below 2048) and the other low ones (below the low limit) as 16-bit
// values, eight to a unit, then the high ones as 32-bit values, four to a unit,
// each class padded to whole units; behind the hub columns of a row with many
// of them, their bitmap.  The in-edges of k (the rows i > k that hold column k)
// are entries {first unit, list units | bitmap << 14 | high units << 15} of
// what row i holds below k.
struct TriGraph {
    int64_t m = 0, E = 0;
    const uint4 *units = nullptr;
    const uint32_t *vstart = nullptr;  // [m + 1] first unit of every row
    const uint2 *shape = nullptr;      // [m] {hub columns | low columns << 16, columns} of every row
    const uint32_t *urp = nullptr;     // [m + 1] in-edge entries of every row
    const uint2 *uent = nullptr;
};

constexpr uint32_t TRI_HUB = 2048;          // columns below it are hubs
constexpr uint32_t TRI_MAP = TRI_HUB / 128;  // units of a hub bitmap
constexpr uint32_t TRI_MAP_MIN = 6;          // units of hub columns from which their bitmap is read instead

// Shape of a row's storage: hub columns, other low columns and high columns,
// each padded to whole units; a row with at least TRI_MAP_MIN units of hub
// columns keeps their bitmap behind them.
struct TriShape {
    uint32_t hubs, lows, n;  // columns: hubs, hubs and other low ones, all
    __device__ __forceinline__ uint32_t hub_units() const { return (hubs + 7) / 8; }
    __device__ __forceinline__ uint32_t map_units() const { return hub_units() >= TRI_MAP_MIN ? TRI_MAP : 0; }
    __device__ __forceinline__ uint32_t mid_units() const { return (lows - hubs + 7) / 8; }
    __device__ __forceinline__ uint32_t high_units() const { return (n - lows + 3) / 4; }
    __device__ __forceinline__ uint32_t units() const {
        return hub_units() + map_units() + mid_units() + high_units();
    }
};

// The input of an orientation: rows [0, m) of a strict lower triangle whose row
// pointers run from ebase and whose columns run from vbase (the block-diagonal
// batch's groups; 0 for one graph).
struct TriInput {
    DevCsr L;
    int64_t ebase = 0, vbase = 0;
    const int32_t *key = nullptr;    // batch: graph of vertex vbase + r
    const int64_t *gvbase = nullptr; // batch: first vertex of every graph
    int nkeys = 1;                   // graphs of the batch
    int64_t max_m = 0;               // vertices of the largest of them
};

// Triangle count of the input by degree order, added to sums[0] (or, with
// keys, to sums[key]).  facts: the content check's counters; sample: what
// tri_sample added up.  *done is false, and nothing is added, where the product
// over the given order is the better or only choice.
int tri_count(const TriInput &in, const CsrCheckOut &facts, unsigned long long sample, unsigned long long *sums,
              cudaStream_t s, bool *done);
// Adds nnz(L_k) over the columns k of min(nnz, TRI_SAMPLE) entries to *sum (the
// work of the product per entry); reads nothing through a matrix that the check
// refused (chk, may be null).
constexpr int TRI_SAMPLE = 16384;
int tri_sample(const TriInput &in, const CsrCheckOut *chk, unsigned long long *sum, cudaStream_t s);

// Support of every edge (the triangles it lies on) of the graph whose strict
// lower triangle is L.  An edge's number is the place of its column in its row's
// storage: unit * 8 + position in the unit (find it with tri_edge); rows keep
// no hub class here.  false in *done: numbers beyond 32 bits (no room: GK_ERR_OOM).
struct TriSupport {
    TriGraph g;
    const uint32_t *rank = nullptr;  // of every vertex
    int32_t *sup = nullptr;          // per edge number
    int64_t numbers = 0;             // edge numbers lie below it
};
int tri_support(const DevCsr &L, TriSupport *out, cudaStream_t s, Scratch &scr, bool *done);

// Number of the edge between the vertices of rank a and b, which exists.
__device__ __forceinline__ uint32_t tri_edge(const TriGraph &g, uint32_t a, uint32_t b) {
    const uint32_t i = a > b ? a : b, k = a > b ? b : a;
    const uint2 w = __ldg(g.shape + i);
    const uint32_t lows = w.x >> 16, v0 = __ldg(g.vstart + i);
    const uint16_t *lc = reinterpret_cast<const uint16_t *>(g.units + v0);
    uint32_t lo = 0, hi = lows;
    while (lo < hi) {
        const uint32_t md = (lo + hi) >> 1;
        if ((__ldg(lc + md) ^ 31u) < k) lo = md + 1;
        else hi = md;
    }
    if (lo < lows) return 8 * v0 + lo;
    const uint32_t v1 = v0 + (lows + 7) / 8;
    const uint32_t *hc = reinterpret_cast<const uint32_t *>(g.units + v1);
    lo = 0;
    hi = w.y - lows;
    while (lo < hi) {
        const uint32_t md = (lo + hi) >> 1;
        if (__ldg(hc + md) < k) lo = md + 1;
        else hi = md;
    }
    return 8 * (v1 + (lo >> 2)) + (lo & 3u);
}

// Sum of C<L> = L·L over the given order, for graphs small enough
// (tri_small_fits); any square pattern.  Everything is queued without a
// synchronisation: chk is the content check's result, whose defects keep the
// kernels from reading L (null: not checked), sample a zeroed word.
bool tri_small_fits(int64_t m, int64_t nnz);
int tri_count_small(const DevCsr &L, const CsrCheckOut *chk, unsigned long long *sample, unsigned long long *sum,
                    cudaStream_t s);

// Graphs of a batch (device arrays, not yet checked): the sampled work per entry
// of each, by which a graph is walked (below the limit) or reordered.  One graph
// pays the orientation's launches for itself, a batch's graphs share them (409
// uneven graphs, GPU time: limit 80 16.5 ms, 40 15.9, 20 16.0).
constexpr int TRI_WALK_WORK = 80, TRI_WALK_WORK_BATCH = 40;
struct TriGraphRef {
    const int64_t *rp;
    const int32_t *col;
    int64_t m, nnz;
};
int tri_sample_graphs(const TriGraphRef *graphs, int n, float *per_entry, cudaStream_t s);

}  // namespace gk
