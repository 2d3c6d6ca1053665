// k-truss on the GPU: gk_ktruss.
//
// Reference: k_truss (src/main.cpp:94-141): repeat Tmp<C> = C·C, drop the
// entries with support < k-2 (keeping the others with value 1), until nnz
// stops changing, at most n passes.  The reference compacts serially on the
// host (:110-119); here one pass is
//   1. support  S<C> = C·C (plus-pair) with the masked SpGEMM engine (EPI_WRITE);
//               for a symmetric C only its lower triangle is computed (below)
//   2. flag     keep[j] = S[j] >= k-2
//   3. scan     exclusive prefix of keep over all entries (one device scan)
//   4. compact  new_rp[i] = pos[rp[i]], new_col[pos[j]] = col[j] for kept j
//   5. copy the pruned matrix back over the current one
// and the loop stops when the kept count equals nnz.  Compaction preserves the
// order within rows, so rows stay sorted and the edge set is bit-exact with the
// reference (whose View-size defect at :99/:118 is not reproduced).
// A symmetric pattern without diagonal entries (an undirected graph) takes
// another way to the same passes (ktruss_peel below): the support of every edge
// is computed once, in degree order (tri.cu), and a pass then only visits the
// edges that the pass before left below k-2, taking their triangles off the
// other two edges.  These passes are short, so several are queued at once.
// For other patterns every pass reads its sizes on the device, so the loop is one
// CUDA graph: a conditional while node around one captured pass, the condition
// set by the pass's last kernel; the host waits once, at the end.  With profiling
// on (its events cannot be captured) the host runs the passes itself.
#include <cub/cub.cuh>

#include <algorithm>

#include "gk_common.cuh"
#include "gk_device.cuh"
#include "gk_spgemm.cuh"
#include "gk_tri.cuh"

namespace gk {

// Loop state in device memory, so that a pass needs no host value.
struct KtState {
    long long iters;   // passes run
    long long kept;    // nnz after the last pass
};

// keep[j] = S[j] >= k-2 for j < nnz (nnz = rp[m]); 0 up to the capacity, so
// that a scan over capacity+1 entries yields the kept count at pos[cap].
__global__ void k_keep_flags(const int32_t *sup, const int64_t *rp, int64_t m, int64_t cap, int thresh,
                             int32_t *keep) {
    const int64_t nnz = rp[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j <= cap; j += stride)
        keep[j] = j < nnz ? (sup[j] >= thresh) : 0;
}

__global__ void k_compact(int64_t m, const int64_t *rp, const int32_t *col, const int32_t *keep, const int64_t *pos,
                          int64_t *nrp, int32_t *ncol) {
    const int64_t nnz = rp[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += stride)
        if (keep[j]) ncol[pos[j]] = col[j];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= m; i += stride) nrp[i] = pos[rp[i]];
}

// End of a pass: count it and decide whether another pass follows (the edge
// count changed and fewer than max_iters passes ran).  Inside the graph the
// decision drives the conditional while node.
__global__ void k_pass_end(const int64_t *rp, const int64_t *nrp, int64_t m, long long max_iters, KtState *st,
                           cudaGraphConditionalHandle h, int in_graph) {
    const long long old = rp[m], kept = nrp[m];
    const long long it = st->iters + 1;
    st->iters = it;
    st->kept = kept;
    if (in_graph) cudaGraphSetConditional(h, (kept != old && it < max_iters) ? 1u : 0u);
}

// The pruned matrix becomes the current one.
__global__ void k_copy_back(int64_t m, const int64_t *nrp, const int32_t *ncol, int64_t *rp, int32_t *col) {
    const int64_t nnz = nrp[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= m; i += stride) rp[i] = nrp[i];
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += stride) col[j] = ncol[j];
}

// ---- symmetric input: support on the lower triangle only -------------------
// For a symmetric C, S = C·C is symmetric (S_ij = |N(i) ∩ N(j)| = S_ji), so the
// pass computes S<L> = C·C with L the strict lower triangle of C and reads the
// support of an upper entry (i, j > i) at its mirror (j, i) in L.  The B rows
// streamed for row i then stop at row i's largest lower column (the engine
// ends a B row past the mask's last column), which roughly halves the streamed
// entries.  The values are the same integers, so the truss is unchanged.

// Row index of every entry (warp per row, coalesced stores).  The per-entry
// kernels below then spread their work over entries, not rows: with a warp per
// row, a hub row of 10^5 entries is one warp's serial loop of binary searches
// and sets the kernel's duration.  (An equal part of the entries per warp took
// longer here, RMAT-20 0.27 ms against 0.19: the searches for the row.)
__global__ void k_row_of(int64_t m, const int64_t *rp, int32_t *row) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < m; i += warps)
        for (int64_t p = rp[i] + lane; p < rp[i + 1]; p += 32) row[p] = static_cast<int32_t>(i);
}

// Whether every entry (i, j) has its mirror (j, i): a thread per entry, a binary
// search in row j.  Only the entries that lead to a shorter row (to a smaller
// index among equals) are searched for: one of every pair, and if all of them
// have a mirror and are half of the entries off the diagonal, the mirrors are
// the other half (RMAT-20 1.03 -> 0.66 ms).
struct SymFacts {
    unsigned long long searched, diagonal, missing;
    bool symmetric(int64_t nnz) const {
        return missing == 0 && 2 * searched + diagonal == static_cast<unsigned long long>(nnz);
    }
};

__global__ void __launch_bounds__(256) k_sym_check(int64_t m, const int64_t *rp, const int32_t *col,
                                                   const int32_t *row, SymFacts *facts) {
    __shared__ unsigned long long red[8];
    const int64_t nnz = rp[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    unsigned int searched = 0, diagonal = 0, missing = 0;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += stride) {
        const int i = row[p], j = col[p];
        int64_t lo = rp[j], hi = rp[j + 1];
        const int64_t end = hi, mine = rp[i + 1] - rp[i];
        diagonal += i == j;
        if (hi - lo > mine || (hi - lo == mine && j >= i)) continue;
        ++searched;
        while (lo < hi) {
            const int64_t md = (lo + hi) >> 1;
            if (col[md] < i) lo = md + 1;
            else hi = md;
        }
        missing += lo == end || col[lo] != i;
    }
    const unsigned long long s = block_sum(static_cast<unsigned long long>(searched), red);
    const unsigned long long d = block_sum(static_cast<unsigned long long>(diagonal), red);
    const unsigned long long x = block_sum(static_cast<unsigned long long>(missing), red);
    if (threadIdx.x == 0) {
        if (s) atomicAdd(&facts->searched, s);
        if (d) atomicAdd(&facts->diagonal, d);
        if (x) atomicAdd(&facts->missing, x);
    }
}

// Entries of row i below the diagonal (a prefix of the sorted row).
__global__ void k_lower_len(int64_t m, const int64_t *rp, const int32_t *col, int64_t *len) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
        int64_t lo = rp[i], hi = rp[i + 1];
        while (lo < hi) {
            const int64_t md = (lo + hi) >> 1;
            if (col[md] < i) lo = md + 1;
            else hi = md;
        }
        len[i] = lo - rp[i];
    }
}

// Lower-triangle columns, a thread per entry of C (balanced over entries).
__global__ void k_lower_fill(int64_t m, const int64_t *rp, const int32_t *col, const int32_t *row,
                             const int64_t *lrp, int32_t *lcol) {
    const int64_t nnz = rp[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += stride) {
        const int i = row[p], j = col[p];
        const int64_t off = p - rp[i];  // below llen[i] for every j < i of a sorted row
        if (j < i && off < lrp[i + 1] - lrp[i]) lcol[lrp[i] + off] = j;
    }
}

// keep[p] for every entry of C from the lower supports, a thread per entry: a
// lower entry reads its own position in L, an upper entry (i, j) the position
// of i in L's row j (binary search).
__global__ void k_keep_sym(int64_t m, int64_t cap, const int64_t *rp, const int32_t *col, const int32_t *row,
                           const int64_t *lrp, const int32_t *lcol, const int32_t *sup, int thresh, int32_t *keep) {
    const int64_t nnz = rp[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += stride) {
        const int i = row[p], j = col[p];
        int64_t q;
        if (j < i) {
            q = lrp[i] + (p - rp[i]);
        } else {
            int64_t lo = lrp[j], hi = lrp[j + 1];
            const int64_t end = hi;
            while (lo < hi) {
                const int64_t md = (lo + hi) >> 1;
                if (lcol[md] < i) lo = md + 1;
                else hi = md;
            }
            q = (lo < end && lcol[lo] == i) ? lo : -1;
        }
        keep[p] = (q >= 0 && sup[q] >= thresh) ? 1 : 0;
    }
    for (int64_t p = nnz + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p <= cap; p += stride) keep[p] = 0;
}

// keep[p] for every entry off the diagonal.
__global__ void k_keep_edges(int64_t m, int64_t cap, const int64_t *rp, const int32_t *col, const int32_t *row,
                             int32_t *keep) {
    const int64_t nnz = rp[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p <= cap; p += stride)
        keep[p] = p < nnz && row[p] != col[p];
}

struct KtBuffers {
    int64_t m, cap;            // rows, nnz of the input (capacity of every edge array)
    int64_t *rp, *nrp;         // current / pruned row pointers
    int32_t *col, *ncol;       // current / pruned columns
    int32_t *sup, *keep;       // support per entry, keep flags (cap + 1)
    int64_t *pos;              // exclusive scan of keep (cap + 1)
    void *scan_tmp;
    size_t scan_bytes;
    void *arena;               // scratch of the support SpGEMM
    size_t arena_bytes;
    KtState *st;
    int k, sched;
    bool sym;                  // symmetric input: support on the lower triangle
    int64_t *llen, *lrp;       // lower-triangle lengths (m + 1) and row pointers (m + 1)
    int32_t *lcol;             // lower-triangle columns
    int32_t *row;              // row index of every entry of the current matrix
};

// One pass: support S<C> = C·C, flags, scan, compaction, pass end, copy back.
// Every size is read on the device, so the same launches serve every pass.
static int ktruss_pass(const KtBuffers &b, cudaStream_t s, cudaGraphConditionalHandle h, bool in_graph) {
    const int sms = ctx().num_sms;
    Scratch pass(s, b.arena, b.arena_bytes);
    SpgemmRequest rq;
    DevCsr c{b.m, b.m, b.cap, b.rp, b.col, nullptr};
    rq.A = rq.B = rq.M = c;
    rq.epi = EPI_WRITE;
    rq.sched = b.sched;
    rq.c_val = b.sup;
    rq.stream = s;
    size_t scan_bytes = b.scan_bytes;
    if (b.sym) {
        k_row_of<<<sms * 8, 256, 0, s>>>(b.m, b.rp, b.row);
        k_lower_len<<<sms * 4, 256, 0, s>>>(b.m, b.rp, b.col, b.llen);
        GK_CUDA(cub::DeviceScan::ExclusiveSum(b.scan_tmp, scan_bytes, b.llen, b.lrp, b.m + 1, s));
        k_lower_fill<<<sms * 8, 256, 0, s>>>(b.m, b.rp, b.col, b.row, b.lrp, b.lcol);
        rq.M = DevCsr{b.m, b.m, b.cap, b.lrp, b.lcol, nullptr};
        GK_CHECK(run_spgemm(rq, pass));
        k_keep_sym<<<sms * 8, 256, 0, s>>>(b.m, b.cap, b.rp, b.col, b.row, b.lrp, b.lcol, b.sup, b.k - 2, b.keep);
        note_launches(4);
    } else {
        GK_CHECK(run_spgemm(rq, pass));
        k_keep_flags<<<sms * 8, 256, 0, s>>>(b.sup, b.rp, b.m, b.cap, b.k - 2, b.keep);
        note_launches(1);
    }
    scan_bytes = b.scan_bytes;
    GK_CUDA(cub::DeviceScan::ExclusiveSum(b.scan_tmp, scan_bytes, b.keep, b.pos, b.cap + 1, s));
    k_compact<<<sms * 8, 256, 0, s>>>(b.m, b.rp, b.col, b.keep, b.pos, b.nrp, b.ncol);
    k_pass_end<<<1, 1, 0, s>>>(b.rp, b.nrp, b.m, static_cast<long long>(b.m), b.st, h, in_graph ? 1 : 0);
    k_copy_back<<<sms * 8, 256, 0, s>>>(b.m, b.nrp, b.ncol, b.rp, b.col);
    note_launches(5);
    GK_CUDA(cudaGetLastError());
    return GK_OK;
}

// A loop as one CUDA graph: a conditional while node whose body is `pass`
// (captured once: pass(stream, handle) queues it and returns a status), launched
// on s.  Returns GK_ERR_UNSUPPORTED where the graph cannot be built (the caller
// then runs the passes from the host).
template <class F>
static int while_graph(cudaStream_t s, int *launches_per_pass, F pass) {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t cs = nullptr;
    int status = GK_OK;
    do {
        if (cudaGraphCreate(&g, 0) != cudaSuccess) { status = GK_ERR_UNSUPPORTED; break; }
        cudaGraphConditionalHandle h;
        if (cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault) != cudaSuccess) {
            status = GK_ERR_UNSUPPORTED;
            break;
        }
        cudaGraphNodeParams np = {};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        cudaGraphNode_t node;
        if (cudaGraphAddNode(&node, g, nullptr, 0, &np) != cudaSuccess) { status = GK_ERR_UNSUPPORTED; break; }
        cudaGraph_t body = np.conditional.phGraph_out[0];
        if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) { status = GK_ERR_UNSUPPORTED; break; }
        if (cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) !=
            cudaSuccess) {
            status = GK_ERR_UNSUPPORTED;
            break;
        }
        const int64_t before = launches_noted();
        const int ps = pass(cs, h);
        *launches_per_pass = static_cast<int>(launches_noted() - before);
        cudaGraph_t captured = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(cs, &captured);
        if (ps != GK_OK) { status = ps; break; }
        if (ce != cudaSuccess) { status = cuda_fail(ce, "k-truss pass capture"); break; }
        if (cudaGraphInstantiate(&exec, g, 0) != cudaSuccess) {
            cudaGetLastError();
            status = GK_ERR_UNSUPPORTED;
            break;
        }
        const cudaError_t le = cudaGraphLaunch(exec, s);
        if (le != cudaSuccess) status = cuda_fail(le, "k-truss graph launch");
    } while (false);
    if (exec) cudaGraphExecDestroy(exec);
    if (g) cudaGraphDestroy(g);
    if (cs) cudaStreamDestroy(cs);
    return status;
}

// ---- undirected graphs: support once, then peeling ---------------------------
// The support product of one pass costs the same whatever the pass before
// removed, and every pass needed it again (RMAT-20, k = 5: 11 passes, 45 ms
// each).  Here: support once 3.3 ms, all passes 3.1 ms, the call 500 -> 10.7 ms;
// RMAT-13, k = 4: 20 -> 0.63 ms.
// Loop state: pass t works on the list of the edges removed in it (support
// below k-2 after the passes before), mark[e] = t for those; an edge with mark 0
// or above t is still there when pass t starts.
struct PeelState {
    unsigned int pass, iters, done, fetch;
    unsigned int n[2];           // edges of pass t at [t & 1], of pass t + 1 at the other
};

struct PeelArgs {
    int64_t m;
    const int64_t *rp;
    const int32_t *col, *row;
    const uint32_t *eid;  // edge number of every entry
    int32_t *sup;
    uint32_t *mark;
    uint32_t *list[2];    // entries (one of an edge's two) of the edges of a pass
    int thresh;
    PeelState *st;
};

// Edge numbers of all entries; the edges below the threshold are pass 1's.
__global__ void __launch_bounds__(256) k_peel_begin(PeelArgs a, TriGraph g, const uint32_t *__restrict__ rank,
                                                    uint32_t *eid) {
    const int64_t nnz = a.rp[a.m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); b < nnz; b += stride) {
        const int64_t p = b + lane;
        bool low = false;
        uint32_t e = 0;
        if (p < nnz) {
            const int i = a.row[p], j = a.col[p];
            e = tri_edge(g, __ldg(rank + i), __ldg(rank + j));
            eid[p] = e;
            low = j < i && a.sup[e] < a.thresh;
        }
        const unsigned lm = __ballot_sync(0xFFFFFFFFu, low);
        uint32_t at = 0;
        if (lane == 0 && lm) at = atomicAdd(&a.st->n[1], static_cast<unsigned>(__popc(lm)));
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(lm & ((1u << lane) - 1u));
        if (low) {
            a.mark[e] = 1;
            a.list[1][at] = static_cast<uint32_t>(p);
        }
    }
}

// One triangle less on edge e (entry p); falling below the threshold it joins
// the next pass.
__device__ __forceinline__ void peel_take(const PeelArgs &a, uint32_t e, int64_t p, uint32_t t) {
    if (atomicSub(a.sup + e, 1) == a.thresh) {
        a.mark[e] = t + 1;
        a.list[(t + 1) & 1][atomicAdd(&a.st->n[(t + 1) & 1], 1u)] = static_cast<uint32_t>(p);
    }
}

// Pass t: a warp per removed edge (u, v).  Its triangles are the neighbours w of
// the endpoint with the shorter row that the other row holds (binary search),
// both edges still there when the pass started.  A triangle that loses several
// edges in this pass is taken off once, by the one with the smallest number.
// An edge without triangles left needs no visit, and a visit ends when all of
// them are found.
__global__ void __launch_bounds__(256) k_peel_pass(PeelArgs a) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    if (a.st->done) return;
    const uint32_t t = a.st->pass, n = a.st->n[t & 1];
    const uint32_t *__restrict__ list = a.list[t & 1];
    const int lane = threadIdx.x & 31;
    for (;;) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&a.st->fetch, 32u);
        at = __shfl_sync(FULL, at, 0);
        if (at >= n) break;
        // 32 edges: those with triangles left, one by one
        uint32_t mine = 0, e0 = 0;
        int left = 0;
        if (at + lane < n) {
            mine = list[at + lane];
            e0 = a.eid[mine];
            left = a.sup[e0];
        }
        for (unsigned todo = __ballot_sync(FULL, left > 0); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const uint32_t p0 = __shfl_sync(FULL, mine, src), e = __shfl_sync(FULL, e0, src);
            int need = __shfl_sync(FULL, left, src);
            int u = a.row[p0], v = a.col[p0];
            int64_t u0 = a.rp[u], u1 = a.rp[u + 1], v0 = a.rp[v], v1 = a.rp[v + 1];
            if (u1 - u0 > v1 - v0) {
                int64_t z = u0;
                u0 = v0;
                v0 = z;
                z = u1;
                u1 = v1;
                v1 = z;
                const int y = u;
                u = v;
                v = y;
            }
            for (int64_t b = u0; b < u1 && need > 0; b += 32) {
                const int64_t p1 = b + lane;
                bool tri = false;
                uint32_t e1 = 0, e2 = 0, m1 = 0, m2 = 0;
                int64_t p2 = 0;
                if (p1 < u1) {
                    const int w = __ldg(a.col + p1);
                    e1 = __ldg(a.eid + p1);
                    m1 = a.mark[e1];
                    if (w != v && (m1 == 0 || m1 >= t)) {
                        int64_t lo = v0, hi = v1;
                        while (lo < hi) {
                            const int64_t md = (lo + hi) >> 1;
                            if (__ldg(a.col + md) < w) lo = md + 1;
                            else hi = md;
                        }
                        if (lo < v1 && __ldg(a.col + lo) == w) {
                            p2 = lo;
                            e2 = __ldg(a.eid + p2);
                            m2 = a.mark[e2];
                            tri = m2 == 0 || m2 >= t;
                        }
                    }
                }
                need -= __popc(__ballot_sync(FULL, tri));
                if (tri) {
                    const bool in1 = m1 == t, in2 = m2 == t;
                    if (!in1 && (!in2 || e < e2)) peel_take(a, e1, p1, t);
                    if (!in2 && (!in1 || e < e1)) peel_take(a, e2, p2, t);
                }
            }
        }
    }
}

// End of a pass: a pass that removed nothing, or the m-th, is the last one.
__global__ void k_peel_end(PeelState *st, unsigned int max_iters) {
    if (st->done) return;
    const unsigned int t = st->pass, n = st->n[t & 1];
    st->iters = t;
    if (n > 0 && t < max_iters) {
        st->n[t & 1] = 0;
        st->fetch = 0;
        st->pass = t + 1;
    } else {
        st->done = 1;
    }
}

__global__ void __launch_bounds__(256) k_peel_keep(PeelArgs a, int64_t cap, int32_t *keep) {
    const uint32_t last = a.st->iters;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p <= cap; p += stride) {
        int k = 0;
        if (p < cap) {
            const uint32_t mk = a.mark[a.eid[p]];
            k = mk == 0 || mk > last;
        }
        keep[p] = k;
    }
}

// Passes queued before the host looks whether the last one is among them; more
// once there are many (half as many as have run, so that few are queued in vain).
// A pass queued behind the last one does nothing (4 us); a graph with the loop in
// it took 0.3 ms to build (RMAT-13, five passes: the call 0.78 -> 0.63 ms).
constexpr int PEEL_AHEAD = 8;

// What the passes work on, and the truss's arrays (in scr, which outlives the call's
// own scratch).
struct PeelBuffers {
    TriSupport ts;
    PeelArgs a;
    uint32_t *eid;
    int32_t *keep;
    int64_t *pos;
    char *scan_tmp;
    size_t scan_bytes;
    int64_t *rp_res;
    int32_t *col_res;
    bool ok = false;
};

// The supports, and every allocation.
static int peel_prepare(int64_t m, int64_t nnz, const int64_t *rp, const int32_t *col, const int32_t *row, int k,
                        PeelBuffers *out, cudaStream_t s, Scratch &own, Scratch &scr) {
    const int sms = ctx().num_sms;
    const int64_t E = nnz / 2;
    int64_t *len, *lrp;
    int32_t *lcol;
    size_t sb = 0, kb = 0;
    GK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, sb, static_cast<int64_t *>(nullptr),
                                          static_cast<int64_t *>(nullptr), m + 1, s));
    GK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, kb, static_cast<int32_t *>(nullptr),
                                          static_cast<int64_t *>(nullptr), nnz + 1, s));
    out->scan_bytes = kb;
    GK_CHECK(own.alloc(&out->scan_tmp, sb > kb ? sb : kb));
    Scratch low(s);  // the lower triangle, needed for the support only
    GK_CHECK(low.alloc(&len, m + 1));
    GK_CHECK(low.alloc(&lrp, m + 1));
    GK_CHECK(low.alloc(&lcol, E));
    GK_CUDA(cudaMemsetAsync(len + m, 0, sizeof(int64_t), s));
    k_lower_len<<<sms * 4, 256, 0, s>>>(m, rp, col, len);
    GK_CUDA(cub::DeviceScan::ExclusiveSum(out->scan_tmp, sb, len, lrp, m + 1, s));
    k_lower_fill<<<sms * 8, 256, 0, s>>>(m, rp, col, row, lrp, lcol);
    note_launches(2);
    GK_CUDA(cudaGetLastError());
    GK_CHECK(tri_support(DevCsr{m, m, E, lrp, lcol, nullptr}, &out->ts, s, own, &out->ok));
    if (!out->ok) return GK_OK;
    low.release();
    PeelArgs &a = out->a;
    a.m = m;
    a.rp = rp;
    a.col = col;
    a.row = row;
    a.sup = out->ts.sup;
    a.thresh = k - 2;
    GK_CHECK(own.alloc(&out->eid, nnz));
    GK_CHECK(own.alloc(&a.mark, out->ts.numbers));
    GK_CHECK(own.alloc(&a.list[0], E));
    GK_CHECK(own.alloc(&a.list[1], E));
    GK_CHECK(own.alloc(&a.st, 1));
    GK_CHECK(own.alloc(&out->keep, nnz + 1));
    GK_CHECK(own.alloc(&out->pos, nnz + 1));
    GK_CHECK(scr.alloc(&out->rp_res, m + 1));
    return scr.alloc(&out->col_res, nnz);
}

// k-truss of an undirected graph (rp, col: symmetric, sorted, no diagonal; row:
// every entry's row); the truss is left in rp_res / col_res (scratch).  false in
// *done: no room for it, and what it took has been given back.
static int ktruss_peel(int64_t m, int64_t nnz, const int64_t *rp, const int32_t *col, const int32_t *row, int k,
                       int *iters_out, int64_t *nnz_out, int64_t **rp_res, int32_t **col_res, cudaStream_t s,
                       Scratch &scr, bool *done) {
    *done = false;
    if (nnz >= (int64_t(1) << 32)) return GK_OK;
    const int sms = ctx().num_sms;
    Scratch own(s);
    PeelBuffers b;
    const int status = peel_prepare(m, nnz, rp, col, row, k, &b, s, own, scr);
    if (status == GK_ERR_OOM) {
        own.release();
        scratch_reclaim(s);
        return GK_OK;
    }
    GK_CHECK(status);
    if (!b.ok) return GK_OK;
    PeelArgs &a = b.a;
    const TriSupport &ts = b.ts;
    uint32_t *eid = b.eid;
    int32_t *keep = b.keep;
    int64_t *pos = b.pos;
    char *tmp = b.scan_tmp;
    size_t kb = b.scan_bytes;
    *rp_res = b.rp_res;
    *col_res = b.col_res;
    a.eid = eid;
    GK_CUDA(cudaMemsetAsync(a.mark, 0, sizeof(uint32_t) * ts.numbers, s));
    PeelState init{};
    init.pass = 1;
    GK_CUDA(cudaMemcpyAsync(a.st, &init, sizeof(init), cudaMemcpyHostToDevice, s));
    k_peel_begin<<<sms * 8, 256, 0, s>>>(a, ts.g, ts.rank, eid);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    const unsigned int max_iters = static_cast<unsigned int>(m);
    PeelState h{};
    while (!h.done) {
        const int ahead = std::max(PEEL_AHEAD, static_cast<int>(h.iters / 2));
        for (int t = 0; t < ahead; ++t) {
            k_peel_pass<<<sms * 8, 256, 0, s>>>(a);
            k_peel_end<<<1, 1, 0, s>>>(a.st, max_iters);
        }
        note_launches(2 * ahead);
        GK_CUDA(cudaGetLastError());
        GK_CUDA(cudaMemcpyAsync(&h, a.st, sizeof(h), cudaMemcpyDeviceToHost, s));
        GK_CUDA(cudaStreamSynchronize(s));
    }
    k_peel_keep<<<sms * 8, 256, 0, s>>>(a, nnz, keep);
    GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, kb, keep, pos, nnz + 1, s));
    k_compact<<<sms * 8, 256, 0, s>>>(m, rp, col, keep, pos, *rp_res, *col_res);
    note_launches(2);
    GK_CUDA(cudaGetLastError());
    GK_CUDA(cudaMemcpyAsync(nnz_out, pos + nnz, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    GK_CUDA(cudaStreamSynchronize(s));
    *iters_out = static_cast<int>(h.iters);
    *done = true;
    return GK_OK;
}

int ktruss_device(int64_t m, int64_t nnz0, int64_t *rp_a, int32_t *col_a, int k, int sched, int *iters_out,
                  int64_t *nnz_out, int64_t **rp_res, int32_t **col_res, cudaStream_t s, Scratch &scr) {
    NvtxRange range("gk:ktruss");
    *rp_res = rp_a;
    *col_res = col_a;
    if (nnz0 == 0 || m == 0) {  // the reference counts one pass over the empty matrix
        *iters_out = m > 0 ? 1 : 0;
        *nnz_out = 0;
        return GK_OK;
    }
    KtBuffers b;
    b.m = m;
    b.cap = nnz0;
    b.rp = rp_a;
    b.col = col_a;
    b.k = k;
    b.sched = sched;
    GK_CHECK(scr.alloc(&b.row, nnz0));
    bool loops = false;  // self-loops of a symmetric pattern
    {
        SymFacts *facts, h{};
        GK_CHECK(scr.alloc(&facts, 1));
        GK_CUDA(cudaMemsetAsync(facts, 0, sizeof(SymFacts), s));
        k_row_of<<<ctx().num_sms * 8, 256, 0, s>>>(m, rp_a, b.row);
        k_sym_check<<<ctx().num_sms * 8, 256, 0, s>>>(m, rp_a, col_a, b.row, facts);
        note_launches(2);
        GK_CUDA(cudaMemcpyAsync(&h, facts, sizeof(h), cudaMemcpyDeviceToHost, s));
        GK_CUDA(cudaStreamSynchronize(s));
        // the supports on the lower triangle leave self-loops out, which the product
        // counts (a loop at i supports every edge of i): those take the full mask
        b.sym = h.symmetric(nnz0) && h.diagonal == 0;
        loops = h.symmetric(nnz0) && h.diagonal > 0;
        if (b.sym) {
            bool done = false;
            GK_CHECK(sched_prepare(sched, GK_ACCUM_AUTO));
            GK_CHECK(ktruss_peel(m, nnz0, rp_a, col_a, b.row, k, iters_out, nnz_out, rp_res, col_res, s, scr, &done));
            if (done) return GK_OK;
        }
    }
    GK_CHECK(scr.alloc(&b.nrp, m + 1));
    GK_CHECK(scr.alloc(&b.ncol, nnz0));
    GK_CHECK(scr.alloc(&b.sup, nnz0));
    GK_CHECK(scr.alloc(&b.keep, nnz0 + 1));
    GK_CHECK(scr.alloc(&b.pos, nnz0 + 1));
    GK_CHECK(scr.alloc(&b.st, 1));
    GK_CHECK(scr.alloc(&b.llen, m + 1));
    GK_CHECK(scr.alloc(&b.lrp, m + 1));
    GK_CHECK(scr.alloc(&b.lcol, nnz0));
    GK_CUDA(cudaMemsetAsync(b.llen + m, 0, sizeof(int64_t), s));
    b.scan_bytes = 0;
    GK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b.scan_bytes, b.keep, b.pos, nnz0 + 1, s));
    {
        size_t lb = 0;
        GK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, lb, b.llen, b.lrp, m + 1, s));
        if (lb > b.scan_bytes) b.scan_bytes = lb;
    }
    GK_CHECK(scr.alloc(reinterpret_cast<char **>(&b.scan_tmp), b.scan_bytes));
    b.arena_bytes = spgemm_scratch_bytes(m);
    GK_CHECK(scr.alloc(reinterpret_cast<char **>(&b.arena), b.arena_bytes));
    GK_CUDA(cudaMemsetAsync(b.st, 0, sizeof(KtState), s));
    GK_CHECK(spgemm_prepare(EPI_WRITE, false, sched, GK_ACCUM_AUTO));

    int status = GK_ERR_UNSUPPORTED;
    int per_pass = 0;
    if (!prof_any())
        status = while_graph(s, &per_pass, [&](cudaStream_t cs, cudaGraphConditionalHandle gh) {
            return ktruss_pass(b, cs, gh, true);
        });
    KtState h{};
    if (status == GK_OK) {
        GK_CUDA(cudaMemcpyAsync(&h, b.st, sizeof(KtState), cudaMemcpyDeviceToHost, s));
        GK_CUDA(cudaStreamSynchronize(s));
        note_launches(static_cast<int>(per_pass * (h.iters - 1)));  // replays beyond the captured pass
    } else if (status == GK_ERR_UNSUPPORTED) {
        // passes driven from the host (profiling on, or no conditional graphs)
        long long prev = nnz0;
        for (int64_t t = 0; t < m; ++t) {
            GK_CHECK(ktruss_pass(b, s, cudaGraphConditionalHandle{}, false));
            GK_CUDA(cudaMemcpyAsync(&h, b.st, sizeof(KtState), cudaMemcpyDeviceToHost, s));
            GK_CUDA(cudaStreamSynchronize(s));
            if (h.kept == prev) break;
            prev = h.kept;
        }
    } else {
        return status;
    }
    *iters_out = static_cast<int>(h.iters);
    *nnz_out = h.kept;
    if (!loops) return GK_OK;
    // the truss of an undirected graph has no loops
    const int sms = ctx().num_sms;
    size_t scan_bytes = b.scan_bytes;
    k_row_of<<<sms * 8, 256, 0, s>>>(m, b.rp, b.row);
    k_keep_edges<<<sms * 8, 256, 0, s>>>(m, b.cap, b.rp, b.col, b.row, b.keep);
    GK_CUDA(cub::DeviceScan::ExclusiveSum(b.scan_tmp, scan_bytes, b.keep, b.pos, b.cap + 1, s));
    k_compact<<<sms * 8, 256, 0, s>>>(m, b.rp, b.col, b.keep, b.pos, b.nrp, b.ncol);
    note_launches(3);
    GK_CUDA(cudaGetLastError());
    GK_CUDA(cudaMemcpyAsync(nnz_out, b.pos + nnz0, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    GK_CUDA(cudaStreamSynchronize(s));
    *rp_res = b.nrp;
    *col_res = b.ncol;
    return GK_OK;
}

}  // namespace gk

using namespace gk;

extern "C" int gk_ktruss(gk_csr_mut *inout, int k, int *iters, int sched, void *stream) {
    if (!inout || !iters) return fail(GK_ERR_ARG, "gk_ktruss: null argument");
    if (k < 3) return fail(GK_ERR_ARG, "gk_ktruss: k must be >= 3");
    if (inout->m != inout->n) return fail(GK_ERR_ARG, "gk_ktruss: matrix must be square");
    if (inout->m < 0 || inout->nnz < 0 || !inout->rowptr || (inout->nnz > 0 && !inout->col))
        return fail(GK_ERR_ARG, "gk_ktruss: bad matrix");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Scratch scr(s);
    const int64_t m = inout->m, nnz0 = inout->nnz;
    const bool dev = is_device_pointer(inout->rowptr);
    int64_t *rp;
    int32_t *col;
    GK_CHECK(scr.alloc(&rp, m + 1));
    GK_CHECK(scr.alloc(&col, nnz0 > 0 ? nnz0 : 1));
    GK_CUDA(cudaMemcpyAsync(rp, inout->rowptr, sizeof(int64_t) * (m + 1), cudaMemcpyDefault, s));
    if (nnz0) GK_CUDA(cudaMemcpyAsync(col, inout->col, sizeof(int32_t) * nnz0, cudaMemcpyDefault, s));
    GK_CHECK(check_csr(DevCsr{m, m, nnz0, rp, col, nullptr}, CSR_SORTED, "graph", s, scr));
    int64_t nnz = 0;
    int64_t *rp_res;
    int32_t *col_res;
    GK_CHECK(ktruss_device(m, nnz0, rp, col, k, sched, iters, &nnz, &rp_res, &col_res, s, scr));
    GK_CUDA(cudaMemcpyAsync(inout->rowptr, rp_res, sizeof(int64_t) * (m + 1),
                            dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s));
    if (nnz) GK_CUDA(cudaMemcpyAsync(inout->col, col_res, sizeof(int32_t) * nnz,
                                     dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s));
    GK_CUDA(cudaStreamSynchronize(s));
    inout->nnz = nnz;
    return GK_OK;
}
