// Complement-masked product C<!M> = A·B: gk_mxmm_cmask.
//
// Reference: mxmm_msa_cmask (include/matrix_la.h:733-934).  Row i of C holds
// every column j reached by some product A(i,k)·B(k,j) — structurally, kept
// even where the sum is zero — that is not a column of M's row i, in
// ascending order, with the sum of the products.  The reference sizes C with
// a symbolic pass over a dense per-thread state array and then scans all B.n
// columns for every row to emit them in order (:834-843).
//
// Here a row is one CTA's (or warp's) work in shared memory, by its number of
// products (k_cmask_classes):
//   up to 256, or 2,048   k_cmask_hash: a hash of the columns and their sums;
//                         the columns that M's row does not hold are sorted
//   more                  k_cmask_map: windows of the columns as a bitmap;
//                         products set bits, M's row clears them, and prefix
//                         counts over the words give every column its place, at
//                         which a second reading of the products adds them up
// Such a row costs at least its windows, whatever it holds: calls with several
// windows a row and too few products for them take the sort of cmask_sort.cu
// (cm_sorts).
// A's entries are taken 32 at a time per warp and their B rows' elements packed
// onto the lanes, so that short B rows leave no lanes idle.  Nothing is written
// to memory but C itself: expanding all products as 64-bit keys, sorting and
// reducing them took 10.6 ms for the distance-two pairs of RMAT-13 (edge factor
// 8; both calls), 0.72 ms here.
// Two calls, as the reference's symbolic and numeric passes: without C_col the
// row pointers are computed; with them (and C_rowptr from the first call) the
// columns and values are written.
#include <cub/cub.cuh>

#include <algorithm>

#include "gk_cmask.cuh"
#include "gk_common.cuh"
#include "gk_device.cuh"

namespace gk {

constexpr int64_t CM_ROW_LIMIT = int64_t(1) << 31;  // products of a row (counts within a row are 32-bit)
constexpr int CM_WARP_WORK = 256, CM_CTA_WORK = 2048;  // products of the hash classes
// A window's CTA: 128 threads where a row's window is small, so that many rows
// are in flight (a row is a chain of a dozen dependent loads and barriers:
// RMAT-13's rows, symbolic call, 0.29 ms with 512 threads, 0.21 with 128); 512
// where a window's words alone are thousands.
constexpr int CM_SMALL_WIN = 15;
constexpr int CM_DENSE_WIN = 13;  // 32 KB of sums: six CTAs of 256 threads an SM
// Entries of a window summed in shared memory; wider ones are summed in C itself.
__host__ __device__ constexpr int cm_acc(int nt) { return 16 * nt; }
constexpr int CM_WIN_MAX = 19;  // log2 columns of a window at most (64 KB of bits, 64 KB of prefix counts)

struct CmaskState {
    CsrCheckOut chk[3];
    unsigned int n[3];      // rows of each class
    unsigned int fetch[3];  // next row of each class
    unsigned int mismatch;  // C_rowptr is not this product's
    unsigned int too_long;  // a row has CM_ROW_LIMIT products or more
    unsigned long long work, long_work, max_work;  // products: all, those of rows in windows, the longest row's
};

struct CmaskArgs {
    DevCsr A, B, M;
    bool values;
    const int64_t *crp;  // numeric call: C's row pointers
    int64_t *cnt;        // symbolic call: entries of every row
    int32_t *c_col, *c_val;
    uint32_t *rows;  // three lists of up to m rows
    int64_t *work;   // products of every row, where cm_sorts may want them (else null)
    CmaskState *st;
    int checked;  // the checks ran: nothing is read through a matrix that one of them refused
    int win;      // log2 columns of a window

    __device__ __forceinline__ bool ready() const {
        return !checked || (st->chk[0].sound() && st->chk[1].sound() && st->chk[2].sound());
    }
};

// Products of every row and its class.
__global__ void __launch_bounds__(256) k_cmask_classes(CmaskArgs a) {
    if (!a.ready()) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long all = 0, in_windows = 0, longest = 0;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < a.A.m; i += warps) {
        int64_t w = 0;
        for (int64_t t = a.A.rp[i] + lane; t < a.A.rp[i + 1]; t += 32) {
            const int k = a.A.col[t];
            w += a.B.rp[k + 1] - a.B.rp[k];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xFFFFFFFFu, w, o);
        if (lane != 0) continue;
        if (a.work) a.work[i] = w;
        if (w >= CM_ROW_LIMIT) {
            a.st->too_long = 1;
            continue;
        }
        if (w == 0) {
            if (a.cnt) a.cnt[i] = 0;
            else if (a.crp[i + 1] != a.crp[i]) a.st->mismatch = 1;
            continue;
        }
        // a window that covers all columns in few words is the cheaper structure
        // from a warp's work on
        const int c = w <= CM_WARP_WORK ? 0 : (w <= CM_CTA_WORK && a.B.n > (1 << 15) ? 1 : 2);
        a.rows[c * a.A.m + atomicAdd(&a.st->n[c], 1u)] = static_cast<uint32_t>(i);
        all += w;
        if (c == 2) in_windows += w;
        longest = max(longest, static_cast<unsigned long long>(w));
    }
    if (a.work && all) {
        atomicAdd(&a.st->work, all);
        atomicAdd(&a.st->long_work, in_windows);
        atomicMax(&a.st->max_work, longest);
    }
}

// f(column, product) for the products of A's entries t0 .. t1 - 1, dealt 32 at a
// time to the CTA's NW warps; each lane takes four elements of a B row.
template <int NW, class F>
__device__ __forceinline__ void cm_products(const CmaskArgs &a, int64_t t0, int64_t t1, F f) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t tb = t0 + 32 * warp; tb < t1; tb += 32 * NW) {
        const int64_t t = tb + lane;
        int64_t b0 = 0;
        uint32_t n = 0, av = 1;
        if (t < t1) {
            const int k = __ldg(a.A.col + t);
            b0 = __ldg(a.B.rp + k);
            n = static_cast<uint32_t>(__ldg(a.B.rp + k + 1) - b0);
            if (a.values && a.A.val) av = static_cast<uint32_t>(__ldg(a.A.val + t));
        }
        const uint32_t u = (n + 3) / 4;
        uint32_t incl = u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        for (uint32_t b = 0; b < total; b += 32) {
            const uint32_t at = b + lane;
            int j = 0;
#pragma unroll
            for (int s = 16; s > 0; s >>= 1)
                if (__shfl_sync(FULL, incl, j + s - 1) <= at) j += s;
            j &= 31;
            const uint32_t z = 4 * (at - __shfl_sync(FULL, incl - u, j));
            const uint32_t nj = __shfl_sync(FULL, n, j), aj = __shfl_sync(FULL, av, j);
            const int64_t bj = __shfl_sync(FULL, b0, j);
            if (at < total) {
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c)
                    if (z + c < nj) {
                        const int64_t p = bj + z + c;
                        const uint32_t bv = a.values && a.B.val ? static_cast<uint32_t>(__ldg(a.B.val + p)) : 1u;
                        f(static_cast<uint32_t>(__ldg(a.B.col + p)), aj * bv);
                    }
            }
        }
    }
}

// Whether the row's place in C is this product's: its length and, since the
// pointers are the caller's, the bounds of what is written.
__device__ __forceinline__ bool cm_place(const CmaskArgs &a, int64_t i, int64_t found) {
    const int64_t c0 = a.crp[i], c1 = a.crp[i + 1];
    return c1 - c0 == found && c0 >= 0 && c1 <= a.crp[a.A.m];
}

// A row in a hash of CAP slots (load at most one half): columns and their sums.
template <int NT, int CAP, int CLASS, bool FILL>
__global__ void __launch_bounds__(NT) k_cmask_hash(CmaskArgs a) {
    if (!a.ready()) return;
    extern __shared__ unsigned long long cm_list[];  // CAP / 2 sorted entries (numeric call), then the table
    unsigned long long *list = cm_list;
    int *keys = reinterpret_cast<int *>(cm_list + (FILL ? CAP / 2 : 0));
    uint32_t *sums = reinterpret_cast<uint32_t *>(keys + CAP);
    __shared__ uint32_t s_row, s_n;
    const uint32_t n = a.st->n[CLASS];
    for (;;) {
        if (threadIdx.x == 0) {
            s_row = atomicAdd(&a.st->fetch[CLASS], 1u);
            s_n = 0;
        }
        for (int z = threadIdx.x; z < CAP; z += NT) {
            keys[z] = -1;
            if (FILL) sums[z] = 0;
        }
        __syncthreads();
        if (s_row >= n) break;
        const int64_t i = a.rows[CLASS * a.A.m + s_row];
        cm_products<NT / 32>(a, a.A.rp[i], a.A.rp[i + 1], [&](uint32_t x, uint32_t prod) {
            uint32_t h = (x * 0x9E3779B1u) >> (32 - __builtin_ctz(CAP));
            for (int probe = 0; probe < CAP; ++probe, h = (h + 1) & (CAP - 1)) {
                const int old = atomicCAS(keys + h, -1, static_cast<int>(x));
                if (old == -1 || old == static_cast<int>(x)) {
                    if (FILL) atomicAdd(sums + h, prod);
                    break;
                }
            }
        });
        __syncthreads();
        const int64_t m0 = a.M.rp[i], m1 = a.M.rp[i + 1];
        for (int z = threadIdx.x; z < CAP; z += NT) {
            const int x = keys[z];
            if (x < 0) continue;
            int64_t lo = m0, hi = m1;
            while (lo < hi) {
                const int64_t md = (lo + hi) >> 1;
                if (__ldg(a.M.col + md) < x) lo = md + 1;
                else hi = md;
            }
            if (lo < m1 && __ldg(a.M.col + lo) == x) continue;
            const uint32_t at = atomicAdd(&s_n, 1u);
            if (FILL) list[at] = (static_cast<unsigned long long>(x) << 32) | sums[z];
        }
        __syncthreads();
        const uint32_t found = s_n;
        if (!FILL) {
            if (threadIdx.x == 0) a.cnt[i] = found;
        } else if (cm_place(a, i, found)) {
            uint32_t len = 2;
            while (len < found) len <<= 1;
            for (uint32_t z = found + threadIdx.x; z < len; z += NT) list[z] = ~0ull;
            __syncthreads();
            for (uint32_t size = 2; size <= len; size <<= 1)
                for (uint32_t d = size >> 1; d > 0; d >>= 1) {
                    for (uint32_t z = threadIdx.x; z < len / 2; z += NT) {
                        const uint32_t p = 2 * z - (z & (d - 1)), q = p + d;
                        const unsigned long long x = list[p], y = list[q];
                        if ((x > y) == ((p & size) == 0)) {
                            list[p] = y;
                            list[q] = x;
                        }
                    }
                    __syncthreads();
                }
            const int64_t c0 = a.crp[i];
            for (uint32_t z = threadIdx.x; z < found; z += NT) {
                a.c_col[c0 + z] = static_cast<int32_t>(list[z] >> 32);
                if (a.c_val) a.c_val[c0 + z] = static_cast<int32_t>(list[z] & 0xFFFFFFFFu);
            }
        } else if (threadIdx.x == 0) {
            a.st->mismatch = 1;
        }
        __syncthreads();
    }
}

// A row by windows of 2^win columns.
// With DENSE the sums of all columns of the window are kept, and the products
// are read once (RMAT-13's rows, numeric call: 0.76 -> 0.26 ms).
template <int NT, bool FILL, bool DENSE>
__global__ void __launch_bounds__(NT) k_cmask_map(CmaskArgs a) {
    if (!a.ready()) return;
    constexpr int NW = NT / 32, ACC = cm_acc(NT);
    extern __shared__ uint32_t cm_smem[];
    const uint32_t words = 1u << (a.win - 5);
    uint32_t *bits = cm_smem, *pre = bits + words, *acc = pre + words;  // pre, acc: numeric call
    __shared__ uint32_t s_row, s_warp[NW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t n = a.st->n[2];
    const uint32_t per = (words + NT - 1) / NT;  // words a thread counts
    for (;;) {
        if (threadIdx.x == 0) s_row = atomicAdd(&a.st->fetch[2], 1u);
        __syncthreads();
        if (s_row >= n) break;
        const int64_t i = a.rows[2 * a.A.m + s_row];
        const int64_t t0 = a.A.rp[i], t1 = a.A.rp[i + 1], m0 = a.M.rp[i], m1 = a.M.rp[i + 1];
        const int64_t c0 = FILL ? a.crp[i] : 0, room = FILL ? a.crp[i + 1] - c0 : 0;
        const bool fits = !FILL || (room >= 0 && c0 >= 0 && a.crp[i + 1] <= a.crp[a.A.m]);
        int64_t found = 0;
        for (int64_t w0 = 0; w0 < a.B.n; w0 += int64_t(1) << a.win) {
            const uint32_t base = static_cast<uint32_t>(w0);
            for (uint32_t z = threadIdx.x; z < words; z += NT) bits[z] = 0;
            if (FILL && DENSE)
                for (uint32_t z = threadIdx.x; z < 32 * words; z += NT) acc[z] = 0;
            __syncthreads();
            cm_products<NW>(a, t0, t1, [&](uint32_t x, uint32_t prod) {
                const uint32_t y = x - base;
                if (y < 32 * words) {
                    const uint32_t bit = 1u << (y & 31);
                    if (!(bits[y >> 5] & bit)) atomicOr(bits + (y >> 5), bit);
                    if (FILL && DENSE) atomicAdd(acc + y, prod);
                }
            });
            __syncthreads();
            // M's columns of the window
            int64_t lo = m0, hi = m1;
            while (lo < hi) {
                const int64_t md = (lo + hi) >> 1;
                if (__ldg(a.M.col + md) < w0) lo = md + 1;
                else hi = md;
            }
            for (int64_t q = lo + threadIdx.x; q < m1; q += NT) {
                const uint32_t y = static_cast<uint32_t>(__ldg(a.M.col + q)) - base;
                if (y >= 32 * words) break;
                atomicAnd(bits + (y >> 5), ~(1u << (y & 31)));
            }
            __syncthreads();
            // places: thread t counts its words, a scan over the threads
            const uint32_t z0 = min(threadIdx.x * per, words), z1 = min(z0 + per, words);
            uint32_t mine = 0;
            for (uint32_t z = z0; z < z1; ++z) mine += __popc(bits[z]);
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            uint32_t at = incl - mine, total = 0;
            for (int z = 0; z < NW; ++z) {
                if (z < warp) at += s_warp[z];
                total += s_warp[z];
            }
            if (FILL) {
                const bool write = fits && found + total <= room;
                const int64_t o = c0 + found;
                const bool local = total <= ACC;
                for (uint32_t z = z0; z < z1; ++z) {
                    pre[z] = at;
                    at += __popc(bits[z]);
                }
                if (write) {
                    if (!DENSE && a.c_val) {
                        if (local)
                            for (uint32_t z = threadIdx.x; z < total; z += NT) acc[z] = 0;
                        else
                            for (uint32_t z = threadIdx.x; z < total; z += NT) a.c_val[o + z] = 0;
                    }
                    __syncthreads();
                    // a word per warp, its columns side by side
                    for (uint32_t z = warp; z < words; z += NW) {
                        const uint32_t w = bits[z];
                        if (!((w >> lane) & 1u)) continue;
                        const int64_t place = o + pre[z] + __popc(w & ((1u << lane) - 1u));
                        a.c_col[place] = static_cast<int32_t>(base + 32 * z + lane);
                        if (DENSE && a.c_val) a.c_val[place] = static_cast<int32_t>(acc[32 * z + lane]);
                    }
                    if (!DENSE && a.c_val) {
                        cm_products<NW>(a, t0, t1, [&](uint32_t x, uint32_t prod) {
                            const uint32_t y = x - base;
                            if (y >= 32 * words) return;
                            const uint32_t w = bits[y >> 5], bit = 1u << (y & 31);
                            if (!(w & bit)) return;
                            const uint32_t place = pre[y >> 5] + __popc(w & (bit - 1));
                            if (local) atomicAdd(acc + place, prod);
                            else atomicAdd(reinterpret_cast<unsigned int *>(a.c_val + o + place), prod);
                        });
                        __syncthreads();
                        if (local)
                            for (uint32_t z = threadIdx.x; z < total; z += NT)
                                a.c_val[o + z] = static_cast<int32_t>(acc[z]);
                    }
                }
            }
            found += total;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            if (!FILL) a.cnt[i] = found;
            else if (!fits || found != room) a.st->mismatch = 1;
        }
        __syncthreads();
    }
}

template <int NT, int CAP, int CLASS, bool FILL>
static int launch_hash(const CmaskArgs &a, int per_sm, cudaStream_t s) {
    const size_t smem = FILL ? 12 * CAP : 4 * CAP;
    GK_CUDA(cudaFuncSetAttribute(k_cmask_hash<NT, CAP, CLASS, FILL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    k_cmask_hash<NT, CAP, CLASS, FILL><<<ctx().num_sms * per_sm, NT, smem, s>>>(a);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    return GK_OK;
}

template <int NT, bool FILL, bool DENSE>
static int launch_map(const CmaskArgs &a, cudaStream_t s) {
    const size_t words = size_t(1) << (a.win - 5);
    const size_t smem = FILL ? 8 * words + (DENSE ? 128 * words : 4 * cm_acc(NT)) : 4 * words;
    GK_CUDA(cudaFuncSetAttribute(k_cmask_map<NT, FILL, DENSE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    int per_sm = 0;
    GK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cmask_map<NT, FILL, DENSE>, NT, smem));
    k_cmask_map<NT, FILL, DENSE><<<ctx().num_sms * std::max(per_sm, 1), NT, smem, s>>>(a);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    return GK_OK;
}

static int launch_classes(const CmaskArgs &a, cudaStream_t s) {
    k_cmask_classes<<<ctx().num_sms * 8, 256, 0, s>>>(a);
    note_launches(1);
    GK_CUDA(cudaGetLastError());
    return GK_OK;
}

// Whether the sort is the better path for these rows: the estimates of both calls'
// times in us, fitted to the figures below (2^18 columns or fewer: never).  Windows
// cost 0.4 ms, a row 0.72 us a window spread over the SMs (clearing, counting and
// writing 2^14 words) and at least one SM's share of that, 9 us per million products a
// window, hashed rows 120; the sort 0.8 ms and 260 us per million products, and in
// every batch of 2^26 products the warp of the longest row is waited for (20 ms per
// million of its products).  ms, windows / sort, rows x products at columns:
//   20,000 x 2,400 at 2^19  15.4 / 11.8   2,000 x 3,000 at 2^20   3.6 / 2.2
//   20,000 x 4,500 at 2^19  17.3 / 23     2,000 x 3,000 at 2^24  47.4 / 2.2
//   20,000 x 12,000 at 2^20 35.8 / 66     2,000 x 30,000 at 2^24 62.4 / 15.3
//   5,000 x 40,000 at 2^21  27.8 / 71       200 x 500,000 at 2^24  51 / 105
constexpr int CM_SORT_WIN = 19;  // windows from which the question is asked
static bool cm_sorts(const CmaskState &st, int64_t n, int win, int sms) {
    if (st.n[2] == 0) return false;
    const double windows = static_cast<double>((n + (int64_t(1) << win) - 1) >> win);
    const double rows = std::max<double>(st.n[2], sms), work = static_cast<double>(st.work);
    const double by_windows = 400.0 + windows * (0.72 * rows + 9e-6 * st.long_work) + 1.2e-4 * (work - st.long_work);
    const double batches = std::max(1.0, work / double(1 << 26));
    const double by_sort = 800.0 + 2.6e-4 * work + 2.0 * batches * 0.02 * st.max_work;
    return by_sort < by_windows;
}

// All rows of a, read from its state as ready, by the sort.
static int cmask_by_sort(const CmaskArgs &a, cudaStream_t s, Scratch &scr) {
    int64_t *cnt = a.cnt;
    if (!cnt) GK_CHECK(scr.alloc(&cnt, a.A.m + 1));  // numeric call
    return cmask_by_sort(a.A, a.B, a.M, a.values, a.work, cnt, a.crp, a.crp ? a.c_col : nullptr, a.c_val,
                         &a.st->mismatch, s, scr);
}

template <bool FILL>
static int launch_rows(const CmaskArgs &a, cudaStream_t s) {
    // the class of the longest rows first
    if (FILL && a.win <= CM_DENSE_WIN) GK_CHECK((launch_map<256, FILL, FILL>(a, s)));
    else if (a.win <= CM_SMALL_WIN) GK_CHECK((launch_map<128, FILL, false>(a, s)));
    else GK_CHECK((launch_map<512, FILL, false>(a, s)));
    if (a.B.n > (1 << 15)) GK_CHECK((launch_hash<128, 2 * CM_CTA_WORK, 1, FILL>(a, 4, s)));
    GK_CHECK((launch_hash<32, 2 * CM_WARP_WORK, 0, FILL>(a, 32, s)));
    return GK_OK;
}

}  // namespace gk

using namespace gk;

extern "C" int gk_mxmm_cmask(const gk_csr *A, const gk_csr *B, const gk_csr *M, int semiring, int64_t *C_rowptr,
                             int32_t *C_col, int32_t *C_val, void *stream) {
    NvtxRange range("gk:mxmm_cmask");
    GK_CHECK(validate_csr_shape(A, "A"));
    GK_CHECK(validate_csr_shape(B, "B"));
    GK_CHECK(validate_csr_shape(M, "M"));
    if (A->m != M->m || A->n != B->m || B->n != M->n)
        return fail(GK_ERR_ARG, "shape mismatch: need A.m == M.m, A.n == B.m, B.n == M.n");
    if (semiring != GK_PLUS_TIMES && semiring != GK_PLUS_PAIR) return fail(GK_ERR_ARG, "unknown semiring");
    if (!C_rowptr) return fail(GK_ERR_ARG, "C_rowptr is null");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Scratch scr(s);
    CmaskArgs a{};
    GK_CHECK(stage_csr(A, &a.A, scr, s, nullptr, 0, "A"));
    GK_CHECK(stage_csr(B, &a.B, scr, s, nullptr, 0, "B"));
    GK_CHECK(stage_csr(M, &a.M, scr, s, nullptr, 0, "M"));
    a.values = semiring == GK_PLUS_TIMES;
    const int64_t m = A->m;
    const bool fill = C_col != nullptr;
    const bool check = csr_check_active(s);
    GK_CHECK(scr.alloc(&a.st, 1));
    GK_CUDA(cudaMemsetAsync(a.st, 0, sizeof(CmaskState), s));
    a.checked = check ? 1 : 0;
    // the checks and the rows are queued together and read back with one
    // synchronisation
    if (check) {
        GK_CHECK(launch_csr_check(a.A, CSR_STRUCTURE, &a.st->chk[0], s));
        GK_CHECK(launch_csr_check(a.B, CSR_STRUCTURE, &a.st->chk[1], s));
        GK_CHECK(launch_csr_check(a.M, CSR_SORTED, &a.st->chk[2], s));
    }
    GK_CHECK(scr.alloc(&a.rows, 3 * (m > 0 ? m : 1)));
    a.win = 10;
    while (a.win < CM_WIN_MAX && (int64_t(1) << a.win) < B->n) ++a.win;
    int64_t cnnz = 0;  // entries of C (numeric call with host outputs)
    int32_t *dcol = C_col, *dval = C_val;
    int64_t ends[2] = {0, 0};
    if (fill) {
        const bool rp_dev = is_device_pointer(C_rowptr);
        int64_t *drp = C_rowptr;
        if (!rp_dev) {
            GK_CHECK(scr.alloc(&drp, m + 1));
            GK_CUDA(cudaMemcpyAsync(drp, C_rowptr, sizeof(int64_t) * (m + 1), cudaMemcpyHostToDevice, s));
        }
        a.crp = drp;
        GK_CUDA(cudaMemcpyAsync(&ends[0], C_rowptr, sizeof(int64_t), cudaMemcpyDefault, s));
        GK_CUDA(cudaMemcpyAsync(&ends[1], C_rowptr + m, sizeof(int64_t), cudaMemcpyDefault, s));
        const bool host_col = !is_device_pointer(C_col), host_val = C_val && !is_device_pointer(C_val);
        if (host_col || host_val) {
            GK_CUDA(cudaStreamSynchronize(s));
            cnnz = ends[1] > 0 ? ends[1] : 0;
            if (ends[0] != 0) return fail(GK_ERR_ARG, "C_rowptr[0] must be 0 (pass the first call's row pointers)");
            if (host_col && cnnz > 0) GK_CHECK(scr.alloc(&dcol, cnnz));
            if (host_val && cnnz > 0) GK_CHECK(scr.alloc(&dval, cnnz));
        }
        a.c_col = dcol;
        a.c_val = dval;
    } else {
        GK_CHECK(scr.alloc(&a.cnt, m + 1));
        GK_CUDA(cudaMemsetAsync(a.cnt + m, 0, sizeof(int64_t), s));
    }
    const bool may_sort = m > 0 && a.win >= CM_SORT_WIN;
    if (may_sort) GK_CHECK(scr.alloc(&a.work, m));
    CmaskState h{};
    auto read_state = [&]() -> int {  // its defects, too
        GK_CUDA(cudaMemcpyAsync(&h, a.st, sizeof(h), cudaMemcpyDeviceToHost, s));
        GK_CUDA(cudaStreamSynchronize(s));
        if (check && !(h.chk[0].sound() && h.chk[1].sound() && h.chk[2].sound())) {
            GK_CHECK(check_csr(a.A, CSR_STRUCTURE, "A", s, scr));  // names the defect
            GK_CHECK(check_csr(a.B, CSR_STRUCTURE, "B", s, scr));
            GK_CHECK(check_csr(a.M, CSR_SORTED, "M", s, scr));
            return fail(GK_ERR_INVALID_CSR, "defect found by the content check");
        }
        if (h.too_long) return fail(GK_ERR_UNSUPPORTED, "complement-masked product: a row has >= 2^31 products");
        return GK_OK;
    };
    if (m > 0) GK_CHECK(launch_classes(a, s));
    if (may_sort) GK_CHECK(read_state());
    bool done = m == 0;
    if (may_sort && cm_sorts(h, B->n, a.win, ctx().num_sms)) {
        if (fill && ends[0] != 0)
            return fail(GK_ERR_ARG, "C_rowptr[0] must be 0 (pass the first call's row pointers)");
        // without room for the products (nothing is written before it is known) the windows serve
        Scratch own(s);
        const int status = cmask_by_sort(a, s, own);
        if (status == GK_ERR_OOM) {
            own.release();
            scratch_reclaim(s);
        } else {
            GK_CHECK(status);
            done = true;
        }
    }
    if (!done) GK_CHECK(fill ? launch_rows<true>(a, s) : launch_rows<false>(a, s));
    GK_CHECK(read_state());
    if (fill) {
        if (ends[0] != 0) return fail(GK_ERR_ARG, "C_rowptr[0] must be 0 (pass the first call's row pointers)");
        if (h.mismatch)
            return fail(GK_ERR_ARG, "C_rowptr does not match this product (pass the first call's row pointers)");
        if (cnnz > 0 && dcol != C_col)
            GK_CUDA(cudaMemcpyAsync(C_col, dcol, sizeof(int32_t) * cnnz, cudaMemcpyDeviceToHost, s));
        if (cnnz > 0 && C_val && dval != C_val)
            GK_CUDA(cudaMemcpyAsync(C_val, dval, sizeof(int32_t) * cnnz, cudaMemcpyDeviceToHost, s));
        if (cnnz > 0) GK_CUDA(cudaStreamSynchronize(s));
        return GK_OK;
    }
    const bool rp_dev = is_device_pointer(C_rowptr);
    int64_t *drp = C_rowptr;
    if (!rp_dev) GK_CHECK(scr.alloc(&drp, m + 1));
    size_t tb = 0;
    GK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, a.cnt, drp, m + 1, s));
    char *tmp;
    GK_CHECK(scr.alloc(&tmp, tb));
    GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, a.cnt, drp, m + 1, s));
    if (!rp_dev) {
        GK_CUDA(cudaMemcpyAsync(C_rowptr, drp, sizeof(int64_t) * (m + 1), cudaMemcpyDeviceToHost, s));
        GK_CUDA(cudaStreamSynchronize(s));
    }
    return GK_OK;
}
