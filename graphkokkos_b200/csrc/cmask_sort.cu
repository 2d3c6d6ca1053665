// Complement-masked product by expanding, sorting and reducing all products: the
// path of gk_mxmm_cmask (cmask.cu) for long rows over very many columns, whose
// cost does not depend on the number of columns.
//   1. per batch of rows whose products fit a fixed budget, the products' offsets
//      (a scan over the batch's A entries) and one warp per row writing a 64-bit
//      key (row << 32 | column) and the product for every B element, the key of a
//      column of M's row replaced by a sentinel that sorts last;
//   2. one radix sort of (key, product) and one reduce-by-key: the runs are C's
//      entries in CSR order, so the batch's run j is entry rp[r0] + j.
// About 0.25 us per 1,000 products and both calls, bound by the sort's passes
// over memory (2,000 rows x 3,000 products, any number of columns: 2.2 ms).
#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "gk_cmask.cuh"
#include "gk_common.cuh"

namespace gk {

constexpr int64_t CMASK_BUDGET = int64_t(1) << 26;  // products per batch
constexpr unsigned long long CMASK_SENTINEL = ~0ull;

__global__ void k_cmask_entry_len(DevCsr A, DevCsr B, int64_t t0, int64_t t1, int64_t *len) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = t0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < t1; t += stride) {
        const int k = A.col[t];
        len[t - t0] = B.rp[k + 1] - B.rp[k];
    }
}

// One warp per row of [r0, r1): every product of the row at off[t - t0] + q.
__global__ void k_cmask_expand(DevCsr A, DevCsr B, DevCsr M, int64_t r0, int64_t r1, int64_t t0, const int64_t *off,
                               bool values, unsigned long long *keys, int32_t *prods) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = r0 + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < r1; i += warps) {
        const int64_t m0 = M.rp[i], m1 = M.rp[i + 1];
        for (int64_t t = A.rp[i]; t < A.rp[i + 1]; ++t) {
            const int k = A.col[t];
            const uint32_t a = (values && A.val) ? static_cast<uint32_t>(A.val[t]) : 1u;
            const int64_t b0 = B.rp[k], b1 = B.rp[k + 1], o = off[t - t0] - b0;
            for (int64_t j = b0 + lane; j < b1; j += 32) {
                const int c = B.col[j];
                int64_t lo = m0, hi = m1;  // is c a column of M's row i?
                while (lo < hi) {
                    const int64_t md = (lo + hi) >> 1;
                    if (M.col[md] < c) lo = md + 1;
                    else hi = md;
                }
                const bool masked = lo < m1 && M.col[lo] == c;
                const uint32_t b = (values && B.val) ? static_cast<uint32_t>(B.val[j]) : 1u;
                keys[o + j] = masked ? CMASK_SENTINEL
                                     : ((static_cast<unsigned long long>(i) << 32) | static_cast<uint32_t>(c));
                prods[o + j] = static_cast<int32_t>(a * b);
            }
        }
    }
}

// Entries per row from the sorted unique keys (the sentinel run excluded): a row's
// last run and its first one, so that a long row is two atomics (one an entry took
// a quarter of the call at 30,000 products a row).
__global__ void k_cmask_row_counts(const unsigned long long *uniq, const int64_t *nruns, unsigned long long *cnt) {
    const int64_t n = *nruns;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const unsigned long long k = uniq[r], row = k >> 32;
        if (k == CMASK_SENTINEL) continue;
        if (r == 0 || uniq[r - 1] >> 32 != row) atomicAdd(cnt + row, static_cast<unsigned long long>(-r));
        if (r + 1 == n || uniq[r + 1] >> 32 != row) atomicAdd(cnt + row, static_cast<unsigned long long>(r + 1));
    }
}

__global__ void k_cmask_write(const unsigned long long *uniq, const int32_t *sums, const int64_t *nruns, int64_t base,
                              int32_t *c_col, int32_t *c_val) {
    const int64_t n = *nruns;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const unsigned long long k = uniq[r];
        if (k == CMASK_SENTINEL) continue;
        c_col[base + r] = static_cast<int32_t>(k & 0xFFFFFFFFull);
        if (c_val) c_val[base + r] = sums[r];
    }
}

// wrapping int32 sum, as the reference accumulates int values
struct WrapSum {
    __device__ __forceinline__ int32_t operator()(int32_t a, int32_t b) const {
        return static_cast<int32_t>(static_cast<uint32_t>(a) + static_cast<uint32_t>(b));
    }
};

// Numeric call: the entries found in a row against its place in C.
__global__ void k_cmask_compare(int64_t m, const int64_t *cnt, const int64_t *crp, unsigned int *mismatch) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride)
        if (crp[i + 1] - crp[i] != cnt[i]) *mismatch = 1;
}

int cmask_by_sort(const DevCsr &a, const DevCsr &b, const DevCsr &mk, bool values, const int64_t *work, int64_t *cnt,
                  const int64_t *crp, int32_t *c_col, int32_t *c_val, unsigned int *mismatch, cudaStream_t s,
                  Scratch &scr) {
    const int64_t m = a.m;
    const bool fill = c_col != nullptr;
    const int sms = ctx().num_sms;
    // the batches are cut on the host
    std::vector<int64_t> hwork(m), arp(m + 1), hcrp(m + 1, 0);
    GK_CUDA(cudaMemcpyAsync(hwork.data(), work, sizeof(int64_t) * m, cudaMemcpyDeviceToHost, s));
    GK_CUDA(cudaMemcpyAsync(arp.data(), a.rp, sizeof(int64_t) * (m + 1), cudaMemcpyDeviceToHost, s));
    if (fill) GK_CUDA(cudaMemcpyAsync(hcrp.data(), crp, sizeof(int64_t) * (m + 1), cudaMemcpyDeviceToHost, s));
    GK_CUDA(cudaStreamSynchronize(s));
    auto batch_end = [&](int64_t r0, int64_t *products) {  // a row above the budget is a batch of its own
        int64_t r1 = r0, acc = 0;
        while (r1 < m && (r1 == r0 || acc + hwork[r1] <= CMASK_BUDGET)) acc += hwork[r1++];
        *products = acc;
        return r1;
    };
    int64_t maxb = 0, max_entries = 1;
    for (int64_t r0 = 0, n = 0; r0 < m;) {
        const int64_t r1 = batch_end(r0, &n);
        maxb = std::max(maxb, n);
        max_entries = std::max(max_entries, arp[r1] - arp[r0] + 1);
        r0 = r1;
    }
    GK_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (m + 1), s));
    if (maxb > 0) {
        unsigned long long *keys, *keys2, *uniq;
        int32_t *prods, *prods2, *sums;
        int64_t *len, *off, *nruns;
        char *tmp;
        GK_CHECK(scr.alloc(&keys, maxb));
        GK_CHECK(scr.alloc(&keys2, maxb));
        GK_CHECK(scr.alloc(&uniq, maxb));
        GK_CHECK(scr.alloc(&prods, maxb));
        GK_CHECK(scr.alloc(&prods2, maxb));
        GK_CHECK(scr.alloc(&sums, maxb));
        GK_CHECK(scr.alloc(&nruns, 1));
        GK_CHECK(scr.alloc(&len, max_entries));
        GK_CHECK(scr.alloc(&off, max_entries));
        size_t sort_bytes = 0, red_bytes = 0, scan_bytes = 0;
        const int nmax = static_cast<int>(maxb);  // a row has fewer than 2^31 products
        GK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, keys, keys2, prods, prods2, nmax, 0, 64, s));
        GK_CUDA(cub::DeviceReduce::ReduceByKey(nullptr, red_bytes, keys2, uniq, prods2, sums, nruns, WrapSum(), nmax,
                                               s));
        GK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, len, off, max_entries, s));
        const size_t tmp_bytes = std::max(std::max(sort_bytes, red_bytes), scan_bytes);
        GK_CHECK(scr.alloc(&tmp, tmp_bytes));
        for (int64_t r0 = 0, n = 0; r0 < m;) {
            const int64_t r1 = batch_end(r0, &n), t0 = arp[r0], t1 = arp[r1];
            if (n > 0) {
                k_cmask_entry_len<<<sms * 4, 256, 0, s>>>(a, b, t0, t1, len);
                GK_CUDA(cudaMemsetAsync(len + (t1 - t0), 0, sizeof(int64_t), s));
                size_t tb = tmp_bytes;
                GK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, len, off, t1 - t0 + 1, s));
                k_cmask_expand<<<sms * 8, 256, 0, s>>>(a, b, mk, r0, r1, t0, off, values, keys, prods);
                tb = tmp_bytes;
                GK_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, keys, keys2, prods, prods2, static_cast<int>(n), 0, 64,
                                                        s));
                tb = tmp_bytes;
                GK_CUDA(cub::DeviceReduce::ReduceByKey(tmp, tb, keys2, uniq, prods2, sums, nruns, WrapSum(),
                                                       static_cast<int>(n), s));
                k_cmask_row_counts<<<sms * 4, 256, 0, s>>>(uniq, nruns,
                                                         reinterpret_cast<unsigned long long *>(cnt));
                note_launches(3);
                GK_CUDA(cudaGetLastError());
                if (fill) {  // nothing is written unless the batch's entries are those its row pointers announce
                    int64_t runs = 0;
                    unsigned long long last = 0;
                    GK_CUDA(cudaMemcpyAsync(&runs, nruns, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
                    GK_CUDA(cudaStreamSynchronize(s));
                    if (runs > 0)
                        GK_CUDA(cudaMemcpyAsync(&last, uniq + runs - 1, sizeof(last), cudaMemcpyDeviceToHost, s));
                    GK_CUDA(cudaStreamSynchronize(s));
                    const int64_t got = runs - (runs > 0 && last == CMASK_SENTINEL ? 1 : 0);
                    if (got != hcrp[r1] - hcrp[r0] || hcrp[r0] < 0 || hcrp[r1] > hcrp[m]) {
                        GK_CUDA(cudaMemsetAsync(mismatch, 1, sizeof(*mismatch), s));
                        return GK_OK;
                    }
                    k_cmask_write<<<sms * 4, 256, 0, s>>>(uniq, sums, nruns, hcrp[r0], c_col, c_val);
                    note_launches(1);
                    GK_CUDA(cudaGetLastError());
                }
            }
            r0 = r1;
        }
    }
    if (fill) {
        k_cmask_compare<<<sms * 4, 256, 0, s>>>(m, cnt, crp, mismatch);
        note_launches(1);
        GK_CUDA(cudaGetLastError());
    }
    return GK_OK;
}

}  // namespace gk
