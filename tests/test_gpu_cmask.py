"""The complement-masked product's row classes (csrc/cmask.cu) against the CPU
oracle: hashed rows of a warp and of a CTA, bitmap rows, windows with more
columns than the shared-memory sums hold, several windows, empty rows, and row
pointers that are not the product's."""
import ctypes

import numpy as np
import pytest

from tests import graphs as G

pytestmark = pytest.mark.gpu


def csr(m, n, rows, cols, seed, values=True):
    key = np.unique(np.asarray(rows, dtype=np.int64) * n + cols)
    rp = np.zeros(m + 1, dtype=np.int64)
    np.cumsum(np.bincount(key // n, minlength=m), out=rp[1:])
    val = np.random.default_rng(seed).integers(-4, 5, len(key)).astype(np.int32) if values else None
    return G.Csr(m, n, rp, (key % n).astype(np.int32), val, len(key))


def case(k, n, long_rows, seed):
    """A with rows of 0, 1, a few, and long_rows entries; B's rows uneven, one of
    them long."""
    rng = np.random.default_rng(seed)
    m = 40
    lens = [0, 1, 3, 9, 40] * 7 + long_rows
    lens = (lens + [2] * m)[:m]
    ar = np.repeat(np.arange(m), lens)
    A = csr(m, k, ar, rng.integers(0, k, len(ar)), seed)
    br = np.concatenate([rng.integers(0, k, 12 * k), np.zeros(min(n, 9000), dtype=np.int64)])
    B = csr(k, n, br, rng.integers(0, n, len(br)), seed + 1)
    mr = rng.integers(0, m, 6 * m)
    M = csr(m, n, mr, rng.integers(0, n, len(mr)), seed + 2, values=False)
    # some columns that the products surely reach are masked too
    hit = B.col[: min(len(B.col), 200)]
    M = csr(m, n, np.concatenate([np.repeat(np.arange(m), np.diff(M.rowptr)), np.arange(len(hit)) % m]),
            np.concatenate([M.col, hit]), seed + 3, values=False)
    return A, B, M


@pytest.mark.parametrize("k,n,long_rows", [
    (300, 700, [250, 290]),                     # one small window
    (900, 32768, [700, 880]),                   # the widest window that takes every longer row
    (900, 32769, [150, 700, 880]),              # CTA hash and bitmap rows
    (4000, 300000, [180, 3000, 3990]),          # windows with thousands of columns
    (3000, (1 << 19) + 77, [170, 2000]),        # two windows, the second nearly empty
    (3000, 1300001, [2900]),                    # three windows
])
def test_row_classes(gk, orc, cuda, k, n, long_rows):
    A, B, M = case(k, n, long_rows, n)
    for semiring in ("plus_times", "plus_pair"):
        a, b = (A, B) if semiring == "plus_times" else (G.Csr(A.m, A.n, A.rowptr, A.col, None, A.nnz),
                                                         G.Csr(B.m, B.n, B.rowptr, B.col, None, B.nnz))
        rp, col, val = orc.mxmm_cmask(a, b, M)
        for C in (gk.mxmm_cmask(A.to("cuda"), B.to("cuda"), M.to("cuda"), semiring=semiring).numpy(),
                  gk.mxmm_cmask(A, B, M, semiring=semiring)):
            np.testing.assert_array_equal(C.rowptr, rp)
            np.testing.assert_array_equal(C.col, col)
            np.testing.assert_array_equal(C.val, val)


def test_foreign_row_pointers(gk, cuda):
    """Row pointers of another product are refused, and nothing is written
    beyond the entries they announce."""
    A, B, M = case(900, 40000, [150, 700, 880], 5)
    lib = gk.load()
    C = gk.mxmm_cmask(A, B, M)
    ga, gb, gm = A.as_gk(), B.as_gk(), M.as_gk()
    for bad in (np.concatenate([C.rowptr[:3] , C.rowptr[3:] + 1]), np.minimum(C.rowptr, 100),
                np.concatenate([C.rowptr[:-1] * 0, C.rowptr[-1:]])):
        bad = np.ascontiguousarray(bad, dtype=np.int64)
        n = int(bad[-1])
        col = np.full(n + 64, -7, dtype=np.int32)
        val = np.full(n + 64, -7, dtype=np.int32)
        rc = lib.gk_mxmm_cmask(ctypes.byref(ga), ctypes.byref(gb), ctypes.byref(gm), 0, bad.ctypes.data,
                               col.ctypes.data, val.ctypes.data, None)
        assert rc == gk._lib.GK_ERR_ARG
        assert (col[n:] == -7).all() and (val[n:] == -7).all()


@pytest.mark.parametrize("entries", [5000, 1 << 19])
def test_row_of_too_many_products(gk, cuda, entries):
    """A row of 2^31 products is refused, a shorter one is not (A's order and
    duplicates do not matter)."""
    n, b = 1 << 15, 1 << 12
    A = G.Csr(2, 1, np.array([0, 1, 1 + entries]), np.zeros(1 + entries, dtype=np.int32), None)
    B = G.Csr(1, n, np.array([0, b]), np.arange(b, dtype=np.int32) * 3, None)
    M = G.Csr(2, n, np.array([0, 0, 1]), np.array([6], dtype=np.int32), None)
    if entries * b < 1 << 31:
        C = gk.mxmm_cmask(A.to("cuda"), B.to("cuda"), M.to("cuda"), semiring="plus_pair").numpy()
        np.testing.assert_array_equal(C.rowptr, [0, b, 2 * b - 1])
        np.testing.assert_array_equal(C.col[b:], np.delete(np.arange(b) * 3, 2))
        np.testing.assert_array_equal(C.val, [1] * b + [entries] * (b - 1))
    else:
        with pytest.raises(gk.GkError) as e:
            gk.mxmm_cmask(A.to("cuda"), B.to("cuda"), M.to("cuda"), semiring="plus_pair")
        assert e.value.code == gk._lib.GK_ERR_UNSUPPORTED


def random_rows(m, n, per_row, seed, values=True):
    rng = np.random.default_rng(seed)
    return csr(m, n, np.repeat(np.arange(m), per_row), rng.integers(0, n, m * per_row), seed, values)


def test_long_rows_over_very_many_columns(gk, orc, cuda):
    """Rows of some thousand products over 2^23 columns, which are sorted (in
    windows where that finds no memory), among short and empty ones."""
    n, k = (1 << 23) + 5, 2000
    A = csr(60, k, np.concatenate([np.repeat(np.arange(40), 90), np.arange(40, 58)]),
            np.random.default_rng(1).integers(0, k, 3618), 1)
    B, M = random_rows(k, n, 40, 2), random_rows(60, n, 30, 3, values=False)
    M = csr(60, n, np.concatenate([np.repeat(np.arange(60), np.diff(M.rowptr)), np.arange(4000) % 60]),
            np.concatenate([M.col, B.col[:4000]]), 4, values=False)
    rp, col, val = orc.mxmm_cmask(A, B, M)
    dev = [x.to("cuda") for x in (A, B, M)]
    lib = gk.load()
    failures = 0
    for after in [-1] + list(range(40)):
        lib.gk_inject_alloc_failure(after)
        try:
            C = gk.mxmm_cmask(*dev).numpy()
        except gk.GkError as e:
            assert e.code == gk._lib.GK_ERR_OOM
            failures += 1
            continue
        finally:
            lib.gk_inject_alloc_failure(-1)
        np.testing.assert_array_equal(C.rowptr, rp)
        np.testing.assert_array_equal(C.col, col)
        np.testing.assert_array_equal(C.val, val)
    assert failures < 12  # the calls' own few arrays
    # foreign row pointers
    ga, gb, gm = (x.as_gk() for x in (A, B, M))
    for bad in (np.concatenate([rp[:3], rp[3:] + 1]), np.concatenate([rp[:-1] * 0, rp[-1:]]),
                np.concatenate([rp[:5], rp[4:5], rp[6:]])):
        bad = np.ascontiguousarray(bad, dtype=np.int64)
        c, v = np.full(int(bad[-1]) + 64, -7, dtype=np.int32), np.full(int(bad[-1]) + 64, -7, dtype=np.int32)
        rc = lib.gk_mxmm_cmask(ctypes.byref(ga), ctypes.byref(gb), ctypes.byref(gm), 0, bad.ctypes.data, c.ctypes.data,
                               v.ctypes.data, None)
        assert rc == gk._lib.GK_ERR_ARG
        assert (c[int(bad[-1]):] == -7).all() and (v[int(bad[-1]):] == -7).all()


def test_time_does_not_grow_with_the_columns(gk, cuda):
    """The same number of products over 2^24 columns took 60 times as long as over
    2^17, window by window; the sort takes some three times as long."""
    import torch

    def best(n):
        args = [x.to("cuda") for x in (random_rows(2000, 20000, 100, 5), random_rows(20000, n, 30, 6),
                                       random_rows(2000, n, 20, 7, values=False))]
        ts = []
        for _ in range(5):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            gk.mxmm_cmask(*args)
            t1.record()
            torch.cuda.synchronize()
            ts.append(t0.elapsed_time(t1))
        return min(ts)

    assert best(1 << 24) < 15 * best(1 << 17)
