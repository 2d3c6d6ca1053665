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
