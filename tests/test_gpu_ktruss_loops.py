"""k-truss of symmetric patterns with self-loops: the loops count in the supports of
every pass, as the product S<C> = C·C counts them, and are left out of the truss."""
import numpy as np
import pytest

from tests import graphs as G

pytestmark = pytest.mark.gpu


def with_loops(A, share, seed):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(A.m), np.diff(A.rowptr))
    loops = np.flatnonzero(rng.random(A.m) < share)
    key = np.unique(np.concatenate([rows * A.m + np.asarray(A.col), loops * A.m + loops]))
    rp = np.zeros(A.m + 1, dtype=np.int64)
    np.cumsum(np.bincount(key // A.m, minlength=A.m), out=rp[1:])
    return G.Csr(A.m, A.m, rp, (key % A.m).astype(np.int32), None, len(key))


CASES = {
    "all ones": lambda gk: with_loops(G.complete(3), 1.0, 0),
    "clique, one loop": lambda gk: with_loops(G.complete(7), 0.2, 1),
    "rmat, few loops": lambda gk: with_loops(gk.gen_rmat(9, 6, seed=2), 0.1, 2),
    "rmat, all loops": lambda gk: with_loops(gk.gen_rmat(10, 4, seed=3), 1.0, 3),
    "path, all loops": lambda gk: with_loops(G.path(50), 1.0, 4),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("k", [3, 4, 5, 7])
def test_off_diagonal_truss_and_passes(gk, orc, cuda, name, k):
    A = CASES[name](gk)
    rp, col, iters, _ = orc.ktruss(A, k)
    rows = np.repeat(np.arange(A.m), np.diff(rp))
    edge = rows != col
    want = np.zeros(A.m + 1, dtype=np.int64)
    np.cumsum(np.bincount(rows[edge], minlength=A.m), out=want[1:])
    for X in (A.to("cuda"), A):
        T, it = gk.ktruss(X, k)
        T = T.numpy() if X is not A else T
        assert it == iters
        np.testing.assert_array_equal(T.rowptr, want)
        np.testing.assert_array_equal(T.col, col[edge])
