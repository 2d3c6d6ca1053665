"""Small graphs with very uneven rows in the triangle count's one-kernel path
(csrc/tri.cu): a long row that many short ones name, rows of nearly all columns."""
import numpy as np
import pytest

from tests import graphs as G
from tests.test_gpu_tri import lower

pytestmark = pytest.mark.gpu


def long_row(m):
    """Vertex m/2 joined to everybody: half of the edges in its row, the others one a row."""
    v = m // 2
    return np.stack([np.delete(np.arange(m), v), np.full(m - 1, v)], 1)


def hub_rows(m, h):
    """The last h vertices joined to all others."""
    return np.stack([np.repeat(np.arange(m - h, m), m - h), np.tile(np.arange(m - h), h)], 1)


def extra(m, count, seed):
    return np.random.default_rng(seed).integers(0, m, (count, 2))


CASES = {
    "long row": lambda: (long_row(40000), 40000),
    "long row, others": lambda: (np.concatenate([long_row(12000), extra(12000, 30000, 1)]), 12000),
    "long row and cliques": lambda: (np.concatenate([long_row(16384), extra(300, 9000, 2) + 8000]), 16384),
    "hub rows": lambda: (hub_rows(16384, 32), 16384),
    "hub rows, others": lambda: (np.concatenate([hub_rows(16384, 25), extra(16384, 3000, 3)]), 16384),
    "hub rows, many others": lambda: (np.concatenate([hub_rows(9000, 20), extra(9000, 60000, 4)]), 9000),
    # L_i and L_k around the ratio and the mapped length at which the lookup turns round
    "around the ratio": lambda: (np.concatenate(
        [np.stack([np.full(n, 5000 + i), np.arange(n)], 1) for i, n in
         enumerate([1023, 1024, 1025, 1055, 1056, 1057, 1058, 1087, 1088, 1089, 2111, 2112, 2113, 4000])] +
        [np.stack([np.full(1 + i % 3, 6000 + i), np.arange(1 + i % 3)], 1) for i in range(300)] +
        [np.stack([np.arange(6000, 6300), 5000 + np.arange(300) % 14], 1)]), 6300),
}


@pytest.mark.parametrize("name", CASES)
def test_counts(gk, orc, cuda, name):
    e, m = CASES[name]()
    L = lower(e, m)
    assert gk.tc_count(L.to("cuda")) == orc.tc_merge(L)
    sums = gk.tc_row_sums(L.to("cuda")).cpu().numpy()
    assert int(sums.astype(np.int64).sum()) == orc.tc_merge(L)


def test_patterns_that_are_no_triangle(gk, orc, cuda):
    e, m = np.concatenate([long_row(3000), extra(3000, 4000, 5)]), 3000
    key = np.unique(np.concatenate([e[:, 0] * m + e[:, 1], e[:1700, 1] * m + e[:1700, 0]]))
    rp = np.zeros(m + 1, dtype=np.int64)
    np.cumsum(np.bincount(key // m, minlength=m), out=rp[1:])
    A = G.Csr(m, m, rp, (key % m).astype(np.int32), None, len(key))
    assert gk.tc_count(A.to("cuda")) == int(orc.mxmm(A, A, A).astype(np.int64).sum())


@pytest.mark.parametrize("name", ["long row", "hub rows"])
def test_no_slower_than_the_row_sums(gk, cuda, name):
    """The engine's product of the same matrix took a fraction of the one-kernel
    count's time where a warp read a whole long row for a few columns."""
    import torch
    e, m = CASES[name]()
    L = lower(e, m).to("cuda")

    def best(fn):
        ts = []
        for _ in range(8):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            fn(L)
            t1.record()
            torch.cuda.synchronize()
            ts.append(t0.elapsed_time(t1))
        return min(ts)

    assert best(gk.tc_count) < 1.5 * best(gk.tc_row_sums)
