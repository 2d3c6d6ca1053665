"""Few edges on many vertices: runs of empty rows of every length around the 32 that
are passed at once, in the one-kernel count, the walk, the degree order, the k-truss
and BC's entry walks."""
import numpy as np
import pytest

from tests import graphs as G
from tests.test_gpu_tri import lower, symmetric

pytestmark = pytest.mark.gpu

GAPS = [1, 2, 30, 31, 32, 33, 34, 63, 64, 65, 66, 97, 1000, 1055, 1056, 1057]


def spread(m, clique, seed):
    """Cliques whose vertices lie the given gaps apart, up to m vertices."""
    rng = np.random.default_rng(seed)
    edges, v = [], 0
    while True:
        ids = [v]
        for _ in range(clique - 1):
            ids.append(ids[-1] + int(rng.choice(GAPS)))
        if ids[-1] >= m:
            return np.array(edges)
        edges += [(b, a) for i, a in enumerate(ids) for b in ids[i + 1:]]
        v = ids[-1] + int(rng.choice(GAPS))


@pytest.mark.parametrize("m", [300, 10856, 16384, 40000, 65536, 65537, 300000])
@pytest.mark.parametrize("clique", [2, 3, 9, 40])
def test_counts(gk, orc, cuda, m, clique):
    e = spread(m, clique, m + clique)
    if not len(e):
        pytest.skip("no room for one clique")
    L = lower(e, m)
    want = orc.tc_merge(L)
    D = L.to("cuda")
    assert gk.tc_count(D) == want
    for head in (0, 1, 2):  # the first, a middle and the last entries alone
        part = lower(e[:3] if head == 0 else e[len(e) // 2:len(e) // 2 + 40] if head == 1 else e[-3:], m)
        assert gk.tc_count(part.to("cuda")) == orc.tc_merge(part)
    np.testing.assert_array_equal(gk.tc_count_batched([D, part.to("cuda"), D]), [want, orc.tc_merge(part), want])
    A = symmetric(L)
    rp, col, iters, _ = orc.ktruss(A, 4)
    T, it = gk.ktruss(A.to("cuda"), 4)
    assert it == iters
    np.testing.assert_array_equal(T.rowptr.cpu().numpy(), rp)
    np.testing.assert_array_equal(T.col.cpu().numpy(), col)
    src = np.unique(e[:20].ravel())[:8].astype(np.int32)
    G.assert_bc_close(gk.bc_batch(A.to("cuda"), src).cpu().numpy(), orc.bc_f64(A, src))


def test_empty_rows_are_passed_in_no_time(gk, cuda):
    """64 edges on 16,000 vertices took fifteen times as long as on 64."""
    import torch

    def best(m):
        rng = np.random.default_rng(m)
        L = lower(np.stack([rng.permutation(m)[:64], rng.permutation(m)[:64]], 1), m).to("cuda")
        ts = []
        for _ in range(10):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            gk.tc_count(L)
            t1.record()
            torch.cuda.synchronize()
            ts.append(t0.elapsed_time(t1))
        return min(ts)

    assert best(16000) < 4 * best(64)
