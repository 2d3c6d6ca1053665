"""A few long rows among rows that the packed kinds take: each is a CTA's work of its
own, not eight of them one CTA's."""
import numpy as np
import pytest

from tests import graphs as G
from tests.test_gpu_packed import rows_csr

pytestmark = pytest.mark.gpu


def operands(long_rows):
    k, n = 3000, 1900  # masks of more than a twentieth of the columns: no packed kind for the long rows
    B = rows_csr(n, [30] * k, 1)
    A = rows_csr(k, [1200] * long_rows + [3] * (400 - long_rows), 2)
    M = rows_csr(n, [100] * 400, 3, values=False)
    return A, B, M


@pytest.mark.parametrize("long_rows", [0, 1, 7, 8, 9, 64, 400])
def test_values(gk, orc, cuda, long_rows):
    A, B, M = operands(long_rows)
    want = orc.mxmm(A, B, M)
    for sched in ("plain", "learned"):
        if sched == "learned":
            from graphkokkos_b200 import sched as s
            s.load_model()
        got = gk.mxmm_masked(A.to("cuda"), B.to("cuda"), M.to("cuda"), sched=sched).cpu().numpy()
        np.testing.assert_array_equal(got, want)
    pat = G.Csr(A.m, A.n, A.rowptr, A.col, None, A.nnz), G.Csr(B.m, B.n, B.rowptr, B.col, None, B.nnz)
    for variant in (3, 4, 5, 18, 6):  # the kinds that take several items a fetch
        got = gk.mxmm_masked_variant(pat[0].to("cuda"), pat[1].to("cuda"), M.to("cuda"), variant).cpu().numpy()
        np.testing.assert_array_equal(got, orc.mxmm(*pat, M))


def test_eight_long_rows_take_hardly_longer_than_one(gk, cuda):
    import torch

    def best(long_rows):
        args = [x.to("cuda") for x in operands(long_rows)]
        ts = []
        for _ in range(8):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            gk.mxmm_masked(*args)
            t1.record()
            torch.cuda.synchronize()
            ts.append(t0.elapsed_time(t1))
        return min(ts)

    assert best(8) < 2.5 * best(1)
