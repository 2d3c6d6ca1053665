"""The first bad row of a batch, numbered in the caller's order whichever way its
graphs are counted: device graphs are walked or reordered in two groups, host
graphs go in the order given."""
import re

import numpy as np
import pytest

from tests import graphs as G

pytestmark = pytest.mark.gpu


def skewed(gk, seed):
    return gk.lower_host(gk.gen_rmat(12, 24, seed=seed))  # reordered


def flat(gk, seed):
    return gk.lower_host(gk.gen_er(3000, 9000, seed=seed))  # walked


def spoil(L, row):
    """L with the first two columns of its first row of two or more from `row` on exchanged."""
    r = int(np.flatnonzero(np.diff(L.rowptr)[row:] > 1)[0]) + row
    col = L.col.copy()
    p = int(L.rowptr[r])
    col[p], col[p + 1] = col[p + 1], col[p]
    return G.Csr(L.m, L.m, L.rowptr, col, None, L.nnz), r


@pytest.mark.parametrize("kinds", ["sfsf", "fsfs", "ssff", "ffss", "ssss", "ffff"])
@pytest.mark.parametrize("bad", [(0,), (1,), (2,), (3,), (1, 2), (0, 3), (2, 3)])
def test_first_bad_row(gk, cuda, kinds, bad):
    graphs = [skewed(gk, i) if k == "s" else flat(gk, i) for i, k in enumerate(kinds)]
    first = None
    base = 0
    for i, L in enumerate(graphs):
        if i in bad:
            graphs[i], r = spoil(L, 700 + 50 * i)
            first = base + r if first is None else first
        base += L.m
    for batch in (graphs, [x.to("cuda") for x in graphs]):
        with pytest.raises(gk.GkError) as e:
            gk.tc_count_batched(batch)
        assert e.value.code == gk._lib.GK_ERR_INVALID_CSR
        assert int(re.search(r"first at row (\d+)", str(e.value)).group(1)) == first


def test_defect_before_the_mode(gk, cuda):
    """A bad graph in the second group is named before an unknown schedule."""
    import ctypes
    graphs = [flat(gk, 1).to("cuda"), spoil(skewed(gk, 2), 300)[0].to("cuda")]
    arr = (gk._lib.GkCsr * 2)(*[x.as_gk() for x in graphs])
    out = np.zeros(2, dtype=np.uint64)
    assert gk.load().gk_tc_count_batched(arr, 2, out.ctypes.data_as(ctypes.c_void_p), 7, None) == \
        gk._lib.GK_ERR_INVALID_CSR
    good = [flat(gk, 1).to("cuda"), skewed(gk, 2).to("cuda")]
    arr = (gk._lib.GkCsr * 2)(*[x.as_gk() for x in good])
    assert gk.load().gk_tc_count_batched(arr, 2, out.ctypes.data_as(ctypes.c_void_p), 7, None) == gk._lib.GK_ERR_ARG
