"""Calls with device outputs wait for their stream once: the content check's result
and the kernels to launch are read together."""
import ctypes

import numpy as np
import pytest

from tests import graphs as G

pytestmark = pytest.mark.gpu


def waits(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        fn()
    return sum(e.count for e in prof.key_averages() if e.key == "cudaStreamSynchronize")


def test_one_wait_a_call(gk, cuda):
    import torch
    lib = gk.load()
    A = gk.gen_rmat(12, 16, seed=2)
    L = gk.lower_host(A).to("cuda")
    A = A.to("cuda")
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    g = L.as_gk()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert waits(lambda: gk.tc_row_sums(L)) == 1
    assert waits(lambda: gk.tc_vertex(A, sched="plain")) == 1
    assert waits(lambda: gk.mxmm_masked(L, L, L)) == 1
    assert waits(lambda: lib.gk_tc_count_noalloc(ctypes.byref(g), ctypes.c_void_p(out.data_ptr()), 0, stream)) == 1


@pytest.mark.parametrize("defect", ["column", "order", "rowptr", "ends"])
def test_defects_are_named(gk, cuda, defect):
    """The check that is read with the plan: every defect, its row, and the library
    usable afterwards; a defect comes before an unknown schedule."""
    L = gk.lower_host(gk.gen_rmat(9, 16, seed=4))
    rp, col = np.array(L.rowptr), np.array(L.col)
    row = int(np.flatnonzero(np.diff(rp) > 3)[5])
    p = int(rp[row])
    if defect == "column":
        col[p + 1] = L.m
    elif defect == "order":
        col[p], col[p + 1] = col[p + 1], col[p]
    elif defect == "rowptr":
        rp[row + 1] = rp[row] - 1
    else:
        rp[0] = 1
    bad = G.Csr(L.m, L.m, rp, col, None, L.nnz).to("cuda")
    good = L.to("cuda")
    lib = gk.load()
    want = gk.tc_row_sums(good).cpu().numpy()
    out = np.zeros(L.m, dtype=np.uint64)
    g = bad.as_gk()
    for fn in (lambda: lib.gk_tc_row_sums(ctypes.byref(g), out.ctypes.data, 0, None),
               lambda: lib.gk_tc_row_sums(ctypes.byref(g), out.ctypes.data, 7, None),
               lambda: lib.gk_tc_vertex(ctypes.byref(g), out.ctypes.data, 0, None),
               lambda: lib.gk_tc_count_variant(ctypes.byref(g), 6, out.ctypes.data, None),
               lambda: lib.gk_tc_count_noalloc(ctypes.byref(g), out.ctypes.data, 0, None),
               lambda: lib.gk_tc_count_noalloc(ctypes.byref(g), out.ctypes.data, 7, None)):
        assert fn() == gk._lib.GK_ERR_INVALID_CSR
        text = lib.gk_last_error_string().decode()
        if defect in ("column", "order"):
            assert f"first at row {row})" in text, text
        np.testing.assert_array_equal(gk.tc_row_sums(good).cpu().numpy(), want)
    gg = good.as_gk()
    assert lib.gk_tc_row_sums(ctypes.byref(gg), out.ctypes.data, 7, None) == gk._lib.GK_ERR_ARG
