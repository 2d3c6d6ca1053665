"""The 24 variants of the masked product keep their kernels: a forced variant, a
forced accumulator and a model's choice never run the packed kinds, which are no
variants (csrc/gk_sched.cuh)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kernels(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = fn()
        torch.cuda.synchronize()
    return out, [e.key for e in prof.key_averages()]


def test_forced_choices(gk, orc, cuda):
    A = gk.gen_rmat(10, 12, seed=5)
    L = gk.lower_host(A)
    D = L.to("cuda")
    want = orc.mxmm(L, L, L)
    for accum in ("hash", "msa", "mca"):
        got, names = kernels(lambda: gk.mxmm_masked(D, D, D, accum=accum))
        np.testing.assert_array_equal(got.cpu().numpy(), want)
        assert any("k_group" in n or "k_block" in n for n in names)
        assert not any("k_packed" in n for n in names), accum
    for variant in (0, 1, 2):
        got, names = kernels(lambda: gk.mxmm_masked_variant(D, D, D, variant))
        np.testing.assert_array_equal(got.cpu().numpy(), want)
        assert any("k_group" in n for n in names) and not any("k_packed" in n for n in names), variant
        assert gk.tc_count_variant(D, variant) == orc.tc_lower(L)
    assert gk.num_variants() == 24
    with pytest.raises(gk.GkError):
        gk.tc_count_variant(D, 24)


def test_model_choices_run_the_catalogue(gk, orc, cuda):
    """A model that predicts one variant far below the others: every bin that admits
    it runs that variant's kernel."""
    import ctypes
    from graphkokkos_b200 import sched
    lib = gk.load()
    nv, nf, _ = sched.dims()
    h = sched.MLP_H
    size = sched.model_size()
    A = gk.gen_rmat(10, 12, seed=5)
    L = gk.lower_host(A)
    D = L.to("cuda")
    want = orc.mxmm(L, L, L)
    try:
        for variant in (1, 2):
            w = np.zeros(size, dtype=np.float32)
            b3 = h * nf + h + h * h + h + nv * h
            w[b3:b3 + nv] = 10.0
            w[b3 + variant] = 0.0
            w[size - nf:] = 1.0  # sigma
            assert lib.gk_sched_set_model(w.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), ctypes.c_size_t(size)) == 0
            got, names = kernels(lambda: gk.mxmm_masked(D, D, D, sched="learned"))
            np.testing.assert_array_equal(got.cpu().numpy(), want)
            assert any(f"k_group<{8 if variant == 1 else 32}," in n.replace("(int)", "") for n in names), names
    finally:
        sched.load_model()
