"""No call asks the driver how much memory is free: now and then that takes tens of
milliseconds.  What does not fit shows when it is allocated."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_calls_do_not_ask(gk, cuda):
    import torch
    from torch.profiler import ProfilerActivity, profile
    A = gk.gen_rmat(17, 8, seed=1, device="cuda")
    L = gk.extract_lower(A)
    src = np.arange(300, dtype=np.int32) * 11
    calls = [lambda: gk.bc_batch(A, src), lambda: gk.tc_count(L), lambda: gk.tc_count_batched([L] * 3),
             lambda: gk.ktruss(A, 4)]
    for fn in calls:
        fn()
    torch.cuda.synchronize()
    for fn in calls:
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
            fn()
        assert not any("MemGetInfo" in e.key for e in prof.key_averages())
