"""The reference's per-vertex and L·U counts where its library was not built: the
restatement's, so that the GPU tests that compare with them still run."""
import numpy as np
import pytest

import oracle
from tests import graphs as G


@pytest.mark.parametrize("built", [False, None])
def test_reference_counts_without_its_library(gk, monkeypatch, tmp_path, built):
    if built is False:
        monkeypatch.setattr(oracle, "REF_PATH", str(tmp_path / "missing.so"))
    A = gk.gen_rmat(9, 16, seed=4)
    tri = oracle.tc_lower(gk.lower_host(A))
    got = oracle.ref_tc_vertex(A)
    np.testing.assert_array_equal(got, oracle.tc_vertex(A))
    assert int(got.astype(np.int64).sum()) == 3 * tri
    assert oracle.ref_tc_lu(A) == tri
    assert oracle.ref_tc_lu(G.complete(6)) == 20
