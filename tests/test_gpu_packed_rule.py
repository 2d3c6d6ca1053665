"""Which rows the packed kinds take under the learned schedule (csrc/spgemm.cu): for
sums only those of flat products with enough work a row, for written values by the
row's size; and that written values are right whichever way they go."""
import numpy as np
import pytest

from tests import graphs as G
from tests.test_gpu_catalogue import kernels
from tests.test_gpu_packed import rows_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def model(gk):
    from graphkokkos_b200 import sched
    sched.load_model()


@pytest.mark.parametrize("graph,packed", [("few", False), ("flat", True), ("long", False)])
def test_row_sums(gk, orc, cuda, graph, packed):
    if graph == "few":  # a dozen products a row
        A = gk.gen_er(20000, 70000, seed=1)
    elif graph == "flat":
        A = gk.gen_er(4000, 60000, seed=2)
    else:  # every row names one of the long ones
        n = 3000
        rng = np.random.default_rng(3)
        e = [np.stack([np.repeat(np.arange(400, 420), 390), np.tile(np.arange(390), 20)], 1),
             np.stack([np.repeat(np.arange(420, n), 2), np.concatenate([rng.choice(20, 2, False) + 400
                                                                        for _ in range(420, n)])], 1)]
        A = G.from_edges(n, [tuple(x) for x in np.concatenate(e).tolist()])
    L = gk.lower_host(A)
    D = L.to("cuda")
    got, names = kernels(lambda: gk.tc_row_sums(D, sched="learned"))
    np.testing.assert_array_equal(got.cpu().numpy().astype(np.uint64), orc.tc_row_sums(L))
    assert any("k_packed" in x for x in names) == packed
    got, names = kernels(lambda: gk.tc_row_sums(D))  # plain: by the row's size alone
    np.testing.assert_array_equal(got.cpu().numpy().astype(np.uint64), orc.tc_row_sums(L))
    assert any("k_packed" in x for x in names)


@pytest.mark.parametrize("n", [3000, 21000])
def test_written_values_learned(gk, orc, cuda, n):
    """The learned schedule's written values, rows on both sides of the rule's limits."""
    k, blen = 700, 33
    masks = [0, 1, 31, 33, 151, 255, 256, 257, 1024, 1025]
    works = [1, 33, 511, 513, 2047, 2049, 65536, 65537]
    lens = [(a, max(1, min(w // blen, k))) for a in masks for w in works]
    A, B = rows_csr(k, [x for _, x in lens], 2), rows_csr(n, [blen] * (k - 1) + [900], 1)
    M = rows_csr(n, [x for x, _ in lens], 3, values=False)
    got = gk.mxmm_masked(A.to("cuda"), B.to("cuda"), M.to("cuda"), sched="learned").cpu().numpy()
    np.testing.assert_array_equal(got, orc.mxmm(A, B, M))


def test_copies_of_an_operand_are_one_mask(gk, orc, cuda):
    """The mask is recognised as an operand in host arrays, which are staged one by
    one, and in copies: no CTA kind for triangles."""
    L = gk.lower_host(gk.gen_rmat(11, 16, seed=3))
    want = orc.mxmm(L, L, L)
    D = L.to("cuda")
    copy = L.to("cuda")
    for args in ((D, D, D), (D, D, copy), (L, L, L)):
        got, names = kernels(lambda: gk.mxmm_masked(*args, sched="learned"))
        np.testing.assert_array_equal(got.cpu().numpy() if hasattr(got, "cpu") else got, want)
        assert not any("k_packed_cta" in x for x in names)


@pytest.mark.parametrize("m,groups", [(131071, False), (131072, True)])
def test_plain_rows_of_a_few_products(gk, orc, cuda, m, groups):
    """Of very many rows of a few products each, most are left to the groups of four
    threads (not the rows of 32 products and more); of fewer, none."""
    L = gk.lower_host(gk.gen_er(m, 2 * m, seed=4))
    D = L.to("cuda")
    got, names = kernels(lambda: gk.tc_row_sums(D))
    np.testing.assert_array_equal(got.cpu().numpy().astype(np.uint64), orc.tc_row_sums(L))
    assert any("k_group" in x for x in names) == groups
    got, names = kernels(lambda: gk.mxmm_masked(D, D, D))
    np.testing.assert_array_equal(got.cpu().numpy(), orc.mxmm(L, L, L))
    assert any("k_group" in x for x in names) == groups
