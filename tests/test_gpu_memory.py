"""Calls that find no memory for the faster path's scratch take the one that needs
less: the failing allocation is made to fail on the host (gk_inject_alloc_failure)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def failures(gk, op, check, tries):
    """How many of the first `tries` allocations, failing one at a time, fail the
    call; the others' results are checked."""
    lib = gk.load()
    op()  # what is allocated once per process
    failed = []
    for after in range(tries):
        lib.gk_inject_alloc_failure(after)
        try:
            out = op()
        except gk.GkError as e:
            assert e.code == gk._lib.GK_ERR_OOM, str(e)
            failed.append(after)
            continue
        finally:
            lib.gk_inject_alloc_failure(-1)
        check(out)
    return failed


def test_count_without_room_for_the_degree_order(gk, orc, cuda):
    L = gk.extract_lower(gk.gen_rmat(17, 16, seed=3, device="cuda"))
    want = orc.tc_merge(L.numpy())

    def same(got):
        assert got == want

    # the result's word alone cannot do without its allocation
    assert failures(gk, lambda: gk.tc_count(L), same, 45) == [0]


def test_batch_without_room_for_the_degree_order(gk, orc, cuda):
    host = [gk.lower_host(gk.gen_rmat(12, 24, seed=i)) for i in range(3)]
    host += [gk.lower_host(gk.gen_er(3000, 9000, seed=i)) for i in range(3)]
    graphs = [x.to("cuda") for x in host]
    want = np.array([orc.tc_lower(x) for x in host], dtype=np.uint64)
    failed = failures(gk, lambda: gk.tc_count_batched(graphs), lambda got: np.testing.assert_array_equal(got, want), 60)
    assert len(failed) <= 12, failed  # the combined matrix, the tables and a word per group


def test_ktruss_without_room_for_the_peeling(gk, orc, cuda):
    """The product loop takes over, whichever of the peeling's allocations fails."""
    A = gk.gen_rmat(11, 16, seed=6)
    rp, col, iters, _ = orc.ktruss(A, 5)
    G = A.to("cuda")

    def same(got):
        T, it = got
        assert it == iters
        np.testing.assert_array_equal(T.rowptr.cpu().numpy(), rp)
        np.testing.assert_array_equal(T.col.cpu().numpy(), col)

    failed = failures(gk, lambda: gk.ktruss(G, 5), same, 60)
    # the matrix's copies, the check's word, the entries' rows and the symmetry's counters
    assert failed == list(range(5)), failed


@pytest.mark.parametrize("nsrc", [100, 600])
def test_bc_without_room_for_a_wide_chunk(gk, orc, cuda, nsrc):
    """A chunk whose allocations fail is narrowed; one of 32 sources needs them all
    (one reservation and the eight arrays carved from it)."""
    from tests import graphs as G
    A = gk.gen_rmat(11, 8, seed=6)
    src = np.random.default_rng(1).permutation(A.m)[:nsrc]
    want, want20 = orc.bc_f64(A, src), orc.bc_f64(A, src[:20])
    D = A.to("cuda")
    wide = failures(gk, lambda: gk.bc_batch(D, src).cpu().numpy(), lambda got: G.assert_bc_close(got, want), 60)
    narrow = failures(gk, lambda: gk.bc_batch(D, src[:20]).cpu().numpy(), lambda got: G.assert_bc_close(got, want20), 60)
    assert len(wide) == len(narrow) - 9, (wide, narrow)
