"""GPU: the cluster kernel (lnt_cluster.cu), one test over the CTAs of a cluster.

Every digit against the oracle at every length and cluster size it serves, both modes, both
run lengths; states handed over from and to the two-pass kernels; several tests in one launch.
"""
import numpy as np
import pytest

from oracle import bigint_model as B

pytestmark = pytest.mark.gpu


def random_digits(q, n, seed):
    rng = np.random.default_rng(seed)
    w = np.array(B.widths(q, n), dtype=np.uint64)
    return (rng.integers(0, 2**62, size=n, dtype=np.uint64) % (np.uint64(1) << w)).astype(np.uint64)


# the policy's exponents of each length, and (second of a length) short words: runs of eight
@pytest.mark.parametrize("q,n", [(9689, 512), (4253, 512), (21701, 1024), (44021, 2048), (20011, 2048),
                                 (86243, 4096), (160001, 8192), (60013, 8192), (316003, 16384), (620009, 32768)])
@pytest.mark.parametrize("prp", [False, True])
def test_digits_equal_oracle(lnt, oracle_mod, q, n, prp):
    start = random_digits(q, n, q)
    with lnt.LucasTest(q, n, prp) as g, oracle_mod.OracleTest(q, n, prp) as o:
        assert "cluster_square_loop" in g.profile_iterations(1)
        g.set_digits(start)
        o.set_digits(start)
        for k in (1, 2, 5):
            g.iterate(k)
            o.iterate(k)
            assert np.array_equal(g.digits(), o.digits()), (q, n, prp, k)


@pytest.mark.parametrize("n", [512, 8192, 32768])
def test_extreme_digits(lnt, oracle_mod, n):
    """All digits at their maximum, and all zero."""
    q = {512: 9689, 8192: 160001, 32768: 620009}[n]
    top = ((np.uint64(1) << np.array(B.widths(q, n), dtype=np.uint64)) - np.uint64(1)).astype(np.uint64)
    for start in (top, np.zeros(n, np.uint64)):
        with lnt.LucasTest(q, n, True) as g, oracle_mod.OracleTest(q, n, True) as o:
            g.set_digits(start)
            o.set_digits(start)
            g.iterate(3)
            o.iterate(3)
            assert np.array_equal(g.digits(), o.digits())


def test_pending_carries_of_the_two_pass_kernels(lnt):
    """The Gerbicz products (two-pass kernels) leave run carries that the next squarings take in."""
    with lnt.LucasTest(160001, 8192, prp=True) as a, lnt.LucasTest(160001, 8192, prp=True) as b:
        a.gerbicz_enable(4)
        for k in (3, 10, 20, 32):
            a.iterate(k)
            b.iterate(k)
            assert np.array_equal(a.digits(), b.digits())
        assert a.gerbicz_stats()["checks"] >= 3 and a.gerbicz_stats()["errors"] == 0


@pytest.mark.parametrize("count", [1, 7, 24, 60, 160])
def test_batches_of_every_cluster_size(lnt, count):
    """Mixed lengths in one launch: clusters of eight, four, and one CTA per test (fewer tests than SMs, and
    more), against the same tests alone."""
    qs = [(9689, 21701, 44021, 86243)[i % 4] + 2 * i for i in range(count)]
    with lnt.Batch() as b:
        ids = [b.submit(q, prp=bool(i & 1), iterations=300) for i, q in enumerate(qs)]
        b.run(300)
        got = {r["id"]: r for r in b.poll()}
    for i, q in enumerate(qs[:8]):
        with lnt.LucasTest(q, prp=bool(i & 1)) as t:
            for _ in range(3):
                t.iterate(100)
            assert got[ids[i]]["res64"] == t.res64() and got[ids[i]]["status"] == 0


def test_two_pass_groups_take_over(lnt):
    """Batches of 8K words and more run on the two-pass kernels from the first squaring on, and end on
    the residues that the cluster kernel gives."""
    with lnt.Batch() as b:
        ids = [b.submit(q, prp=True, iterations=50) for q in (160001, 160033, 316003)]
        b.run(50)
        got = {r["id"]: r["res64"] for r in b.poll()}
    for i, q in zip(ids, (160001, 160033, 316003)):
        with lnt.LucasTest(q, prp=True) as t:
            t.iterate(50)
            assert got[i] == t.res64()


@pytest.mark.parametrize("q,n", [(9689, 512), (44021, 2048), (160001, 8192), (620009, 32768)])
@pytest.mark.parametrize("squaring", [0, 1, 6])
def test_a_wait_that_gives_up(lnt, oracle_mod, q, n, squaring):
    """A CTA that leaves early: the others give up at waits of 50 ms, the readout reports it, and
    the GPU runs on.  A launch that ends before that squaring is not touched."""
    start = random_digits(q, n, q + 1)
    with lnt.LucasTest(q, n, True) as t:
        t.set_digits(start)
        if squaring:
            t.debug_cluster_quit(squaring)
            t.iterate(squaring)
            t.synchronize()
        t.debug_cluster_quit(squaring)
        t.iterate(20)
        with pytest.raises(lnt.LucasNTTError, match="cluster kernel timed out") as e:
            t.digits()
        assert e.value.status == 3
    with lnt.LucasTest(q, n, True) as t, oracle_mod.OracleTest(q, n, True) as o:
        t.set_digits(start)
        o.set_digits(start)
        t.iterate(4)
        o.iterate(4)
        assert np.array_equal(t.digits(), o.digits())
