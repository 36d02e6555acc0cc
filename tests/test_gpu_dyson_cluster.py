"""The cluster Householder reduction and the eigenvector kernel of orders beyond 160: just
above that order, with rows beyond shared memory, on every cluster size."""
import numpy as np
import pytest

from helpers import strong_diffs

pytestmark = pytest.mark.gpu


# 161: one row a CTA more than 160 / 16; 163: a remainder in every split; 688 and 1 100: the
# first keeps all rows in shared memory, the second does not; D = 1 and 4
@pytest.mark.parametrize("n,ish", [(161, 1), (163, 0), (337, 2), (688, 0), (1100, 5)])
def test_large_orders_against_lapack(bdmod, problems, n, ish):
    p = problems(6, 20.0, 1, 50)
    rng = np.random.default_rng(n)
    ctx = bdmod.Context().upload(p)
    D = int(p.ms.no[ish])
    nb = (n - D) // 4
    nf = n - D - nb
    fw, bk = np.zeros((nf, 2 + D)), np.zeros((nb, 2 + D))
    fw[:, 0], bk[:, 0] = rng.uniform(20.0, 300.0, nf), -rng.uniform(60.0, 250.0, nb)
    fw[:, 2:], bk[:, 2:] = rng.standard_normal((nf, D)) * 0.3, rng.standard_normal((nb, D)) * 0.3
    s1, hf = np.diag(np.linspace(-20.0, 60.0, D)), np.zeros((D, D))
    r = ctx.dyson_rows(ish, 2, fw, bk, sig1b=s1, sighf=hf, efermi=-50.0)
    A = np.diag(np.concatenate([np.zeros(D), fw[:, 0], bk[:, 0]]))
    A[:D, :D] = s1
    A[D:, :D] = np.concatenate([fw[:, 2:], bk[:, 2:]])
    A[:D, D:] = A[D:, :D].T
    w, v = np.linalg.eigh(A)
    got = np.concatenate([r["qp"], r["qh"]])
    assert len(got) == n
    # the bisection stops at max(1e-12 |W|, 1e-13 |T|); double-float rounding is below it
    np.testing.assert_allclose(np.sort(got[:, 0]), w, rtol=1e-11, atol=1e-11 * np.abs(A).sum(0).max())
    ref = np.concatenate([w[:, None], (v[:D] ** 2).sum(0)[:, None], v[:D].T], 1)
    e, z = strong_diffs(ref, got)
    assert e < 1e-10 and z < 1e-8
    # the rows of Q stay orthonormal: sum_k x_k x_k^T = 1
    x = got[:, 2:]
    assert np.abs(x.T @ x - np.eye(D)).max() < 1e-11
    ctx.close()


def test_cluster_sizes_agree(bdmod, problems):
    """Batched, orders up to 203 (D = 3, both directions 100 rows): clusters of 1 to 16 CTAs."""
    p = problems(4, 20.0, 0, 40)
    ctx = bdmod.Context().upload(p)
    ctx.run_all(lanczos=True)
    ctx.dressed_propagator(1e-3, 1)
    got = {}
    for c in (8, 1, 2, 4, 16):
        ctx.set_tuning(dy_cluster=c)
        ctx.run_all(lanczos=True)
        got[c] = [ctx.result(i) for i in range(p.ms.nsubsh)]
        for a, b in zip(got[8], got[c]):
            for tag in ("qp", "qh"):
                assert len(a[tag]) == len(b[tag])
                e, z = strong_diffs(a[tag], b[tag])
                assert e < 1e-10 and z < 1e-8, c
            np.testing.assert_allclose(a["koltun"], b["koltun"], rtol=1e-10, atol=1e-11)
    ctx.close()


# the smallest order one matrix takes the whole GPU for and one less, orders that are no multiple
# of its CTAs, rows beyond shared memory; D from the channel
@pytest.mark.parametrize("n,ish", [(383, 1), (384, 1), (511, 1), (512, 1), (531, 5), (760, 2), (1901, 0)])
def test_one_matrix_on_the_whole_gpu(bdmod, problems, n, ish):
    p = problems(6, 20.0, 1, 50)
    rng = np.random.default_rng(n)
    ctx = bdmod.Context().upload(p)
    D = int(p.ms.no[ish])
    nb = (n - D) // 3
    nf = n - D - nb
    fw, bk = np.zeros((nf, 2 + D)), np.zeros((nb, 2 + D))
    fw[:, 0], bk[:, 0] = rng.uniform(20.0, 300.0, nf), -rng.uniform(60.0, 250.0, nb)
    fw[:, 2:], bk[:, 2:] = rng.standard_normal((nf, D)) * 0.3, rng.standard_normal((nb, D)) * 0.3
    s1, hf = np.diag(np.linspace(-20.0, 60.0, D)), np.zeros((D, D))
    r = ctx.dyson_rows(ish, 2, fw, bk, sig1b=s1, sighf=hf, efermi=-50.0)
    A = np.diag(np.concatenate([np.zeros(D), fw[:, 0], bk[:, 0]]))
    A[:D, :D] = s1
    A[D:, :D] = np.concatenate([fw[:, 2:], bk[:, 2:]])
    A[:D, D:] = A[D:, :D].T
    w, v = np.linalg.eigh(A)
    got = np.concatenate([r["qp"], r["qh"]])
    assert len(got) == n
    # the tolerances of the cluster kernel's test above: the arithmetic is the same
    np.testing.assert_allclose(np.sort(got[:, 0]), w, rtol=1e-11, atol=1e-11 * np.abs(A).sum(0).max())
    ref = np.concatenate([w[:, None], (v[:D] ** 2).sum(0)[:, None], v[:D].T], 1)
    e, z = strong_diffs(ref, got)
    assert e < 1e-10 and z < 1e-8
    x = got[:, 2:]
    assert np.abs(x.T @ x - np.eye(D)).max() < 1e-11
    ctx.close()


def test_whole_gpu_reductions_of_two_threads(bdmod, problems):
    """Two contexts on two host threads, each solving large matrices that take every SM: the same
    bits as alone."""
    import threading
    p = problems(4, 20.0, 0, 20)
    D = int(p.ms.no[0])
    rng = np.random.default_rng(3)
    jobs = []
    for n in (600, 777):
        rows = np.zeros((n, 2 + D))
        rows[:, 0], rows[:, 2:] = rng.uniform(20.0, 300.0, n), rng.standard_normal((n, D)) * 0.3
        ctx = bdmod.Context().upload(p)

        def solve(ctx=ctx, rows=rows):
            r = ctx.dyson_rows(0, 2, rows, np.zeros((0, 2 + D)), sig1b=np.diag(np.linspace(-20.0, 60.0, D)),
                               sighf=np.zeros((D, D)), efermi=-50.0)
            return np.concatenate([r["qp"], r["qh"]])
        jobs.append((ctx, solve, solve()))
    bad = []

    def work(solve, want):
        for _ in range(5):
            if not np.array_equal(solve(), want):
                bad.append(len(want))
    threads = [threading.Thread(target=work, args=j[1:]) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for j in jobs:
        j[0].close()


def test_orders_beyond_2300_in_fp64(bdmod, problems):
    """The eigenvector components of an order that is reduced in FP64: off by LAPACK's own rounding in the median
    (about 1e-15), where double-float's 2^-48 leaves 1.8e-14."""
    p = problems(6, 20.0, 1, 50)
    n, ish = 2403, 0
    rng = np.random.default_rng(n)
    ctx = bdmod.Context().upload(p)
    D = int(p.ms.no[ish])
    nb = n // 5
    nf = n - D - nb
    fw, bk = np.zeros((nf, 2 + D)), np.zeros((nb, 2 + D))
    fw[:, 0], bk[:, 0] = rng.uniform(20.0, 300.0, nf), -rng.uniform(60.0, 250.0, nb)
    fw[:, 2:], bk[:, 2:] = (rng.standard_normal((k, D)) * (4.0 / np.sqrt(nf)) for k in (nf, nb))
    s1, hf = np.diag(np.linspace(-20.0, 60.0, D)), np.zeros((D, D))
    r = ctx.dyson_rows(ish, 2, fw, bk, sig1b=s1, sighf=hf, efermi=-50.0)
    ctx.close()
    A = np.diag(np.concatenate([np.zeros(D), fw[:, 0], bk[:, 0]]))
    A[:D, :D] = s1
    A[D:, :D] = np.concatenate([fw[:, 2:], bk[:, 2:]])
    A[:D, D:] = A[D:, :D].T
    w, v = np.linalg.eigh(A)
    got = np.concatenate([r["qp"], r["qh"]])
    got, ref = got[np.argsort(got[:, 0])], v[:D].T
    x = got[:, 2:] * np.where((got[:, 2:] * ref).sum(1) < 0.0, -1.0, 1.0)[:, None]
    assert np.median(np.abs(x - ref).max(1)) < 6e-15


# more orbitals than the model spaces above have, on the cluster kernel and on the whole GPU (a row of Q each)
@pytest.mark.parametrize("n,nmax,D", [(203, 12, 7), (305, 14, 8), (400, 12, 7), (611, 14, 8)])
def test_seven_and_eight_orbitals(bdmod, synth, n, nmax, D):
    ms = synth.make_modspace(nmax, 20.0)
    prop = synth.make_unperturbed_propagator(ms)
    none = synth.Interaction(np.zeros(1, np.int32), np.zeros(1, np.int32), np.zeros(1))
    ctx = bdmod.Context().upload(synth.Problem(ms, prop, none, synth.make_pivots(ms, prop, 1), 0, 1.0), with_pivots=False)
    assert int(ms.no[0]) == D
    rng = np.random.default_rng(n)
    nb = n // 4
    nf = n - D - nb
    fw, bk = np.zeros((nf, 2 + D)), np.zeros((nb, 2 + D))
    fw[:, 0], bk[:, 0] = rng.uniform(20.0, 300.0, nf), -rng.uniform(60.0, 250.0, nb)
    fw[:, 2:], bk[:, 2:] = rng.standard_normal((nf, D)) * 0.3, rng.standard_normal((nb, D)) * 0.3
    s1, hf = np.diag(np.linspace(-20.0, 60.0, D)), np.zeros((D, D))
    r = ctx.dyson_rows(0, 2, fw, bk, sig1b=s1, sighf=hf, efermi=-50.0)
    ctx.close()
    A = np.diag(np.concatenate([np.zeros(D), fw[:, 0], bk[:, 0]]))
    A[:D, :D] = s1
    A[D:, :D] = np.concatenate([fw[:, 2:], bk[:, 2:]])
    A[:D, D:] = A[D:, :D].T
    w, v = np.linalg.eigh(A)
    got = np.concatenate([r["qp"], r["qh"]])
    # as test_large_orders_against_lapack
    np.testing.assert_allclose(np.sort(got[:, 0]), w, rtol=1e-11, atol=1e-11 * np.abs(A).sum(0).max())
    ref = np.concatenate([w[:, None], (v[:D] ** 2).sum(0)[:, None], v[:D].T], 1)
    e, z = strong_diffs(ref, got)
    assert e < 1e-10 and z < 1e-8
    x = got[:, 2:]
    assert np.abs(x.T @ x - np.eye(D)).max() < 1e-11
