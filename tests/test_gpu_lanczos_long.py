"""The FP64 Lanczos reduction of long chains (fixed-point sweeps) against numpy and against
the kernel of shorter chains."""
import dataclasses

import numpy as np
import pytest

from helpers import strong_diffs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _reference(E, M, nit):
    """Rows of the multi-pivot reduction with unit pivots, three Gram-Schmidt sweeps a step."""
    D = len(M)
    V, rows, last = [], [], []
    for p in range(D):
        for k in range(nit):
            w = M[p].copy() if k == 0 else E * V[-1]
            for _ in range(3):
                if V:
                    B = np.array(V)
                    w = w - (B @ w) @ B
            beta = np.linalg.norm(w)
            u = w / beta
            g = [float(np.dot(V[t], E * u)) for t in last]
            row = np.zeros(2 * D + 1)
            row[0], row[1] = np.dot(u, E * u), g[-1] if k == 0 and g else beta
            row[2:2 + len(g)] = g
            row[D + 1:] = M @ u
            V.append(u)
            rows.append(row)
        last.append(len(V) - 1)
    return np.array(rows)


def _run(bdmod, E, M, nit):
    D, N = M.shape
    tE, tM = torch.from_numpy(E).cuda(), torch.from_numpy(M).cuda()
    out = torch.full((min(N, D * nit), 2 * D + 1), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    L, ipiv, piv, nits = bdmod.lanczos_chain_noalloc(tE.data_ptr(), tM.data_ptr(), N, D, np.eye(D),
                                                     np.full(D, nit, np.int32), out.data_ptr(), len(out))
    return out.cpu().numpy()[:L]


# the shortest chain it takes and one less; remainders of the 16 slices and of the four poles a
# thread; more vectors than the 64 a round of warps takes; D = 1 and 8
@pytest.mark.parametrize("N,D,nit", [(2047, 2, 9), (2048, 2, 9), (2049, 1, 30), (4099, 8, 9), (20011, 4, 17)])
def test_rows_against_numpy(bdmod, N, D, nit):
    rng = np.random.default_rng(N)
    E = np.sort(rng.uniform(20.0, 300.0, N))
    M = rng.standard_normal((D, N)) * np.exp(-E / 100.0)
    got, ref = _run(bdmod, E, M, nit), _reference(E, M, nit)
    scale = np.maximum(np.abs(ref).max(0), 1e-300)
    # FP64 rounding of E v (a few hundred eps of a coupling) over the steps
    assert (np.abs(got - ref) / scale).max() < 1e-11


@pytest.mark.parametrize("kind", ["zeros", "huge", "tiny", "few"])
def test_unusual_chains(bdmod, kind):
    """Poles no vector reaches; energies and couplings outside the fixed-point range (left to
    the other kernel); a space of fewer directions than rows (its restart vectors too)."""
    rng = np.random.default_rng(5)
    N, D, nit = 3001, 2, 10
    E = np.sort(rng.uniform(20.0, 300.0, N))
    M = rng.standard_normal((D, N))
    scale = 1.0
    if kind == "zeros":
        M[:, 1::3] = 0.0
    elif kind == "huge":
        scale = 1e14
        E = E * scale
    elif kind == "tiny":
        M = M * 1e-14
    else:
        M[:, 12:] = 0.0                # twelve reachable poles: both chains end early
        nit = 40
    got = _run(bdmod, E, M, nit)
    assert np.isfinite(got).all() and len(got) == D * nit
    if kind == "few":
        # the twelve poles the couplings reach and rows that couple to nothing: sum of m m^T kept
        G = got[:, D + 1:].T @ got[:, D + 1:]
        np.testing.assert_allclose(G, M @ M.T, rtol=1e-10)
        return
    ref = _reference(E, M, nit)
    s = np.maximum(np.abs(ref).max(0), 1e-300)
    assert (np.abs(got - ref) / s).max() < 1e-11


def test_dressed_chains_vectors_and_slices(bdmod, problems):
    """A context's long chains: the stored basis read back (two integer planes a vector), and
    clusters of 2 CTAs, whose slices do not fit in shared memory, against 8."""
    p = problems(6, 20.0, 1, 12)
    ctx = bdmod.Context().upload(p)
    ctx.run_all(lanczos=True)
    ctx.dressed_propagator(1e-3, 2)
    ish = max(range(p.ms.nsubsh), key=lambda i: ctx.count_poles(i)[0])
    n = ctx.count_poles(ish)
    assert n[0] > 20000
    ctx.run_all(lanczos=True)
    a = ctx.result(ish)
    pv = p.piv
    fw, _ = ctx.sigma2_build(ish)
    lz = ctx.lanczos_reduce(ish, pv.vec[ish], pv.n_fw[ish], pv.n_bk[ish])
    V = ctx.lanczos_vectors(ish, 0, len(lz["lz_fw"]), n[0])
    assert np.abs(V @ V.T - np.eye(len(V))).max() < 1e-13
    E = np.sort(fw[:, 0])
    alpha = np.einsum("ti,i,ti->t", V, E, V)
    assert np.abs(alpha - lz["lz_fw"][:, 0]).max() < 1e-12 * np.abs(E).max()
    ctx.set_tuning(lz_cluster=2)
    ctx.run_all(lanczos=True)
    b = ctx.result(ish)
    for tag in ("qp", "qh"):
        e, z = strong_diffs(a[tag], b[tag])
        assert e < 1e-10 and z < 1e-9
    ctx.close()


@pytest.mark.parametrize("D,nq", [(1, 300), (3, 300), (7, 270), (8, 129), (3, 128)])
def test_unreached_directions_of_many_groups(bdmod, D, nq):
    """Groups of 1 to 24 equal energies, more (and just as many) energies than are ranked by
    whole warps: an exhausted chain's rows take each group's m - rank(M) directions in order."""
    rng = np.random.default_rng(D)
    m = np.arange(nq) % 24 + 1
    Eq = np.sort(rng.uniform(20.0, 300.0, nq))
    E = np.repeat(Eq, m)
    first = np.concatenate([[0], np.cumsum(m)])
    M = np.zeros((D, len(E)))
    expect = []
    for q in range(nq):
        s = slice(first[q], first[q + 1])
        if q % 40 == 7:                                    # full rank
            M[:, s] = rng.standard_normal((D, m[q]))
        elif q % 40 == 23:                                 # rank one (24 poles)
            M[:, s] = np.outer(rng.standard_normal(D), rng.standard_normal(m[q]))
        rank = np.linalg.matrix_rank(M[:, s]) if M[:, s].any() else 0
        expect += [Eq[q]] * (m[q] - int(rank))
    got = _run(bdmod, E, M, 60)
    defl = got[np.abs(got[:, 1:]).max(1) == 0, 0]
    assert len(defl) > 20
    assert np.array_equal(defl, np.array(expect)[:len(defl)])


def _run_pivots(bdmod, E, M, piv, nits):
    D, N = M.shape
    tE, tM = torch.from_numpy(E).cuda(), torch.from_numpy(np.ascontiguousarray(M)).cuda()
    out = torch.full((int(sum(nits)), len(piv) + 1 + D), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    L, *_ = bdmod.lanczos_chain_noalloc(tE.data_ptr(), tM.data_ptr(), N, D, piv, np.array(nits, np.int32), out.data_ptr(),
                                        len(out))
    return out.cpu().numpy()[:L]


# the second orbital's couplings below the first's by as much as FP32's squares hold, and beyond (|M p|^2 from
# 2^-90 down); a second pivot in which couplings cancel down to their last bits (an exact difference); a second
# pivot that lives on poles next to zero (|E v|^2)
@pytest.mark.parametrize("kind,size", [("orbital", 1e-11), ("orbital", 1e-14), ("orbital", 1e-20), ("orbital", 1e-24),
                                       ("orbital", 1e-40), ("cancelling", 1e-11), ("energies", 1e-24)])
def test_weakly_coupled_orbital(bdmod, kind, size):
    rng = np.random.default_rng(11)
    N, nit = 2500, 8
    E = np.sort(rng.uniform(20.0, 300.0, N))
    M = rng.standard_normal((2, N))
    piv = np.eye(2)
    if kind == "orbital":
        M[1] *= size
    elif kind == "cancelling":
        M = np.concatenate([M * size, np.zeros((2, N))])
        M[1] = M[0] * (1.0 + 2.0 ** -52 * rng.integers(-3, 4, N))
        piv = np.array([[1.0, 0.0, 0.0, 0.0], [0.5, -0.5, 0.5, -0.5]])
    else:
        E[:40] = np.sort(rng.uniform(1.0, 2.0, 40)) * size
        M[0, :40] = 0.0
        M[1, 40:] = 0.0
    got = _run_pivots(bdmod, E, M, piv, [nit, nit])
    ref = _reference(E, piv @ M, nit)
    for c in (0, 1):   # every chain on the scale of the energies it lives on
        r = slice(c * nit, (c + 1) * nit)
        scale = np.abs(ref[r, 0]).max()
        assert np.abs(got[r, 0] - ref[r, 0]).max() < 1e-11 * scale, c
        assert np.abs(got[r, 1][1:] - ref[r, 1][1:]).max() < 1e-11 * scale, c
        assert np.abs(got[r, 2] - ref[r, 2]).max() < 1e-11 * 300.0, c


# A vector of equal elements against one of two values: the fixed-point words of all elements have one sign, so
# neither their cross products (1 and 4 times 2^63) nor the products of their low words (4e-14 |w|) cancel.
@pytest.mark.parametrize("overlap", [0.694, 0.678])
def test_elements_of_one_size(bdmod, overlap):
    N = 111230   # (an element 1 / sqrt(N) whose low word is the largest there is)
    rng = np.random.default_rng(1)
    E = np.sort(rng.uniform(20.0, 300.0, N))
    s = np.where(np.arange(N) < N // 2, 1.0, -1.0)
    M = np.array([np.ones(N), overlap + np.sqrt(1.0 - overlap ** 2) * s])
    got = _run_pivots(bdmod, E, M, np.eye(2), [1, 3])
    u = M[1] - M[1].mean()
    u = u / np.linalg.norm(u)
    g = np.dot(np.full(N, 1.0 / np.sqrt(N)), E * u)
    # FP64 sums of a hundred thousand terms over a tree of at most some 64 additions in a row: 64 eps of the terms' sizes
    tol = 64 * 2.2e-16
    assert abs(got[1, 0] - np.dot(u, E * u)) < tol * 300.0
    assert abs(got[1, 1] - g) < tol * 300.0
    assert abs(got[1, 3]) < tol * np.sqrt(N)          # <M_0|u>, nothing
    assert abs(got[1, 4] - np.dot(M[1], u)) < tol * np.sqrt(N)


# pivots whose couplings depend on one another: exactly, through a combination, but for 1e-5 of them (the FP64 sums
# tell), by an orbital that couples to nothing
@pytest.mark.parametrize("kind", ["twice", "difference", "close", "none"])
@pytest.mark.parametrize("N", [2500, 20011])
def test_dependent_pivots(bdmod, N, kind):
    rng = np.random.default_rng(N)
    nit = 8
    E = np.sort(rng.uniform(20.0, 300.0, N))
    M = rng.standard_normal((3, N))
    if kind == "twice":
        M[2] = 2.0 * M[0]
    elif kind == "difference":
        M[2] = M[0] - M[1]
    elif kind == "close":
        M[2] = M[0] - M[1] + 1e-5 * M[2]
    else:
        M[2] = 0.0
    got = _run(bdmod, E, M, nit)
    assert got.shape == (3 * nit, 7) and np.isfinite(got).all()
    n = 3 if kind == "close" else 2              # (the third chain's are restart vectors otherwise)
    ref = _reference(E, M[:n], nit)
    r = n * nit
    # FP64 rounding of E v over the steps, of the couplings' remainder where they are close
    tol = 1e-11 if kind != "close" else 1e-9
    assert np.abs(got[:r, 0] - ref[:, 0]).max() < tol * 300.0
    assert np.abs(got[:r, 2:1 + n] - ref[:, 2:1 + n]).max() < tol * 300.0
    assert np.abs(got[:r, 4:4 + n] - ref[:, 1 + n:]).max() < tol * np.sqrt(N)


# many chains in a launch: the longest below the length from which k_lz_long takes them all, and above it
@pytest.mark.parametrize("nmax,frag,long", [(6, 1, False), (4, 2, True)])
def test_batches_on_both_sides_of_the_rule(bdmod, problems, nmax, frag, long):
    p = problems(nmax, 20.0, 1, 12)
    ctx = bdmod.Context().upload(p)
    ctx.run_all(lanczos=True)
    ctx.dressed_propagator(1e-3, frag)
    n = [max(ctx.count_poles(i)) for i in range(p.ms.nsubsh)]
    assert p.ms.nsubsh > 15 and max(n) > 2048 and (max(n) >= 8192) == long
    got = []
    for mode in (0, 1):   # 1: k_lanczos alone
        ctx.set_lanczos_slices(mode)
        ctx.run_all(lanczos=True)
        got.append([ctx.result(i) for i in range(p.ms.nsubsh)])
    for a, b in zip(*got):
        for tag in ("qp", "qh"):
            assert len(a[tag]) == len(b[tag])
            e, z = strong_diffs(b[tag], a[tag])
            assert e < 1e-10 and z < 1e-9
        np.testing.assert_allclose(a["koltun"], b["koltun"], rtol=1e-10, atol=1e-11)
    ctx.close()
