"""The Lanczos reduction in the space the couplings span (chains of few distinct energies)
against the reduction over all poles, which bd_set_lanczos_slices(1) keeps."""
import numpy as np
import pytest

from helpers import strong_diffs

pytestmark = pytest.mark.gpu


# h-bar omega values whose shell energies round to one and to several doubles; groups smaller
# and larger than a rotation keeps; one step a pivot, truncated and exhausted chains; L = N
# (every backward chain at N_max = 2, where some need a restart vector and are left to the
# full space); odd N_max
@pytest.mark.parametrize("nmax,hw,nit", [(2, 20.0, 10), (3, 13.7, 7), (4, 27.3, 3), (5, 20.0, 1), (6, 11.9, 50),
                                         (7, 23.1, 30)])
def test_compact_reduction_equals_full(bdmod, problems, nmax, hw, nit):
    p = problems(nmax, hw, 3, nit)
    ctx = bdmod.Context().upload(p)
    pv = p.piv
    built = 0
    for ish in range(p.ms.nsubsh):
        D = int(p.ms.no[ish])
        s1 = np.diag(p.ms.orb_xe[p.ms.orb_start[ish]:p.ms.orb_start[ish] + D])
        got = []
        for mode in (0, 1):
            ctx.set_lanczos_slices(mode)
            ctx.sigma2_build(ish, copy=False)
            lz = ctx.lanczos_reduce(ish, pv.vec[ish], pv.n_fw[ish], pv.n_bk[ish])
            got.append((lz, ctx.lanczos_stored()[ish].copy(), ctx.dyson_solve(ish, s1)))
            if mode == 0:
                # the stored vectors, formed over the poles: orthonormal, and T = V E V^T on the rows
                fw, bk = ctx.sigma2_build(ish)
                for d, sig, tag in ((0, fw, "lz_fw"), (1, bk, "lz_bk")):
                    L, N = len(lz[tag]), len(sig)
                    if L == 0:
                        continue
                    V = ctx.lanczos_vectors(ish, d, L, N)
                    on = np.abs(V).max(1) > 0
                    Vs = V[on]
                    # a factor's error grows with its pivots' loss, at most 1e3 eps (kPivot)
                    assert np.abs(Vs @ Vs.T - np.eye(len(Vs))).max() < 1e-12
                    E = sig[np.argsort(sig[:, 0] if d == 0 else -sig[:, 0], kind="stable"), 0]
                    alpha = np.einsum("ti,i,ti->t", Vs, E, Vs)
                    assert np.abs(alpha - lz[tag][on, 0]).max() < 1e-10 * np.abs(E).max()
                    built += len(Vs)
        (la, sa, ra), (lb, sb, rb) = got
        assert np.array_equal(sa, sb), ish                      # as many vectors built
        for tag in ("lz_fw", "lz_bk"):
            assert la[tag].shape == lb[tag].shape
            na = np.abs(la[tag][:, 1:]).max(1) == 0              # the same deflated rows
            nb = np.abs(lb[tag][:, 1:]).max(1) == 0
            assert np.array_equal(na, nb) and np.array_equal(la[tag][na], lb[tag][nb]), (ish, tag)
        for tag in ("qp", "qh"):
            assert len(ra[tag]) == len(rb[tag])
            e, z = strong_diffs(rb[tag], ra[tag])
            assert e < 1e-10 and z < 1e-10, (ish, tag, e, z)
        np.testing.assert_allclose(ra["koltun"], rb["koltun"], rtol=1e-10, atol=1e-11)
    assert built > 0
    ctx.close()


@pytest.mark.parametrize("nmax,hw,kind", [(2, 20.0, "batched"), (3, 13.7, "channel"), (4, 27.3, "batched"),
                                          (4, 20.0, "channel"), (4, 20.0, "dressed")])
def test_rotated_full_dyson_equals_plain_rows(bdmod, problems, nmax, hw, kind):
    """The un-reduced solve, its equal energies rotated, against the same rows handed in by the
    caller (bd_dyson_rows solves them as they are)."""
    p = problems(nmax, hw, 3, 1)
    ctx = bdmod.Context().upload(p)
    if kind == "dressed":                       # distinct energies: nothing to rotate
        ctx.run_all(lanczos=False)
        ctx.dressed_propagator(0.5, 1)
    ctx.run_all(lanczos=False, graph=(kind == "batched"))
    for ish in range(0, p.ms.nsubsh, 3):
        D = int(p.ms.no[ish])
        s1 = np.diag(p.ms.orb_xe[p.ms.orb_start[ish]:p.ms.orb_start[ish] + D])
        a = ctx.result(ish)
        hf = ctx.ehf(ish)
        fw, bk = ctx.sigma2_build(ish)
        if kind == "channel":
            a = ctx.dyson_solve(ish, s1, hf)
        ctx2 = bdmod.Context().upload(p)
        ef = float((a["qp"][-1, 0] + a["qh"][0, 0]) / 2) if len(a["qh"]) else float(a["qp"][-1, 0]) - 1.0
        b = ctx2.dyson_rows(ish, 2, fw, bk, sig1b=s1, sighf=hf, efermi=ef)
        ctx2.close()
        for tag in ("qp", "qh"):
            assert len(a[tag]) == len(b[tag])
            assert np.all(np.diff(a[tag][:, 0]) <= 0)
            # every energy, the unreached directions' among them
            np.testing.assert_allclose(a[tag][:, 0], b[tag][:, 0], rtol=1e-10, atol=1e-10)
            e, z = strong_diffs(b[tag], a[tag])
            assert e < 1e-10 and z < 1e-10, (ish, tag, e, z)
        np.testing.assert_allclose(a["koltun"], b["koltun"], rtol=1e-10, atol=1e-11)
    ctx.close()


@pytest.mark.parametrize("lead", [False, True])
def test_pivot_of_zeros_as_in_the_full_space(bdmod, problems, lead):
    """A pivot without direction (the chain's first, or a later one): its rows are not finite, as those of the
    reduction over the poles, and not an exhausted chain's."""
    p = problems(4, 20.0, 3, 4)
    ctx = bdmod.Context().upload(p)
    ish = 0
    D = int(p.ms.no[ish])
    piv = np.eye(D)
    piv[0 if lead else D - 1] = 0.0
    rows = []
    for mode in (0, 1):
        ctx.set_lanczos_slices(mode)
        ctx.sigma2_build(ish, copy=False)
        lz = ctx.lanczos_reduce(ish, piv, np.full(D, 4), np.full(D, 4))
        rows.append((lz["lz_fw"], lz["lz_bk"]))
    for a, b in zip(*rows):
        assert not np.isfinite(b).all()
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
    ctx.close()


@pytest.mark.parametrize("shift", [0.0, 1500.0, 2500.0])
def test_norms_of_vectors_short_beside_the_energies(bdmod, synth, shift):
    """Energies far from zero: w is E v less its projections and much shorter (down to 2^-6, where the sweep is
    repeated), so |w|^2 is made of the low words.  The stored vectors' norms are off by the rounding of 1/|w|
    and of the elements and of the sum's terms only: a few eps."""
    p = synth.make_problem(8, 16.0, 1, 6)
    p.prop.ep[:] += shift
    p.prop.eh[:] += shift
    ctx = bdmod.Context().upload(p)
    D = int(p.ms.no[0])
    ctx.sigma2_build(0, copy=False)
    nit = np.full(D, 6, np.int32)
    lz = ctx.lanczos_reduce(0, np.eye(D), nit, nit)
    V = ctx.lanczos_vectors(0, 0, len(lz["lz_fw"]), ctx.count_poles(0)[0]).astype(np.longdouble)
    assert np.abs((V ** 2).sum(1) - 1.0).max() < 8 * 2.2e-16
    ctx.close()


def _close_orbitals(synth, p, delta):
    """The problem with matrix elements that hardly depend on the radial quantum numbers: every subshell's
    orbitals couple alike but for the part delta."""
    v, sh = p.vpp, p.ms.orb_sh
    J = v.iabJ % synth.JMULT
    (a, b), (c, d) = ((k // synth.JMULT // synth.ABMULT, k // synth.JMULT % synth.ABMULT) for k in (v.iabJ, v.icdJ))
    k1, k2 = sh[a] * 64 + sh[b], sh[c] * 64 + sh[d]
    key = (np.minimum(k1, k2).astype(np.int64) * 4096 + np.maximum(k1, k2)) * synth.JMULT + J
    u, inv = np.unique(key, return_inverse=True)
    rng = np.random.default_rng(len(u))
    z = rng.standard_normal(len(u))[inv]
    z[((sh[a] == sh[b]) | (sh[c] == sh[d])) & (J % 2 == 1)] = 0.0   # (sign changes under exchange)
    p.vpp = synth.Interaction(v.iabJ, v.icdJ, z * (1.0 + delta * rng.standard_normal(len(z))))
    return p


def _reference_rows(E, M, nit):
    """Rows of the reduction with unit pivots in extended precision, two Gram-Schmidt sweeps a step."""
    E, M = E.astype(np.longdouble), M.astype(np.longdouble)
    D = len(M)
    V, rows, last = [], [], []
    for p in range(D):
        for k in range(nit):
            w = M[p].copy() if k == 0 else E * V[-1]
            for _ in range(2):
                for t in V:
                    w = w - (t * w).sum() * t
            beta = np.sqrt((w * w).sum())
            u = w / beta
            g = [(V[t] * E * u).sum() for t in last]
            row = np.zeros(2 * D + 1, np.longdouble)
            row[0], row[1] = (u * E * u).sum(), g[-1] if k == 0 and g else beta
            row[2:2 + len(g)] = g
            row[D + 1:] = M @ u
            V.append(u)
            rows.append(row)
        last.append(len(V) - 1)
    return np.array(rows)


# orbitals whose couplings are alike: pivots of the groups' Gram matrices at about delta^2 of their diagonal entries,
# from those that are taken as they are to just above the least one that is rotated at all (1e-6)
@pytest.mark.parametrize("nmax,hw,delta", [(4, 20.0, 1.0), (4, 23.1, 3e-3), (6, 17.3, 0.3), (6, 20.0, 3e-2), (6, 13.7, 3e-3),
                                           (8, 16.0, 3e-3)])
def test_rows_of_close_orbitals(bdmod, synth, nmax, hw, delta):
    p = synth.make_problem(nmax, hw, 3, 3)
    if delta < 1.0:
        _close_orbitals(synth, p, delta)
    ctx = bdmod.Context().upload(p)
    D = int(p.ms.no[0])
    nit = np.full(D, 3, np.int32)
    err = []
    for mode in (0, 1):
        ctx.set_lanczos_slices(mode)
        fw, bk = ctx.sigma2_build(0)
        lz = ctx.lanczos_reduce(0, np.eye(D), nit, nit)
        for sig, tag in ((fw, "lz_fw"), (bk, "lz_bk")):
            E, M = sig[:, 0], np.ascontiguousarray(sig[:, 2:].T)
            d = np.abs(lz[tag] - _reference_rows(E, M, 3))
            err.append([float(d[:, :D + 1].max() / np.abs(E).max()), float(d[:, D + 1:].max() / np.abs(lz[tag][:, D + 1:]).max())])
    ctx.close()
    # what the reduction over the poles makes of the same rows, within the scatter of two roundings
    assert np.all(np.array(err[:2]) <= 8 * np.array(err[2:]) + 1e-15), err


# steps of energies that are rounding's one by one (3 eps) and not as a run, and steps just beyond rounding
@pytest.mark.parametrize("step", [3.0, 12.0])
def test_energies_a_few_eps_apart(bdmod, synth, step):
    """Levels of a shell a few eps apart: no pole's energy moves by more than its own rounding."""
    p = synth.make_problem(4, 20.0, 3, 3)
    p.prop.ep[:] += (np.arange(len(p.prop.ep)) % 3) * step * 2.0 ** -52 * 200.0
    ctx = bdmod.Context().upload(p)
    D = int(p.ms.no[0])
    nit = np.full(D, 3, np.int32)
    fw, _ = ctx.sigma2_build(0)
    lz = ctx.lanczos_reduce(0, np.eye(D), nit, nit)["lz_fw"]
    ctx.close()
    E = fw[:, 0]
    ref = _reference_rows(E, np.ascontiguousarray(fw[:, 2:].T), 3)
    # alpha is a mean of the energies: their half span in a group (2 eps), and the rounding of its sum
    assert np.abs(lz[:, 0] - ref[:, 0]).max() < 6 * 2.2e-16 * np.abs(E).max()


@pytest.mark.parametrize("ref_order", [False, True])
@pytest.mark.parametrize("nmax,hw,nit", [(3, 13.7, 7), (5, 20.0, 3)])
def test_vectors_keep_the_reduction_s_order(bdmod, problems, nmax, hw, nit, ref_order):
    """The stored vectors read back before and after the sorted poles were put in another order of their equal
    energies: the same, pole by pole."""
    p = problems(nmax, hw, 3, nit)
    ctx = bdmod.Context().upload(p)
    pv = p.piv
    for ish in range(p.ms.nsubsh):
        n = ctx.count_poles(ish)
        ctx.sigma2_build(ish, copy=False)
        lz = ctx.lanczos_reduce(ish, pv.vec[ish], pv.n_fw[ish], pv.n_bk[ish], ref_order=ref_order)
        L = (len(lz["lz_fw"]), len(lz["lz_bk"]))
        before = [ctx.lanczos_vectors(ish, d, L[d], n[d]) for d in (0, 1) if L[d]]
        sorted_rows = ctx.sigma2_sorted(ish)
        after = [ctx.lanczos_vectors(ish, d, L[d], n[d]) for d in (0, 1) if L[d]]
        for a, b in zip(before, after):
            assert np.array_equal(a, b), ish
        for a, b in zip(sorted_rows, ctx.sigma2_sorted(ish)):
            assert np.array_equal(a, b), ish
    ctx.close()
