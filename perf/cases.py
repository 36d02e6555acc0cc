"""The work that a user of this framework has it do, as cases that can be timed.

A case is one call pattern of the public interface (``bd.Context``, the C ABI behind it and
``bd.lanczos_chain_noalloc``) on seeded synthetic inputs in the reference's formats:

* ``step``      the whole chain for every channel with the problem resident (``bd_run_all``), and every
                channel's solutions and Koltun sums read back, as each iteration of a self-consistent run does;
                on the unperturbed propagator (first iterations) or a dressed one (the following iterations)
* ``channel``   the reference's per-channel calls: static self-energy, Sigma(2) with its rows, the Lanczos
                reduction and the Dyson solve of one channel
* ``rows``      the Dyson solve of self-energy rows the caller brings (one loaded from a file, say)
* ``chain``     the Lanczos reduction of one pole set in caller-owned device memory
* ``upload``    a new problem from host memory, its chain and its results: what a scan over problems repeats
"""
import ctypes
import functools
import importlib
import math

import numpy as np
import torch

synth = importlib.import_module("boccadorata-public_gb300.synth")
bd = importlib.import_module("boccadorata-public_gb300.bd")


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    step = dict(kind="step", lanczos=True, mixed=False, graph=False, frag=0, sigma=2.0)
    return [
        # the smallest problem anyone runs: a first look at a nucleus, or one of many in a parameter scan
        dict(step, name="nmax4_lanczos20", nmax=4, hw=20.0, nit=20),
        # the same problem without the Lanczos reduction: the reference solution that a reduced one is held to
        dict(step, name="nmax4_full", nmax=4, hw=20.0, nit=1, lanczos=False),
        # ordinary production sizes, the step replayed as a captured graph
        dict(step, name="nmax8_lanczos100", nmax=8, hw=20.0, nit=100, graph=True),
        dict(step, name="nmax10_lanczos100", nmax=10, hw=16.0, nit=100, graph=True),
        # the mixed form at the benchmark's size
        dict(step, name="nmax10_lanczos100_mixed", nmax=10, hw=16.0, nit=100, mixed=True, graph=True),
        # the largest configuration: 50 channels, D up to 7
        dict(step, name="nmax12_lanczos100", nmax=12, hw=16.0, nit=100, graph=True),
        # a later iteration of a self-consistent run: two fragments a subshell and side, all pole energies distinct
        dict(step, name="nmax6_dressed", nmax=6, hw=20.0, nit=20, frag=2),
        # a later iteration of the many-problem run: one fragment a subshell and side, the mixed form
        dict(step, name="nmax8_dressed_mixed", nmax=8, hw=20.0, nit=20, frag=1, mixed=True, graph=True),
        # the calls that replace the reference's, channel by channel, with the rows it keeps on the host
        dict(kind="channel", name="nmax8_channel", nmax=8, hw=20.0, nit=100, sigma=2.0, ish=0, frag=0),
        # a stored self-energy solved again: a dense spectrum of about a thousand poles
        dict(kind="rows", name="dyson_rows_1000", nmax=4, hw=20.0, ish=0, nfw=800, nbk=197),
        # one long pole set with distinct energies, reduced in the caller's own buffers
        dict(kind="chain", name="chain_20000", poles=20000, d=4, nit=20, mixed=False),
        # a new problem every time: upload, chain and read-back
        dict(kind="upload", name="nmax8_upload", nmax=8, hw=20.0, nit=100, sigma=2.0, mixed=False),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "dressed", "dressed", "channel", "rows", "chain", "upload"])
    hw, sigma = round(rng.uniform(10.0, 30.0), 2), round(rng.uniform(1.0, 3.0), 2)
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    if kind == "step":
        full = rng.random() < 0.2
        return dict(kind="step", lanczos=not full, mixed=not full and rng.random() < 0.3, graph=rng.random() < 0.5, frag=0,
                    sigma=sigma, nmax=rng.choice([2, 3, 4] if full else [4, 5, 6, 7, 8, 9, 10]), hw=hw,
                    nit=1 if full else log(20, 100))
    if kind == "dressed":
        frag = rng.choice([1, 1, 2])
        return dict(kind="step", lanczos=True, mixed=rng.random() < 0.3, graph=rng.random() < 0.5, frag=frag, sigma=sigma,
                    nmax=rng.choice([4, 5, 6, 7, 8] if frag == 1 else [4, 5, 6]), hw=hw, nit=rng.randint(8, 20))
    if kind == "channel":
        nmax, frag = rng.choice([4, 5, 6, 7, 8, 9]), 0
        return dict(kind="channel", nmax=nmax, hw=hw, nit=log(20, 100), sigma=sigma, ish=rng.randrange(2 * nmax + 1), frag=frag)
    if kind == "rows":
        n = log(60, 1000)
        nbk = rng.randint(0, n // 3)
        return dict(kind="rows", nmax=rng.choice([4, 5, 6]), hw=hw, ish=rng.randrange(6), nfw=n - nbk, nbk=nbk)
    if kind == "chain":
        return dict(kind="chain", poles=log(300, 20000), d=rng.randint(1, 6), nit=rng.randint(5, 20), mixed=rng.random() < 0.3)
    return dict(kind="upload", nmax=rng.choice([4, 5, 6, 7, 8]), hw=hw, nit=log(20, 100), sigma=sigma, mixed=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------ the inputs
@functools.lru_cache(maxsize=2)
def _structure(nmax):
    """The canonical pair list of a model space (independent of the seed): keys and size factors."""
    ms = synth.make_modspace(nmax, 1.0)
    nosc = (2 * ms.orb_n + ms.l[ms.orb_sh]).astype(np.float64)
    iab, icd, size = [], [], []
    for _, _, J, pairs in synth.two_body_channels(ms):
        p = np.array(pairs, np.int64)
        key = ((p[:, 0] * synth.ABMULT + p[:, 1]) * synth.JMULT + J).astype(np.int32)
        f = np.exp(-(nosc[p[:, 0]] + nosc[p[:, 1]]) / 8.0)
        i, j = np.triu_indices(len(p))
        iab.append(key[i])
        icd.append(key[j])
        size.append(f[i] * f[j])
    return np.concatenate(iab), np.concatenate(icd), torch.from_numpy(np.concatenate(size)).cuda()


def _interaction(nmax, sigma, seed, pinned=False):
    iab, icd, size = _structure(nmax)
    g = torch.Generator("cuda").manual_seed(seed)
    v = size * torch.randn(len(iab), dtype=torch.float64, device="cuda", generator=g) * sigma
    host = torch.empty(v.shape, dtype=v.dtype, pin_memory=pinned).copy_(v).numpy()
    if pinned:  # the arrays that a program uploading problem after problem keeps page-locked
        iab, icd = (torch.from_numpy(a).pin_memory().numpy() for a in (iab, icd))
    return synth.Interaction(iab, icd, host)


def _dressed(ms, frag, seed):
    """A propagator as a truncated update leaves it: `frag` fragments a subshell and side, strong where the subshell has
    that side's orbits and weak where it has not, energies spread about the orbits', amplitudes mixed over the orbits."""
    rng = np.random.default_rng(seed)
    nspb = ms.nspb_mx
    out = {0: ([], []), 1: ([], [])}  # side (0 particles, 1 holes): energies, amplitudes
    for s in range(ms.nsubsh):
        o, d = int(ms.orb_start[s]), int(ms.no[s])
        for side in (0, 1):
            own = [k for k in range(d) if int(ms.orb_F[o + k]) == side]
            rows = []
            for f in range(frag):
                if f < len(own):
                    k, z, e = own[f], rng.uniform(0.6, 0.95), ms.orb_xe[o + own[f]] + rng.normal(0.0, 1.5)
                else:
                    k, z = int(rng.integers(d)), rng.uniform(0.005, 0.03)
                    e = -60.0 - 40.0 * rng.random() if side else 80.0 + 60.0 * rng.random()
                a = 0.25 * rng.standard_normal(d)
                a[k] += 1.0
                amp = np.zeros(nspb)
                amp[:d] = a * math.sqrt(z) / np.linalg.norm(a)
                rows.append((e, amp))
            for e, amp in sorted(rows, key=lambda r: -r[0]):
                out[side][0].append(e)
                out[side][1].append(amp)
    n = np.full(ms.nsubsh, frag, np.int32)
    return synth.propagator_from_arrays(nspb, n, n, out[0][0], out[1][0], np.array(out[0][1]), np.array(out[1][1]))


def _problem(case, seed, pinned=False):
    ms = synth.make_modspace(case["nmax"], case["hw"])
    prop = synth.make_unperturbed_propagator(ms)
    piv = synth.make_pivots(ms, prop, max(1, case.get("nit", 1)))
    vpp = _interaction(case["nmax"], case.get("sigma", 2.0), seed, pinned)
    return synth.Problem(ms, prop, vpp, piv, seed, case.get("sigma", 2.0))


def _rows(case, seed):
    rng = np.random.default_rng(seed)
    ms = synth.make_modspace(case["nmax"], case["hw"])
    o, d = int(ms.orb_start[case["ish"]]), int(ms.no[case["ish"]])
    fw, bk = (np.zeros((n, 2 + d)) for n in (case["nfw"], case["nbk"]))
    fw[:, 0] = np.sort(rng.uniform(20.0, 300.0, len(fw)))
    bk[:, 0] = -np.sort(rng.uniform(60.0, 250.0, len(bk)))
    for r in (fw, bk):
        r[:, 2:] = rng.standard_normal((len(r), d)) * (4.0 / math.sqrt(len(fw)))
        r[:, 1] = (r[:, 2:] ** 2).sum(1)
    hf = rng.standard_normal((d, d))
    return ms, fw, bk, np.diag(ms.orb_xe[o:o + d]), 0.5 * (hf + hf.T)


def _chain(case, seed):
    rng = np.random.default_rng(seed)
    n, d = case["poles"], case["d"]
    e = np.sort(rng.uniform(20.0, 300.0, n))
    m = rng.standard_normal((d, n)) * np.exp(-e / 120.0) * (4.0 / math.sqrt(n))
    return e, m, np.eye(d), np.full(d, case["nit"], np.int32)


class _State:
    pass


def _room(s, ctx, case):
    """The arrays that a program reading every iteration's results keeps."""
    ms, rows = s.prob.ms, 0
    for i in range(ms.nsubsh):
        n = list(ctx.count_poles(i))
        if case.get("lanczos", True):
            n = [min(k, int(sum(v[i]))) for k, v in zip(n, (s.prob.piv.n_fw, s.prob.piv.n_bk))]
        rows += (int(ms.no[i]) + sum(n)) * (2 + int(ms.no[i]))
    s.sol, s.cnt, s.kol = np.zeros(rows), np.zeros(2 * ms.nsubsh, np.int32), np.zeros(3 * ms.nsubsh)


def prepare(case, seed):
    s = _State()
    s.case, kind = case, case["kind"]
    if kind == "chain":
        e, m, s.piv, s.nit = _chain(case, seed)
        s.e, s.m = torch.from_numpy(e).cuda(), torch.from_numpy(m).cuda()
        s.rows = torch.zeros((min(int(s.nit.sum()), len(e)), 2 * case["d"] + 1), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return s
    s.ctx = bd.Context(0)
    if kind == "rows":
        s.ctx.upload(_problem(case, seed))
        _, s.fw, s.bk, s.s1, s.hf = _rows(case, seed)
        return s
    s.prob = _problem(case, seed, pinned=kind == "upload")
    s.ctx.upload(s.prob)
    if case.get("frag", 0):
        s.ctx.upload_propagator(_dressed(s.prob.ms, case["frag"], seed))
    if kind != "channel":
        _room(s, s.ctx, case)
    return s


# ------------------------------------------------------------------------------------------------ the calls
def _signed(rows):
    """Solution rows [W, Z, x_0 ..] with the eigenvector's free sign chosen: its largest component positive."""
    x = rows[:, 2:]
    top = np.take_along_axis(x, np.abs(x).argmax(1)[:, None], 1)
    return np.concatenate([rows[:, :2], np.where(top < 0.0, -x, x)], 1)


def _fetch(s):
    p = lambda a, t: a.ctypes.data_as(ctypes.POINTER(t))  # noqa: E731
    rc = s.ctx.lib.bd_result_fetch_all(s.ctx.h, p(s.sol, ctypes.c_double), len(s.sol), p(s.cnt, ctypes.c_int),
                                       p(s.kol, ctypes.c_double))
    if rc != bd.BD_OK:
        raise bd.BDError(rc, s.ctx.lib.bd_last_error(s.ctx.h).decode())
    sol = s.sol
    if not s.case.get("lanczos", True):  # the un-reduced matrix: nothing else fixes the eigenvectors' signs
        sol, o = [], 0
        for i, d in enumerate(int(d) for d in s.prob.ms.no):
            n = int(s.cnt[2 * i] + s.cnt[2 * i + 1]) * (2 + d)
            sol.append(_signed(s.sol[o:o + n].reshape(-1, 2 + d)).reshape(-1))
            o += n
        sol = np.concatenate(sol)
    return dict(solutions=sol, counts=s.cnt, koltun=s.kol)


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "step":
        s.ctx.run_all(lanczos=case["lanczos"], mixed=case["mixed"], graph=case["graph"])
        return _fetch(s)
    if kind == "upload":
        s.ctx.upload(s.prob)
        s.ctx.run_all(mixed=case["mixed"])
        return _fetch(s)
    if kind == "channel":
        i, piv = case["ish"], s.prob.piv
        hf = s.ctx.ehf(i)
        fw, bk = s.ctx.sigma2_build(i)
        lz = s.ctx.lanczos_reduce(i, piv.vec[i], piv.n_fw[i], piv.n_bk[i])
        o, d = int(s.prob.ms.orb_start[i]), int(s.prob.ms.no[i])
        r = s.ctx.dyson_solve(i, np.diag(s.prob.ms.orb_xe[o:o + d]), hf)
        return dict(hf=hf, sigma_fw=fw, sigma_bk=bk, lanczos_fw=lz["lz_fw"], lanczos_bk=lz["lz_bk"], qp=r["qp"], qh=r["qh"],
                    koltun=r["koltun"])
    if kind == "rows":
        r = s.ctx.dyson_rows(case["ish"], 2, s.fw, s.bk, sig1b=s.s1, sighf=s.hf, efermi=-50.0)
        return dict(qp=_signed(r["qp"]), qh=_signed(r["qh"]), koltun=r["koltun"])
    n, ipiv, piv, nit = bd.lanczos_chain_noalloc(s.e.data_ptr(), s.m.data_ptr(), case["poles"], case["d"], s.piv, s.nit,
                                                 s.rows.data_ptr(), len(s.rows), mixed=case["mixed"])
    return dict(rows=s.rows, ipiv=ipiv, n=n)


# ------------------------------------------------------------------------------------------------ what they need
@functools.lru_cache(maxsize=64)
def _poles(nmax, frag):
    """(poles, D, pivots' count D) of every channel and direction: three fragments with the triangle and parity rules."""
    ms = synth.make_modspace(nmax, 1.0)
    prop = synth.make_unperturbed_propagator(ms)
    npv, nhv = (np.full(ms.nsubsh, frag), np.full(ms.nsubsh, frag)) if frag else (prop.np_, prop.nh)
    pairs = {}  # (charge, parity, J) -> number of pairs a <= b on each side
    for side, n in ((0, npv), (1, nhv)):
        for a in range(ms.nsubsh):
            for b in range(a, ms.nsubsh):
                for J in range(abs(ms.j2[a] - ms.j2[b]) // 2, (ms.j2[a] + ms.j2[b]) // 2 + 1):
                    k = n[a] * n[b] if a != b else n[a] * (n[a] + (1 if J % 2 == 0 else -1)) // 2
                    key = (side, int(ms.ch[a] + ms.ch[b]), int(ms.ip[a] + ms.ip[b]) % 2, J)
                    pairs[key] = pairs.get(key, 0) + int(k)
    out = []
    for i in range(ms.nsubsh):
        for side, third in ((0, nhv), (1, npv)):
            tot = 0
            for (sd, ch, par, J), k in pairs.items():
                if sd != side:
                    continue
                for g in range(ms.nsubsh):
                    if ch - ms.ch[g] == ms.ch[i] and (par + ms.ip[g]) % 2 == ms.ip[i] and abs(ms.j2[g] - ms.j2[i]) <= 2 * J <= ms.j2[g] + ms.j2[i]:
                        tot += k * int(third[g])
            out.append((i, tot, int(ms.no[i])))
    return out


def work(case):
    """Bytes: every pole's energy and couplings formed once from as many matrix elements, the solutions written once (and
    the interaction copied in, where the call does).  Flops: the couplings' contraction, what the reduction of a pole set
    needs at least (the pairwise products of its vectors), and the eigenproblem of the reduced order."""
    kind = case["kind"]
    if kind == "chain":
        n, d = case["poles"], case["d"]
        r = min(n, d * case["nit"])
        return dict(bytes=8.0 * (n * (1 + d) + r * (2 * d + 1)), flops=2.0 * n * r * r)
    if kind == "rows":
        n = case["nfw"] + case["nbk"] + 3
        return dict(bytes=8.0 * n * 10, flops=4.0 / 3.0 * n ** 3)
    by = fl = 0.0
    for i, n, d in _poles(case["nmax"], case["frag"] if "frag" in case else 0):
        if kind == "channel" and i != case["ish"]:
            continue
        rows = min(n, d * case["nit"]) if case.get("lanczos", True) else n
        by += 8.0 * (n * (1 + 2 * d) + rows * (2 + d))
        if case.get("frag", 0):
            fl += 2.0 * n * rows * rows + 4.0 / 3.0 * rows ** 3
        else:  # few distinct energies: the products of each pole's couplings hold all that the reduction needs
            fl += n * d * (d + 1.0)
    if kind == "upload":
        by += 16.0 * len(_structure(case["nmax"])[0])
    return dict(bytes=by, flops=fl)


def _split(w, x, ef):
    """Solutions as the solve returns them: quasiparticles, then quasiholes, each by descending energy."""
    rows = np.concatenate([w[:, None], (x ** 2).sum(1)[:, None], x], 1)[np.argsort(-w, kind="stable")]
    return rows[rows[:, 0] > ef], rows[rows[:, 0] <= ef]


def exact(case, seed):
    """The caller's rows and the single chain from numpy; a whole chain has no value that numpy gives in this time."""
    if case["kind"] == "rows":
        ms, fw, bk, s1, hf = _rows(case, seed)
        d = len(s1)
        a = np.diag(np.concatenate([np.zeros(d), fw[:, 0], bk[:, 0]]))
        a[:d, :d] = s1 + hf
        a[d:, :d] = np.concatenate([fw[:, 2:], bk[:, 2:]])
        a[:d, d:] = a[d:, :d].T
        w, v = np.linalg.eigh(a)
        qp, qh = _split(w, v[:d].T, -50.0)
        j = float(ms.j2[case["ish"]] + 1)
        x = qh[:, 2:]
        kol = [np.einsum("ka,ab,kb->", x, s1, x), (qh[:, 1] * qh[:, 0]).sum(), qh[:, 1].sum()]
        return dict(qp=_signed(qp), qh=_signed(qh), koltun=np.array(kol) * j)
    if case["kind"] == "chain" and not case["mixed"] and case["poles"] > 4 * case["d"] * case["nit"]:
        e, m, piv, nit = _chain(case, seed)
        d, v, out = len(m), [], []
        last = []  # the last vector of every earlier chain
        for p in range(d):
            for k in range(int(nit[p])):
                w = (piv[p] @ m) if k == 0 else e * v[-1]
                for _ in range(3):
                    if v:
                        b = np.array(v)
                        w = w - (b @ w) @ b
                beta = np.linalg.norm(w)
                u = w / beta
                row = np.zeros(2 * d + 1)
                g = [float(np.dot(v[t], e * u)) for t in last]
                row[0] = np.dot(u, e * u)
                row[1] = (g[-1] if k == 0 and g else beta)
                row[2:2 + len(g)] = g
                row[d + 1:] = m @ u
                v.append(u)
                out.append(row)
            last.append(len(v) - 1)
        return dict(rows=np.array(out), ipiv=None, n=None)
    return None
