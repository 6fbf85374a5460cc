"""Workloads of the Koopmans + SC/PC-NEVPT2 library, as a program that uses it
runs them: the stage-1 driver, its resident builders, the reader of the 4-RDM,
the A-matrices of the (+-1') classes and the energy stage.

Wavefunctions.  The states are equal-weight mixtures of 2 nact determinants in
random orbitals.  Their spin-free RDMs are exact, complete and mutually
consistent and cost a few products instead of a CI expansion.  Closed-shell
determinants make a singlet, whose PC metrics have a few exact null vectors;
with orbitals of their own for each spin the metrics keep every eigenvalue, as
those of the random determinant expansions of the benchmark configurations do.  Density-fitted integrals,
orbital energies and the off-diagonal Fock elements follow the distributions
of ``nevpt2_gb300.synth``.  The energy stage gets Koopmans matrices of the form
D^1/2 S D^1/2 with the class's metric S and positive excitation energies D:
the positive spectra of a converged reference state, so that no denominator
vanishes and energies are defined to rounding.

Array layouts are the library's: Fortran order, state index first (the packed
4-RDM has it last).  A tensor x[i, j, ...] of this file is stored that way as
the C-ordered tensor with its axes reversed (``_fortran``).
"""
from __future__ import annotations

import ctypes
import itertools
import math

import numpy as np
import torch

F64 = torch.float64
KINDS = ("driver", "front", "unfold", "bamat", "energies")


def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


# --------------------------------------------------------------------- cases
def listed():
    return [
        # the whole of stage 1 through the host API on a minimal active space (a molecule's HOMO/LUMO region):
        # a few hundred bytes to megabytes in and out, all launch and call latency
        {"name": "driver_cas4", "kind": "driver", "nact": 4, "nele": 4, "ncore": 4, "nvirt": 12, "states": 1},
        # everything of stage 1 but the A-matrices, resident, on the CAS(8,8) configuration
        {"name": "front_cas8", "kind": "front", "nact": 8, "nele": 8, "ncore": 10, "nvirt": 40, "states": 1},
        # the same for two roots of an odd, large active space
        {"name": "front_cas13_2", "kind": "front", "nact": 13, "nele": 12, "ncore": 20, "nvirt": 150, "states": 2},
        # unfolding of a QCMaquis 4-RDM label/value list (the DMRG hand-off), resident
        {"name": "unfold_cas9", "kind": "unfold", "nact": 9, "fill": 1.0},
        # A-matrices: a small, an odd two-root, and the benchmark's active space
        {"name": "bamat_cas8", "kind": "bamat", "nact": 8, "nele": 8, "ncore": 10, "states": 1, "split": False},
        {"name": "bamat_cas11_2", "kind": "bamat", "nact": 11, "nele": 10, "ncore": 10, "states": 2, "split": False},
        {"name": "bamat_cas16", "kind": "bamat", "nact": 16, "nele": 16, "ncore": 30, "states": 1, "split": False},
        # the same in split precision on the CAS(14,14) configuration's active space
        {"name": "bamat_cas14_split", "kind": "bamat", "nact": 14, "nele": 14, "ncore": 20, "states": 1, "split": True},
        # the energy stage through the host API: one of the small three-root problems that come in batches
        {"name": "energies_cas6_3", "kind": "energies", "nact": 6, "nele": 6, "ncore": 12, "nvirt": 75, "states": 3,
         "split": False, "host": True, "singlet": True},
        # the energy stage, resident: the middle of the range, and the CAS(14,14) configuration
        {"name": "energies_cas10_2", "kind": "energies", "nact": 10, "nele": 10, "ncore": 15, "nvirt": 90, "states": 2,
         "split": False, "host": False, "singlet": True},
        {"name": "energies_cas14", "kind": "energies", "nact": 14, "nele": 14, "ncore": 20, "nvirt": 150, "states": 1,
         "split": False, "host": False, "singlet": False},
        # the energy stage in split precision
        {"name": "energies_cas12_split", "kind": "energies", "nact": 12, "nele": 12, "ncore": 20, "nvirt": 120,
         "states": 1, "split": True, "host": False, "singlet": False},
    ]


def draw(rng):
    kind = rng.choice(("driver", "front", "unfold", "bamat", "bamat", "energies", "energies"))
    if kind == "unfold":
        # the writer leaves out entries that are zero by symmetry or below its threshold
        return {"kind": kind, "nact": rng.randint(6, 11), "fill": round(rng.uniform(0.2, 1.0), 3)}
    lo, hi = {"driver": (3, 6), "front": (6, 14), "bamat": (6, 15), "energies": (4, 13)}[kind]
    n = rng.randint(lo, hi)
    nele = 2 * max(2, min(n - 1, (n + rng.randint(-1, 1)) // 2))
    case = {"kind": kind, "nact": n, "nele": nele, "ncore": rng.randint(3, 30),
            "states": rng.randint(1, 3 if n <= 10 else 1)}
    if kind != "bamat":
        case["nvirt"] = int(round(math.exp(rng.uniform(math.log(12), math.log(160)))))
    if kind == "energies":
        case["host"] = n <= 8 and rng.random() < 0.5
        case["singlet"] = rng.random() < 0.5
    if kind in ("bamat", "energies"):
        case["split"] = n >= 8 and rng.random() < 0.3
    return case


# -------------------------------------------------------------------- inputs
def _generator(seed, stream):
    return torch.Generator(device="cpu").manual_seed(1_000_003 * int(seed) + 7919 * stream + 17)


def _gauss(gen, *shape):
    # small arrays come from the CPU generator, large ones from one seeded by it on the device
    if math.prod(shape) < 1 << 16 or _device().type == "cpu":
        return torch.randn(*shape, generator=gen, dtype=F64).to(_device())
    dev = torch.Generator(device=_device()).manual_seed(int(torch.randint(1 << 40, (1,), generator=gen)))
    return torch.randn(*shape, generator=dev, dtype=F64, device=_device())


def _uniform(gen, lo, hi, k):
    return (lo + (hi - lo) * torch.rand(k, generator=gen, dtype=F64)).to(_device())


def _orbitals(gen, n, nele, count):
    return torch.linalg.qr(_gauss(gen, count, n, nele // 2))[0]


def _mixture(gen, n, nele, pure=True):
    """(weights, alpha and beta 1-RDMs) of a state: 2n determinants, closed-shell (a singlet, whose PC metrics have
    the null vectors of a spin eigenfunction) or with orbitals of their own for each spin (metrics of full rank)."""
    ca = _orbitals(gen, n, nele, 2 * n)
    cb = ca if pure else _orbitals(gen, n, nele, 2 * n)
    return torch.full((2 * n,), 1.0 / (2 * n), dtype=F64, device=ca.device), (ca @ ca.mT, cb @ cb.mT)


def _transition(gen, n, nele):
    """The same of a pair of states: overlapping pairs of determinants C and D, whose transition densities obey the
    determinant formula with gamma = C (D^T C)^-1 D^T."""
    g = []
    for _ in range(2):
        c = _orbitals(gen, n, nele, 4)
        d = torch.linalg.qr(c + 0.3 * _gauss(gen, *c.shape))[0]
        g.append(c @ torch.linalg.solve(d.mT @ c, d.mT))
    return 0.1 * _gauss(gen, 4), tuple(g)


def _holes(state):
    """The holes of a mixture of determinants: gamma -> 1 - gamma for each spin."""
    w, g = state
    return w, tuple(torch.eye(x.shape[-1], dtype=F64, device=x.device) - x for x in g)


def _permutations(k):
    """(permutation, its cycles, sign) of the determinant formula."""
    for p in itertools.permutations(range(k)):
        cycles, seen = [], set()
        for i in range(k):
            if i not in seen:
                cycles.append([])
                while i not in seen:
                    seen.add(i)
                    cycles[-1].append(i)
                    i = p[i]
        yield p, cycles, (-1.0) ** (k - len(cycles))


def _rdm(state, k):
    """Dense spin-free k-RDM [p1..pk, q1..qk], k <= 3: the determinant formula with one spin for each cycle."""
    w, g = state
    n = g[0].shape[-1]
    out = torch.zeros((n,) * (2 * k), dtype=F64, device=w.device)
    cre, ann = "abc"[:k], "def"[:k]
    for p, cycles, sign in _permutations(k):
        for spins in itertools.product((0, 1), repeat=len(cycles)):
            spin = {i: s for cyc, s in zip(cycles, spins) for i in cyc}
            terms = ",".join("m" + cre[i] + ann[p[i]] for i in range(k))
            x = [g[spin[i]] for i in range(k)]
            out += torch.einsum(f"{terms}->{cre}{ann}", sign * w[:, None, None] * x[0], *x[1:])
    return out


def _rdm4_rows(state, rows):
    """Spin-free 4-RDM of a singlet for the creator quadruples `rows` (r, 4): [r, q1, q2, q3, q4]."""
    w, g = state[0], 2.0 * state[1][0]
    n = g.shape[-1]
    coef = {p: sign * 2.0 ** (len(cycles) - 4) for p, cycles, sign in _permutations(4)}
    out = torch.empty((rows.shape[0], n, n, n, n), dtype=F64, device=g.device)
    for r0 in range(0, rows.shape[0], 512):
        r = rows[r0:r0 + 512]
        x = [g[:, r[:, i], :].permute(1, 0, 2) for i in range(4)]  # [r, m, q]
        u, v = [], []
        for i, j in itertools.permutations(range(4), 2):  # q1 <- i, q2 <- j; q3, q4 <- the other two
            a, b = (t for t in range(4) if t not in (i, j))
            signs = []
            for t, s in ((a, b), (b, a)):
                p = [0] * 4
                p[i], p[j], p[t], p[s] = 0, 1, 2, 3
                signs.append(coef[tuple(p)])
            u.append((x[i][..., :, None] * x[j][..., None, :]).flatten(2))
            v.append((w[None, :, None, None] * (signs[0] * x[a][..., :, None] * x[b][..., None, :]
                                                + signs[1] * x[b][..., :, None] * x[a][..., None, :])).flatten(2))
        out[r0:r0 + 512] = (torch.cat(u, 1).mT @ torch.cat(v, 1)).view(-1, n, n, n, n)
    return out


def _keys(n):
    """The packed key quadruples (descending), in the order of their index."""
    k = [(a, b, c, d) for a in range(n) for b in range(a + 1) for c in range(b + 1) for d in range(c + 1)]
    return torch.tensor(k, device=_device())


def _fortran(tensors):
    """Flat Fortran-order array (slot, i, j, ...) of one tensor [i, j, ...] per slot."""
    return torch.stack([t.permute(*range(t.dim() - 1, -1, -1)) for t in tensors], -1).reshape(-1)


def _packed_rdm4(states):
    return torch.stack([_rdm4_rows(s, _keys(s[1][0].shape[-1])).permute(4, 3, 2, 1, 0) for s in states]).reshape(-1)


def _pairs(norb):
    p, q = torch.tril_indices(norb, norb, device=_device())
    return p, q


def _integrals(case, gen, state):
    """oneint, the Cholesky array [pair, Q] and the target orbital energies."""
    nc, na = case["ncore"], case["nact"]
    nv = case.get("nvirt", 0)
    norb = nc + na + nv
    p, q = _pairs(norb)
    chol = _gauss(gen, p.numel(), 4 * norb) * (0.05 * torch.exp(-(p - q) / 8.0))[:, None]
    eps = torch.cat([_uniform(gen, lo, hi, k).sort()[0] for lo, hi, k in ((-2.0, -0.5, nc), (-0.5, 0.5, na),
                                                                          (0.5, 5.0, nv))])
    off = 1e-3 * _gauss(gen, norb, norb)
    fock = torch.diag(eps) + off.triu(1) + off.triu(1).mT
    b = _dense_df(chol, norb)
    h = fock - _fock2(b, nc, na, _rdm(state, 1))
    return h[p, q].contiguous(), chol


def _dense_df(chol, norb):
    p, q = _pairs(norb)
    b = torch.empty(chol.shape[1], norb, norb, dtype=F64, device=chol.device)
    b[:, p, q] = chol.mT
    b[:, q, p] = chol.mT
    return b


def _fock2(b, nc, na, g1):
    """Two-electron part of the core and virtual Fock operators."""
    c, a = slice(0, nc), slice(nc, nc + na)
    j = 2.0 * torch.einsum("xkk->x", b[:, c, c]) + torch.einsum("xab,ba->x", b[:, a, a], g1)
    k = torch.einsum("xpk,xkq->pq", b[:, :, c], b[:, c, :])
    return torch.einsum("x,xpq->pq", j, b) - k - 0.5 * torch.einsum("xpb,ba,xaq->pq", b[:, :, a], g1, b[:, a, :])


def _states(case, seed):
    pure = case.get("singlet", True)
    return [_mixture(_generator(seed, 10 + s), case["nact"], case["nele"], pure) for s in range(case["states"])]


def _accessors(state, three=True):
    """Normal-ordered products of a state as dense tensors: g1, g2, g3 and <EE>, <EEE>."""
    g1, g2 = _rdm(state, 1), _rdm(state, 2)
    n = g1.shape[0]
    d = torch.eye(n, dtype=F64, device=g1.device)
    ee = g2.permute(0, 2, 1, 3) + torch.einsum("bc,ad->abcd", d, g1)
    if not three:
        return g1, g2, ee, d
    g3 = _rdm(state, 3)
    eee = g3.permute(0, 3, 1, 4, 2, 5).clone()
    eee += torch.einsum("ed,acbf->abcdef", d, g2) + torch.einsum("eb,acfd->abcdef", d, g2)
    eee += torch.einsum("bc,aedf->abcdef", d, g2) + torch.einsum("bc,ed,af->abcdef", d, d, g1)
    return g1, g2, g3, ee, eee, d


def _hole2(g1, g2, d):
    """2-hole RDM [ap, bp, a, b]."""
    x = g2.permute(2, 3, 0, 1).clone()
    x += -2.0 * torch.einsum("pa,bq->pqab", d, g1) - 2.0 * torch.einsum("qb,ap->pqab", d, g1)
    x += torch.einsum("pb,aq->pqab", d, g1) + torch.einsum("qa,bp->pqab", d, g1)
    return x + 4.0 * torch.einsum("pa,qb->pqab", d, d) - 2.0 * torch.einsum("pb,qa->pqab", d, d)


def _scaled(s, d):
    """D^1/2 S D^1/2 over matching row and column index sets of s."""
    r = d.sqrt()
    return r.reshape(d.shape + (1,) * d.dim()) * s * r


def _koopmans(case, gen, state):
    """The datasets of one state that the energy stage reads, with positive pencils."""
    n = case["nact"]
    g1, g2, g3, ee, eee, d = _accessors(state)
    e1, e2, e2b, e3, e3b = (_uniform(gen, 0.3, 1.5, n) for _ in range(5))
    two = e2[:, None] + e2[None, :]
    exc = 0.5 * (e2[:, None] + e2b[None, :])
    three = e3[:, None, None] + e3b[None, :, None] + e3[None, None, :]
    o = {"1-RDM": g1, "2-RDM": g2, "3-RDM": g3, "2-HRDM": _hole2(g1, g2, d)}
    o["1-IPKO"], o["1-EAKO"] = 2.0 * _scaled(g1, e1), 2.0 * _scaled(2.0 * d - g1, e1)
    o["2-IPKO"], o["2-EAKO"] = _scaled(g2, two), _scaled(o["2-HRDM"], two)
    north = ee.permute(1, 0, 2, 3)                               # <E_ba^+ E_cd> at [a, b, c, d] of (bp, ap, a, b)
    south = -g2.permute(3, 1, 0, 2) + 2.0 * torch.einsum("pa,qb->pqab", d, g1)
    o["gk0pa"] = 2.0 * _scaled(north, exc).permute(1, 0, 2, 3)
    o["gk0pd"] = _scaled(south, exc).permute(1, 0, 2, 3)
    o["gk0pf"] = torch.zeros_like(g1)                            # F vanishes for an eigenstate
    for tag, w3, w2, rho in (("IP", eee, ee, g1),
                             ("EA", 2.0 * torch.einsum("cd,abef->abcdef", d, ee) - eee.permute(0, 1, 3, 2, 4, 5),
                              2.0 * torch.einsum("cd,ab->abcd", d, g1) - ee.permute(0, 1, 3, 2), 2.0 * d - g1)):
        s3 = w3.permute(1, 2, 0, 4, 3, 5)                        # [ap, bp, cp, a, b, c] of w3(cp, ap, bp, b, a, c)
        s2 = w2.permute(1, 2, 0, 3) * three.sqrt()[..., None] * e3.sqrt()
        o["amat" + tag], o["dmat" + tag] = _scaled(s3, three), _scaled(rho, e3)
        o["bmat" + tag], o["cmat" + tag] = s2, s2.permute(3, 0, 1, 2)
    return o


KOOP = ("1-RDM", "2-RDM", "3-RDM", "2-HRDM", "1-IPKO", "1-EAKO", "2-IPKO", "2-EAKO", "gk0pa", "gk0pd", "gk0pf",
        "amatIP", "amatEA", "bmatIP", "bmatEA", "cmatIP", "cmatEA", "dmatIP", "dmatEA")


class _State:
    """What a program holds between calls: buffers, sizes and the library's handle."""


def _context(split=False):
    from nevpt2_gb300._native import Context
    ctx = Context(0)
    if split:
        ctx.call("nvpt_set_precision", 1)
    return ctx


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _problem(case, ro4, oneint, chol):
    """The host-side problem description of the Python API."""
    from nevpt2_gb300 import synth
    n, m = case["nact"], case["states"]
    z = np.zeros(1)
    w = synth.nwords(n)
    return synth.Problem(nact=n, nele=case["nele"], ncore=case["ncore"], nvirt=case["nvirt"], metat=m,
                         nchovec=chol.shape[1], seed=0, amask=z, bmask=z, coef=z, dal=z, taa=z, daaa=z,
                         ro4=None if ro4 is None else ro4.cpu().numpy().reshape((w,) + (n,) * 4 + (m,), order="F"),
                         oneint=oneint.cpu().numpy(), chol=np.asfortranarray(chol.cpu().numpy().T), eps=z)


def prepare(case, seed):
    s = _State()
    s.case = case
    kind, n = case["kind"], case["nact"]
    new = lambda k: torch.zeros(k, dtype=F64, device=_device())
    if kind == "unfold":
        keys = _keys(n)
        # the entries whose creators are the key group, in the file's order: sorted creators, any annihilators
        # of at most their rank
        q = torch.cartesian_prod(*([torch.arange(n, device=_device())] * 4))
        q = q[(_rank(q)[None, :] <= torch.arange(keys.shape[0], device=_device())[:, None]).nonzero()[:, 1]]
        k = keys.repeat_interleave(torch.bincount(_rank(torch.cartesian_prod(*([torch.arange(n, device=_device())] * 4))),
                                                  minlength=keys.shape[0]).cumsum(0), 0)
        gen = _generator(seed, 1)
        pick = _gauss(gen, k.shape[0]).argsort()[:max(1, int(case["fill"] * k.shape[0]))].sort()[0]
        s.labels = torch.cat([k, q], 1)[pick].to(torch.int32).contiguous()
        s.values = _gauss(gen, s.labels.shape[0])
        s.ro4 = new(keys.shape[0] * n**4)
        s.ctx, s.stream = _context(), torch.cuda.Stream()
        return s
    m, nc = case["states"], case["ncore"]
    states = _states(case, seed)
    if kind == "energies":
        return _prepare_energies(s, case, seed, states)
    oneint, chol = _integrals(case, _generator(seed, 2), states[0])
    s.ro4 = _packed_rdm4(states)
    if kind == "driver":
        s.problem = _problem(case, s.ro4, oneint, chol)
        return s
    norb = nc + n + case.get("nvirt", 0)
    npair = norb * (norb + 1) // 2
    s.ctx, s.stream = _context(case.get("split", False)), torch.cuda.Stream()
    s.norb, s.chol, s.oneint = norb, chol.contiguous(), oneint
    s.f, s.aj, s.atwo = new(npair), new(npair), new(n**4)
    if kind == "front":
        s.rdm = {k: new(m * n**e) for k, e in (("3-RDM", 6), ("2-RDM", 4), ("1-RDM", 2))}
        s.koop = {k: new(m * n**e) for k, e in (("1-IPKO", 2), ("1-EAKO", 2), ("2-HRDM", 4), ("2-IPKO", 4),
                                                ("2-EAKO", 4), ("gk0pa", 4), ("gk0pd", 4), ("gk0pf", 2))}
        s.lower = {k + t: new(m * n**e) for k, e in (("bmat", 4), ("cmat", 4), ("dmat", 2)) for t in ("IP", "EA")}
    else:
        atwo, aj = _active_integrals(case, oneint, chol)
        s.atwo = _fortran([atwo])
        p, q = _pairs(norb)
        full = _square(oneint, norb)
        full[nc:nc + n, nc:nc + n] = aj
        s.aj = full[p, q].contiguous()
        s.rdm = {"3-RDM": _fortran([_rdm(x, 3) for x in states]), "2-RDM": _fortran([_rdm(x, 2) for x in states]),
                 "1-RDM": _fortran([_rdm(x, 1) for x in states])}
        s.amat, s.atmat = new(m * n**6), new(m * n**6)
    return s


def _rank(q):
    """0-based packed index of the descending-sorted quadruples."""
    k = q.sort(1, descending=True)[0] + 1
    a, b, c, d = k.unbind(1)
    return (a - 1) * a * (a + 1) * (a + 2) // 24 + (b - 1) * b * (b + 1) // 6 + (c - 1) * c // 2 + d - 1


def _prepare_energies(s, case, seed, states):
    n, m, nc, nv = case["nact"], case["states"], case["ncore"], case["nvirt"]
    oneint, chol = _integrals(case, _generator(seed, 2), states[0])
    koop = [_koopmans(case, _generator(seed, 50 + i), x) for i, x in enumerate(states)]
    s.koop = {k: _fortran([o[k] for o in koop]) for k in KOOP}
    pairs = [_transition(_generator(seed, 100 + i), n, case["nele"]) for i in range(m * (m - 1) // 2)]
    s.trdm = [_fortran([_rdm(p, k) for p in pairs]) for k in (1, 2, 3)] if pairs else []
    if case["host"]:
        s.problem = _problem(case, None, oneint, chol)
        shape = lambda k: (m,) + (n,) * round(math.log(s.koop[k].numel() // m, n))
        s.koop = {k: v.cpu().numpy().reshape(shape(k), order="F") for k, v in s.koop.items()}
        s.trdm = [t.cpu().numpy().reshape((len(pairs),) + (n,) * (2 * k + 2), order="F")
                  for k, t in enumerate(s.trdm)] or None
        from nevpt2_gb300 import koopro
        koopro.context()
        return s
    s.ctx, s.stream = _context(case["split"]), torch.cuda.Stream()
    s.oneint, s.chol, s.norb = oneint, chol.contiguous(), nc + n + nv
    return s


# ---------------------------------------------------------------------- runs
ENERGIES = ("e2mpp", "psimpp", "e2enp", "psienep", "e2mp", "e2en", "psimp", "psien", "epsnew", "nnew")


def run(s):
    case = s.case
    n = case["nact"]
    kind = case["kind"]
    if kind == "driver":
        from nevpt2_gb300 import koopro
        return koopro.koopro4QD(s.problem)
    if kind == "energies":
        return _run_energies(s)
    st = ctypes.c_void_p(s.stream.cuda_stream)
    call = s.ctx.call
    if kind == "unfold":
        call("nvpt_permute_4rdm_d", _ptr(s.ro4), n, _ptr(s.labels), _ptr(s.values), s.values.numel(), st)
        return s.ro4
    m, nc = case["states"], case["ncore"]
    d3, d2, d1 = (_ptr(s.rdm[k]) for k in ("3-RDM", "2-RDM", "1-RDM"))
    atwo, aj, f = _ptr(s.atwo), _ptr(s.aj), _ptr(s.f)
    if kind == "bamat":
        call("nvpt_bamat_d", _ptr(s.amat), _ptr(s.atmat), atwo, _ptr(s.ro4), d3, d2, d1, n, nc, f, aj, s.norb, m, 1, st)
        return {"amatIP": s.amat, "amatEA": s.atmat}
    ne = case["nele"]
    call("nvpt_bro3_d", _ptr(s.ro4), d3, n, ne, m, st)
    call("nvpt_bro2_d", d3, d2, n, ne, m, st)
    call("nvpt_bro1_d", d2, d1, n, ne, m, st)
    call("nvpt_get_aj_atwo_d", atwo, n, nc, s.norb, aj, _ptr(s.oneint), _ptr(s.chol), s.chol.shape[1], st)
    call("nvpt_koop_matrices_ctl_d", m, n, nc, atwo, d3, d2, d1, f, aj, *(_ptr(x) for x in s.koop.values()), st)
    o = {k: _ptr(x) for k, x in s.lower.items()}
    call("nvpt_bbmat_d", atwo, o["bmatIP"], o["bmatEA"], d3, d2, d1, n, nc, f, aj, m, st)
    call("nvpt_bcmat_d", atwo, o["cmatIP"], o["cmatEA"], d3, d2, d1, n, nc, f, aj, m, st)
    call("nvpt_bdmat_d", atwo, o["dmatIP"], o["dmatEA"], d2, d1, n, nc, f, aj, m, st)
    return {**s.rdm, "atwo": s.atwo, "aj": s.aj, **s.koop, **s.lower}


def _run_energies(s):
    from nevpt2_gb300 import qdnevpt as gq
    case = s.case
    m = case["states"]
    if case["host"]:
        res = gq.qdnevpt(s.problem, s.koop, transition=s.trdm)
        return {k: getattr(res, k) for k in ENERGIES}
    gq._bind(s.ctx)
    inp = gq._In(case["ncore"], case["nact"], case["nvirt"], m, s.chol.shape[1], 1e-6, 0, 0xFF, None, _ptr(s.oneint),
                 _ptr(s.chol), *(_ptr(s.koop[k]) for k in KOOP), *(map(_ptr, s.trdm) if s.trdm else (None,) * 3))
    res = {k: np.zeros((8, m), order="F") for k in ENERGIES[:4]}
    res.update({k: np.zeros((m, m), order="F") for k in ENERGIES[4:6]})
    res.update({k: np.zeros(m) for k in ENERGIES[6:8]})
    res["epsnew"], res["nnew"] = np.zeros((s.norb, m), order="F"), np.zeros((10, m), np.int64, order="F")
    out = gq._Out(*(ctypes.c_void_p(res[k].ctypes.data) for k in ENERGIES))
    s.ctx.check(s.ctx._lib.nvpt_qdnevpt_d(s.ctx.handle, ctypes.byref(inp), ctypes.byref(out),
                                          ctypes.c_void_p(s.stream.cuda_stream)), "nvpt_qdnevpt_d")
    return res


# ---------------------------------------------------------------------- work
def work(case):
    """Each input read once (of the packed 4-RDM the entries that are defined), each output written once; the flops
    of the contractions after the permutational symmetry of the RDMs and integrals is used."""
    n = case["nact"]
    w = n * (n + 1) * (n + 2) * (n + 3) // 24
    packed = 8 * w * n**4 // 2
    if case["kind"] == "unfold":
        entries = int(case["fill"] * packed) // 8
        return {"bytes": entries * (8 * 4 + 8) + entries * 8, "flops": 0}
    m, nc = case["states"], case["ncore"]
    norb = nc + n + case.get("nvirt", 0)
    pair, nchol = norb * (norb + 1) // 2, 4 * norb
    nn = n * (n + 1) // 2
    # A-matrices: one n^9 contraction over unordered excitation pairs and (d f) pairs
    a_flops = m * 2 * (n * n * (n * n + 1) // 2) * n * (nn * n) * n
    a_bytes = m * (packed + 8 * n**6 + 2 * 8 * n**6) + 8 * n**4
    if case["kind"] == "bamat":
        return {"bytes": a_bytes, "flops": a_flops}
    act = nn + n * nc + nc  # Cholesky columns of the active and core-active pairs
    front = {"bytes": m * (packed + 8 * (n**6 + 12 * n**4)) + 8 * (act * nchol + 2 * pair + n**4),
             "flops": nn * nn * nchol + m * 2 * 10 * n**7}
    if case["kind"] == "front":
        return front
    if case["kind"] == "driver":
        return {"bytes": front["bytes"] + a_bytes, "flops": front["flops"] + a_flops}
    nv, n3 = case["nvirt"], n**3
    half = 0.5 * nchol * 2
    eri = half * ((nc * nv) ** 2 + (nc * n) ** 2 + (n * nv) ** 2) + 2 * half * n * nc * (nc * nv + n * n + n * nv)
    eri += 2 * half * (nc * nv * n * nv + nc * nv * n * n + n * n * n * nv)
    half_transform = 2 * nchol * (nc * nc * nv + nc * nv * nv + n * nv * nv + nc * nc * n)
    pencil = 2 * (n3**3 // 3 + n3**3 + 4 * n3**3 // 3) + (nv + nc) * (2 + m) * 3 * n3 * n3
    small = 2 * 9 * ((2 * n * n) ** 3 + 2 * (n * n) ** 3)
    return {"bytes": 8 * (nchol * pair + m * (3 * n**6 + 9 * n**4) + m * (m - 1) // 2 * n**6),
            "flops": eri + m * (half_transform + pencil + small)}


# --------------------------------------------------- plain 64-bit evaluation
def exact(case, seed):
    kind = case["kind"]
    if kind == "unfold":
        return None  # values are copied, halved or doubled, nothing is computed
    states = _states(case, seed)
    oneint, chol = _integrals(case, _generator(seed, 2), states[0])
    if kind == "energies":
        return _exact_energies(case, seed, states, oneint, chol)
    atwo, aj = _active_integrals(case, oneint, chol)
    if kind == "bamat":
        a, at = zip(*(_exact_bamat(x, atwo, aj) for x in states))
        return {"amatIP": _fortran(a), "amatEA": _fortran(at)}
    out = [_exact_front(x, atwo, aj) for x in states]
    if kind == "driver":
        for x, o in zip(states, out):
            o["amatIP"], o["amatEA"] = _exact_bamat(x, atwo, aj)
    res = {k: _fortran([o[k] for o in out]) for k in out[0]}
    nc, n, norb = case["ncore"], case["nact"], case["ncore"] + case["nact"] + case["nvirt"]
    full = _square(oneint, norb)
    full[nc:nc + n, nc:nc + n] = aj
    res["aj"], res["atwo"] = full[_pairs(norb)], _fortran([atwo])
    if kind == "driver":  # host arrays (state, i, j, ...), Fortran order
        m = case["states"]
        for k, v in res.items():
            v = v.cpu().numpy()
            if k == "atwo":
                v = v.reshape((n,) * 4, order="F")
            elif k != "aj":
                v = v.reshape((m,) + (n,) * round(math.log(v.size // m, n)), order="F")
            res[k] = v
    return res


def _square(tri, norb):
    p, q = _pairs(norb)
    h = torch.empty(norb, norb, dtype=F64, device=tri.device)
    h[p, q] = tri
    h[q, p] = tri
    return h


def _active_integrals(case, oneint, chol):
    """(ab|cd) over the active orbitals and the core-dressed one-electron operator."""
    nc, n = case["ncore"], case["nact"]
    norb = nc + n + case.get("nvirt", 0)
    b = _dense_df(chol, norb)
    c, a = slice(0, nc), slice(nc, nc + n)
    atwo = torch.einsum("xab,xcd->abcd", b[:, a, a], b[:, a, a])
    aj = _square(oneint, norb)[a, a] + 2.0 * torch.einsum("xab,xkk->ab", b[:, a, a], b[:, c, c])
    return atwo, aj - torch.einsum("xak,xkb->ab", b[:, a, c], b[:, c, a])


def _exact_front(state, T, h):
    es = torch.einsum
    g1, g2, g3, ee, eee, d = _accessors(state)
    jx = es("accb->ab", T)
    f1, f2 = h - 0.5 * jx, h - jx
    o = {"3-RDM": g3, "2-RDM": g2, "1-RDM": g1}
    ip = -2.0 * (es("ac,pc->pa", h, g1) + es("cead,pcde->pa", T, g2))
    o["1-IPKO"] = ip
    o["1-EAKO"] = ip + 2.0 * (2.0 * h + 2.0 * es("depa,de->pa", T, g1) - es("peda,de->pa", T, g1))
    h2 = o["2-HRDM"] = _hole2(g1, g2, d)
    h3 = _rdm(_holes(state), 3)
    # 2-IP
    x = -es("ad,pqdb->pqab", f1, g2) - es("bd,pqad->pqab", f1, g2)
    y = g3 + 0.5 * es("df,pqeb->pqdfbe", d, g2) + 0.5 * es("db,pqfe->pqdfbe", d, g2)
    x -= es("deaf,pqdfbe->pqab", T, y)
    y = g3 + 0.5 * es("da,pqef->pqdafe", d, g2) + 0.5 * es("df,pqae->pqdafe", d, g2)
    o["2-IPKO"] = x - es("debf,pqdafe->pqab", T, y)
    # 2-EA
    x = es("ac,pqcb->pqab", f1, h2) + es("bc,pqac->pqab", f1, h2)
    y = -h3 + 2.0 * es("ce,pqdb->pqedbc", d, h2) - 0.5 * es("de,pqcb->pqedbc", d, h2)
    x += es("ceda,pqedbc->pqab", T, y - 0.5 * es("be,pqdc->pqedbc", d, h2))
    y = -h3 + 2.0 * es("ce,pqad->pqeadc", d, h2) - 0.5 * es("ae,pqcd->pqeadc", d, h2)
    o["2-EAKO"] = x + es("cedb,pqeadc->pqab", T, y - 0.5 * es("de,pqac->pqeadc", d, h2))
    # 0': A [q, p, a, b] of <E_qp ...>
    x = 2.0 * (es("ca,qpcb->qpab", f1, ee) - es("bc,qpac->qpab", f1, ee))
    x += es("ceda,qpcedb->qpab", T, eee) + es("ceda,qpdbce->qpab", T, eee)
    o["gk0pa"] = x - es("becd,qpaecd->qpab", T, eee) - es("becd,qpcdae->qpab", T, eee)
    d1 = -ee.permute(2, 1, 0, 3) + 2.0 * es("ap,qc->qpac", d, g1) + es("qp,ac->qpac", d, g1)
    x = -es("bc,qpac->qpab", f1, d1) + es("ca,qpcb->qpab", f1, d1)
    # D operand over (c, e, a, q, p, d)
    y = -es("ceapqd->ceapqd", eee) - es("apqdce->ceapqd", eee)
    y = y + 2.0 * (es("pa,ceqd->ceapqd", d, ee) + es("pa,qdce->ceapqd", d, ee))
    y = y + es("qp,cead->ceapqd", d, ee) + es("qp,adce->ceapqd", d, ee)
    y = y - es("pc,aeqd->ceapqd", d, ee) + 2.0 * es("pc,ea,qd->ceapqd", d, d, g1)
    y = y + es("qe,apcd->ceapqd", d, ee) - 2.0 * es("qe,pa,cd->ceapqd", d, d, g1)
    o["gk0pd"] = x - 0.5 * es("cebd,ceapqd->qpab", T, y) + 0.5 * es("ceda,cedpqb->qpab", T, y)
    x = 2.0 * (es("ca,cb->ab", f1, g1) - es("bc,ac->ab", f1, g1))
    x += es("ceda,cedb->ab", T, ee) + es("ceda,dbce->ab", T, ee)
    o["gk0pf"] = x - es("becd,aecd->ab", T, ee) - es("becd,cdae->ab", T, ee)
    # B, C, D of the (+-1') classes
    et = 2.0 * es("ab,cd->abcd", d, g1) - ee.permute(1, 0, 2, 3)          # <E~_ab E_cd>
    etr = 2.0 * es("cd,ab->abcd", d, g1) - ee.permute(0, 1, 3, 2)         # <E_ab E~_cd>
    eet = 2.0 * es("cd,abef->abcdef", d, ee) - eee.permute(0, 1, 3, 2, 4, 5)
    etl = 2.0 * es("ab,cdef->abcdef", d, ee) - eee.permute(1, 0, 2, 3, 4, 5)
    o["bmatIP"] = -es("ca,rpqc->pqra", f2, ee) - es("rpqecf,aecf->pqra", eee, T)
    o["bmatEA"] = es("ca,rpqc->pqra", h, etr) + es("rpqecf,aecf->pqra", eet, T)
    kx = es("deea->da", T)
    fm, fp = f1 - 0.5 * kx, f1 + 0.5 * kx
    x = es("da,pbdc->pabc", fm, ee) - es("cd,pbad->pabc", fp, ee) - es("bd,pdac->pabc", fm, ee)
    x += es("pbde,ceda->pabc", ee, T) + es("pbdfec,dfea->pabc", eee, T)
    o["cmatIP"] = x - es("pbdfae,dfce->pabc", eee, T) - es("pedfac,dfbe->pabc", eee, T)
    x = es("da,pbdc->pabc", fm, et) - es("cd,pbad->pabc", fp, et) + es("bd,pdac->pabc", fp, et)
    x += es("pbde,ceda->pabc", et, T) + es("pbdfec,dfea->pabc", etl, T)
    o["cmatEA"] = x - es("pbdfae,dfce->pabc", etl, T) + es("pedfac,dfbe->pabc", etl, T)
    o["dmatIP"] = -es("ca,pc->pa", f2, g1) - es("pecf,aecf->pa", ee, T)
    o["dmatEA"] = es("ca,pc->pa", h, 2.0 * d - g1) + es("pecf,aecf->pa", et, T)
    return o


def _exact_bamat(state, T, h):
    """A and A~ [ap, bp, cp, a, b, c], one cp at a time."""
    es = torch.einsum
    g1, g2, g3, ee, eee, d = _accessors(state)
    n = g1.shape[0]
    kx = es("deea->da", T)
    f = h - 0.5 * kx
    fm, fp = f - 0.5 * kx, f + 0.5 * kx
    A, At = (torch.empty((n,) * 6, dtype=F64, device=g1.device) for _ in range(2))
    rest = torch.cartesian_prod(*([torch.arange(n, device=g1.device)] * 3))
    for r in range(n):
        rows = torch.cat([torch.full_like(rest[:, :1], r), rest], 1)
        g4 = _rdm4_rows(state, rows).view((n,) * 7)               # creators c, e, g of r; annihilators b, d, f, h
        x = g4.permute(3, 0, 4, 1, 5, 2, 6).contiguous()          # <E_rb E_cd E_ef E_gh> at [b, c, d, e, f, g, h]
        del g4
        t3, t2, t1 = g3[r], g2[r], g1[r]
        x += es("bc,egdfh->bcdefgh", d, t3)
        x += es("be,cgfdh->bcdefgh", d, t3)
        x += es("bg,cehdf->bcdefgh", d, t3)
        x += es("de,gcbhf->bcdefgh", d, t3)
        x += es("dg,cebhf->bcdefgh", d, t3)
        x += es("fg,ecbhd->bcdefgh", d, t3)
        x += es("bc,de,gfh->bcdefgh", d, d, t2)
        x += es("bc,dg,ehf->bcdefgh", d, d, t2)
        x += es("bc,fg,edh->bcdefgh", d, d, t2)
        x += es("be,dg,cfh->bcdefgh", d, d, t2)
        x += es("be,fg,chd->bcdefgh", d, d, t2)
        x += es("bg,de,chf->bcdefgh", d, d, t2)
        x += es("de,fg,cbh->bcdefgh", d, d, t2)
        x += es("bc,de,fg,h->bcdefgh", d, d, d, t1)
        # p = ap, q = bp: <E_rp E_qb E_df E_wz> = x[p, q, b, d, f, w, z]
        t_1 = es("pqbdfec,dfea->pqabc", x, T)
        t_2 = es("pqbdfae,dfce->pqabc", x, T)
        t_3 = es("pqedfac,dfbe->pqabc", x, T)
        t_4 = es("peqdfac,dfbe->pqabc", x, T)
        del x
        e3, e2 = eee[r], ee[r]                                    # [p, q, b, d, c, ...]
        a = es("pqbdc,da->pqabc", e3, fm) - es("pqbad,cd->pqabc", e3, fp) - es("pqdac,bd->pqabc", e3, fm)
        a += es("pqbde,ceda->pqabc", e3, T) + t_1 - t_2 - t_3
        e3t = 2.0 * es("qb,pdc->pqbdc", d, e2) - e3.permute(0, 2, 1, 3, 4)
        at = es("pqbdc,da->pqabc", e3t, f) - es("pqbad,cd->pqabc", e3t, f) + es("pqdac,bd->pqabc", e3t, fp)
        m1 = 2.0 * es("qb,pde->pqbde", d, e2) - es("pbqde->pqbde", e3)
        at += es("pqbde,ceda->pqabc", m1, T) - 0.5 * es("pqbdc,da->pqabc", m1, kx) - 0.5 * es("pqbae,ce->pqabc", m1, kx)
        e4t = es("pdfac,dfbq->pqabc", e3, T)                      # 2 sum <E_rp E_df E_ac> (df|bq) of the E~ product
        at += 2.0 * e4t - t_4
        at += 2.0 * es("qb,pdfec,dfea->pqabc", d, e3, T) - 2.0 * es("qb,pdfae,dfce->pqabc", d, e3, T)
        at -= (t_1 - t_2).permute(0, 3, 2, 1, 4)
        A[:, :, r], At[:, :, r] = a, at
    return A, At


def _pc(S, K, thr=1e-6):
    """PC basis of a metric: eigenvectors of K in the kept eigenspace of S, and its energies."""
    w, u = torch.linalg.eigh(S)
    keep = w >= thr
    x = u[:, keep] / w[keep].sqrt()
    e, v = torch.linalg.eigh(x.mT @ K @ x)
    return x @ v, e


def _exact_energies(case, seed, states, oneint, chol):
    nc, n, nv, m = case["ncore"], case["nact"], case["nvirt"], case["states"]
    norb = nc + n + nv
    b0, h0 = _dense_df(chol, norb), _square(oneint, norb)
    out = {k: np.zeros((8, m)) for k in ENERGIES[:4]}
    out["epsnew"], out["nnew"] = np.zeros((norb, m)), None
    for i, state in enumerate(states):
        ko = _koopmans(case, _generator(seed, 50 + i), state)
        fock = h0 + _fock2(b0, nc, n, ko["1-RDM"])
        eps = torch.zeros(norb, dtype=F64, device=h0.device)
        u = torch.eye(norb, dtype=F64, device=h0.device)
        for o in (slice(0, nc), slice(nc + n, norb)):
            eps[o], u[o, o] = torch.linalg.eigh(fock[o, o])
        b, h = u.mT @ b0 @ u, u.mT @ h0 @ u
        out["epsnew"][:, i] = eps.cpu().numpy()
        for cls, r in enumerate(_class_energies(ko, b, h, eps, nc, n)):
            for k, v in zip(ENERGIES[:4], r):
                out[k][cls, i] = float(v)
    out["psimp"], out["psien"] = out["psimpp"].sum(0), out["psienep"].sum(0)
    one = m == 1  # the off-diagonal elements of several states have no plain counterpart here
    out["e2mp"] = out["e2mpp"].sum(0, keepdims=True) if one else None
    out["e2en"] = out["e2enp"].sum(0, keepdims=True) if one else None
    return out


def _sc(dn, dk, base):
    """Strongly contracted energy and norm over the labels."""
    ok = dn.abs() > 1e-14
    dn, dk, base = dn[ok], dk[ok], base[ok]
    den = base - dk / dn
    return (dn / den).sum(), (dn / den**2).sum()


def _pc_sums(r2, w, shift):
    """Partially contracted energy and norm from squared numerators [label, mu]."""
    den = w[None, :] + shift[:, None]
    return -(r2 / den).sum(), (r2 / den**2).sum()


def _class_energies(ko, b, h, eps, nc, n):
    """(E_SC, norm_SC, E_PC, norm_PC) of the eight classes (0) +1 -1 +2 -2 +1' -1' 0'."""
    es = torch.einsum
    c, a, v = slice(0, nc), slice(nc, nc + n), slice(nc + n, None)
    bcc, bca, bcv, baa, bav = b[:, c, c], b[:, c, a], b[:, c, v], b[:, a, a], b[:, a, v]
    ec, ev = eps[c], eps[v]
    eri = lambda x, y: es("xpq,xrs->pqrs", x, y)
    g1 = ko["1-RDM"]
    nv = ev.numel()
    d = torch.eye(n, dtype=F64, device=b.device)
    up = lambda k, o: torch.triu_indices(k, k, offset=o, device=b.device)
    res = []
    # (0)
    g = eri(bcv, bcv).permute(0, 2, 1, 3)                           # [i, j, r, s] = (i r | j s)
    ab1, ab2 = g.permute(1, 0, 2, 3), g
    zi = torch.eye(nc, dtype=torch.bool, device=b.device)[:, :, None, None]
    zr = torch.eye(nv, dtype=torch.bool, device=b.device)[None, None]
    x = torch.where(zi & zr, ab1, torch.where(zi ^ zr, math.sqrt(2.0) * ab1,
                                              2.0 * (ab1**2 + ab2**2 - ab1 * ab2).clamp_min(0).sqrt()))
    den = ev[None, None, :, None] + ev[None, None, None, :] - ec[:, None, None, None] - ec[None, :, None, None]
    (i, j), (r, s) = up(nc, 0), up(nv, 0)
    x, den = x[i, j][:, r, s], den[i, j][:, r, s]
    co = -x / den
    res.append(((x * co).sum(), (co * co).sum()) * 2)
    # (+-1)
    for plus in (True, False):
        if plus:
            t = eri(bca, bcv)                                      # [i, a, j, r]
            p, q = i, j
            tj, tk = t[p, :, q, :].permute(0, 2, 1), t[q, :, p, :].permute(0, 2, 1)   # [pair, r, a]
            base = (ec[p] + ec[q])[:, None] - ev[None, :]
            ro, gk = 2.0 * d - g1, ko["1-EAKO"]
        else:
            t = eri(bcv, bav)                                      # [i, r, a, s]
            p, q = r, s
            tj = t[:, p][torch.arange(nc)[:, None], torch.arange(p.numel())[None], :, q[None]].permute(1, 0, 2)
            tk = t[:, q][torch.arange(nc)[:, None], torch.arange(p.numel())[None], :, p[None]].permute(1, 0, 2)
            base = ec[None, :] - (ev[p] + ev[q])[:, None]
            ro, gk = g1, ko["1-IPKO"]
        same = (p == q)[:, None, None].to(F64)
        form = lambda m: (es("lea,ab,leb->le", tj, m, tj) + es("lea,ab,leb->le", tk, m, tk)
                          - 0.5 * es("lea,ab,leb->le", tj, m, tk) - 0.5 * es("lea,ab,leb->le", tk, m, tj)) \
            * torch.where(p == q, 0.5, 1.0)[:, None].to(F64)
        sc = _sc((2.0 * form(ro)).reshape(-1), form(gk).reshape(-1), base.reshape(-1))
        cc, w = _pc(ro, 0.5 * gk)
        sm = ro.mT @ cc
        vp, vm = (tj + tk) * (1.0 - same * (1.0 - math.sqrt(0.5))), (tj - tk) * (1.0 - same)
        r2 = 0.5 * (vp @ sm) ** 2 + 1.5 * (vm @ sm) ** 2
        res.append(sc + _pc_sums(r2.reshape(-1, w.numel()), w, -base.reshape(-1)))
    # (+-2)
    for plus in (True, False):
        t = eri(bca, bca) if plus else eri(bav, bav)
        t = t.permute(0, 2, 1, 3) if plus else t.permute(1, 3, 0, 2)   # [p, q, a, b]: (p a | q b), (a p | b q)
        N = t.shape[0]
        dm, km = (ko["2-HRDM"], ko["2-EAKO"]) if plus else (ko["2-RDM"], ko["2-IPKO"])
        e = ec if plus else -ev
        p, q = up(N, 1)
        ne, eq = t[p, q], t[torch.arange(N), torch.arange(N)]
        sne = ne if plus else t[q, p]
        form = lambda x, m: es("lab,abcd,lcd->l", x, m, x)
        dn = torch.cat([form(sne, dm), form(0.5 * eq, dm + dm.permute(0, 1, 3, 2))])
        dk = torch.cat([form(sne, km), form(0.5 * eq, km + km.permute(1, 0, 2, 3))])
        base = torch.cat([e[p] + e[q], 2.0 * e])
        sc = _sc(dn, dk, base)
        S, K = dm.reshape(n * n, n * n), km.reshape(n * n, n * n)
        cc, w = _pc(S, K)
        x = (ne.permute(0, 2, 1) if plus else ne).reshape(-1, n * n)
        e1, s1 = _pc_sums((x @ (S.mT @ cc)) ** 2, w, -(e[p] + e[q]))
        ia, ib = up(n, 0)
        pick = lambda m: (m + m.permute(0, 1, 3, 2))[ia, ib][:, ia, ib]
        S, K = pick(dm), pick(km)
        cc, w = _pc(S, K)
        y = (eq.permute(0, 2, 1) if plus else eq)[:, ia, ib] * torch.where(ia == ib, 1.0, 2.0).to(F64)
        e2, s2 = _pc_sums((y @ (0.5 * S.mT @ cc)) ** 2, w, -2.0 * e)
        res.append(sc + (e1 + e2, s1 + s2))
    # (+1') and (-1')
    ee = ko["2-RDM"].permute(0, 2, 1, 3) + es("bc,ad->abcd", d, g1)
    g2 = ko["2-RDM"]
    eee = ko["3-RDM"].permute(0, 3, 1, 4, 2, 5) + es("ed,acbf->abcdef", d, g2) + es("eb,acfd->abcdef", d, g2)
    eee = eee + es("bc,aedf->abcdef", d, g2) + es("bc,ed,af->abcdef", d, d, g1)
    jc = es("xkk->x", bcc)
    for minus in (False, True):
        if minus:
            hd = h[a, v] + 2.0 * es("x,xar->ar", jc, bav) - es("xka,xkr->ar", bca, bcv) - es("xab,xbr->ar", baa, bav)
            hd = hd.mT
            vd = eri(baa, bav).permute(3, 0, 2, 1)                     # [r, ap, bp, cp] of (ap cp | bp r)
            w3, w2, rho, tag, base = eee, ee, g1, "IP", -ev
        else:
            hd = h[c, a] + 2.0 * es("x,xia->ia", jc, bca) - es("xki,xka->ia", bcc, bca)
            vd = eri(baa, bca).permute(2, 0, 3, 1)                     # [i, ap, bp, cp] of (ap cp | i bp)
            w3 = 2.0 * es("cd,abef->abcdef", d, ee) - eee.permute(0, 1, 3, 2, 4, 5)
            w2 = 2.0 * es("cd,ab->abcd", d, g1) - ee.permute(0, 1, 3, 2)
            rho, tag, base = 2.0 * d - g1, "EA", ec
        n3 = n**3
        vd = vd.reshape(-1, n3)
        S = w3.permute(1, 2, 0, 4, 3, 5).reshape(n3, n3)
        W2 = w2.permute(1, 2, 0, 3).reshape(n3, n)
        A, bc = ko["amat" + tag].reshape(n3, n3), ko["bmat" + tag] + ko["cmat" + tag].permute(1, 2, 3, 0)
        quad = lambda x, m, y: ((x @ m) * y).sum(1)
        dn = quad(hd, rho, hd) + 2.0 * quad(vd, W2, hd) + quad(vd, S, vd)
        dk = quad(hd, ko["dmat" + tag], hd) + quad(vd, bc.reshape(n3, n), hd) + quad(vd, A, vd)
        sc = _sc(dn, dk, base)
        cc, w = _pc(S, A)
        z = vd @ S + hd @ W2.mT
        res.append(sc + _pc_sums((z @ cc) ** 2, w, -base))
    # (0')
    hd = (h[c, v] + 2.0 * es("x,xir->ir", jc, bcv) - es("xki,xkr->ir", bcc, bcv)).reshape(-1)
    nn = n * n
    dj = eri(bcv, baa).reshape(-1, nn)
    dk_ = eri(bca, bav).permute(0, 3, 1, 2).reshape(-1, nn)            # [i, r, a, b] of (i a | b r)
    etr = 2.0 * es("cd,ab->abcd", d, g1) - ee.permute(0, 1, 3, 2)
    m1 = ee.permute(1, 0, 2, 3).reshape(nn, nn)
    m2 = (etr.permute(2, 0, 3, 1) + es("ab,qp->pqab", d, g1)).reshape(nn, nn)
    k1, k2 = (ko[k].permute(1, 0, 2, 3).reshape(nn, nn) for k in ("gk0pa", "gk0pd"))
    form = lambda x, m, y: ((x @ m) * y).sum(1)
    both = lambda p, q, w0: (2.0 * form(dj, p, dj) - form(dj, p, dk_) - form(dk_, p, dj)) * w0 + form(dk_, q, dk_)
    di = 2.0 * dj - dk_
    dn = both(m1, m2, 1.0) + 2.0 * hd * (di @ g1.mT.reshape(-1)) + 2.0 * hd**2
    dk = both(k1, k2, 0.5) + 0.5 * hd * (di @ ko["gk0pf"].reshape(-1))
    base = (ec[:, None] - ev[None, :]).reshape(-1)
    sc = _sc(dn, dk, base)
    north = ee.permute(2, 3, 1, 0).reshape(nn, nn)
    south = (-g2.permute(1, 2, 3, 0) + 2.0 * es("ap,qb->abpq", d, g1)).reshape(nn, nn)
    south2 = (-g2.permute(2, 1, 0, 3) + 2.0 * es("pa,bq->abpq", d, g1)).reshape(nn, nn)
    S = torch.cat([torch.cat([2.0 * north, -north], 1), torch.cat([-north, south], 1)])
    K = torch.cat([torch.cat([k1, -0.5 * k1], 1), torch.cat([-0.5 * k1, k2], 1)])
    cc, w = _pc(S, K)
    top, bot = cc[:nn], cc[nn:]
    gba = g1.mT.reshape(1, nn)
    z = di @ (north @ top) - dj @ (north @ bot) + dk_ @ (south2 @ bot) + hd[:, None] * (gba @ (2.0 * top - bot))
    res.append(sc + _pc_sums(z**2, w, -base))
    return res
