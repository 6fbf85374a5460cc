"""The A-matrices of the (+-1') classes from one n^9 contraction.

CPU: the route's sums (the ones csrc/bamat_sym.cu evaluates) in numpy against
the oracle's restatement of src/koopro4QD.F90:3974-4104.
GPU: both routes against the oracle -- RDMs and integrals with their physical
symmetries, and inputs without one of them, which the device has to notice
and send through the general route.  Tolerance 1e-10 of the largest element,
the bound every Koopmans matrix is held to (FP64 sums of at most n^3 terms in
another order: below 1e-13)."""
import numpy as np
import pytest

from conftest import rel_err
from nevpt2_gb300 import synth
from oracle import oracle as orc

es = np.einsum


def _inputs(n, ne, metat, seed, ndet=None):
    p = synth.make_problem(n, ne, 2, 3, metat=metat, ndet=ndet, seed=seed)
    atwo, aj = orc.get_aj_atwo(p.oneint, p.chol, n, 2, p.norb)
    return p, np.asarray(atwo), aj


def _oracle(p, atwo, aj):
    f = np.zeros(p.norb * (p.norb + 1) // 2)
    return orc.bamat(atwo, p.ro4, p.daaa, p.taa, p.dal, p.nact, 2, f, aj, p.norb, p.metat)


def _dense4(p, s):
    """Gamma4[p1..p4, q1..q4] from the packed array."""
    n = p.nact
    out = np.zeros((n,) * 8)
    keys = [(a, b, c, d) for a in range(n) for b in range(a + 1) for c in range(b + 1) for d in range(c + 1)]
    rank = {k: i for i, k in enumerate(keys)}
    for c in np.ndindex(*(n,) * 4):
        for a in np.ndindex(*(n,) * 4):
            kc, ka = (rank[tuple(sorted(x, reverse=True))] for x in (c, a))
            k, o = (c, a) if kc >= ka else (a, c)
            order = sorted(range(4), key=lambda i: -k[i])
            out[c + a] = p.ro4[(max(kc, ka),) + tuple(o[i] for i in order) + (s,)]
    return out


@pytest.mark.parametrize("n,ne", [(3, 4), (4, 4)])
def test_one_contraction_equals_the_loop(n, ne):
    p, T, aj = _inputs(n, ne, 1, 40 + n)
    A0, At0 = (np.asarray(x)[0] for x in _oracle(p, T, aj))
    D1, D2, D3, D4 = p.dal[0], p.taa[0], p.daaa[0], _dense4(p, 0)
    d = np.eye(n)
    h = np.array([[aj[synth.tri(i + 3, j + 3) - 1] for j in range(n)] for i in range(n)])  # f + K/2 = aj
    F = es("pqdersfc,dfea->prqsca", D4, T, optimize=True) + es("pqdrsc,da->prqsca", D3, h)  # [A, B, c, a]
    J = es("pqdrsf,dfxy->prqsxy", D3, T) + es("pqrs,xy->prqsxy", D2, h)
    Kx = es("pqdrse,dxye->prqsxy", D3, T)
    Wca, Waa = es("pqefrs,xfey->pqrsxy", D3, T), es("pqtfre,xfye->pqrtxy", D3, T)
    G1, G3 = es("pqecea->pqca", J), es("peqrxe->pqrx", J)
    Q1 = es("ptfe,xfye->ptxy", D2, T)
    J2 = es("pdqf,dfxy->pqxy", D2, T) + es("pq,xy->pqxy", D1, h)
    JW = J2 + es("pefs,xfey->psxy", D2, T)
    Z = 2 * J2 - es("pecf,qfbe->pcqb", D2, T)
    Q2 = es("pece->pc", J2)
    o = "->jkialc"  # i, j, k, l = cp, ap, bp, b
    A = es("ijklca" + o, F) - es("jilkac" + o, F) - es("jicakl" + o, F)
    A += es("iklcja" + o, Wca) + es("icklja" + o, J) - es("iklajc" + o, Waa) - es("kijalc" + o, Waa)
    A -= es("iackjl" + o, Waa) + es("la,kijc" + o, d, G3) + es("la,ikjc" + o, d, Q1)
    A += es("jk,ilca" + o, d, G1) - es("jk,liac" + o, d, G1) - es("jk,iacl" + o, d, G3) - es("jk,ialc" + o, d, Q1)
    A -= es("ja,iklc" + o, d, G3) + es("ja,kicl" + o, d, G3) + es("ja,kilc" + o, d, Q1) + es("jk,la,ic" + o, d, d, Q2)
    assert rel_err(A, A0) < 1e-12
    B = es("jiklac" + o, F) - es("ijlkca" + o, F) - es("ijackl" + o, F)
    B = B + es("ilkajc" + o, Waa) + es("lijakc" + o, Waa) - es("cjikal" + o, Waa)
    B -= es("ilkcja" + o, Wca) + es("lijcka" + o, Wca) + es("iackjl" + o, Wca)
    B += 2 * es("ijaclk" + o, J) - es("iclkja" + o, J) - es("ijlcka" + o, J) - es("ikacjl" + o, J) - es("ijaclk" + o, Kx)
    B += 2 * es("idjc,dalk" + o, D2, T) - es("iejc,kale" + o, D2, T)
    B += 2 * es("iaec,jelk" + o, D2, T) - es("iafc,kflj" + o, D2, T)
    B -= es("ilfc,jfka" + o, D2, T) + es("ilcf,kfja" + o, D2, T) + es("idkc,dalj" + o, D2, T) + es("ieck,jale" + o, D2, T)
    B += 2 * es("ic,jalk" + o, D1, T) - es("ic,kalj" + o, D1, T)
    B += es("ja,ilkc" + o, d, G3) + es("ja,likc" + o, d, Q1) - es("ja,ickl" + o, d, G1) + es("ja,ickl" + o, d, Z)
    B += es("jl,kiac" + o, d, G1) - es("jl,ikca" + o, d, G1) - es("jl,icka" + o, d, JW) + es("jl,iakc" + o, d, Q1)
    B += es("jl,ka,ic" + o, d, d, Q2) + es("ka,lijc" + o, d, G3) + es("ka,iljc" + o, d, Q1)
    B -= es("ka,ijcl" + o, d, G1) + es("ka,icjl" + o, d, JW)
    D = G1 + es("icja->ijca", JW) - es("aijc->ijca", G3) - es("iajc->ijca", Q1) - es("ja,ic->ijca", d, Q2)
    B += 2 * es("lk,ijca" + o, d, D)
    assert rel_err(B, At0) < 1e-12


def _gpu(p, atwo, aj):
    from nevpt2_gb300 import koopro
    f = np.zeros(p.norb * (p.norb + 1) // 2)
    return koopro.bamat(atwo, p.ro4, p.daaa, p.taa, p.dal, p.nact, 2, f, aj, p.norb, p.metat)


# the smallest sizes, both sides of the direct kernel's limit, odd sizes and several states
SIZES = [(1, 2, 1), (2, 2, 2), (3, 4, 1), (5, 4, 2), (6, 6, 1), (7, 6, 3), (8, 8, 1), (9, 8, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,ne,metat", SIZES)
def test_symmetric_inputs(gpu_ctx, n, ne, metat):
    p, atwo, aj = _inputs(n, ne, metat, 60 + n, ndet=300 if n > 6 else None)
    for got, ref in zip(_gpu(p, atwo, aj), _oracle(p, atwo, aj)):
        assert rel_err(got, ref) < 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["atwo_ij", "atwo_exchange", "ro4", "daaa", "taa", "dal", "nan"])
@pytest.mark.parametrize("n,ne", [(4, 4), (6, 6)])
def test_inputs_without_a_symmetry_take_the_general_route(gpu_ctx, n, ne, what):
    """One element moved by 1e-6 of the largest (the second state's, where the array has states): both states
    must follow the reference's loop for exactly these inputs.  The element is one that the loop reads."""
    p, atwo, aj = _inputs(n, ne, 2, 80 + n)
    atwo, ro4, daaa, taa, dal = (np.array(x, order="F") for x in (atwo, p.ro4, p.daaa, p.taa, p.dal))
    if what == "atwo_ij":
        atwo[1, 0, 2, 3] += 1e-6 * abs(atwo).max()
    elif what == "atwo_exchange":  # (ij|kl) = (ji|kl) = (ij|lk) kept
        for i, j, k, l in ((1, 0, 3, 2), (0, 1, 3, 2), (1, 0, 2, 3), (0, 1, 2, 3)):
            atwo[i, j, k, l] += 1e-6 * abs(atwo).max()
    elif what in ("ro4", "nan"):   # the key (2,2,1,0): its first two annihilators no longer exchange
        x = ro4[10, 0, 1, 2, 0, 1]
        ro4[10, 0, 1, 2, 0, 1] = np.nan if what == "nan" else x + 1e-6 * abs(ro4).max()
    elif what == "daaa":
        daaa[1, 0, 1, 2, 3, 2, 1] += 1e-6 * abs(daaa).max()
    elif what == "taa":
        taa[1, 0, 1, 2, 3] += 1e-6 * abs(taa).max()
    else:
        dal[1, 0, 1] += 1e-6 * abs(dal).max()
    p.ro4, p.daaa, p.taa, p.dal = ro4, daaa, taa, dal
    for got, ref in zip(_gpu(p, atwo, aj), _oracle(p, atwo, aj)):
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        for s in range(2):
            keep = np.isfinite(ref[s])
            if keep.any():
                assert abs(got[s][keep] - ref[s][keep]).max() < 1e-10 * abs(ref[s][keep]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6, 10, 11, 12])
def test_split_route_matches_fp64(gpu_ctx, n):
    """Both sides of the size from which split mode takes the digit products, the second state without the
    symmetry of its 4-RDM.  Digit products keep 2^-59 of the row and column maxima: 1e-12 of the largest element."""
    from nevpt2_gb300 import koopro
    p, atwo, aj = _inputs(n, 6, 2, 90 + n, ndet=200)
    p.ro4[10, 0, 1, 2, 0, 1] += 1e-3 * abs(p.ro4).max()
    ref = _gpu(p, atwo, aj)
    with koopro.precision(koopro.SPLIT):
        got = _gpu(p, atwo, aj)
    for g, r in zip(got, ref):
        for s in range(2):
            assert rel_err(g[s], r[s]) < 1e-12
