"""The Koopmans matrices from one n^7 contraction (csrc/koop_sym.cu).

CPU: the route's formulas in numpy against the oracle's restatement of
src/koop_matrices.F90 and src/koopro4QD.F90:4231-4397.  GPU: both routes against
the oracle at the edges of their sizes, with inputs that have their physical
symmetries and with inputs that lack one.  Tolerance 1e-10 of the largest
element, as for every Koopmans matrix."""
import numpy as np
import pytest

from conftest import rel_err
from nevpt2_gb300 import synth
from oracle import oracle as orc

es = np.einsum


def _inputs(n, ne, metat, seed, ndet=None, ncore=2):
    p = synth.make_problem(n, ne, ncore, 3, metat=metat, ndet=ndet, seed=seed, with_ro4=False)
    atwo, aj = orc.get_aj_atwo(p.oneint, p.chol, n, ncore, p.norb)
    return p, np.asarray(atwo), aj


def _oracle(p, atwo, aj):
    n, M, nc = p.nact, p.metat, p.ncore
    f = np.zeros(p.norb * (p.norb + 1) // 2)
    o = dict(orc.koop_matrices_ctl(M, n, nc, atwo, p.daaa, p.taa, p.dal, f, aj))
    o["f"] = f.copy()
    o["bmatIP"], o["bmatEA"] = orc.bbmat(atwo, p.daaa, p.taa, p.dal, n, nc, f, aj, M)
    o["cmatIP"], o["cmatEA"] = orc.bcmat(atwo, p.daaa, p.taa, p.dal, n, nc, f, aj, M)
    o["dmatIP"], o["dmatEA"] = orc.bdmat(atwo, p.taa, p.dal, n, nc, f, aj, M)
    return o


def _gpu(p, atwo, aj):
    from nevpt2_gb300 import koopro
    n, M, nc = p.nact, p.metat, p.ncore
    f = np.zeros(p.norb * (p.norb + 1) // 2)
    o = dict(koopro.koop_matrices_ctl(M, n, nc, atwo, p.daaa, p.taa, p.dal, f, aj))
    names = {"1-IPKO": "ipko1", "1-EAKO": "eako1", "2-HRDM": "hrdm2", "2-IPKO": "ipko2", "2-EAKO": "eako2"}
    o = {names.get(k, k): v for k, v in o.items()}
    o["f"] = f.copy()
    o["bmatIP"], o["bmatEA"] = koopro.bbmat(atwo, p.daaa, p.taa, p.dal, n, nc, f, aj, M)
    o["cmatIP"], o["cmatEA"] = koopro.bcmat(atwo, p.daaa, p.taa, p.dal, n, nc, f, aj, M)
    o["dmatIP"], o["dmatEA"] = koopro.bdmat(atwo, p.taa, p.dal, n, nc, f, aj, M)
    return o


@pytest.mark.parametrize("n,ne", [(3, 4), (4, 4)])
def test_one_contraction_equals_the_loops(n, ne):
    p, T, aj = _inputs(n, ne, 1, 20 + n)
    ref = {k: np.asarray(v)[0] for k, v in _oracle(p, T, aj).items()}
    D1, D2, D3 = p.dal[0], p.taa[0], p.daaa[0]
    d = np.eye(n)
    h = np.array([[aj[synth.tri(i + 3, j + 3) - 1] for j in range(n)] for i in range(n)])
    F3 = es("pdeqfc,dfea->pqca", D3, T) + es("pdqc,da->pqca", D2, h)
    J2 = es("pdqf,dfxy->pqxy", D2, T) + es("pq,xy->pqxy", D1, h)
    W2, X2 = es("pefs,xfey->psxy", D2, T), es("pdqe,dxye->pqxy", D2, T)
    Q1 = es("ptfe,xfye->ptxy", D2, T)
    Q2, G1, T1 = es("pece->pc", J2), es("ecea->ca", J2), es("pf,xyzf->pxyz", D1, T)
    Y = G1 - 2 * es("df,dfxy->xy", D1, T) + es("ef,xfey->xy", D1, T) - 2 * h
    x = "->pqca"
    F3R = 2 * (J2 + es("pq,ca" + x, d, Y) + es("cqpa" + x, T1) + es("pcaq" + x, T1) + es("qcap" + x, T1) + es("cpqa" + x, T))
    F3R = F3R - F3 - es("cp,qa" + x, d, Y) - es("pcqa" + x, J2 + W2) - es("pqac" + x, X2) - es("qcpa" + x, Q1)
    F3R = F3R - es("pqac" + x, T1) - es("qcpa" + x, T1) - es("cqap" + x, T1) - 4 * es("qpca" + x, T)
    x = "->ptxy"
    Q1R = Q1 + es("typx" + x, T1) + es("pxty" + x, T1) + 4 * es("xpyt" + x, T)
    Q1R = Q1R - 2 * (es("txpy" + x, T1) + es("pytx" + x, T1) + es("xtyp" + x, T))
    o = {}
    o["ipko2"] = -es("bqpa->pqab", F3) - es("apqb->pqab", F3) - Q1
    o["eako2"] = -es("bqpa->pqab", F3R) - es("apqb->pqab", F3R) - Q1R
    A = es("qpba->qpab", F3) - es("pqab->qpab", F3) + es("qbpa->qpab", J2 + W2) - es("qapb->qpab", Q1)
    o["gk0pa"] = 2 * (A - es("pa,qb->qpab", d, Q2))
    o["gk0pd"] = es("paqb->qpab", F3) - es("qbpa->qpab", F3 - 2 * J2) - es("qbap->qpab", X2) + es("aqpb->qpab", Q1)
    o["gk0pd"] = o["gk0pd"] - 2 * es("pa,qb->qpab", d, Q2)
    o["bmatIP"] = -es("prqa->pqra", F3) - es("rqpa->pqra", Q1) - es("pq,ra->pqra", d, Q2)
    B = 2 * es("rpaq->pqra", J2) - es("rpqa->pqra", F3) - es("rpaq->pqra", X2) - es("rqpa->pqra", W2 + J2)
    o["bmatEA"] = B - es("rapq->pqra", T1) + 2 * es("raqp->pqra", T1)
    C = es("qbca->qabc", F3) - es("bqac->qabc", F3) - es("caqb->qabc", F3) - es("qabc->qabc", Q1)
    o["cmatIP"] = C - es("ab,qc->qabc", d, Q2)
    C = es("qbac->qabc", F3) - es("bqca->qabc", F3) - es("acqb->qabc", F3) - es("bcqa->qabc", J2 + W2)
    C = C + es("baqc->qabc", Q1) - es("acbq->qabc", X2) - es("cqab->qabc", Q1) + 2 * es("acbq->qabc", J2)
    C = C + 2 * es("cbqa->qabc", T1) - es("cqab->qabc", T1) + es("qa,bc->qabc", d, Q2) - es("qa,cb->qabc", d, G1)
    o["cmatEA"] = C + 2 * es("bq,ca->qabc", d, G1) - 2 * es("bq,ac->qabc", d, Q2)
    for k, v in o.items():
        assert rel_err(v, ref[k]) < 1e-12, k


# both sides of the smallest size of the route, odd and largest-tile sizes, more states than one pass takes
SIZES = [(1, 2, 1, 2), (2, 2, 2, 0), (4, 4, 1, 3), (5, 4, 2, 1), (6, 6, 1, 2), (7, 6, 5, 2), (8, 8, 1, 0), (11, 6, 2, 2),
         (13, 4, 1, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,ne,metat,ncore", SIZES)
def test_symmetric_inputs(gpu_ctx, n, ne, metat, ncore):
    p, atwo, aj = _inputs(n, ne, metat, 30 + n, ndet=200 if n > 6 else None, ncore=ncore)
    ref, got = _oracle(p, atwo, aj), _gpu(p, atwo, aj)
    for k, v in got.items():
        assert rel_err(v, ref[k]) < 1e-10, k


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["atwo_ij", "atwo_exchange", "daaa", "taa", "dal"])
@pytest.mark.parametrize("n,ne,metat", [(6, 6, 2), (9, 4, 1)])
def test_inputs_without_a_symmetry_take_the_direct_kernels(gpu_ctx, n, ne, metat, what):
    p, atwo, aj = _inputs(n, ne, metat, 50 + n, ndet=200)
    atwo, daaa, taa, dal = (np.array(x, order="F") for x in (atwo, p.daaa, p.taa, p.dal))
    s = metat - 1
    if what == "atwo_ij":
        atwo[1, 0, 2, 3] += 1e-6 * abs(atwo).max()
    elif what == "atwo_exchange":
        for i, j, k, l in ((1, 0, 3, 2), (0, 1, 3, 2), (1, 0, 2, 3), (0, 1, 2, 3)):
            atwo[i, j, k, l] += 1e-6 * abs(atwo).max()
    elif what == "daaa":
        daaa[s, 0, 1, 2, 3, 2, 1] += 1e-6 * abs(daaa).max()
    elif what == "taa":
        taa[s, 0, 1, 2, 3] += 1e-6 * abs(taa).max()
    else:
        dal[s, 0, 1] += 1e-6 * abs(dal).max()
    p.daaa, p.taa, p.dal = daaa, taa, dal
    ref, got = _oracle(p, atwo, aj), _gpu(p, atwo, aj)
    for k, v in got.items():
        assert rel_err(v, ref[k]) < 1e-10, k
