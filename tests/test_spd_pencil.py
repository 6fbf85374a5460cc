"""The inverse Cholesky factor of the order-n^3 metrics, thresholds around the
smallest metric eigenvalue: far below it (the trace of the inverse decides), just
below it (the trace does not, a factorisation of the shifted metric does) and above
it (eigenvalues are dropped).  Against the oracle, tolerance as for the other
resolvent tests (1e-9)."""
import numpy as np
import pytest

from nevpt2_gb300 import qdnevpt as gq
from nevpt2_gb300 import synth
from oracle import oracle as orc
from oracle import qdnevpt_oracle as q

es = np.einsum
KOOP = {"ipko1": "1-IPKO", "eako1": "1-EAKO", "hrdm2": "2-HRDM", "ipko2": "2-IPKO", "eako2": "2-EAKO"}


def _smallest(p):
    n, d = p.nact, np.eye(p.nact)
    D1, D2, D3 = p.dal[0], p.taa[0], p.daaa[0]
    ee = D2.transpose(0, 2, 1, 3) + es("bc,ad->abcd", d, D1)
    eee = D3.transpose(0, 3, 1, 4, 2, 5) + es("ed,acbf->abcdef", d, D2) + es("eb,acfd->abcdef", d, D2)
    eee = eee + es("bc,aedf->abcdef", d, D2) + es("bc,ed,af->abcdef", d, d, D1)
    hole = 2 * es("cd,abef->abcdef", d, ee) - eee.transpose(0, 1, 3, 2, 4, 5)
    return [np.linalg.eigvalsh(w.transpose(1, 2, 0, 4, 3, 5).reshape(n**3, n**3))[0] for w in (eee, hole)]


@pytest.mark.gpu
@pytest.mark.parametrize("factor", [1 / 400, 0.9, 1.05])
def test_thresholds_around_the_smallest_eigenvalue(gpu_ctx, factor):
    p = synth.make_problem(8, 8, 3, 7, metat=1, ndet=4000, seed=180)
    o = {KOOP.get(k, k): v for k, v in orc.stage1(p).items()}
    o["1-RDM"], o["2-RDM"], o["3-RDM"] = p.dal, p.taa, p.daaa
    thr = factor * min(_smallest(p))
    inp = q.inputs_from(p, o)
    inp.thr_lindep = thr
    ref = q.qdnevpt(inp, classes=[5, 6])
    got = gq.qdnevpt(p, o, thr_lindep=thr, class_mask=0x60)
    for slot, cls in ((6, 5), (7, 6)):
        assert got.nnew[slot, 0] == ref.nnew[(cls, 0)]
        assert (got.nnew[slot, 0] == 512) == (factor < 1)
        np.testing.assert_allclose(got.e2enp[cls], ref.e2enp[cls], rtol=1e-9, atol=1e-9)
        np.testing.assert_allclose(got.psienep[cls], ref.psienep[cls], rtol=1e-9, atol=1e-9)
