"""PC classes whose metric drops eigenvalues: the eigenpairs of the (+-1') pencils are
found on the helper stream (started at the head of the call with one state, within the
class with several), those of the others within their class.  Against the oracle, with
a threshold in a gap of every metric's spectrum, densities included.  Tolerances as for
the resolvent tests: 1e-9 relative, 1e-9 (energies) and 1e-10 (densities) absolute."""
import numpy as np
import pytest

from nevpt2_gb300 import qdnevpt as gq
from nevpt2_gb300 import synth
from oracle import oracle as orc
from oracle import qdnevpt_oracle as q

KOOP = {"ipko1": "1-IPKO", "eako1": "1-EAKO", "hrdm2": "2-HRDM", "ipko2": "2-IPKO", "eako2": "2-EAKO"}
SLOTS = {(3, "a"): 2, (3, "b"): 3, (4, "a"): 4, (4, "b"): 5, (5,): 6, (6,): 7, (7,): 8}


@pytest.mark.gpu
@pytest.mark.parametrize("n,nele,metat,thr", [(5, 5, 1, 0.1), (6, 6, 1, 0.35), (6, 6, 2, 0.15), (5, 4, 3, 1e-6)])
def test_dropped_eigenvalues_against_oracle(gpu_ctx, n, nele, metat, thr):
    p = synth.make_problem(n, nele, 4, 7, metat=metat, seed=700 + 10 * n + metat, with_trdm=metat > 1)
    o = {KOOP.get(k, k): v for k, v in orc.stage1(p).items()}
    o["1-RDM"], o["2-RDM"], o["3-RDM"] = p.dal, p.taa, p.daaa
    tr = p.trdm if metat > 1 else None
    ref = q.qdnevpt(q.inputs_from(p, o, thr_lindep=thr, transition=None if tr is None else tuple(list(t) for t in tr)))
    got = gq.qdnevpt(p, o, transition=tr, thr_lindep=thr, rho1st=True)
    for s in range(metat):
        for k, slot in SLOTS.items():
            assert got.nnew[slot, s] == ref.nnew[(k[0], s) + k[1:]], (slot, s)
        assert min(got.nnew[6, s], got.nnew[7, s]) < n**3
    np.testing.assert_allclose(got.e2enp, ref.e2enp, rtol=1e-9, atol=1e-9)
    np.testing.assert_allclose(got.e2en, ref.e2en, rtol=1e-9, atol=1e-9)
    for block in ("rhoir", "rhoid", "rhodr"):
        np.testing.assert_allclose(np.abs(getattr(got, block)), np.abs(getattr(ref, block)), rtol=1e-9, atol=1e-10)
