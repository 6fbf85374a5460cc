"""The order-n^3 pencils on both sides of the change of form against the oracle's
eigenvector sequence: 512, the largest order in tridiagonal form, and 729 = 22 * 32 +
25 in band form (half bandwidth 32), whose last panel is ragged.
Energies, norms, cross terms of several states, and the densities, whose
solutions are mapped back through the reflectors.  Tolerances as for the other
resolvent tests: 1e-9 relative, 1e-10 (densities) and 1e-9 (energies) absolute."""
import numpy as np
import pytest

from nevpt2_gb300 import qdnevpt as gq
from nevpt2_gb300 import synth
from oracle import oracle as orc
from oracle import qdnevpt_oracle as q

KOOP = {"ipko1": "1-IPKO", "eako1": "1-EAKO", "hrdm2": "2-HRDM", "ipko2": "2-IPKO", "eako2": "2-EAKO"}


@pytest.mark.gpu
@pytest.mark.parametrize("n,nele,metat", [(8, 8, 3), (9, 8, 1), (9, 9, 2)])
def test_band_pencils_against_oracle(gpu_ctx, n, nele, metat):
    p = synth.make_problem(n, nele, 3, 7, metat=metat, ndet=4000, seed=170 + n + metat, with_trdm=metat > 1,
                           with_ro4=True)
    o = {KOOP.get(k, k): v for k, v in orc.stage1(p).items()}
    o["1-RDM"], o["2-RDM"], o["3-RDM"] = p.dal, p.taa, p.daaa
    tr = p.trdm if metat > 1 else None
    ref = q.qdnevpt(q.inputs_from(p, o, transition=None if tr is None else tuple(list(t) for t in tr)), classes=[5, 6])
    got = gq.qdnevpt(p, o, transition=tr, class_mask=0x60, rho1st=True)
    for s in range(metat):
        for slot, key in ((6, (5, s)), (7, (6, s))):
            assert got.nnew[slot, s] == ref.nnew[key] == n**3
    for cls in (5, 6):
        np.testing.assert_allclose(got.e2enp[cls], ref.e2enp[cls], rtol=1e-9, atol=1e-9)
        np.testing.assert_allclose(got.psienep[cls], ref.psienep[cls], rtol=1e-9, atol=1e-9)
    np.testing.assert_allclose(got.e2en, ref.e2en, rtol=1e-9, atol=1e-9)
    for block in ("rhoid", "rhodr"):
        np.testing.assert_allclose(np.abs(getattr(got, block)), np.abs(getattr(ref, block)), rtol=1e-9, atol=1e-10)
