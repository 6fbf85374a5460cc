"""The order-n^3 pencils of the (+-1') classes with the singular metrics of a spin
eigenfunction: the exact null vectors are deflated and the pencil keeps its
resolvent form (nnew = n^3 - null vectors), against the oracle's pseudo-inverse
and eigenvector sequence.  The state is a mixture of closed-shell determinants in
random orbitals (a singlet), whose spin-free RDMs are signed sums over
permutations of 1-RDM products; the Koopmans matrices are symmetric with a
positive pencil, so that the energies are defined to rounding (1e-9 Eh, the
energies' tolerance)."""
import itertools

import numpy as np
import pytest

from nevpt2_gb300 import qdnevpt as gq
from nevpt2_gb300 import synth
from oracle import qdnevpt_oracle as q

es = np.einsum


def _rdms(n, nele, rng):
    out = [np.zeros((n,) * 2), np.zeros((n,) * 4), np.zeros((n,) * 6)]
    for _ in range(2 * n):
        C = np.linalg.qr(rng.standard_normal((n, nele // 2)))[0]
        g = 2.0 * C @ C.T
        for k in (1, 2, 3):
            for p in itertools.permutations(range(k)):
                seen, cyc = set(), 0
                for i in range(k):
                    if i not in seen:
                        cyc += 1
                    while i not in seen:
                        seen.add(i)
                        i = p[i]
                t = ",".join("abc"[i] + "def"[p[i]] for i in range(k))
                out[k - 1] += (-0.5) ** (k - cyc) / (2 * n) * es(f"{t}->{'abc'[:k]}{'def'[:k]}", *[g] * k)
    return out


def _problem(n, nele, metat, seed):
    p = synth.make_problem(n, nele, 4, 9, metat=1, ndet=20, seed=seed, with_ro4=False)
    rng = np.random.default_rng(seed)
    d = np.eye(n)
    p.metat, p.energies = metat, np.zeros(metat)
    states, koop = [], []
    for _ in range(metat):
        D1, D2, D3 = _rdms(n, nele, rng)
        ee = D2.transpose(0, 2, 1, 3) + es("bc,ad->abcd", d, D1)
        eee = D3.transpose(0, 3, 1, 4, 2, 5) + es("ed,acbf->abcdef", d, D2) + es("eb,acfd->abcdef", d, D2)
        eee = eee + es("bc,aedf->abcdef", d, D2) + es("bc,ed,af->abcdef", d, d, D1)
        o = {}
        for tag, w3, w2 in (("IP", eee, ee), ("EA", 2 * es("cd,abef->abcdef", d, ee) - eee.transpose(0, 1, 3, 2, 4, 5),
                                              2 * es("cd,ab->abcd", d, D1) - ee.transpose(0, 1, 3, 2))):
            e = np.sqrt(es("a,b,c->abc", *(rng.uniform(0.5, 1.2, n) for _ in range(3))))
            o["amat" + tag] = es("abc,abcdef,def->abcdef", e, w3.transpose(1, 2, 0, 4, 3, 5), e)
            o["bmat" + tag] = es("abc,abcd->abcd", e, w2.transpose(1, 2, 0, 3))
            o["cmat" + tag] = o["bmat" + tag].transpose(3, 0, 1, 2)
            o["dmat" + tag] = D1 if tag == "IP" else 2 * d - D1
        states.append((D1, D2, D3))
        koop.append(o)
    st = lambda xs: np.asfortranarray(np.stack(xs))
    p.dal, p.taa, p.daaa = (st([s[k] for s in states]) for k in range(3))
    z4, z2 = np.zeros((metat,) + (n,) * 4), np.zeros((metat, n, n))
    o = {k: st([x[k] for x in koop]) for k in koop[0]}
    o.update({"1-RDM": p.dal, "2-RDM": p.taa, "3-RDM": p.daaa, "2-HRDM": z4, "2-IPKO": z4, "2-EAKO": z4, "gk0pa": z4,
              "gk0pd": z4, "1-IPKO": z2, "1-EAKO": z2, "gk0pf": z2})
    pairs = metat * (metat - 1) // 2
    p.trdm = tuple(np.asfortranarray(0.05 * rng.standard_normal((pairs,) + (n,) * (2 * k))) for k in (1, 2, 3)) \
        if pairs else None
    return p, o


@pytest.mark.gpu
@pytest.mark.parametrize("n,nele,metat", [(8, 8, 1), (8, 6, 2), (9, 8, 1), (8, 8, 3)])
def test_null_vectors_are_deflated(gpu_ctx, n, nele, metat):
    p, o = _problem(n, nele, metat, 5 + n + metat)
    got = gq.qdnevpt(p, o, transition=p.trdm, class_mask=0x60)
    ref = q.qdnevpt(q.inputs_from(p, o, transition=None if p.trdm is None else tuple(list(t) for t in p.trdm)),
                    classes=[5, 6])
    for s in range(metat):
        for slot, cls in ((6, 5), (7, 6)):
            assert got.nnew[slot, s] == ref.nnew[(cls, s)] == n**3 - n
    for cls in (5, 6):
        np.testing.assert_allclose(got.e2enp[cls], ref.e2enp[cls], rtol=1e-9, atol=1e-9)
        np.testing.assert_allclose(got.psienep[cls], ref.psienep[cls], rtol=1e-9, atol=1e-9)
    np.testing.assert_allclose(got.e2en, ref.e2en, rtol=1e-9, atol=1e-9)
