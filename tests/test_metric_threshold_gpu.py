"""A threshold below the line that calls a metric eigenvalue null (1e-12 of the largest
diagonal element): an eigenvalue between the two is kept, as the reference keeps it.
One null vector of a singlet's (-1') metric is lifted to 5e-13 of that element and the
threshold put at a tenth of it; the other null eigenvalues are rounding, 1e-15.  The
count nnew is compared, an integer; the energies of such a metric are not defined to
rounding."""
import numpy as np
import pytest

from nevpt2_gb300 import qdnevpt as gq
from oracle import qdnevpt_oracle as q
from test_singlet_pencil import _problem

es = np.einsum


def _lifted(n, nele, seed):
    p, o = _problem(n, nele, 1, seed)
    d, D1, D2, D3 = np.eye(n), p.dal[0], p.taa[0], p.daaa[0]
    eee = D3.transpose(0, 3, 1, 4, 2, 5) + es("ed,acbf->abcdef", d, D2) + es("eb,acfd->abcdef", d, D2)
    eee = eee + es("bc,aedf->abcdef", d, D2) + es("bc,ed,af->abcdef", d, d, D1)
    S = eee.transpose(1, 2, 0, 4, 3, 5).reshape(n**3, n**3)  # [ap, bp, cp, a, b, c] of eee(cp, ap, bp, b, a, c)
    w, v = np.linalg.eigh(0.5 * (S + S.T))
    big = S.diagonal().max()
    assert (abs(w) < 1e-14 * big).sum() == n
    v = v[:, 0].reshape((n,) * 3)
    # + lift v v^T on S through the 3-RDM in it, which the energy stage reads as Gamma3(a2,a4,a6,a1,a3,a5)
    eee = 5e-13 * big * es("pqr,abc->rpqbac", v, v)
    o["3-RDM"] = p.daaa = np.asfortranarray(p.daaa + eee.transpose(1, 3, 5, 0, 2, 4)[None])
    return p, o, 5e-14 * big


@pytest.mark.gpu
@pytest.mark.parametrize("n,nele", [(5, 4), (6, 6), (8, 8)])
def test_eigenvalue_above_a_low_threshold_is_kept(gpu_ctx, n, nele):
    p, o, thr = _lifted(n, nele, 20 + n)
    ref = q.qdnevpt(q.inputs_from(p, o, thr_lindep=thr), classes=[6])
    got = gq.qdnevpt(p, o, thr_lindep=thr, class_mask=0x40)
    assert got.nnew[7, 0] == ref.nnew[(6, 0)] == n**3 - n + 1
    # the same metric under a threshold above the line drops all of them
    assert gq.qdnevpt(p, o, thr_lindep=1e-6, class_mask=0x40).nnew[7, 0] == n**3 - n
