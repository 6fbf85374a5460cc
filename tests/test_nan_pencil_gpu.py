"""A Koopmans matrix with a NaN of the bits that the exchanges of the pencil reductions
use for "not arrived" (all ones, as memory filled with 0xff bytes holds it): the class's
energies are NaN and the call returns, with a tridiagonal form (n = 6) and a band
(n = 9); the next call is right (1e-9, the energies' tolerance)."""
import numpy as np
import pytest

from nevpt2_gb300 import qdnevpt as gq
from nevpt2_gb300 import koopro, synth

NAN = np.uint64(2**64 - 1).view(np.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6, 9])
@pytest.mark.parametrize("key,cls,mask", [("amatIP", 6, 0x40), ("amatEA", 5, 0x20)])
def test_nan_with_all_bits_set(gpu_ctx, n, key, cls, mask):
    p = synth.make_problem(n, 6, 3, 5, metat=1, ndet=None if n == 6 else 2000, seed=60 + n)
    koop = koopro.koopro4QD(p)
    ref = gq.qdnevpt(p, koop, class_mask=mask)
    bad = dict(koop)
    bad[key] = np.array(koop[key], order="F")
    bad[key][0, 0, 0, 0, 0, 0, 0] = NAN
    assert bad[key].view(np.uint64).flat[0] == 2**64 - 1
    got = gq.qdnevpt(p, bad, class_mask=mask)
    assert np.isnan(got.e2enp[cls, 0]) and np.isnan(got.e2mpp[cls, 0])
    assert got.nnew[cls + 1, 0] == ref.nnew[cls + 1, 0] == n**3
    again = gq.qdnevpt(p, koop, class_mask=mask)
    np.testing.assert_allclose(again.e2enp[cls], ref.e2enp[cls], rtol=1e-9, atol=1e-9)
