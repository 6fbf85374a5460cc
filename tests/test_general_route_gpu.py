"""bamat on inputs without a symmetry: one thread group per element (n <= 5) and slabs
with their products (n > 5; a launch per pair of column counts, 6 to 16), every state
flagged.  Small sizes against the oracle.  Large ones against the symmetric route: one
integral moved by 2^-43 of the largest (ii|ii), four times the symmetry tolerance, which
moves the matrices by less than 1e-11.  Bounds: 1e-10 of the largest element, that of
every Koopmans matrix; split mode 1e-12 of FP64 on the same route (digits keep 2^-59 of
the row and column maxima)."""
import numpy as np
import pytest

from conftest import rel_err
from test_bamat_sym import _gpu, _inputs, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ne,metat", [(1, 2, 2), (2, 2, 1), (3, 4, 3), (4, 4, 1), (5, 4, 2), (6, 6, 1), (7, 6, 2),
                                        (8, 6, 1), (9, 6, 1)])
def test_every_state_flagged_against_the_oracle(gpu_ctx, n, ne, metat):
    p, atwo, aj = _inputs(n, ne, metat, 130 + n, ndet=200 if n > 6 else None)
    rng = np.random.default_rng(n)
    # (ij|kl) = (kl|ij) gone (n = 1 has one integral: its states stay symmetric)
    atwo = np.asfortranarray(atwo + 1e-3 * abs(atwo).max() * rng.standard_normal(atwo.shape))
    for got, ref in zip(_gpu(p, atwo, aj), _oracle(p, atwo, aj)):
        assert rel_err(got, ref) < 1e-10


@pytest.mark.parametrize("n", [10, 11, 12, 13, 14, 15, 16])
def test_slabs_agree_with_the_symmetric_route(gpu_ctx, n):
    p, atwo, aj = _inputs(n, 6, 1, 150 + n, ndet=40)
    ref = _gpu(p, atwo, aj)
    moved = np.array(atwo, order="F")
    moved[1, 0, 2, 3] += 2.0**-43 * max(moved[i, i, i, i] for i in range(n))
    for g, r in zip(_gpu(p, moved, aj), ref):
        assert rel_err(g, r) < 1e-10


@pytest.mark.parametrize("n", [6, 8, 13, 16])
def test_split_slabs(gpu_ctx, n):
    from nevpt2_gb300 import koopro
    p, atwo, aj = _inputs(n, 6, 1, 170 + n, ndet=40)
    atwo = np.array(atwo, order="F")
    atwo[1, 0, 2, 3] += 1e-3 * abs(atwo).max()
    ref = _gpu(p, atwo, aj)
    with koopro.precision(koopro.SPLIT):
        got = _gpu(p, atwo, aj)
    for g, r in zip(got, ref):
        assert rel_err(g, r) < 1e-12
