"""Unfolding of label/value lists with more than 16 entries an element, whose claims
look before they write: the last entry of the list wins, as in the sequential loop.
Below and above the rule, both RDMs, straight and transposed.  Bitwise."""
import numpy as np
import pytest

from nevpt2_gb300 import koopro
from oracle import oracle as orc


@pytest.mark.gpu
@pytest.mark.parametrize("n,ne", [(1, 16), (1, 17), (2, 1024), (2, 1040), (3, 11664), (3, 40000)])
def test_last_entry_wins(gpu_ctx, n, ne):
    rng = np.random.default_rng(ne)
    val = rng.standard_normal(ne)
    lab = rng.integers(0, n, (ne, 6)).astype(np.int32)
    for trans in (False, True):
        ref = np.full(n**6, -7.0)
        orc.permute_3rdm(ref, 1, n, lab, val, trans)
        got = koopro.permute_3rdm(np.full((n,) * 6, -7.0, order="F"), lab, val, trans)
        assert np.array_equal(got.reshape(-1, order="F"), ref)
    lab = rng.integers(0, n, (3 * ne, 8)).astype(np.int32)
    val = rng.standard_normal(3 * ne)
    shape = (n * (n + 1) * (n + 2) * (n + 3) // 24,) + (n,) * 4
    ref, _ = orc.permute_4rdm(np.full(shape, -7.0, order="F"), lab, val)
    got = koopro.permute_4rdm(np.full(shape, -7.0, order="F"), lab, val)
    assert np.array_equal(got, ref)
