"""The label/value unfolding's claim keys: lists of 2^26 entries and more (64-bit
keys; all but a few entries below the threshold, so that the oracle reads the kept
ones alone) and labels off the 16-byte boundary.  Bitwise."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc

TOO_LONG = 1 << 26


@pytest.mark.gpu
@pytest.mark.parametrize("k,ne", [(4, TOO_LONG - 1), (4, TOO_LONG), (3, TOO_LONG + 777), (4, 3001), (3, 3001)])
@pytest.mark.parametrize("shift", [0, 1])
def test_unfold_matches_the_sequential_order(gpu_ctx, k, ne, shift):
    import torch
    from nevpt2_gb300.koopro import context
    n = 5
    rng = np.random.default_rng(ne + k)
    at = np.unique(np.concatenate([rng.integers(0, ne, 3000), [0, ne - 1]]))
    lab = rng.integers(0, n, (at.size, 2 * k)).astype(np.int32)
    eq = rng.random(lab.shape) < 0.3
    lab[eq] = lab[np.nonzero(eq)[0], 0]
    val = rng.standard_normal(at.size)
    labels = torch.zeros(ne * 2 * k + shift, dtype=torch.int32, device="cuda")[shift:]
    values = torch.zeros(ne, dtype=torch.float64, device="cuda")
    where = torch.from_numpy(at).cuda()
    labels.view(ne, 2 * k)[where] = torch.from_numpy(lab).cuda()
    values[where] = torch.from_numpy(val).cuda()
    if k == 4:
        shape = (n * (n + 1) * (n + 2) * (n + 3) // 24,) + (n,) * 4
        ref, _ = orc.permute_4rdm(np.full(shape, -7.0, order="F"), lab, val)
        ref = ref.reshape(-1, order="F")
    else:
        ref = np.full(n**6, -7.0)
        orc.permute_3rdm(ref, 1, n, lab, val)
    out = torch.full((ref.size,), -7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    if k == 4:
        context().call("nvpt_permute_4rdm_d", ptr(out), n, ptr(labels), ptr(values), ne, None)
    else:
        context().call("nvpt_permute_3rdm_d", ptr(out), 1, n, ptr(labels), ptr(values), ne, 0, None)
    assert np.array_equal(out.cpu().numpy(), ref)
