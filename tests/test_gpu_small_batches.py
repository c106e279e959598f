"""Small batches of 17 <= n <= 23 without a register tile: one kernel and no device
memory, as at n <= 16, and the bits of a batch that lists its rejected matrices."""
import numpy as np
import pytest

import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 18, 20, 22, 23])
def test_small_batch_in_one_launch(cuda, lufqhe_mod, n):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    A, z = lufqhe_mod.gen_lll(8 * sms + 1, n, seed=n)
    A[5, 0, 1] = float("nan")
    A[9] = 0.0
    A[13, :, n // 2] = 0.0
    large = lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED)
    assert (large.status == lufqhe_mod.ST_FALLBACK).any()
    for batch in (1, 4, 64, 1000, 8 * sms):
        out = lufqhe_mod.batch_lup_det(A[:batch], mode=lufqhe_mod.MODE_MIXED)
        kernels, allocs = launches.captured(cuda, lambda s: lufqhe_mod.batch_lup_det(
            A[:batch], mode=lufqhe_mod.MODE_MIXED, stream=s, out=out))
        assert len(kernels) == 1 and allocs == 0, kernels
        for k in ("logabs", "phase", "parity", "status"):
            a, b = getattr(out, k).cpu().numpy(), getattr(large, k)[:batch].cpu().numpy()
            assert np.array_equal(a, b, equal_nan=True), (batch, k)
