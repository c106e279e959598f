"""LUFQHE_OPT_TILE_WARPS sets the warps per CTA of every kernel of the
register-tiled sizes but the correction pass, and changes no result."""
import numpy as np
import pytest

import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 8, 12, 16, 24, 32])
@pytest.mark.parametrize("batch", [100, 2000])
def test_tile_warps(cuda, lufqhe_mod, n, batch):
    lib = lufqhe_mod.lib()
    A, _ = lufqhe_mod.gen_lll(batch, n, seed=n)
    want = lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED)
    out = lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED)
    old = lib.lufqhe_get_option(2)
    try:
        for warps in (1, 2, 0):
            assert lib.lufqhe_set_option(2, float(warps)) == 0
            kernels, _ = launches.captured(cuda, lambda s: lufqhe_mod.batch_lup_det(
                A, mode=lufqhe_mod.MODE_MIXED, stream=s, out=out))
            lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED, out=out)
            tiles = [k for k in kernels if "correct" not in k[0]]
            assert tiles and all(k[2] == 32 * (warps or (3 if n == 24 else 4)) for k in tiles), kernels
            for k in ("logabs", "phase", "parity", "status"):
                a, b = getattr(out, k).cpu().numpy(), getattr(want, k).cpu().numpy()
                assert np.array_equal(a, b, equal_nan=True), (warps, k)
    finally:
        lib.lufqhe_set_option(2, old)
