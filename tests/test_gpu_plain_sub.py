"""The plain FP64 kernels with several matrices per warp (n <= 32): batch sizes
that pick 32, 16, 8 and 4 lanes per matrix, with a part-filled last warp, and
matrices that leave the factorisation early beside ones that do not. Factors
must equal the CPU restatement's bit for bit, statuses and parity exactly,
log|det| and phase to 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 4, 5, 8, 9, 15, 16, 17, 24, 31, 32])
@pytest.mark.parametrize("batch", [3, 701, 1501, 5003])
@pytest.mark.parametrize("mode", [0, 1])
def test_factors_bit_exact(cuda, lufqhe_mod, oracle, n, batch, mode):
    rng = np.random.default_rng(1000 * n + batch)
    A = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))) / 2
    if batch > 3:
        A[7::50] = 0.0                                   # below the scale limit
        A[9::50, n - 1, 0] = np.nan
        A[11::50, :, n // 2] = 0.0                       # exact zero pivot (n = 1: tiny)
        A[13::50] = np.round(A[13::50].real * 2) / 2 + 0.25j  # equal quotients
    dA = cuda.from_numpy(A.copy()).cuda()
    out = lufqhe_mod.factor_inplace(dA, mode=mode)
    got = {k: getattr(out, k).cpu().numpy() for k in ("logabs", "phase", "parity", "status")}
    F = dA.cpu().numpy()
    want = oracle.lup_det(A, arith=mode, want_factors=True)
    assert (got["status"] == want["status"]).all()
    ok = want["status"] == 0
    assert (F[ok].view(np.uint64) == want["factors"][ok].view(np.uint64)).all()
    left = (want["status"] & 5) != 0                     # not written back
    assert np.array_equal(F[left], A[left], equal_nan=True)
    assert (got["parity"][ok] == want["parity"][ok]).all()
    scale = np.maximum(1.0, np.abs(want["logabs"][ok]))
    assert (np.abs(got["logabs"][ok] - want["logabs"][ok]) / scale).max() < 1e-12
    d = np.angle(np.exp(1j * (got["phase"][ok] - want["phase"][ok])))
    assert np.abs(d).max() < 1e-12


@pytest.mark.parametrize("n,batch", [(33, 1824), (33, 40), (40, 1500), (47, 9), (48, 9), (49, 9),
                                     (63, 9), (64, 9)])
@pytest.mark.parametrize("mode", [0, 1])
def test_group_and_warp_factors_bit_exact(cuda, lufqhe_mod, oracle, n, batch, mode):
    """n > 32: a warp group per matrix (4 or 6 warps), or a warp each in a batch
    that fills its rounds; one matrix with an exact zero pivot, one below the
    scale limit, one with equal quotients in every column's search."""
    rng = np.random.default_rng(n + batch)
    A = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))) / 2
    A[1, :, n // 2] = A[1, :, 0]
    A[2, 3] = 0.0
    A[3] = np.sign(A[3].real) + 1j * A[3].imag
    dA = cuda.from_numpy(A.copy()).cuda()
    out = lufqhe_mod.factor_inplace(dA, mode=mode)
    got = {k: getattr(out, k).cpu().numpy() for k in ("parity", "status")}
    want = oracle.lup_det(A, arith=mode, want_factors=True)
    assert (got["status"] == want["status"]).all()
    ok = want["status"] == 0
    F = dA.cpu().numpy()
    assert (F[ok].view(np.uint64) == want["factors"][ok].view(np.uint64)).all()
    assert (got["parity"][ok] == want["parity"][ok]).all()
