"""The lane-grid FP32 path (several matrices per warp for n <= 16, padded sizes
up to 31): remainders of a warp's matrices, every lane grid and padding, and the
matrices it rejects.

A matrix's result may not depend on its neighbours or on the grid that its batch
size picks, so a batch that ends in a part-filled warp equals its matrices one
call each (a warp each) bit for bit; every finite result is within the mixed
mode's 1e-10 bound of the double-double oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("logabs", "phase", "parity", "status")


def results(out):
    return {k: getattr(out, k).cpu().numpy() for k in FIELDS}


def special(n, rng):
    """Zero entries, extreme scales, a rejected pivot, NaN and Inf."""
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    nan, inf, sing = a.copy(), a.copy(), a.copy()
    nan[0, n - 1] = np.nan
    inf[n - 1, 0] = np.inf
    sing[:, n // 2] = 0.0
    mats = [np.eye(n), a * 1e-280, a * 1e280, np.triu(a), nan, inf, sing,
            a * np.exp2(rng.integers(-60, 60, (n, n)))]
    return np.stack(mats).astype(np.complex128)


@pytest.mark.parametrize("n", [1, 2, 5, 6, 7, 8, 9, 11, 12, 13, 15, 16, 17, 20, 23, 25, 31])
def test_batch_equals_single_calls(cuda, lufqhe_mod, oracle, n):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(n)
    batch = 4 * sms + 3  # past the one-warp-per-matrix limit, not a whole warp's share
    A, _ = lufqhe_mod.gen_lll(batch, n, seed=40 + n)
    A[::3] = lufqhe_mod.gen_gaussian(batch, n, seed=80 + n)[::3]
    sp = special(n, rng)
    A[5:5 + len(sp)] = cuda.from_numpy(sp).cuda()
    got = results(lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED))
    picked = list(range(40)) + list(range(batch - 20, batch))
    for b in picked:
        one = results(lufqhe_mod.batch_lup_det(A[b:b + 1], mode=lufqhe_mod.MODE_MIXED))
        for k in FIELDS:
            assert np.array_equal(one[k], got[k][b:b + 1], equal_nan=True), (b, k)
    bad = got["status"][5 + 4:5 + 6]
    assert (bad == 4).all()  # LUFQHE_ST_NONFINITE
    ok = np.isfinite(got["logabs"])
    ok[5:5 + len(sp)] = False  # extreme scales: not the oracle's range
    la, ph, _ = oracle.logdet_dd(A.cpu().numpy()[ok])
    scale = np.maximum(1.0, np.abs(la))
    assert (np.abs(got["logabs"][ok] - la) / scale).max() < 1e-10
    d = np.abs(np.angle(np.exp(1j * (got["phase"][ok] - ph)))) / scale
    assert d.max() < 1e-10


def test_plan_small_groups_equal_batched_calls(cuda, lufqhe_mod):
    """A mixed plan's small pass: every n <= 16, group counts around a warp's
    share and an item, padded rows, matrices left to refinement and FP64 and not
    finite ones: the batched calls' bits."""
    groups, want, off = [], [], 0
    for n in range(1, 17):
        rng = np.random.default_rng(n)
        for count, pad in ((1, 0), (3, 1), (9, 0), (203, 0)):
            L, _ = lufqhe_mod.gen_lll(count, n, seed=n + count)
            A = cuda.zeros(count, n, n + pad, dtype=cuda.complex128, device="cuda")
            A[:, :, :n] = L
            if count == 9:
                A[:8] = cuda.from_numpy(special(n, rng)).cuda()
            groups.append((A, off))
            off += count
            want.append(results(lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED)))
    out = lufqhe_mod.DetResult(*(cuda.zeros(off, dtype=d, device="cuda")
                                 for d in (cuda.float64, cuda.float64, cuda.int8, cuda.int32)))
    plan = lufqhe_mod.Plan(groups, out, autotune=False)
    for _ in range(2):
        plan.execute()
    got = results(out)
    for k in FIELDS:
        assert np.array_equal(got[k], np.concatenate([w[k] for w in want]), equal_nan=True), k
    plan.close()
