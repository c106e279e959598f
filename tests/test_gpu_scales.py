"""Mixed mode on matrices scaled by powers of two far from 1 (the exponent and
split arithmetic of the lane grids). The method equilibrates columns first, by
powers of two: column scales whose exponents sum to zero leave it the same matrix
and the same log|det|, so every accepted matrix keeps its bits. Other scales move
log|det| by a known multiple of log 2, and each side is within the mode's bound of
1e-10 max(1, |log|det||)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LN2 = 0.6931471805599453


def results(out):
    return {k: getattr(out, k).cpu().numpy() for k in ("logabs", "phase", "parity", "status")}


def zero_sum(rng, n):
    e = rng.integers(-400, 401, n)
    e[0] -= e.sum()
    while abs(e[0]) > 800:  # spread the remainder
        i = rng.integers(1, n)
        step = int(np.sign(e[0])) * int(min(abs(e[0]), 100))
        e[0] -= step
        e[i] += step
    return e


@pytest.mark.parametrize("n", [1, 3, 6, 8, 9, 12, 13, 16, 19, 24, 25, 32])
@pytest.mark.parametrize("batch", [40, 6000])
def test_power_of_two_scales(cuda, lufqhe_mod, n, batch):
    rng = np.random.default_rng(n)
    A = lufqhe_mod.gen_gaussian(batch, n, seed=n).cpu().numpy()

    def run(e):
        B = np.ldexp(A.real, e) + 1j * np.ldexp(A.imag, e)
        return results(lufqhe_mod.batch_lup_det(cuda.from_numpy(B).cuda(),
                                                mode=lufqhe_mod.MODE_MIXED))

    want = run(np.zeros((1, n), int))
    same = run(zero_sum(rng, n)[None, :])
    assert (same["status"] == want["status"]).all() and (want["status"] == 0).mean() > 0.9
    ok = want["status"] == 0
    for k in ("logabs", "phase", "parity"):
        assert np.array_equal(same[k][ok], want[k][ok]), k
    for e, total in ((np.full((1, n), -900), -900 * n), (np.full((1, n), 900), 900 * n),
                     (zero_sum(rng, n)[:, None], 0)):
        got = run(e)
        # (a matrix left to the FP64 route is refused there if a row lies below 1e-24,
        # as the reference refuses it: SCALE_TINY beside FALLBACK)
        tiny = got["status"] == 8 + 1
        assert np.isin(got["status"], (0, 8, 8 + 1)).all() and tiny.mean() < 0.1
        la = want["logabs"] + total * LN2
        scale = np.maximum(1.0, np.abs(la)) + np.maximum(1.0, np.abs(want["logabs"]))
        assert (np.abs(got["logabs"] - la) / scale)[~tiny].max() < 1e-10
        d = np.abs(np.angle(np.exp(1j * (got["phase"] - want["phase"]))))
        assert (d / scale)[~tiny].max() < 1e-10
