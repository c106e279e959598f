"""A mixed plan's small pass with every largest size: each n = 1..16 as the only
group and beside smaller or larger ones, tuned and not, against the batched
calls bit for bit (a tuned plan may send a size to FP64: status FP64 says so)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("logabs", "phase", "parity", "status")
SETS = [(n,) for n in range(1, 17)] + [(9, 12), (7, 11), (10, 24), (9, 16), (10, 13), (3, 9),
                                       (11, 12, 48), tuple(range(1, 13))]


def results(out):
    return {k: getattr(out, k).cpu().numpy() for k in FIELDS}


@pytest.fixture
def share(lufqhe_mod):
    lib = lufqhe_mod.lib()
    old = lib.lufqhe_get_option(3)
    yield lambda v: lib.lufqhe_set_option(3, v)
    lib.lufqhe_set_option(3, old)


@pytest.mark.parametrize("sizes", SETS, ids=lambda s: "_".join(map(str, s)))
@pytest.mark.parametrize("autotune", [False, True])
def test_small_pass_of_every_size(cuda, lufqhe_mod, share, sizes, autotune):
    groups, off = [], 0
    for n in sizes:
        count = 301
        A, _ = lufqhe_mod.gen_lll(count, n, seed=60 + n)
        A[::3] = lufqhe_mod.gen_gaussian(count, n, seed=n)[::3]
        if n <= 16:
            A[7, 0, n - 1] = float("nan")
        groups.append((A, off))
        off += count
    out = lufqhe_mod.DetResult(*(cuda.zeros(off, dtype=d, device="cuda") for d in
                                 (cuda.float64, cuda.float64, cuda.int8, cuda.int32)))
    plan = lufqhe_mod.Plan(groups, out, mode=lufqhe_mod.MODE_MIXED, autotune=autotune)
    for _ in range(2):
        plan.execute()
    got = results(out)
    plan.close()
    for A, o in groups:
        share(-1.0)
        ref = results(lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED))
        share(1.0)
        fp64 = results(lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED))
        mine = {k: got[k][o:o + A.shape[0]] for k in FIELDS}
        routed = (mine["status"] & lufqhe_mod.ST_FP64) != 0
        assert autotune or A.shape[1] > 32 or not routed.any()
        for k in FIELDS:
            want = np.where(routed, fp64[k], ref[k])
            assert np.array_equal(mine[k], want, equal_nan=True), (A.shape[1], k)
