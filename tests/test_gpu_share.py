"""The routed share (LUFQHE_OPT_FP64_SHARE) between 0 and 1: every form that takes
it (a warp per matrix, several per warp with a list, the passes of n = 17..32, a
plan) gives a routed matrix the FP64 route's bits and the others those of a call
without a share, and a routed matrix that is not finite is reported so. What the
hash routes does not depend on the call, so the shares are nested."""
import numpy as np
import pytest

import launches

pytestmark = pytest.mark.gpu

FIELDS = ("logabs", "phase", "parity", "status")


def results(out):
    return {k: getattr(out, k).cpu().numpy() for k in FIELDS}


@pytest.fixture
def share(lufqhe_mod):
    lib = lufqhe_mod.lib()
    old = lib.lufqhe_get_option(3)
    yield lambda v: lib.lufqhe_set_option(3, v)
    lib.lufqhe_set_option(3, old)


def matrices(lufqhe, n, batch):
    A, _ = lufqhe.gen_lll(batch, n, seed=20 + n)
    A[::2] = lufqhe.gen_gaussian(batch, n, seed=n)[::2]
    A[3::40, n - 1, n // 2] = float("nan")
    A[5::40] = 0.0
    return A


def expected(lufqhe, share, A, s):
    """By the status of a call at share s: FP64 or not; not finite as it is."""
    share(0.0)
    ref = results(lufqhe.batch_lup_det(A, mode=lufqhe.MODE_MIXED))
    share(1.0)
    fp64 = results(lufqhe.batch_lup_det(A, mode=lufqhe.MODE_MIXED))
    share(s)
    return ref, fp64


def check(got, ref, fp64, s, name):
    routed = (got["status"] & 16) != 0
    bad = (ref["status"] & 4) != 0
    assert not routed[bad].any() and (got["status"][bad] == 4).all(), name
    assert abs(routed[~bad].mean() - s) < 5 * np.sqrt(s * (1 - s) / (~bad).sum()) + 0.01, name
    for k in FIELDS:
        want = np.where(routed, fp64[k], ref[k])
        assert np.array_equal(got[k], want, equal_nan=True), (name, k)


@pytest.mark.parametrize("n", [1, 5, 6, 8, 9, 12, 15, 16, 17, 23, 24, 31, 32])
@pytest.mark.parametrize("s", [0.1, 0.5, 0.9])
def test_batched_share(cuda, lufqhe_mod, share, n, s):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    A = matrices(lufqhe_mod, n, 32 * sms + 5)
    ref, fp64 = expected(lufqhe_mod, share, A, s)
    for batch in (7, 1001, 32 * sms, 32 * sms + 5):
        got = results(lufqhe_mod.batch_lup_det(A[:batch], mode=lufqhe_mod.MODE_MIXED))
        cut = [{k: v[:batch] for k, v in r.items()} for r in (ref, fp64)]
        if batch > 1000:
            check(got, *cut, s, (n, batch))
        else:
            whole = np.where((got["status"] & 16) != 0, cut[1]["logabs"], cut[0]["logabs"])
            assert np.array_equal(got["logabs"], whole, equal_nan=True)


@pytest.mark.parametrize("n", [2, 6, 11, 12, 16, 24])
def test_plan_share(cuda, lufqhe_mod, share, n):
    A = matrices(lufqhe_mod, n, 1501)
    ref, fp64 = expected(lufqhe_mod, share, A, 0.5)
    out = lufqhe_mod.DetResult(*(cuda.zeros(1501, dtype=d, device="cuda") for d in
                                 (cuda.float64, cuda.float64, cuda.int8, cuda.int32)))
    plan = lufqhe_mod.Plan([(A, 0)], out, mode=lufqhe_mod.MODE_MIXED, autotune=False)
    plan.execute()
    check(results(out), ref, fp64, 0.5, n)
    plan.close()


@pytest.mark.parametrize("n", [5, 6, 8, 11, 12, 16])
def test_routed_matrices_skip_the_fp32_path(cuda, lufqhe_mod, share, n):
    """At n <= 16 a routed matrix does not wait for its neighbours' FP32 path: up to
    32 matrices per SM a warp takes one matrix at a time, above that the routed
    ones are listed for a kernel of their own."""
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    share(0.5)
    for batch in (1001, 32 * sms, 32 * sms + 1):
        A = lufqhe_mod.gen_gaussian(batch, n, seed=n)
        out = lufqhe_mod.batch_lup_det(A, mode=lufqhe_mod.MODE_MIXED)
        kernels, allocs = launches.captured(cuda, lambda s: lufqhe_mod.batch_lup_det(
            A, mode=lufqhe_mod.MODE_MIXED, stream=s, out=out))
        names = [k[0] for k in kernels]
        if batch <= 32 * sms:
            assert len(kernels) == 1 and allocs == 0, names
            assert 2 * kernels[0][1] * kernels[0][2] // 32 >= batch  # one each, two at most
            assert kernels[0][1] * kernels[0][2] // 32 >= min(batch, 8 * sms)
        else:
            assert len(kernels) == 2 and "lup_mixed_routed_kernel" in names[1], names
