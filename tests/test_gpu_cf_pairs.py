"""The CF builder's pair table: the written-out matrices equal the oracle's bit
for bit on both sides of the rule that picks it (at most half the batch's
terms, np <= 1024), with a repeated particle and an entry out of range."""
import numpy as np
import pytest

import cf_oracle as co

pytestmark = pytest.mark.gpu

K = (1.0, 0.5, 0.5, 1.0)


@pytest.mark.parametrize("n,np_,batch", [
    (3, 3, 2), (3, 3, 3),                # 18 terms of the table against 12 and 18 of the batch
    (11, 11, 2), (11, 11, 3),            # 242 against 220 and 330
    (5, 64, 409), (5, 64, 410),          # 8192 against 8180 and 8200
    (25, 1024, 3600), (25, 1025, 3600),  # the largest table, and one particle more
])
def test_pair_table_bits(cuda, lufqhe_mod, n, np_, batch):
    phi, theta = co.random_config(np_, 7)
    cfg = lufqhe_mod.CfConfig(phi, theta, *K, 0, 1)
    perm = co.random_perms(batch, n, np_, 8)
    perm[1, 0] = perm[1, n - 1]
    dperm = cuda.from_numpy(perm).cuda()
    got = lufqhe_mod.gen_cf(cfg, dperm, n).cpu().numpy()
    uv, tab = lufqhe_mod.cf_tables(cfg, n)
    want = co.matrices(uv, tab, perm, n, *K, 0, 1)
    assert np.array_equal(got.view(np.float64), want.view(np.float64), equal_nan=True)
    perm[0, 2] = 0
    bad = lufqhe_mod.cf_det(cfg, cuda.from_numpy(perm).cuda(), n, mode=2).status.cpu().numpy()
    assert bad[0] == bad[1] == 4 and (bad[2:] != 4).all()
