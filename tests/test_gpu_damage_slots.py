"""The damage update with 1, 2, 4, 16 and 32 points a warp and some, half or all
of them beyond yield (one point alone, two, and groups of up to four teams with
idle ones at the end), or the last point alone (the threads without a point have
no part in it): against the oracle, tolerances as in test_gpu_damage_teams."""
import numpy as np
import pytest

from test_gpu_damage_teams import KEYS, agree, case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nip", [33, 320])
@pytest.mark.parametrize("share", ["last", 0.05, 0.5, 1.0])
@pytest.mark.parametrize("dims", [(3, 1, 1), (12, 4, 4), (12, 6, 6), (16, 8, 8), (24, 10, 10)], ids=lambda d: "x".join(map(str, d)))
def test_shares_of_plastic_points(xt, orc, dims, share, nip):
    ne, nn, ins, st = case(xt, dims, nip, "all")
    ngp = 8 * ne
    rng = np.random.default_rng(5)
    soft = rng.random(ngp) >= share if share != "last" else np.arange(ngp) < ngp - 1
    ins[6] = np.where(soft, 1.0e5, 2.0e5)  # the soft points stay elastic
    st["ws"] = rng.uniform(31.7, 31.8, ngp)
    ref = {k: v.copy() for k, v in st.items()}
    for _ in range(2):
        xt.damage(ne, nn, nip, *ins, st)
        orc.damage(ne, nn, nip, *ins, ref)
        agree(st, ref)
    if nip > 300:
        n = np.count_nonzero(ref["p"])
        assert n == 1 if share == "last" else n >= 0.9 * np.count_nonzero(~soft)
    assert sorted(st) == sorted(KEYS)
