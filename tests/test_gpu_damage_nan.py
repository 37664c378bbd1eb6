"""A NaN in the temporal shape table reaches every point, as in the oracle,
wherever it lies: at a run's first step, inside a run, in a later chunk, at the
last step, on points whose stress never comes near yield (the bounds over runs
and chunks of steps must not pass over it)."""
import numpy as np
import pytest

from test_gpu_damage_teams import KEYS, case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [0, 64, 77, 1024, 1500, 2099])
@pytest.mark.parametrize("scale", [0.1, 1.0], ids=["elastic", "plastic"])
def test_nan_reaches_the_state(xt, orc, scale, step):
    ne, nn, ins, st = case(xt, (3, 1, 1), 2100, "all")
    ins[5] = ins[5] * scale
    ins[4] = np.array(ins[4], dtype=float).copy()
    ins[4].reshape(-1, 6)[step, 4] = np.nan
    ref = {k: v.copy() for k, v in st.items()}
    xt.damage(ne, nn, 2100, *ins, st)
    orc.damage(ne, nn, 2100, *ins, ref)
    assert np.isnan(ref["p"]).all()
    for k in KEYS:
        assert np.array_equal(np.isnan(st[k]), np.isnan(ref[k])), k
        f = ~np.isnan(ref[k])
        assert np.max(np.abs(st[k][f] - ref[k][f]), initial=0.0) <= 1e-8 * max(np.max(np.abs(ref[k][f]), initial=0.0), 1e-300) + 1e-14, k
