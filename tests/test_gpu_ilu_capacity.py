"""The triangular sweeps at the edges of their layouts, against the oracle's
kronlusol: rows on both sides of the step capacities (20 entries at one lane a
row, 24 and 32 at two and four; beyond, the formats of the fallback), one
factor and four row blocks, more warps than the levels need up to the most a
layout takes, and more than fit in shared memory (the plans then take fewer).
Tolerances as in test_gpu_parity: 1e-10 in FP64, 1e-4 in FP32."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem, temporal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(12, 4, 4), (6, 12, 12)], ids=lambda p: "x".join(map(str, p)))
def rod(request, xt):
    pr = rod_problem(xt, *request.param)
    xyz, _ = pr.mesh()
    pr.apply_bc(clamp_mask(xyz))
    yield dict(K=pr.K(), M=pr.M(), A=temporal(xt)[0], f={})
    pr.close()


def factor(xt, rod, lfil, blocks):
    if (lfil, blocks) not in rod["f"]:
        rod["f"][lfil, blocks] = xt.ilut(rod["K"], lfil, 1e-6, blocks=blocks)
    return rod["f"][lfil, blocks]


def check(xt, orc, rod, f, group, blocks, fp32):
    x = np.random.default_rng(7).standard_normal(rod["K"].n * 6)
    ref = orc.kronlusol(rod["A"], *f, x)
    s = xt.SpaceTimeSystem(rod["K"], rod["M"])
    s.set_ilu(*f, group=group, blocks=blocks)
    for _ in range(2):
        y = s.lusol(rod["A"], x, fp32=fp32)
        assert np.linalg.norm(y - ref) <= (1e-4 if fp32 else 1e-10) * np.linalg.norm(ref)
    s.close()


@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("group,blocks", [(3, 1), (3, 4), (1, 1)])
@pytest.mark.parametrize("lfil", [20, 21, 24, 25, 32, 33, 40])
def test_row_lengths_around_the_capacities(xt, orc, rod, lfil, group, blocks, fp32):
    check(xt, orc, rod, factor(xt, rod, lfil, blocks), group, blocks, fp32)


@pytest.mark.parametrize("shares", [1, 2, 4])
@pytest.mark.parametrize("warps", [4, 5, 6, 7, 16])
@pytest.mark.parametrize("group,fp32", [(3, False), (1, False), (3, True), (1, True)])
def test_many_warps(xt, orc, rod, monkeypatch, group, fp32, warps, shares):
    monkeypatch.setenv("XTFEM_ILU_WARPS", str(warps))
    monkeypatch.setenv("XTFEM_ILU_SHARES" if fp32 else "XTFEM_ILU_ROW_H", str(shares))
    check(xt, orc, rod, factor(xt, rod, 20, 1), group, 1, fp32)


@pytest.mark.parametrize("blocks", [1, 4])
def test_sixteen_warps_of_long_rows_keep_the_register_sweep(xt, orc, monkeypatch, capfd, blocks):
    """16 warps of 16 steps beside a window of several hundred nodes do not fit
    in four parts of the ring: fewer warps do, and each row block keeps its own
    thread block."""
    pr = rod_problem(xt, 12, 24, 24)
    xyz, _ = pr.mesh()
    pr.apply_bc(clamp_mask(xyz))
    rod = dict(K=pr.K(), M=pr.M(), A=temporal(xt)[0], f={})
    pr.close()
    monkeypatch.setenv("XTFEM_ILU_WARPS", "16")
    monkeypatch.setenv("XTFEM_TRACE", "1")
    check(xt, orc, rod, factor(xt, rod, 30, blocks), 3, blocks, True)
    err = capfd.readouterr().err
    assert ("register sweep over 4 row blocks: H 2, steps 16" if blocks > 1 else "register sweep: H 2, steps 16") in err
    assert "warps 16" not in err
