"""The triangular sweeps of FP64 factors (row records) and of FP32 factors of
one unknown per node (register sweep) against the oracle's kronlusol: every
number of lanes per row, one warp (each level split in sub-levels) and the
default, one, three and six temporal blocks, on rods whose level widths fall
below, on and above the groups of a warp.  Tolerances as in test_gpu_parity: 1e-10 in FP64 (the same
factor and inverted diagonal blocks in another summation order), 1e-4 in FP32
(the factor itself is rounded)."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem, temporal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(3, 1, 1), (12, 4, 4), (9, 5, 7)], ids=lambda p: "x".join(map(str, p)))
def rod(request, xt):
    pr = rod_problem(xt, *request.param)
    xyz, _ = pr.mesh()
    pr.apply_bc(clamp_mask(xyz))
    K, M = pr.K(), pr.M()
    yield dict(K=K, M=M, f=xt.ilut(K, 20, 1e-4), A=temporal(xt)[0])
    pr.close()


@pytest.mark.parametrize("q", [1, 3, 6])
@pytest.mark.parametrize("warps", [None, 1])
@pytest.mark.parametrize("shares", [None, 1, 2, 4])
@pytest.mark.parametrize("group,fp32", [(1, False), (3, False), (1, True)])
def test_row_sweep_matches_oracle(xt, orc, rod, monkeypatch, group, fp32, shares, warps, q):
    if shares:
        monkeypatch.setenv("XTFEM_ILU_SHARES" if fp32 else "XTFEM_ILU_ROW_H", str(shares))
    if warps:
        monkeypatch.setenv("XTFEM_ILU_WARPS", str(warps))
    A = rod["A"][:q, :q]
    x = np.random.default_rng(q).standard_normal(rod["K"].n * q)
    ref = orc.kronlusol(A, *rod["f"], x)
    s = xt.SpaceTimeSystem(rod["K"], rod["M"], q=q)
    s.set_ilu(*rod["f"], group=group)
    for _ in range(2):  # built, then reused
        y = s.lusol(A, x, fp32=fp32)
        assert np.linalg.norm(y - ref) <= (1e-4 if fp32 else 1e-10) * np.linalg.norm(ref)
    s.close()
