"""A wait for a level's data that runs out in the default triangular sweeps (FP64
row records; the FP32 register sweep with three and with one row a group; the
row blocks of a block-Jacobi factor): the call returns XT_ERR_CUDA with the
"gave up" message, and the applies after it, with the normal limit, agree with
the oracle's kronlusol again (1e-10 in FP64, 1e-4 in FP32, as in
test_gpu_parity).  XTFEM_ILU_SPIN_LIMIT=1 gives up at the first wait, before
anything has been read."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem, temporal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 1, 1), (24, 8, 8)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("group,blocks,fp32", [(3, 1, False), (1, 1, False), (3, 1, True), (1, 1, True), (3, 4, True)])
def test_default_sweeps_report_a_wait_that_runs_out(xt, orc, monkeypatch, dims, group, blocks, fp32):
    pr = rod_problem(xt, *dims)
    xyz, _ = pr.mesh()
    pr.apply_bc(clamp_mask(xyz))
    K, M = pr.K(), pr.M()
    f = xt.ilut(K, 20, 1e-4, blocks=blocks)
    A = temporal(xt)[0]
    x = np.random.default_rng(3).standard_normal(K.n * 6)
    ref = orc.kronlusol(A, *f, x)
    s = xt.SpaceTimeSystem(K, M)
    s.set_ilu(*f, group=group, blocks=blocks)
    for _ in range(2):
        monkeypatch.setenv("XTFEM_ILU_SPIN_LIMIT", "1")
        with pytest.raises(xt.XtError) as e:
            s.lusol(A, x, fp32=fp32)
        assert "status -11" in str(e.value) and "gave up" in str(e.value)
        monkeypatch.delenv("XTFEM_ILU_SPIN_LIMIT")
        for _ in range(2):
            y = s.lusol(A, x, fp32=fp32)
            assert np.linalg.norm(y - ref) <= (1e-4 if fp32 else 1e-10) * np.linalg.norm(ref)
    s.close()
    pr.close()
