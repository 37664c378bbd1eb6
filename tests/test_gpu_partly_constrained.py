"""One clamped component of an otherwise free node (a roller, a symmetry plane):
the pair K, M has no node-block form then and runs through the CSR kernels."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem, temporal
from test_gpu_kron_sizes import compare

pytestmark = pytest.mark.gpu


def clamp_one_component(xt, dims):
    """A rod whose free end has one node with a single clamped component (a
    roller): M then lacks that component's entries."""
    pr = rod_problem(xt, *dims)
    xyz, _ = pr.mesh()
    bc = clamp_mask(xyz)
    node = int(np.argmax(xyz[:, 0]))
    assert not bc[3 * node: 3 * node + 3].any()
    bc[3 * node + 1] = 1
    pr.apply_bc(bc)
    K, M = pr.K(), pr.M()
    pr.close()
    return K, M, bc


@pytest.mark.parametrize("nb", ["2", "1"])
def test_partly_constrained_node(xt, orc, monkeypatch, nb):
    """Such a system has no node-block form (M is no longer one scalar a block)
    and runs through the CSR kernels: FP64 apply and a mode-2 solve, whose
    estimate is the true residual (1e-4 of it, as in test_gpu_kron_staged)."""
    monkeypatch.setenv("XTFEM_KRON_NB", nb)
    K, M, bc = clamp_one_component(xt, (12, 4, 4))
    compare(xt, orc, K, M, 6, 2.0)
    A, B = temporal(xt)[:2]
    s = xt.SpaceTimeSystem(K, M)
    s.set_ilu(*xt.ilut(K, 20, 1e-4))
    s.set_temporal(A, B)
    rhs = np.random.default_rng(2).standard_normal(K.n * 6)
    rhs[np.tile(bc, 6) == 1] = 0.0
    sol, info = s.solve(rhs, im=40, tol=1e-7, maxits=200, precision=2)
    s.close()
    r = rhs - orc.kronspmv(A, B, K, M, sol)
    assert info["relres"] <= 1e-7
    assert abs(np.linalg.norm(r) / np.linalg.norm(rhs) - info["relres"]) <= 1e-4 * info["relres"]
