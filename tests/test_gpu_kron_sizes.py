"""The FP64 Kronecker apply's two kernels over the sizes where one takes over
from the other (q times the nodes, 10,500 from three temporal blocks on and
16,000 below) and, forced by XTFEM_KRON_NB=2, the node blocks on the smallest
meshes: against the oracle (1e-12 in the max norm, as in test_gpu_parity)."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem

pytestmark = pytest.mark.gpu


def systems(xt, dims):
    pr = rod_problem(xt, *dims)
    xyz, _ = pr.mesh()
    pr.apply_bc(clamp_mask(xyz))
    K, M = pr.K(), pr.M()
    pr.close()
    return K, M


def compare(xt, orc, K, M, q, beta):
    rng = np.random.default_rng(q)
    A, B, x, y = rng.standard_normal((q, q)), rng.standard_normal((q, q)), rng.standard_normal(K.n * q), rng.standard_normal(K.n * q)
    s = xt.SpaceTimeSystem(K, M, q=q)
    ref = orc.kronspgemv(A, B, 1.5, beta, K, M, x, y)
    got = s.apply(A, B, x, alpha=1.5, beta=beta, y=y)
    s.close()
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("beta", [0.0, 2.0])
@pytest.mark.parametrize("q", range(1, 9))
@pytest.mark.parametrize("dims", [(1, 1, 1), (12, 1, 1), (4, 2, 3), (12, 4, 4)], ids=lambda p: "x".join(map(str, p)))
def test_blocks_on_small_meshes(xt, orc, monkeypatch, dims, q, beta):
    monkeypatch.setenv("XTFEM_KRON_NB", "2")
    compare(xt, orc, *systems(xt, dims), q, beta)


@pytest.mark.parametrize("q,nodes", [(1, 16000), (2, 8000), (3, 3500), (6, 1750), (8, 1313)])
@pytest.mark.parametrize("side", [-1, 1])
def test_both_sides_of_the_rule(xt, orc, q, nodes, side):
    nx = nodes // 36 - 1  # rods of 6 x 6 nodes a section
    while side * ((nx + 1) * 36 - nodes) < 0:
        nx += side
    compare(xt, orc, *systems(xt, (nx, 5, 5)), q, 0.0)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("dims", [(4, 2, 3), (12, 4, 4)], ids=lambda p: "x".join(map(str, p)))
def test_non_finite_entries_reach_the_same_rows(xt, monkeypatch, dims, value):
    K, M = systems(xt, dims)
    rng = np.random.default_rng(1)
    A, B, x = rng.standard_normal((6, 6)), rng.standard_normal((6, 6)), rng.standard_normal(K.n * 6)
    x[rng.integers(0, x.size, 3)] = value
    s = xt.SpaceTimeSystem(K, M)
    got = []
    for nb in "20":
        monkeypatch.setenv("XTFEM_KRON_NB", nb)
        got.append(s.apply(A, B, x))
    s.close()
    assert np.array_equal(np.isfinite(got[0]), np.isfinite(got[1]))
    f = np.isfinite(got[1])
    assert np.max(np.abs(got[0][f] - got[1][f]), initial=0.0) <= 1e-12 * max(1.0, np.max(np.abs(got[1][f]), initial=0.0))
