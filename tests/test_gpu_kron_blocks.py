"""The FP64 Kronecker apply in node blocks against the oracle and the CSR
kernel (XTFEM_KRON_NB=0): one to eight temporal blocks, alpha and beta, node
counts around a thread block's share, constrained nodes (blocks with missing
entries), infinite and NaN entries of x (a missing entry multiplies nothing),
and pairs without a node-block form (a column listed twice, an M that couples
components).  Tolerance as in test_gpu_parity: 1e-12 in the max norm."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(1, 1, 1), (12, 1, 1), (4, 2, 3), (12, 4, 4)], ids=lambda p: "x".join(map(str, p)))
def pair(request, xt):
    pr = rod_problem(xt, *request.param)
    xyz, _ = pr.mesh()
    bc = clamp_mask(xyz)
    bc[-2] = 1  # one component of one node alone
    pr.apply_bc(bc)
    yield pr.K(), pr.M()
    pr.close()


@pytest.mark.parametrize("q", range(1, 9))
def test_blocks_match_oracle(xt, orc, pair, q):
    K, M = pair
    rng = np.random.default_rng(q)
    A, B, x, y = rng.standard_normal((q, q)), rng.standard_normal((q, q)), rng.standard_normal(K.n * q), rng.standard_normal(K.n * q)
    s = xt.SpaceTimeSystem(K, M, q=q)
    for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):
        ref = orc.kronspgemv(A, B, alpha, beta, K, M, x, y)
        got = s.apply(A, B, x, alpha=alpha, beta=beta, y=y)
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    s.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_entries_reach_the_same_rows(xt, pair, monkeypatch, value):
    K, M = pair
    q = 6
    rng = np.random.default_rng(1)
    A, B, x = rng.standard_normal((q, q)), rng.standard_normal((q, q)), rng.standard_normal(K.n * q)
    x[rng.integers(0, x.size, 3)] = value
    s = xt.SpaceTimeSystem(K, M)
    got = s.apply(A, B, x)
    monkeypatch.setenv("XTFEM_KRON_NB", "0")
    ref = s.apply(A, B, x)
    s.close()
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    f = np.isfinite(ref)
    assert np.max(np.abs(got[f] - ref[f]), initial=0.0) <= 1e-12 * max(1.0, np.max(np.abs(ref[f]), initial=0.0))


@pytest.mark.parametrize("form", ["twice", "mixed"])
def test_pairs_without_block_form(xt, orc, pair, form):
    K, M = pair
    rng = np.random.default_rng(2)
    if form == "twice":  # the first row's first entry in two halves
        ia = K.ia.copy()
        ia[1:] += 1
        K = xt.Csr(ia, np.insert(K.ja, 0, K.ja[0]), np.concatenate([[K.a[0] / 2, K.a[0] / 2], K.a[1:]]))
    else:
        M = K
    A, B, x = rng.standard_normal((6, 6)), rng.standard_normal((6, 6)), rng.standard_normal(K.n * 6)
    ref = orc.kronspmv(A, B, K, M, x)
    got = xt.kronspmv(A, B, K, M, x)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
