"""Rounding of the FP64 Kronecker apply in node blocks: its error against
extended precision is at most 1.05 times the CSR kernel's (XTFEM_KRON_NB=0; 2
takes the blocks at any size), the
2-norm over four inputs on a mesh of full and of constrained node rows.  The
ratio is about 0.95 for sums of nine terms, 1.5 for one sum of 81; the mean over
18,000 and more rounded entries leaves it within a percent or two."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem, temporal

pytestmark = pytest.mark.gpu


def exact(A, B, K, M, x):
    """K X A^T + M X B^T in long double (64 or 113 bits of mantissa)."""
    X = x.reshape(A.shape[0], -1).T.astype(np.longdouble)

    def times(C):
        Y = np.zeros_like(X)
        np.add.at(Y, np.repeat(np.arange(C.n), np.diff(C.ia)), C.a.astype(np.longdouble)[:, None] * X[C.ja - 1])
        return Y

    return (times(K) @ A.T.astype(np.longdouble) + times(M) @ B.T.astype(np.longdouble)).T.ravel()


@pytest.mark.parametrize("q", [3, 6])
def test_no_more_rounding_than_the_csr_kernel(xt, monkeypatch, q):
    pr = rod_problem(xt, 18, 8, 6)
    xyz, _ = pr.mesh()
    pr.apply_bc(clamp_mask(xyz))
    K, M = pr.K(), pr.M()
    pr.close()
    s = xt.SpaceTimeSystem(K, M, q=q)
    err = np.zeros(2)
    for seed in range(4):
        A, B = (T[:q, :q].copy() for T in temporal(xt, t1=0.5 * seed)[:2])
        x = np.random.default_rng(seed).standard_normal(K.n * q)
        ref = exact(A, B, K, M, x)
        for k, nb in enumerate("02"):
            monkeypatch.setenv("XTFEM_KRON_NB", nb)
            err[k] += float(np.sum((s.apply(A, B, x) - ref) ** 2) / np.sum(ref ** 2))
    s.close()
    assert np.sqrt(err[1] / err[0]) <= 1.05
