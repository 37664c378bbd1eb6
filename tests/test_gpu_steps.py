"""The Arnoldi step and the reassembly at the edges of their kernels' shares.

FP64 GMRES: basis sizes around the eight vectors a warp sums at once and the
restart, vectors shorter than a block's rows up to several blocks; a wrong dot
or update breaks the Arnoldi relation, so the last estimate then leaves the
true residual.  Both are rounded at about 1e-13 of the right-hand side and the
estimates compared stay above 1e-9 of it: they agree to about 1e-5, asserted to
1e-4.

Mode 2: the coming step's first half enters the stream before the host has
seen the step, so a cycle may end with it issued, with it held back, at the
restart, at maxits or at the first step; each gives the device-driven loop's
bits.

Reassembly: element counts around a block's eight elements, a modulus for
every Gauss point, against the element integral (1e-11 of the largest entry,
as for one element)."""
import numpy as np
import pytest

from conftest import clamp_mask, rod_problem, temporal
from test_gpu_assembly import element_k, make

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(3, 1, 1), (12, 4, 4), (9, 5, 7)], ids=lambda p: "x".join(map(str, p)))
def rod(request, xt):
    pr = rod_problem(xt, *request.param)
    xyz, _ = pr.mesh()
    bc = clamp_mask(xyz)
    pr.apply_bc(bc)
    K, M = pr.K(), pr.M()
    A, B, _, _ = temporal(xt)
    yield dict(K=K, M=M, bc=bc, f=xt.ilut(K, 20, 1e-4), A=A, B=B)
    pr.close()


def system(xt, rod, q):
    s = xt.SpaceTimeSystem(rod["K"], rod["M"], q=q)
    s.set_ilu(*rod["f"])
    s.set_temporal(rod["A"][:q, :q], rod["B"][:q, :q])
    rhs = np.random.default_rng(q).standard_normal(rod["K"].n * q)
    rhs[np.tile(rod["bc"], q) == 1] = 0.0
    return s, rhs


@pytest.mark.parametrize("q", [1, 3, 6])
@pytest.mark.parametrize("im", [1, 7, 8, 9, 17])
def test_fp64_estimate_is_the_true_residual(xt, orc, rod, im, q):
    s, rhs = system(xt, rod, q)
    x, info = s.gmres(rhs, im=im, eps=1e-8, maxits=40, hist_len=64)  # 40 or the cycle's end
    s.close()
    r = rhs - orc.kronspmv(rod["A"][:q, :q], rod["B"][:q, :q], rod["K"], rod["M"], x)
    est = info["hist"][info["its"] - 1]
    assert abs(np.linalg.norm(r) / np.linalg.norm(rhs) - est) <= 1e-4 * est


@pytest.mark.parametrize("tol", [1e-1, 1e-3, 1e-10])
@pytest.mark.parametrize("maxits", [1, 2, 11, 300])
@pytest.mark.parametrize("im", [1, 2, 6])
def test_early_issued_half_steps_keep_the_bits(xt, rod, monkeypatch, im, maxits, tol):
    s, rhs = system(xt, rod, 6)
    got = []
    for flag in "01":
        monkeypatch.setenv("XTFEM_DEVICE_GMRES", flag)
        got.append(s.solve(rhs, im=im, tol=tol, maxits=maxits, precision=2))
    s.close()
    assert got[0][1] == got[1][1]
    assert np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("ne", [1, 7, 8, 9, 17])
def test_reassembly_around_a_blocks_elements(xt, ne):
    pr, s, _, _, xyz, conn, _ = make(xt, ne, 1, 1, clamp=False)
    rng = np.random.default_rng(ne)
    ym, nu = rng.uniform(1e5, 3e5, (ne, 8)), rng.uniform(0.2, 0.35, (ne, 8))
    s.assemble_k(ym, nu)
    got = s.get_k().to_scipy().toarray()
    ref = np.zeros_like(got)
    for e in range(ne):
        dofs = (3 * (conn[e] - 1)[:, None] + np.arange(3)).ravel()
        ref[np.ix_(dofs, dofs)] += element_k(xyz[conn[e] - 1], ym[e], nu[e])
    s.close()
    pr.close()
    assert np.max(np.abs(got - ref)) <= 1e-11 * np.max(np.abs(ref))
