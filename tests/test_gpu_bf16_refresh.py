"""New values of K reach its BF16 copy (precision mode 3), which a solve before
them has made: after a reassembly with other moduli, mode 3 gives the bits and
the iteration count of a system created from the new K."""
import numpy as np
import pytest

from conftest import temporal
from test_gpu_assembly import E, NU, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 1, 1), (12, 4, 4)], ids=lambda d: "x".join(map(str, d)))
def test_mode3_after_a_reassembly_is_a_fresh_systems(xt, dims):
    pr, s, K, M, _, conn, bc = make(xt, *dims)
    ne = conn.shape[0]
    f = xt.ilut(K, 20, 1e-4)
    A, B, _, _ = temporal(xt)
    rhs = np.random.default_rng(21).standard_normal(K.n * 6)
    rhs[np.tile(bc, 6) == 1] = 0.0
    s.set_ilu(*f)
    s.set_temporal(A, B)
    s.solve(rhs, im=30, tol=1e-8, precision=3)
    ym = np.full((ne, 8), E)
    ym[::2] *= 0.2
    s.assemble_k(ym, np.full((ne, 8), NU))
    got = s.solve(rhs, im=30, tol=1e-8, precision=3)
    t = xt.SpaceTimeSystem(s.get_k(), M)
    t.set_ilu(*f)
    t.set_temporal(A, B)
    ref = t.solve(rhs, im=30, tol=1e-8, precision=3)
    t.close()
    s.close()
    pr.close()
    assert got[1] == ref[1]
    assert np.array_equal(got[0], ref[0])
