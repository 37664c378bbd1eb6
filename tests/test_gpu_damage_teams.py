"""The damage update's exact steps, taken by teams of lanes, against the
oracle: one point of a warp beyond yield (a whole warp per point), every point
(four points a warp at a time, with idle teams at the end), step counts around
the screening passes and the shape-table chunks, stored energy on both sides of
the damage threshold.  Tolerances as in test_gpu_parity: 1e-6 on D, 1e-8
relative on the rest of the state (the same FP64 formulas with regrouped
sums)."""
import ctypes as C

import numpy as np
import pytest

from conftest import rod_problem

pytestmark = pytest.mark.gpu
KEYS = ["eps_old", "eps_pl", "sig_eff", "sig_back", "p", "D", "ws", "del_po", "sig_d"]


def case(xt, dims, nip, peak, seed=3):
    """Axial strain to `peak` times the yield strain everywhere ("all"), or 0.6
    of it with one node pulled further ("one")."""
    pr = rod_problem(xt, *dims)
    xyz, conn = pr.mesh()
    nn, ne = len(xyz), len(conn)
    rng = np.random.default_rng(seed)
    u = np.zeros((nn, 3))
    if peak == "all":
        u[:, 0] = 1.3e-3 * xyz[:, 0]
    else:
        u[:, 0] = 5e-4 * xyz[:, 0]
        u[conn[ne // 2, 4] - 1, 0] += 2e-3 * 3.0 / dims[0]
    u += rng.standard_normal(u.shape) * 1e-6
    blocks = [0.05 * u.ravel() * rng.uniform(0.5, 1.5) for _ in range(3)]
    blocks += [u.ravel() * rng.uniform(0.9, 1.1) for _ in range(3)]
    ngp = 8 * ne
    st = {k: np.zeros(6 * ngp) for k in KEYS[:4]}
    st.update({k: np.zeros(ngp) for k in KEYS[4:]})
    st["ws"] = rng.uniform(31.7, 31.8, ngp)
    ins = [np.repeat(conn, 8, axis=0).ravel().astype(np.int32), *pr.strain_rows(),
           xt.nt_table(nip, np.array([0.0, 0.125, 0.25]), 2 * np.pi * 20), np.concatenate(blocks),
           np.full(ngp, 2.0e5) * rng.uniform(0.98, 1.02, ngp), np.full(ngp, 0.3) * rng.uniform(0.98, 1.02, ngp)]
    pr.close()
    return ne, nn, ins, st


def agree(got, ref):
    assert np.max(np.abs(got["D"] - ref["D"])) <= 1e-6
    for k in KEYS:
        if k != "D":
            assert np.max(np.abs(got[k] - ref[k])) <= 1e-8 * max(np.max(np.abs(ref[k])), 1e-300) + 1e-14, k


@pytest.mark.parametrize("nip", [1, 31, 33, 256, 1025])
@pytest.mark.parametrize("peak", ["one", "all"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 1, 1), (12, 4, 4)], ids=lambda d: "x".join(map(str, d)))
def test_exact_steps_match_oracle(xt, orc, dims, peak, nip):
    ne, nn, ins, st = case(xt, dims, nip, peak)
    ref = {k: v.copy() for k, v in st.items()}
    for _ in range(2):  # the second slab starts from the first one's state
        xt.damage(ne, nn, nip, *ins, st)
        orc.damage(ne, nn, nip, *ins, ref)
        agree(st, ref)
    if nip >= 256:
        assert np.count_nonzero(ref["p"]) >= (ne * 4 if peak == "all" else 1)


def test_device_tables_off_16_byte_boundaries(xt, orc):
    """xt_damage_device takes arrays aligned to their element only."""
    torch = pytest.importorskip("torch")
    xt.lib().xt_init(0)
    ne, nn, ins, st = case(xt, (3, 1, 1), 256, "all")
    ref = {k: v.copy() for k, v in st.items()}
    orc.damage(ne, nn, 256, *ins, ref)

    def off(a):  # one element past an aligned start
        t = torch.empty(a.size + 1, dtype=torch.from_numpy(a[:1]).dtype, device="cuda")
        t[1:] = torch.from_numpy(np.ascontiguousarray(a))
        return t[1:]

    di, ds = [off(a) for a in ins], {k: off(st[k]) for k in KEYS}
    torch.cuda.synchronize()
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    counts = (C.c_ulonglong * 3)()
    rc = xt.lib().xt_damage_device(ne, nn, 3, 8, 3, 8, 6, 256, *[ptr(t) for t in di],
                                   *[ptr(ds[k]) for k in KEYS], counts)
    assert rc == 0, xt.lib().xt_last_error()
    agree({k: ds[k].cpu().numpy() for k in KEYS}, ref)
    assert counts[0] > 0 and counts[1] + counts[2] == 8 * ne * 256
