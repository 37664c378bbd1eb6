"""Workloads of the space-time solve path, as a program calls it: the
Kronecker operator, the ILUT preconditioner, the FP64 and mixed-precision
solves, a batch of specimens, the slab loops, the fatigue-damage update and
the reassembly of K.

A case is a dict of plain values; `prepare` builds what a program has in
hand before the call, `run` makes one pass through the public entry points,
`work` counts the pass's inputs and outputs, and `exact` gives the same
outputs in plain 64-bit torch or numpy where that is affordable.

Sizes are those of the shipped configurations (xtfem_gb300/configs): the
4 x 4 x 12 rod (C1), the 20 x 20 x 60 rod (C2), the 64 rods n x n x 3n (C4);
the plate (C3) and the panel (C5) appear at reduced sizes.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import xtfem_gb300 as xt
from xtfem_gb300 import meshes

FREQ, DT = 20.0, 0.5          # load frequency and slab length of C1, C2 and C4
OMEGA = 2 * np.pi * FREQ
E0, NU0 = 2.0e5, 0.3
STATE6 = ("eps_old", "eps_pl", "sig_eff", "sig_back")
STATE1 = ("p", "D", "ws", "del_po", "sig_d")


def listed():
    c1 = dict(mesh="rod", nx=12, ny=4, nz=4)
    mid = dict(mesh="rod", nx=30, ny=10, nz=10)
    c2 = dict(mesh="rod", nx=60, ny=20, nz=20)
    return [
        # the smallest call: one operator apply on the C1 rod, all latency
        dict(name="apply_c1", path="apply", beta=0.0, **c1),
        # the operator on the C2 rod, accumulated onto y (a residual, a jump term)
        dict(name="apply_c2", path="apply", beta=1.0, **c2),
        # the FP64 preconditioner on the C2 rod (a caller's own Krylov loop)
        dict(name="lusol_c2", path="lusol", **c2),
        # the Fortran driver's call on C1: operator and factor handed over, FP64 GMRES(30)
        dict(name="kronpgmres_c1", path="kronpgmres", im=30, eps=1e-8, **c1),
        # FP64 GMRES on the largest C4 rod with the operator kept on the GPU
        dict(name="gmres_mid", path="gmres", im=120, eps=1e-8, **mid),
        # the mixed-precision solve of an uneven specimen
        dict(name="solve_odd", path="solve", precision=2, im=60, tol=1e-10, mesh="rod", nx=25, ny=9, nz=7),
        # a slab of the C2 loop (load, jump term, solve), its damage update being damage_c2
        dict(name="slab_c2", path="slab", im=200, tol=1e-12, **c2),
        # the C4 batch: 64 uneven rods solved together
        dict(name="batch_c4", path="batch", count=64, nlo=4, nhi=10, im=120, tol=1e-10),
        # a thermal slab (three temporal blocks, one unknown per node) on the C2 mesh
        dict(name="thermal_c2", path="thermal", im=60, tol=1e-10, precision=2, **c2),
        # the driver's damage call on C1 with host arrays, ten load cycles (after the first deletion)
        dict(name="damage_c1", path="damage_host", nip=2560, amp=130.0, **c1),
        # the damage update of a full C2 slab, a hundred cycles, state on the GPU
        dict(name="damage_c2", path="damage", nip=25600, amp=115.0, **c2),
        # reassembly of K from new moduli and its first use (coupled runs, once per slab)
        dict(name="assemble_c2", path="assemble", **c2),
    ]


def _rod(rng, lo, hi):
    """A rod of lo .. hi nodes (log-uniform), three times as long as wide, uneven sides."""
    nodes = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = (nodes / 3) ** (1 / 3)
    ny, nz = (max(2, round(n * rng.uniform(0.85, 1.2))) for _ in range(2))
    nx = max(4, min(60, round(nodes / ((ny + 1) * (nz + 1))) - 1))
    return dict(mesh="rod", nx=nx, ny=min(ny, 20), nz=min(nz, 20))


def _any_mesh(rng, lo, hi):
    r = rng.random()
    if r < 0.2:  # notched plate, two elements thick
        s = rng.uniform(0.15, 0.45)
        return dict(mesh="sent", nx=round(106 * s), ny=round(212 * s) // 2 * 2, nz=2)
    if r < 0.4:  # holed panel, one element thick
        return dict(mesh="panel", nx=4 * rng.randint(6, 24), ny=rng.randint(6, 24), nz=1)
    return _rod(rng, lo, hi)


def draw(rng):
    path = rng.choice(["apply", "apply", "lusol", "lusol", "kronpgmres", "gmres", "solve", "solve", "slab", "batch",
                       "thermal", "damage_host", "damage", "assemble"])
    if path == "apply":
        return dict(path=path, beta=rng.choice([0.0, 1.0]), **_any_mesh(rng, 300, 26000))
    if path == "lusol":
        return dict(path=path, **_any_mesh(rng, 300, 26000))
    if path == "kronpgmres":
        return dict(path=path, im=rng.choice([30, 60]), eps=1e-8, **_rod(rng, 150, 1200))
    if path == "gmres":
        return dict(path=path, im=rng.choice([60, 120]), eps=1e-8, **_rod(rng, 300, 3500))
    if path == "solve":
        return dict(path=path, precision=rng.choice([0, 2, 2, 2]), im=rng.choice([60, 120, 200]), tol=1e-10, **_rod(rng, 300, 4000))
    if path == "slab":
        return dict(path=path, im=rng.choice([120, 200]), tol=1e-12, **_rod(rng, 1500, 20000))
    if path == "batch":
        lo = rng.randint(3, 6)
        return dict(path=path, count=rng.randint(5, 40), nlo=lo, nhi=rng.randint(lo + 1, 9), im=rng.choice([60, 120]), tol=1e-10)
    if path == "thermal":
        return dict(path=path, im=rng.choice([30, 60]), tol=1e-10, precision=rng.choice([0, 2, 2]), **_rod(rng, 500, 26000))
    if path == "damage_host":
        return dict(path=path, nip=256 * rng.randint(1, 20), amp=round(rng.uniform(100, 150), 1), **_rod(rng, 150, 2000))
    if path == "damage":
        return dict(path=path, nip=256 * rng.randint(4, 100), amp=round(rng.uniform(100, 125), 1), **_rod(rng, 1000, 26000))
    return dict(path=path, **_rod(rng, 300, 26000))


# ---------------------------------------------------------------- models
@functools.lru_cache(maxsize=8)
def _mesh(mesh, nx, ny, nz):
    if mesh == "rod":
        return xt.Problem.rod(nx, ny, nz, 3.0, 1.0, 1.0)
    xyz, conn = meshes.sent_plate(nx, ny, nz) if mesh == "sent" else meshes.holed_panel(nx, ny, nz, ratio=1.02, order="rays")
    return xt.Problem.from_mesh(xyz, conn)


@functools.lru_cache(maxsize=8)
def _model(mesh, nx, ny, nz):
    """Mesh, clamped K and M and constrained DOFs: the same for every seed."""
    pr = _mesh(mesh, nx, ny, nz)
    xyz, conn = pr.mesh()
    axis = 0 if mesh == "rod" else 1
    bc = np.repeat(xyz[:, axis] == xyz[:, axis].min(), 3).astype(np.int32)
    pr.apply_bc(bc)
    face = np.zeros(3 * len(xyz))
    face[axis::3] = xyz[:, axis] == xyz[:, axis].max()
    return dict(K=pr.K(), M=pr.M(), xyz=xyz, conn=conn, bc=bc, face=face)


@functools.lru_cache(maxsize=8)
def _factor(mesh, nx, ny, nz):
    return xt.ilut(_model(mesh, nx, ny, nz)["K"], 20, 1e-4)


def _at(case):
    return case["mesh"], case["nx"], case["ny"], case["nz"]


def _temporal(slab=0):
    k, m, kt, mt, _, _ = xt.stcoeff_m(slab * DT, DT, OMEGA)
    return k + kt, m + mt


def _load(m, rng):
    """Load blocks of a traction of seeded amplitude, uneven over the face."""
    f, _ = xt.getfextc_m(0.0, OMEGA, DT)
    r = m["face"] * rng.uniform(50.0, 150.0) * rng.uniform(0.8, 1.2, len(m["face"])) / max(1.0, m["face"].sum())
    return np.concatenate([c * r for c in f])


def _system(at, temporal=True, factor=True):
    m = _model(*at)
    s = xt.SpaceTimeSystem(m["K"], m["M"])
    if factor:
        s.set_ilu(*_factor(*at))
    if temporal:
        s.set_temporal(*_temporal())
    return s


def _rods(case, seed):
    rng = np.random.default_rng(case["count"] * 1000 + case["nlo"])  # the specimens are the program's, loads the seed's
    ns = rng.integers(case["nlo"], case["nhi"] + 1, case["count"])
    return [("rod", 3 * int(n), int(n), int(n)) for n in ns]


def _displacement(case, seed):
    """A loaded rod's displacement over the slab (six temporal blocks): axial
    strain of the applied stress, lateral contraction held back at the clamp,
    and the strain concentration at the clamp's corners that starts fatigue."""
    rng = np.random.default_rng(seed)
    xyz = _model(*_at(case))["xyz"]
    x, y, z = xyz.T
    eps = case["amp"] * rng.uniform(0.98, 1.02) / E0
    free = 1.0 - np.exp(-x / 0.3)
    h = 0.8 / case["ny"]  # the concentration is as sharp as the mesh lets it be
    corner = np.zeros_like(x)
    for cy in (0.0, 1.0):
        for cz in (0.0, 1.0):
            corner += np.exp(-np.hypot(y - cy, z - cz) / h) * rng.uniform(0.95, 1.05)
    u = np.stack([eps * (x + 2.6 * h * corner * (1.0 - np.exp(-x / h))), -NU0 * eps * (y - 0.5) * free, -NU0 * eps * (z - 0.5) * free], 1).ravel()
    u += rng.standard_normal(u.size) * 1e-8
    slow = [0.02 * u * rng.uniform(0.5, 1.5) for _ in range(3)]
    return np.concatenate(slow + [u * rng.uniform(0.97, 1.03) for _ in range(3)])


def _damage_inputs(case, seed):
    pr = _mesh(*_at(case))
    m = _model(*_at(case))
    rng = np.random.default_rng(seed + 1)
    ne, nn = len(m["conn"]), len(m["xyz"])
    ngp = 8 * ne
    st = {k: np.zeros(6 * ngp) for k in STATE6}
    st.update({k: np.zeros(ngp) for k in STATE1})
    st["ws"] = rng.uniform(31.5, 32.0, ngp)  # stored energy around the damage threshold of 31.76
    a = dict(nodes=np.repeat(m["conn"], 8, axis=0).ravel().astype(np.int32))
    a.update(zip(("Nx", "Ny", "Nz"), pr.strain_rows()))
    a["Nt"] = xt.nt_table(case["nip"], np.array([0.0, DT / 2, DT]) * case["nip"] / 25600, OMEGA)
    a["sol"] = _displacement(case, seed)
    a["ym"] = np.full(ngp, E0)
    a["nu"] = np.full(ngp, NU0)
    return ne, nn, a, st


# --------------------------------------------------------------- a pass
def prepare(case, seed):
    path = case["path"]
    rng = np.random.default_rng(seed)
    if path == "batch":
        rods = _rods(case, seed)
        systems = [_system(r) for r in rods]
        return dict(path=path, case=case, b=xt.SystemBatch(systems), rhs=[_load(_model(*r), rng) for r in rods])
    at = _at(case)
    if path in ("damage", "damage_host"):
        xt.lib().xt_init(0)
        ne, nn, a, st = _damage_inputs(case, seed)
        if path == "damage":
            a = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in a.items()}
            st = {k: torch.from_numpy(v).cuda() for k, v in st.items()}
        return dict(path=path, case=case, ne=ne, nn=nn, a=a, st=st)
    if path == "slab":
        cfg = xt.SlabConfig.make(amplitude=float(rng.uniform(50.0, 150.0)), precision=2, im=case["im"], tol=case["tol"],
                                 maxits=4000, gs_passes=1, damage=0)
        return dict(path=path, s=xt.SlabSolver(_mesh(*at), cfg))
    if path == "thermal":
        cfg = xt.ThermalConfig.make(q0=float(rng.uniform(1000.0, 3000.0)), T0=float(rng.uniform(15.0, 25.0)), im=case["im"],
                                    tol=case["tol"], precision=case["precision"])
        return dict(path=path, s=xt.ThermalSolver(_mesh(*at), cfg))
    m = _model(*at)
    d = dict(path=path, case=case)
    if path in ("apply", "lusol", "assemble"):
        d.update(zip("AB", _temporal(seed % 7)))
        d["x"] = rng.standard_normal(6 * m["K"].n)
        d["s"] = _system(at, temporal=False, factor=path == "lusol")
    if path == "apply":
        d["y"] = rng.standard_normal(6 * m["K"].n) if case["beta"] else None
    if path == "assemble":
        d["s"].set_mesh(m["xyz"], m["conn"], m["bc"])
        d["ym"] = E0 * rng.uniform(0.9, 1.0, (len(m["conn"]), 8))
        d["nu"] = NU0 * rng.uniform(0.95, 1.05, (len(m["conn"]), 8))
    if path in ("kronpgmres", "gmres", "solve"):
        d["rhs"] = _load(m, rng)
    if path == "kronpgmres":
        d.update(zip("AB", _temporal()), K=m["K"], M=m["M"], f=_factor(*at))
    if path in ("gmres", "solve"):
        d["s"] = _system(at)
    return d


def run(d):
    path, c = d["path"], d.get("case")
    if path == "apply":
        return d["s"].apply(d["A"], d["B"], d["x"], beta=c["beta"], y=d["y"])
    if path == "lusol":
        return d["s"].lusol(d["A"], d["x"])
    if path == "kronpgmres":
        return xt.kronpgmres(d["A"], d["B"], d["K"], d["M"], *d["f"], d["rhs"], im=c["im"], eps=c["eps"], maxits=4000)
    if path == "gmres":
        sol, info = d["s"].gmres(d["rhs"], im=c["im"], eps=c["eps"], maxits=4000)
        return sol, info["ierr"]
    if path == "solve":
        sol, info = d["s"].solve(d["rhs"], im=c["im"], tol=c["tol"], maxits=4000, precision=c["precision"])
        return sol, info["ierr"]
    if path == "slab":
        d["s"].step()
        return d["s"].state()["disp"]
    if path == "batch":
        sols, _, status = d["b"].solve(d["rhs"], im=c["im"], tol=c["tol"], maxits=4000, precision=2)
        return np.concatenate(sols), status
    if path == "thermal":
        d["s"].step()
        return d["s"].temperature()
    if path == "assemble":
        d["s"].assemble_k(d["ym"], d["nu"])
        return d["s"].apply(d["A"], d["B"], d["x"])
    a, st = d["a"], d["st"]
    inputs = ("nodes", "Nx", "Ny", "Nz", "Nt", "sol", "ym", "nu")
    if path == "damage_host":
        return xt.damage(d["ne"], d["nn"], c["nip"], *[a[k] for k in inputs], st)
    xt.api.check(xt.lib().xt_damage_device(d["ne"], d["nn"], 3, 8, 3, 8, 6, c["nip"],
                                           *[C.c_void_p(a[k].data_ptr()) for k in inputs],
                                           *[C.c_void_p(st[k].data_ptr()) for k in STATE6 + STATE1], None), "damage")
    return st


# ----------------------------------------------------------------- work
def _sizes(mesh, nx, ny, nz):
    """Nodes, elements and stored 3 x 3 blocks (up to 27 neighbours a node)."""
    if mesh == "rod":
        return (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz, (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
    if mesh == "sent":
        return (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz, (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
    return nx * (ny + 1) * (nz + 1), nx * ny * nz, 3 * nx * (3 * ny + 1) * (3 * nz + 1)


def work(case):
    path = case["path"]
    if path == "batch":
        each = [work(dict(path="solve", mesh=r[0], nx=r[1], ny=r[2], nz=r[3])) for r in _rods(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    nn, ne, blocks = _sizes(*_at(case))
    p, q, per = (nn, 3, 1) if path == "thermal" else (3 * nn, 6, 9)
    nk, nm = per * blocks, blocks if path == "thermal" else 3 * blocks
    nlu = 40 * p
    vec = 8 * p * q
    op = 12 * (nk + nm) + 8 * (p + 1)
    op_flops = 2 * q * (nk + nm) + 4 * p * q * q
    lu = 12 * nlu + 8 * p
    lu_flops = 2 * q * nlu + 2 * p * q * q
    if path == "apply":
        return {"bytes": op + (3 if case["beta"] else 2) * vec, "flops": op_flops}
    if path == "lusol":
        return {"bytes": lu + 2 * vec, "flops": lu_flops}
    if path == "assemble":  # mesh, moduli, K's pattern and values, then one apply
        return {"bytes": 24 * nn + 160 * ne + 12 * nk + op + 2 * vec, "flops": 2 * 576 * 8 * ne + op_flops}
    if path in ("damage", "damage_host"):
        ngp = 8 * ne
        # strain rows, nodes and moduli, the state in and out, the solution; one six-term screen per point and step
        return {"bytes": ngp * (8 * 28 + 16 + 2 * 29 * 8) + 8 * 18 * nn + 48 * case["nip"], "flops": ngp * 36 * 12}
    # a solve: the operator and the factor read, load in, solution out; at least one step of the iteration
    return {"bytes": op + lu + 3 * vec, "flops": op_flops + lu_flops}


# ---------------------------------------------------------------- exact
def _csr(A):
    return torch.sparse_csr_tensor(torch.from_numpy(A.ia.astype(np.int64) - 1), torch.from_numpy(A.ja.astype(np.int64) - 1),
                                   torch.from_numpy(A.a), (A.n, A.n)).cuda()


def _kron(K, M, A, B, x):
    X = torch.from_numpy(x).cuda().reshape(A.shape[0], -1).T
    A, B = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (A, B))
    return ((K @ X) @ A.T + (M @ X) @ B.T).T.reshape(-1).cpu().numpy()


def _exact_lusol(alu, jlu, ju, A, x):
    p = len(ju)
    w = np.ascontiguousarray(np.linalg.solve(A, x.reshape(A.shape[0], p)).T)
    j0, u0 = jlu - 1, ju - 1
    for i in range(p):
        a, b = j0[i], u0[i]
        if b > a:
            w[i] -= alu[a:b] @ w[j0[a:b]]
    for i in range(p - 1, -1, -1):
        a, b = u0[i], j0[i + 1]
        w[i] = alu[i] * (w[i] - alu[a:b] @ w[j0[a:b]]) if b > a else alu[i] * w[i]
    return np.ascontiguousarray(w.T).reshape(-1)


_SIGN = torch.tensor([[-1, -1, 1], [-1, -1, -1], [-1, 1, -1], [-1, 1, 1], [1, -1, 1], [1, -1, -1], [1, 1, -1], [1, 1, 1]], dtype=torch.float64)


def _exact_k(m, ym, nu):
    """Clamped stiffness from the Gauss points' moduli: element integrals and their sum."""
    dev = "cuda"
    g = 0.577350269189626
    sg = _SIGN.to(dev)
    xe = torch.from_numpy(m["xyz"][m["conn"] - 1]).to(dev)
    ke = torch.zeros(len(xe), 8, 3, 8, 3, dtype=torch.float64, device=dev)
    eye = torch.eye(3, dtype=torch.float64, device=dev)
    for gp in range(8):
        pt = torch.tensor([g if (gp >> s) & 1 else -g for s in (2, 1, 0)], dtype=torch.float64, device=dev)
        f = 1 + sg * pt
        dn = 0.125 * sg * torch.stack([f[:, 1] * f[:, 2], f[:, 0] * f[:, 2], f[:, 0] * f[:, 1]], 1)
        J = torch.einsum("ia,eim->eam", dn, xe)
        dx = torch.einsum("ema,ia->eim", torch.linalg.inv(J), dn)
        E, v = (torch.from_numpy(a[:, gp].copy()).to(dev) for a in (ym, nu))
        det = torch.linalg.det(J)
        lam, mu = E * v / ((1 + v) * (1 - 2 * v)) * det, E / (2 * (1 + v)) * det
        P = torch.einsum("eia,ejb->eiajb", dx, dx)
        ke += lam[:, None, None, None, None] * P + mu[:, None, None, None, None] * (
            P.transpose(2, 4) + torch.einsum("eicjc,ab->eiajb", P, eye))
    dof = torch.from_numpy((3 * (m["conn"][:, :, None] - 1) + np.arange(3)).reshape(len(xe), 24)).long().to(dev)
    r, c = dof[:, :, None].expand(-1, 24, 24).reshape(-1), dof[:, None, :].expand(-1, 24, 24).reshape(-1)
    bc = torch.from_numpy(m["bc"]).to(dev) != 0
    v = ke.reshape(-1) * ~(bc[r] | bc[c])
    d = torch.nonzero(bc).reshape(-1)
    n = len(m["bc"])
    idx = torch.cat([torch.stack([r, c]), torch.stack([d, d])], 1)
    return torch.sparse_coo_tensor(idx, torch.cat([v, torch.ones(len(d), dtype=torch.float64, device=dev)]), (n, n)).coalesce().to_sparse_csr()


def _exact_damage(case, seed):
    """Every temporal point of every Gauss point in turn: elastic predictor
    and, above the yield stress, the plastic corrector with stored energy and
    damage of the two-scale model."""
    CY, H, SD, SIGF = 1740.0, 0.2, 0.5, 180.0
    WD = (577.0 - SIGF) * 0.08
    ne, nn, a, st = _damage_inputs(case, seed)
    ngp = 8 * ne
    nd = a["nodes"].reshape(ngp, 8) - 1
    sol = a["sol"].reshape(6, nn, 3)
    bx, by, bz = (a[k].reshape(ngp, 8) for k in ("Nx", "Ny", "Nz"))
    basis = np.zeros((6, ngp, 6))
    for k in range(6):
        u0, u1, u2 = (sol[k][nd][:, :, c] for c in range(3))
        for c, v in enumerate((bx * u0, by * u1, bz * u2, by * u0 + bx * u1, bz * u1 + by * u2, bz * u0 + bx * u2)):
            basis[k, :, c] = v.sum(1)
    s = {k: v.reshape(ngp, 6).copy() if k in STATE6 else v.copy() for k, v in st.items()}
    E, v = E0, NU0
    ca, cb = (1 + v) / (3 * (1 - v)), 2 * (4 - 5 * v) / (15 * (1 - v))
    G, Kb, coef = E / (2 * (1 + v)), E / (3 * (1 - 2 * v)), E / ((1 + v) * (1 - 2 * v))
    Dm = np.zeros((6, 6))
    Dm[:3, :3] = coef * v
    Dm[range(3), range(3)] = coef * (1 - v)
    Dm[range(3, 6), range(3, 6)] = coef * (1 - 2 * v) / 2
    wq = np.array([1.5, 1.5, 1.5, 3, 3, 3])
    n3 = np.array([1.0, 1, 1, 0, 0, 0])

    def dev(t):
        return t - np.outer(t[:, :3].sum(1) / 3, n3)

    def equiv(t):
        return np.sqrt((wq * t * t).sum(1))

    Nt = a["Nt"].reshape(-1, 6)
    for j in range(case["nip"]):
        eps = np.tensordot(Nt[j], basis, 1)
        d = s["D"]
        c1, c3 = 1 / (1 - cb * d), cb * (1 - d) / (1 - cb * d)
        c2 = (ca - cb) * d / ((1 - cb * d) * (1 - ca * d))
        tee = c1[:, None] * eps + c3[:, None] * s["eps_pl"] + np.outer(c2 * eps[:, :3].sum(1) / 3, n3) - s["eps_pl"]
        tse = tee @ Dm
        teq = equiv(dev(tse) - s["sig_back"])
        el = teq <= SIGF
        pl = np.flatnonzero(~el)
        new = dict(sig_eff=tse, eps_old=eps, sig_d=teq)
        old = {k: s[k][pl].copy() for k in s}
        for k in new:
            s[k][el] = new[k][el]
        if not len(pl):
            continue
        o, d, ep = old, old["D"], eps[pl]
        de = ep - o["eps_old"]
        c4 = Kb * (ca - cb) * d / ((1 - cb * d) * (1 - ca * d))
        ds = (de @ Dm) / (1 - cb * d)[:, None] + np.outer(c4 * de[:, :3].sum(1), n3)
        qs = o["sig_back"] - o["sig_eff"] - ds
        gam = CY * (1 - d) + 3 * G * (1 - cb) / (1 - cb * d)
        dq, trs = dev(qs), -qs[:, :3].sum(1) / 3
        dp = (equiv(dq) - SIGF) / gam
        dsg = -dq / (1 + gam * dp / SIGF)[:, None]
        dpl = 1.5 * dsg * (dp / SIGF)[:, None]
        o["p"] += dp
        o["eps_pl"] += dpl
        o["sig_back"] += 2 * (CY * (1 - d) / 3)[:, None] * dpl
        o["sig_eff"] = dsg + np.outer(trs, n3) + o["sig_back"]
        seq = equiv(dev(o["sig_eff"]))
        o["ws"] += (np.abs(seq - SIGF) * dp + np.abs(o["sig_d"] - SIGF) * o["del_po"]) / 2
        x = (1 - d) / (1 - H * d)
        sp, sn, tr = np.maximum(o["sig_eff"][:, :3], 0), np.minimum(o["sig_eff"][:, :3], 0), o["sig_eff"][:, :3].sum(1)
        yp = (1 + v) / (2 * E) * ((sp * sp).sum(1) + H * x * x * (sn * sn).sum(1))
        yn = v / (2 * E) * tr * tr * np.where(tr >= 0, 1.0, H * x * x)
        o["D"] = np.where(o["ws"] >= WD, d + np.sqrt(np.maximum(yp - yn, 0) / SD) * dp, 0.0)
        o["eps_old"], o["sig_d"], o["del_po"] = ep, seq, dp
        for k in s:
            s[k][pl] = o[k]
    return {k: s[k].reshape(-1) for k in STATE6 + STATE1}


def exact(case, seed):
    path = case["path"]
    rng = np.random.default_rng(seed)
    if path in ("damage", "damage_host"):
        nn, ne, _ = _sizes(*_at(case))
        return _exact_damage(case, seed) if 8 * ne * case["nip"] < 6e6 else None
    if path in ("slab", "batch", "thermal"):
        return None
    m = _model(*_at(case))
    n = 6 * m["K"].n
    if path in ("apply", "lusol", "assemble"):
        A, B = _temporal(seed % 7)
        x = rng.standard_normal(n)
    if path == "apply":
        y = _kron(_csr(m["K"]), _csr(m["M"]), A, B, x)
        return y + case["beta"] * rng.standard_normal(n) if case["beta"] else y
    if path == "lusol":
        return _exact_lusol(*_factor(*_at(case)), A, x)
    if path == "assemble":
        ym, nu = E0 * rng.uniform(0.9, 1.0, (len(m["conn"]), 8)), NU0 * rng.uniform(0.95, 1.05, (len(m["conn"]), 8))
        return _kron(_exact_k(m, ym, nu), _csr(m["M"]), A, B, x)
    if n > 9000:
        return None
    A, B = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in _temporal())
    S = torch.kron(A, _csr(m["K"]).to_dense()) + torch.kron(B, _csr(m["M"]).to_dense())
    return [torch.linalg.solve(S, torch.from_numpy(_load(m, rng)).cuda()).cpu().numpy(), None]
