"""Cases by which the speed of the library is followed.

A case is one call (or one short analysis) as a user's program makes it, with the
mesh, the model and the matrix structure in hand: the LinearStatic solve of one
mesh with each linear solver, a batch of RVEs with several load cases, Newton
increments of a J2 block and of a batch of damage cubes, and the two element
loops a Newton iteration is made of. Sizes run from the smallest decks of the
tests to the 3-million-DOF cantilever of the benchmark.

`exact` restates the element formulas (8-node hexahedron with 2x2x2 Gauss points,
4-node plane-stress quadrilateral with the shear row taken at the element centre,
4-node tetrahedron; linear elasticity and J2 plasticity with linear hardening) in
plain torch, in 64 bits.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from oofem_gb300 import meshgen as mg
from oofem_gb300 import native

J2 = dict(E=210e9, nu=0.3, sig0=250e6, H=2e9)
EPS_Y = J2["sig0"] / J2["E"]
IDM = dict(E=30e9, nu=0.2, e0=1e-4, gf=100.0)
MAXIT = 200000


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest decks of the test suite: latency and launches only
        dict(name="hex_static_tiny", kind="static", mesh="hex", nx=6, ny=3, nz=3, solver="pcg", precision="fp64",
             rtol=1e-12),
        # a small part model solved with the drop-in FP64 PCG
        dict(name="hex_static_30k", kind="static", mesh="hex", nx=60, ny=12, nz=12, solver="pcg", precision="fp64",
             rtol=1e-12),
        # a mid-sized part, mixed precision, odd sides
        dict(name="hex_static_mixed_130k", kind="static", mesh="hex", nx=101, ny=21, nz=19, solver="pcg",
             precision="mixed", rtol=1e-9),
        # the benchmark's cantilever: the largest single solve
        dict(name="hex_static_mixed_3m", kind="static", mesh="hex", nx=290, ny=58, nz=58, solver="pcg",
             precision="mixed", rtol=1e-8),
        # decks without `lstype` run the direct solver: a small one ...
        dict(name="hex_direct_3k", kind="static", mesh="hex", nx=25, ny=5, nz=6, solver="direct", precision="fp64",
             rtol=1e-12),
        # ... and one at the upper end of what a Skyline factorization is used for
        dict(name="hex_direct_30k", kind="static", mesh="hex", nx=60, ny=12, nz=12, solver="direct",
             precision="fp64", rtol=1e-12),
        # CG with the incomplete-Cholesky preconditioner (lsprecond 4)
        dict(name="hex_ic_5k", kind="static", mesh="hex", nx=33, ny=7, nz=6, solver="ic", precision="fp64",
             rtol=1e-12),
        # homogenisation sweep: RVEs of random sides, three load cases each, one batched solve
        dict(name="rve_batch", kind="rve", count=64, side_min=32, side_max=160, nrhs=3, precision="mixed",
             rtol=1e-11),
        # displacement-driven J2 block, full Newton, three increments into plasticity
        dict(name="j2_block_steps", kind="j2", nx=40, ny=8, nz=8, increments=3, precision="fp64", lin_rtol=1e-10),
        # damage on tets, a batch of seeds, the first increments
        dict(name="idm1_batch_steps", kind="idm1", n=10, seeds=4, increments=2, precision="mixed", lin_rtol=1e-10),
        # residual evaluation of a Newton iteration (radial return at every Gauss point)
        dict(name="j2_forces", kind="forces", mesh="hex", material="j2", nx=101, ny=37, nz=37),
        # tangent assembly of a Newton iteration and one product with it
        dict(name="j2_tangent", kind="tangent", mesh="hex", material="j2", nx=75, ny=31, nz=31),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _beam(rng, lo, hi):
    """nx, ny, nz of a beam with about lo..hi nodes, three to six times as long as wide."""
    nodes, ratio = _log(rng, lo, hi), rng.uniform(3.0, 6.0)
    side = (nodes / ratio) ** (1.0 / 3.0)
    return (max(2, int(ratio * side)), max(2, int(side * rng.uniform(0.8, 1.1))),
            max(2, int(side * rng.uniform(0.8, 1.1))))


def draw(rng):
    kind = rng.choice(["static", "static", "static", "direct", "ic", "rve", "j2", "idm1", "forces", "tangent"])
    if kind == "static":
        mesh = rng.choice(["hex", "hex", "tet", "quad"])
        precision = rng.choice(["fp64", "mixed"])
        c = dict(kind="static", mesh=mesh, solver="pcg", precision=precision,
                 rtol=1e-12 if precision == "fp64" else 1e-9 if mesh == "hex" else 1e-11)
        if mesh == "hex":
            c["nx"], c["ny"], c["nz"] = _beam(rng, 60, 400000 if precision == "mixed" else 100000)
        elif mesh == "tet":
            c["nx"] = c["ny"] = c["nz"] = int(_log(rng, 3, 40))
        else:
            c["nx"] = c["ny"] = int(_log(rng, 8, 257))
            c["nz"] = 0
        return c
    if kind == "direct":
        nx, ny, nz = _beam(rng, 100, 11000)
        return dict(kind="static", mesh="hex", nx=nx, ny=ny, nz=nz, solver="direct", precision="fp64", rtol=1e-12)
    if kind == "ic":
        nx, ny, nz = _beam(rng, 80, 5000)
        return dict(kind="static", mesh="hex", nx=nx, ny=ny, nz=nz, solver="ic", precision="fp64", rtol=1e-12)
    if kind == "rve":
        lo = int(_log(rng, 8, 64))
        return dict(kind="rve", count=int(_log(rng, 2, 96)), side_min=lo, side_max=int(lo * rng.uniform(1.5, 4.0)),
                    nrhs=rng.choice([1, 2, 3, 3, 4]), **rng.choice([dict(precision="mixed", rtol=1e-11)] * 2
                                                                   + [dict(precision="fp64", rtol=1e-12)]))
    if kind == "j2":
        nx, ny, nz = _beam(rng, 80, 12000)
        return dict(kind="j2", nx=nx, ny=ny, nz=nz, increments=rng.choice([2, 3]),
                    precision=rng.choice(["fp64", "mixed"]), lin_rtol=1e-10)
    if kind == "idm1":
        return dict(kind="idm1", n=int(_log(rng, 3, 12)), seeds=rng.randint(1, 6), increments=2,
                    precision=rng.choice(["mixed", "fp64"]), lin_rtol=1e-10)
    mesh = rng.choice(["hex", "hex", "tet"])
    c = dict(kind=kind, mesh=mesh, material=rng.choice(["j2", "j2", "elastic"]))
    if mesh == "hex":
        c["nx"], c["ny"], c["nz"] = _beam(rng, 200, 150000 if kind == "forces" else 80000)
    else:
        c["nx"] = c["ny"] = c["nz"] = int(_log(rng, 4, 48))
    return c


# ----------------------------------------------------------------------------- inputs
_CTX = []


def _context():
    if not _CTX:
        _CTX.append(native.Context(0))
    return _CTX[0]


def _precision(case):
    return native.PREC_MIXED if case["precision"] == "mixed" else native.PREC_FP64


def _static_mesh(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["mesh"] == "hex":
        m = mg.hex_cantilever(nx, ny, nz, jitter=0.2, seed=seed)
        m.nodal_load *= rng.uniform(0.5, 2.0)
    elif case["mesh"] == "tet":
        m = mg.tet_cube_linear(nx, jitter=0.15, seed=seed, end_disp=1e-4 * rng.uniform(0.5, 2.0))
    else:
        m = mg.quad_rve(nx, seed=seed, load_case=seed % 3)
        m.bc_value *= rng.uniform(0.5, 2.0)
    return m


def _field_mesh(case, seed):
    """Mesh of the element-loop cases and two displacement fields on it: the last converged one and the trial one."""
    rng = np.random.default_rng(seed)
    j2 = mg.Material(mg.MAT_MISES, J2["E"], J2["nu"], sig0=J2["sig0"], H=J2["H"])
    mat = j2 if case["material"] == "j2" else mg.Material(mg.MAT_ISOLE, J2["E"], J2["nu"])
    if case["mesh"] == "hex":
        m = mg.hex_block_pull(case["nx"], case["ny"], case["nz"], jitter=0.1, seed=seed, material=mat)
    else:
        m = mg.tet_cube(case["nx"], jitter=0.1, seed=seed, material=mat)
    h = 0.05 if case["mesh"] == "hex" else 1.0 / case["nx"]
    # stretch along x that passes yield over part of the mesh, with a little noise
    x = m.coords[:, 0] / max(m.coords[:, 0].max(), 1e-30)
    s1, s2 = rng.uniform(0.6, 0.9), rng.uniform(1.4, 1.8)
    base = np.zeros((m.nnodes, 3))
    base[:, 0] = EPS_Y * m.coords[:, 0] * (0.5 + x)
    base[:, 1:] = -0.3 * EPS_Y * m.coords[:, 1:]
    noise = lambda: rng.uniform(-0.05, 0.05, (m.nnodes, 3)) * EPS_Y * h  # noqa: E731
    return m, s1 * base + noise(), s2 * base + noise(), rng.uniform(-1.0, 1.0, m.nfree)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    s = dict(case=case, ctx=ctx)
    if kind == "static":
        m = _static_mesh(case, seed)
        s["bc"], s["load"] = _pinned(m.bc_value), _pinned(m.nodal_load)
        s["out"] = (_pinned(np.zeros_like(m.bc_value)), _pinned(np.zeros_like(m.bc_value)))
    elif kind == "rve":
        sides = np.random.default_rng(case["count"]).integers(case["side_min"], case["side_max"] + 1, case["count"])
        meshes = [mg.quad_rve(int(n), seed=seed * 100003 + i) for i, n in enumerate(sides)]
        m, starts = mg.concat_meshes(meshes)
        s["bc"] = np.stack([np.concatenate([mg.rve_bc_values(q, lc % 3) * (1.0 + lc // 3) for q in meshes])
                            for lc in range(case["nrhs"])])
    elif kind == "j2":
        nx = case["nx"]
        m = mg.hex_block_pull(nx, case["ny"], case["nz"], jitter=0.1, seed=seed,
                              material=mg.Material(mg.MAT_MISES, J2["E"], J2["nu"], sig0=J2["sig0"], H=J2["H"]),
                              end_disp=2.0 * EPS_Y * nx * 0.05)
    elif kind == "idm1":
        mat = mg.Material(mg.MAT_IDM1, IDM["E"], IDM["nu"], e0=IDM["e0"], gf=IDM["gf"])
        meshes = [mg.tet_cube(case["n"], jitter=0.15, seed=seed * 1009 + i, material=mat, end_disp=IDM["e0"])
                  for i in range(case["seeds"])]
        m, starts = mg.concat_meshes(meshes)
    else:
        m, u1, u2, x = _field_mesh(case, seed)
    model = native.GpuModel(ctx, m)
    if kind in ("rve", "idm1"):
        model.set_instances(starts)
    A = native.GpuCsrMtrx(ctx)
    if kind != "forces":
        model.build_matrix(A)
    if kind == "static":
        if case["solver"] == "direct":
            A.set_solver(native.LS_DIRECT)
        elif case["solver"] == "ic":
            A.set_preconditioner(4)
    elif kind in ("j2", "idm1"):
        model.set_initial_guess(1)
    elif kind in ("forces", "tangent"):
        # the committed state of the last converged step; the trial field is what an iteration evaluates
        model.internal_forces(u1)
        model.commit_state()
        if kind == "tangent":
            model.internal_forces(u2)
            s["x"] = torch.from_numpy(x).cuda()
            s["y"] = torch.zeros_like(s["x"])
        else:
            s["u"] = torch.from_numpy(u2).cuda()
            s["f"] = torch.zeros_like(s["u"])
    s.update(mesh=m, model=model, A=A)
    torch.cuda.synchronize()
    return s


# ----------------------------------------------------------------------------- one pass
def _check(ctx, code):
    if code != 0:
        raise native.OgbError(code, ctx.lib.ogb_last_error().decode())


def run(s):
    case, kind, m, model, A = s["case"], s["case"]["kind"], s["mesh"], s["model"], s["A"]
    if kind == "static":
        u, reac, info = model.linear_static(A, s["bc"], s["load"], rtol=case["rtol"], maxit=MAXIT,
                                            precision=_precision(case), out=s["out"])
        _check(s["ctx"], info.status)
        return {"u": u, "reactions": reac}
    if kind == "rve":
        u, reac, _, _, status = model.batch_linear_static(A, s["bc"], None, rtol=case["rtol"], maxit=MAXIT,
                                                          precision=_precision(case))
        return {"u": u, "reactions": reac, "status": status}
    if kind in ("j2", "idm1"):
        model.reset_state()
        step = model.nonlinear_step if kind == "j2" else model.batch_nonlinear_step
        outs = []
        for k in range(1, case["increments"] + 1):
            u, reac, _ = step(A, m.bc_value * (k / case["increments"]), None, rtolf=1e-8 if kind == "j2" else 1e-6,
                              maxiter=400, lin_rtol=case["lin_rtol"], precision=_precision(case))
            outs += [u, reac]
        return outs
    lib, p = s["ctx"].lib, lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    if kind == "forces":
        _check(s["ctx"], lib.ogb_model_internal_forces_dev(model.h, p(s["u"]), p(s["f"])))
        return s["f"]
    model.assemble_stiffness(A)
    _check(s["ctx"], lib.ogb_mtrx_times_dev(A.h, p(s["x"]), p(s["y"])))
    return s["y"]


# ----------------------------------------------------------------------------- what a pass cannot do without
def _sizes(case):
    """nodes, elements, DOFs per node, nodes per element, Gauss points, node blocks per row."""
    mesh = case.get("mesh", {"rve": "quad", "idm1": "tet"}.get(case["kind"], "hex"))
    if mesh == "quad":
        if case["kind"] == "rve":
            side = 0.5 * (case["side_min"] + case["side_max"])
            return case["count"] * (side + 1) ** 2, case["count"] * side * side, 2, 4, 4, 9
        return (case["nx"] + 1) ** 2, case["nx"] ** 2, 2, 4, 4, 9
    if mesh == "tet":
        n, k = (case["n"], case["seeds"]) if case["kind"] == "idm1" else (case["nx"], 1)
        return k * (n + 1) ** 3, k * 6 * n ** 3, 3, 4, 1, 15
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz, 3, 8, 8, 27


def work(case):
    nodes, elems, nd, nnpe, ngp, blocks = _sizes(case)
    n, ns = nodes * nd, 3 if nd == 2 else 6
    mesh_bytes = nodes * (8 * nd + 4 * nd) + elems * (nnpe * 4 + 4)
    nnz = n * blocks * nd
    state = elems * ngp * 7 * 8   # plastic strain and hardening variable of a Gauss point
    # element forces: gradients, strain, stress and B^T sigma; element tangents: the two products of B^T D B by
    # their non-zero entries, the symmetric half
    f_forces = elems * ngp * (nnpe * nd * 9 + 120)
    f_tangent = elems * ngp * (nnpe * nd * 2 * ns * 2 + 0.5 * nnpe * nnpe * nd * nd * 6 + 120)
    if case["kind"] == "forces":
        return {"bytes": mesh_bytes + 2 * n * 8 + (2 * state if case["material"] == "j2" else 0)
                + elems * ngp * ns * 16, "flops": f_forces}
    if case["kind"] == "tangent":
        return {"bytes": mesh_bytes + nnz * 8 + 2 * n * 8 + (2 * state if case["material"] == "j2" else 0),
                "flops": f_tangent + 2 * nnz}
    value = 4 if case["precision"] == "mixed" else 8
    # CG iterations grow with the length of the mesh in elements (about 11 per element to 1e-8 on a cantilever)
    if case["kind"] == "static":
        if case["solver"] == "direct":
            bw = nd * (case["nx"] + 1) * (case["ny"] + 1) + 2 * nd
            return {"bytes": mesh_bytes + 2 * n * min(n, bw) * 8 + 4 * n * 8, "flops": n * min(n, bw) ** 2}
        iters = {"hex": 11.0, "tet": 4.5, "quad": 3.5}[case["mesh"]] * case["nx"]
        iters *= 0.3 if case["solver"] == "ic" else 1.0
        per = (nnz * value * (2 if case["solver"] == "ic" else 1), nnz * (4 if case["solver"] == "ic" else 2))
        return {"bytes": mesh_bytes + 4 * n * 8 + iters * per[0], "flops": f_tangent + 2 * f_forces + iters * per[1]}
    if case["kind"] == "rve":
        iters = 3.5 * 0.5 * (case["side_min"] + case["side_max"])
        return {"bytes": mesh_bytes + case["nrhs"] * 2 * n * 8 + iters * nnz * value,
                "flops": f_tangent + case["nrhs"] * (2 * f_forces + iters * 2 * nnz)}
    newton = 4 * case["increments"]
    iters = 11.0 * case["nx"] if case["kind"] == "j2" else 6.0 * case["n"]
    return {"bytes": newton * (mesh_bytes + 2 * state + iters * nnz * value),
            "flops": newton * (f_tangent + f_forces + iters * 2 * nnz)}


# ----------------------------------------------------------------------------- 64-bit values in plain torch
_HEX = [(-1, -1, 1), (-1, 1, 1), (1, 1, 1), (1, -1, 1), (-1, -1, -1), (-1, 1, -1), (1, 1, -1), (1, -1, -1)]
_QUAD = [(1, 1), (-1, 1), (-1, -1), (1, -1)]
_G = 0.577350269189626


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _gradients(x, dn):
    """Gradients (e, node, dim) and Jacobian determinant (e) from nodes x (e, node, dim) and dn (node, dim)."""
    J = torch.einsum("eni,nj->eij", x, dn)
    return torch.einsum("nj,eji->eni", dn, torch.linalg.inv(J)), torch.linalg.det(J)


def _points(m, lo, hi):
    """(B, dV) of every Gauss point of the elements lo..hi: B (e, ns, node * nd), dV (e)."""
    x = _t(m.coords)[_t(m.conn[lo:hi], torch.int64)]
    e = x.shape[0]
    if m.elem_type == mg.ELEM_PLANESTRESS2D:
        corner = _t(np.array(_QUAD, float))

        def dn(p):
            return 0.25 * torch.stack([corner[:, 0] * (1 + p[1] * corner[:, 1]),
                                       corner[:, 1] * (1 + p[0] * corner[:, 0])], 1)
        g0, _ = _gradients(x, dn((0.0, 0.0)))
        for a in (-_G, _G):
            for b in (-_G, _G):
                g, det = _gradients(x, dn((a, b)))
                B = torch.zeros(e, 3, 4, 2, dtype=torch.float64, device="cuda")
                B[:, 0, :, 0], B[:, 1, :, 1] = g[:, :, 0], g[:, :, 1]
                B[:, 2, :, 0], B[:, 2, :, 1] = g0[:, :, 1], g0[:, :, 0]
                yield B.reshape(e, 3, 8), det.abs() * m.thickness
        return
    if m.elem_type == mg.ELEM_LTRSPACE:
        dn = _t([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
        points = [_gradients(x, dn) + (1.0 / 6.0,)]
    else:
        corner = _t(np.array(_HEX, float))
        points = []
        for a in (-_G, _G):
            for b in (-_G, _G):
                for c in (-_G, _G):
                    f = [1 + q * corner[:, i] for i, q in enumerate((a, b, c))]
                    dn = 0.125 * torch.stack([corner[:, 0] * f[1] * f[2], corner[:, 1] * f[0] * f[2],
                                              corner[:, 2] * f[0] * f[1]], 1)
                    points.append(_gradients(x, dn) + (1.0,))
    for g, det, w in points:
        B = torch.zeros(e, 6, g.shape[1], 3, dtype=torch.float64, device="cuda")
        for i in range(3):
            B[:, i, :, i] = g[:, :, i]
        for row, (i, j) in zip((3, 4, 5), ((1, 2), (0, 2), (0, 1))):
            B[:, row, :, i], B[:, row, :, j] = g[:, :, j], g[:, :, i]
        yield B.reshape(e, 6, -1), det.abs() * w


def _elastic(m):
    """D of every material (nmat, ns, ns)."""
    out = []
    for q in m.materials:
        if m.elem_type == mg.ELEM_PLANESTRESS2D:
            f = q.E / (1 - q.nu ** 2)
            out.append(np.array([[f, f * q.nu, 0], [f * q.nu, f, 0], [0, 0, q.E / (2 * (1 + q.nu))]]))
        else:
            G, lam = q.E / (2 * (1 + q.nu)), q.E * q.nu / ((1 + q.nu) * (1 - 2 * q.nu))
            D = np.diag([2 * G] * 3 + [G] * 3)
            D[:3, :3] += lam
            out.append(D)
    return _t(np.stack(out))


def _j2_trial(eps, pl):
    G, K = J2["E"] / (2 * (1 + J2["nu"])), J2["E"] / (3 * (1 - 2 * J2["nu"]))
    el = eps - pl
    mean = el[:, :3].sum(1, keepdim=True) / 3
    s = torch.cat([2 * G * (el[:, :3] - mean), G * el[:, 3:]], 1)
    norm = torch.sqrt((s[:, :3] ** 2).sum(1) + 2 * (s[:, 3:] ** 2).sum(1))
    return s, 3 * K * mean, norm, G, K


def _j2_stress(eps, pl, kappa):
    """Stress, plastic strain and hardening variable after the radial return."""
    s, vol, norm, G, _ = _j2_trial(eps, pl)
    over = math.sqrt(1.5) * norm - (J2["sig0"] + J2["H"] * kappa)
    dk = torch.clamp(over, min=0) / (J2["H"] + 3 * G)
    n = s / torch.where(norm > 0, norm, torch.ones_like(norm))[:, None]
    twice = _t([1, 1, 1, 2, 2, 2])
    pl = pl + math.sqrt(1.5) * dk[:, None] * n * twice
    s = s - math.sqrt(6.0) * G * dk[:, None] * n
    return torch.cat([s[:, :3] + vol, s[:, 3:]], 1), pl, kappa + dk


def _j2_tangent(eps, pl, kappa, D):
    """Consistent tangent of the radial return (the derivative of _j2_stress by eps)."""
    s, _, norm, G, _ = _j2_trial(eps, pl)
    dk = torch.clamp(math.sqrt(1.5) * norm - (J2["sig0"] + J2["H"] * kappa), min=0) / (J2["H"] + 3 * G)
    on = (dk > 0).to(torch.float64)
    norm = torch.where(norm > 0, norm, torch.ones_like(norm))
    n = s / norm[:, None]
    dev = torch.zeros(6, 6, dtype=torch.float64, device="cuda")
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    dev[:3, :3], dev[3:, 3:] = eye - 1.0 / 3.0, 0.5 * eye
    theta = math.sqrt(6.0) * G * dk / norm            # share of the trial deviator that is taken back
    slope = 3.0 * G / (J2["H"] + 3 * G)               # of the norm's own change
    nn = n[:, :, None] * n[:, None, :]
    return (D - (2 * G * theta * on)[:, None, None] * dev + (2 * G * (theta - slope) * on)[:, None, None] * nn)


def _dofs(m, lo, hi):
    c = _t(m.conn[lo:hi], torch.int64)
    return (c[:, :, None] * m.ndofpn + torch.arange(m.ndofpn, device="cuda")).reshape(c.shape[0], -1)


_CHUNK = 1 << 15


def _forces(m, u, state=None):
    """Internal forces (nodes x nd) of the field u; state: list of (plastic strain, kappa) by chunk and point."""
    u, f, D = _t(u).reshape(-1), torch.zeros(m.nnodes * m.ndofpn, dtype=torch.float64, device="cuda"), _elastic(m)
    new = []
    for lo in range(0, m.nelem, _CHUNK):
        hi = min(m.nelem, lo + _CHUNK)
        dof, mat, points = _dofs(m, lo, hi), _t(m.elem_mat[lo:hi], torch.int64), []
        for p, (B, dV) in enumerate(_points(m, lo, hi)):
            eps = torch.einsum("eij,ej->ei", B, u[dof])
            if state is None:
                sig = torch.einsum("eij,ej->ei", D[mat], eps)
            else:
                sig, pl, kappa = _j2_stress(eps, *state[lo // _CHUNK][p])
                points.append((pl, kappa))
            f.index_add_(0, dof.reshape(-1), (torch.einsum("eij,ei->ej", B, sig) * dV[:, None]).reshape(-1))
        new.append(points)
    return f.reshape(m.nnodes, m.ndofpn), new


def _virgin(m):
    z = []
    for lo in range(0, m.nelem, _CHUNK):
        e = min(m.nelem, lo + _CHUNK) - lo
        one = (torch.zeros(e, 6, dtype=torch.float64, device="cuda"), torch.zeros(e, dtype=torch.float64, device="cuda"))
        z.append([one] * (8 if m.elem_type == mg.ELEM_LSPACE else 1))
    return z


def _element_matrices(m, u=None, state=None):
    """(Ke, dofs) by chunk: elastic, or the consistent tangent at the field u from the committed state."""
    D = _elastic(m)
    for lo in range(0, m.nelem, _CHUNK):
        hi = min(m.nelem, lo + _CHUNK)
        dof, K = _dofs(m, lo, hi), 0.0
        Dm = D[_t(m.elem_mat[lo:hi], torch.int64)]
        for p, (B, dV) in enumerate(_points(m, lo, hi)):
            Dp = Dm if state is None else _j2_tangent(torch.einsum("eij,ej->ei", B, _t(u).reshape(-1)[dof]),
                                                      *state[lo // _CHUNK][p], Dm)
            K = K + torch.einsum("eki,ekl,elj->eij", B, Dp * dV[:, None, None], B)
        yield K, dof


def _matrix(m, free):
    """The stiffness of the free DOFs as a CSR tensor, from the elements."""
    number = torch.full((m.nnodes * m.ndofpn,), -1, dtype=torch.int64, device="cuda")
    n = int(free.sum())
    number[free] = torch.arange(n, device="cuda")
    K = torch.sparse_coo_tensor(torch.zeros(2, 0, dtype=torch.int64, device="cuda"),
                                torch.zeros(0, dtype=torch.float64, device="cuda"), (n, n))
    for Ke, dof in _element_matrices(m):
        d = number[dof]
        i, j = d[:, :, None].expand_as(Ke).reshape(-1), d[:, None, :].expand_as(Ke).reshape(-1)
        keep = (i >= 0) & (j >= 0)
        K = (K + torch.sparse_coo_tensor(torch.stack([i[keep], j[keep]]), Ke.reshape(-1)[keep], (n, n))).coalesce()
    return K.to_sparse_csr()


def _solve(K, b):
    """K x = b: Cholesky with two steps of refinement, or diagonal CG run until the residual no longer falls."""
    n = b.shape[0]
    if n <= 12000:
        full = K.to_dense()
        L = torch.linalg.cholesky(full)
        x = torch.zeros_like(b)
        for _ in range(3):
            x = x + torch.cholesky_solve((b - full @ x)[:, None], L)[:, 0]
        return x
    i = torch.repeat_interleave(torch.arange(n, device="cuda"), K.crow_indices().diff())
    on = K.col_indices() == i
    diag = torch.zeros_like(b)
    diag[i[on]] = K.values()[on]
    x = torch.zeros_like(b)
    for _ in range(3):   # restarted from the true residual
        r = b - K @ x
        tol = 1e-15 * float(b.norm())
        z = r / diag
        p, rho, k = z.clone(), torch.dot(r, z), 0
        while k < 20000:
            q = K @ p
            alpha = rho / torch.dot(p, q)
            x, r = x + alpha * p, r - alpha * q
            k += 1
            if k % 50 == 0 and float(r.norm()) <= tol:
                break
            z = r / diag
            new = torch.dot(r, z)
            p, rho = z + (new / rho) * p, new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "static":
        if _sizes(case)[0] * _sizes(case)[2] > 150000:
            return None   # too long in plain torch
        m = _static_mesh(case, seed)
        mask = _t(m.bc_mask.reshape(-1), torch.int64) == 1
        u = torch.where(mask, _t(m.bc_value).reshape(-1), torch.zeros_like(_t(m.bc_value).reshape(-1)))
        load = _t(m.nodal_load).reshape(-1)
        f0, _ = _forces(m, u.cpu().numpy().reshape(m.nnodes, -1))
        u[~mask] = _solve(_matrix(m, ~mask), (load - f0.reshape(-1))[~mask])
        f, _ = _forces(m, u.cpu().numpy().reshape(m.nnodes, -1))
        reac = torch.where(mask, f.reshape(-1) - load, torch.zeros_like(load))
        return {"u": u.reshape(m.nnodes, -1).cpu().numpy(), "reactions": reac.reshape(m.nnodes, -1).cpu().numpy()}
    if kind in ("forces", "tangent"):
        m, u1, u2, x = _field_mesh(case, seed)
        j2 = case["material"] == "j2"
        state = _forces(m, u1, _virgin(m))[1] if j2 else None
        if kind == "forces":
            return _forces(m, u2, state)[0]
        free = _t(m.bc_mask.reshape(-1), torch.int64) == 0
        v = torch.zeros(m.nnodes * m.ndofpn, dtype=torch.float64, device="cuda")
        v[free] = _t(x)
        y = torch.zeros_like(v)
        for Ke, dof in _element_matrices(m, u2, state):
            y.index_add_(0, dof.reshape(-1), torch.einsum("eij,ej->ei", Ke, v[dof]).reshape(-1))
        return y[free]
    return None   # whole Newton analyses and batches: their ends are set by the solvers' own tolerances
