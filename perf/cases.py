"""Timed workloads of the library, from its smallest calls to whole time steps.

Every case goes through the public entry points (the Python mirror, or the
C-ABI with device pointers where the mirror takes host arrays only) with the
settings of the repository's configurations: RosRK3, dt = 2 s (1 s for the
warm bubble), Krylov tolerances 1e-10 (the plain FP64 dynamical steps: 1e-6, the
model's defaults), the synthetic geometries and states of
``asam_gb300.geometry``.  A step case advances its block in place, as a model
run does.
"""
import ctypes as C

import numpy as np
import torch

import asam_gb300
from asam_gb300 import _lib
from asam_gb300 import geometry as G

TOL, TOL_DEFAULT = 1e-10, 1e-6
NOT_FAILED = (0, 1, 2)  # ASAM_OK, ASAM_NOT_CONVERGED, ASAM_BREAKDOWN
TB_COEFS = dict(beta0_dtp=0.5, fac1_l=1.0, fac1_r=1.0, grav_comp=1.0, fac_anela=0.25, fac2_l=1.0, fac2_r=1.0,
                fac3_l=1.0, fac3_r=1.0)


def listed():
    return [
        # the column solver called for one small block: launch and call latency
        {"name": "columns_60x40", "kind": "columns", "ncol": 60, "n1": 40},
        # all columns of a large block at once, the entry's largest call
        {"name": "columns_32768x128", "kind": "columns", "ncol": 32768, "n1": 128},
        # advection right-hand side of a small odd-sized block, 10 components
        {"name": "flux_61x47x33", "kind": "flux", "nx": 61, "ny": 47, "nz": 33},
        # transport step of the moist cut-cell hill, plain FP64, at the largest ensemble member's size
        {"name": "transport_fp64_192x160x96", "kind": "transport", "precision": "fp64", "nx": 192, "ny": 160,
         "nz": 96},
        # transport step of the 256x256x128 hill in the mixed-precision mode
        {"name": "transport_refined_256x256x128", "kind": "transport", "precision": "fp32_refined", "nx": 256,
         "ny": 256, "nz": 128},
        # the dry warm bubble on flat ground: a full dynamical step, plain FP64
        {"name": "bubble_fp64_64x64x32", "kind": "bubble", "precision": "fp64", "nx": 64, "ny": 64, "nz": 32},
        # full dynamical step of the moist hill in the mixed-precision mode
        {"name": "dynamics_refined_256x256x64", "kind": "dynamics", "precision": "fp32_refined", "nx": 256,
         "ny": 256, "nz": 64},
        # full dynamical step of a small odd-sized hill block, plain FP64
        {"name": "dynamics_fp64_61x47x29", "kind": "dynamics", "precision": "fp64", "nx": 61, "ny": 47, "nz": 29},
        # pressure projection alone, of a closed block with odd sizes: hierarchy assembly and one sound solve
        {"name": "project_125x93x61", "kind": "project", "nx": 125, "ny": 93, "nz": 61},
        # checkpointed gradient with respect to the initial tracer (forward, recomputation and reverse sweep)
        {"name": "gradient_128x128x64", "kind": "gradient", "nx": 128, "ny": 128, "nz": 64, "steps": 4, "every": 2},
        # uneven members advanced together, mixed precision
        {"name": "ensemble_refined_4", "kind": "ensemble", "precision": "fp32_refined", "members": 4, "steps": 2,
         "sizes": 4},
        # one V-cycle of the density-coupled 2x2-block preconditioner, parallel order
        {"name": "blockcycle_48x96x80", "kind": "blockcycle", "coupled": False, "n3": 48, "n2": 96, "n1": 80},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    kind = rng.choice(["columns", "flux", "transport", "bubble", "dynamics", "project", "gradient", "ensemble",
                       "blockcycle"])
    if kind == "columns":
        n1 = log(16, 160)
        return {"kind": kind, "ncol": min(log(32, 32768), 4194304 // n1), "n1": n1}
    if kind == "ensemble":
        return {"kind": kind, "precision": rng.choice(["fp64", "fp32_refined"]), "members": rng.randint(2, 4),
                "steps": rng.randint(1, 2), "sizes": rng.randint(0, 999)}
    if kind == "blockcycle":
        return {"kind": kind, "coupled": rng.random() < 0.5, "n3": log(8, 48), "n2": log(16, 96), "n1": log(16, 80)}
    if kind in ("flux", "transport"):
        c = {"kind": kind, "nx": log(24, 192), "ny": log(24, 160), "nz": log(16, 96)}
    elif kind == "bubble":
        c = {"kind": kind, "nx": log(24, 64), "ny": log(24, 64), "nz": log(16, 32)}
    elif kind == "dynamics":
        c = {"kind": kind, "nx": log(24, 64), "ny": log(24, 64), "nz": log(16, 32)}
    else:
        c = {"kind": kind, "nx": log(32, 125), "ny": log(32, 93), "nz": log(24, 61)}
    if kind in ("transport", "bubble", "dynamics"):
        c["precision"] = rng.choice(["fp64", "fp32_refined"])
    if kind == "dynamics" and c["precision"] == "fp32_refined":
        c.update(nx=log(48, 256), ny=log(48, 256), nz=log(24, 64))
    if kind == "gradient":
        c.update(steps=rng.randint(2, 4), every=rng.randint(1, 2))
    return c


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _block(geo, ncomp, precision="fp64", tol=TOL, **kw):
    if precision == "fp32_refined":
        kw["inner_precond"] = "xline"
    return asam_gb300.TransportBlock(geo, ncomp, method="RosRK3", bicgstab_tol=tol, precision=precision, **kw)


def _columns(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ncol, n1 = case["ncol"], case["n1"]

    def uniform(n, lo, hi):
        return lo + (hi - lo) * torch.rand(ncol, n, generator=gen, dtype=torch.float64, device="cuda")

    d, u, lo = uniform(n1, 3.0, 3.5), uniform(n1 - 1, -1.0, 1.0), uniform(n1 - 1, -1.0, 1.0)
    b = torch.randn(ncol, n1, generator=gen, dtype=torch.float64, device="cuda")
    return d, u, lo, b


def _dyn_block(work, precision):
    geo, vel, st, pos, (dx, dy, dz), bound = work
    tol = TOL_DEFAULT if precision == "fp64" else TOL
    blk = _block(geo, st.c.shape[0], precision, tol)
    blk.set_velocity(*vel)
    blk.proj_setup(dx, dy, dz, tol=tol, max_restart=20)
    blk.dyn_setup(pos["th"], pos["mom"], rv_pos=pos.get("qv", -1), bound_cells=bound,
                  scalars=[pos[q] for q in ("qv", "tracer") if q in pos])
    return {"block": blk, "c": _cuda(st.c), "vel": [_cuda(np.empty_like(v)) for v in vel]}


def _member_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    return [(int(rng.integers(64, 193)), int(rng.integers(64, 161)), int(rng.integers(48, 97)))
            for _ in range(case["members"])]


def _box(nx, ny, nz):
    """The adjoint objective's 16x16x8 target box, downstream of the tracer's start."""
    i0, j0, k0 = int(0.3 * nx) + 1, max(1, ny // 2 - 7), max(1, nz // 8)
    return (C.c_int * 6)(i0, min(nx, i0 + 15), j0, min(ny, j0 + 15), k0, min(nz, k0 + 7))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "lib": _lib.load()}
    if kind == "columns":
        s["d"], s["u"], s["l"], s["b"] = _columns(case, seed)
        return s
    if kind == "ensemble":
        s["blocks"], s["states"] = [], []
        rng = np.random.default_rng(seed)
        for m, (nx, ny, nz) in enumerate(_member_sizes(case)):
            geo, vel, st = G.hill_case(nx, ny, nz, seed=1000 * seed + m, height=rng.uniform(0.0, 1500.0),
                                       halfwidth=rng.uniform(2000.0, 8000.0), u0=rng.uniform(5.0, 15.0),
                                       n_bv=rng.uniform(0.008, 0.012))
            blk = _block(geo, st.c.shape[0], case["precision"])
            blk.set_velocity(*vel)
            s["blocks"].append(blk)
            s["states"].append(_cuda(st.c))
        s["batch"] = asam_gb300.Batch(s["blocks"])
        return s
    if kind == "blockcycle":
        rng = np.random.default_rng(seed)
        n3, n2, n1 = case["n3"], case["n2"], case["n1"]

        def field(*shape):
            return rng.uniform(0.2, 2.0, shape)

        s["hier"] = asam_gb300.TriTBHierarchy(
            [field(n3, n2, n1 + 1) for _ in range(4)], [field(n3, n2 + 1, n1) for _ in range(4)],
            [field(n3 + 1, n2, n1) for _ in range(4)], field(n3, n2, n1), field(n3, n2, n1),
            field(n3, n2, n1) if case["coupled"] else None, ref_level=4, **TB_COEFS)
        s["hier"].set_zebra(True)
        s["b"] = _cuda(rng.standard_normal((n3, n2, n1, 2)))
        return s
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind in ("flux", "transport"):
        geo, vel, st = G.hill_case(nx, ny, nz, seed=seed)
        s["block"] = _block(geo, st.c.shape[0], case.get("precision", "fp64"))
        s["block"].set_velocity(*vel)
        s["c"] = _cuda(st.c)
        if kind == "flux":
            s["f"] = torch.empty_like(s["c"])
    elif kind == "bubble":
        s.update(_dyn_block(G.bubble_dyn_case(nx, ny, nz, seed=seed), case["precision"]))
    elif kind == "dynamics":
        s.update(_dyn_block(G.hill_dyn_case(nx, ny, nz, seed=seed), case["precision"]))
    elif kind == "project":
        geo = G.closed_hill_case(nx, ny, nz, seed=seed)
        weights, dx, dy, dz, vel = G.projection_inputs(geo, seed=seed + 1)
        blk = s["block"] = _block(geo, 3)
        blk.proj_setup(dx, dy, dz, tol=TOL, max_restart=20)
        blk.proj_weights(*weights)
        s["start"] = [_cuda(v) for v in vel]
    elif kind == "gradient":
        geo, vel, st = G.hill_case(nx, ny, nz, seed=seed, height=800.0, halfwidth=4000.0, moist=False,
                                   momentum=False)
        s["block"] = _block(geo, st.c.shape[0], bicgstab_maxiter=200)
        s["block"].set_velocity(*vel)
        s["c"] = _cuda(st.c)
        s["grad"] = torch.empty_like(s["c"][0])
    return s


def run(state):
    case, lib = state["case"], state["lib"]
    kind = case["kind"]
    if kind == "columns":
        x = state["b"].clone()
        _lib.check(lib.asam_tri_solve_noalloc(case["ncol"], case["n1"], _ptr(state["d"]), _ptr(state["u"]),
                                              _ptr(state["l"]), _ptr(x), torch.cuda.current_stream().cuda_stream),
                   "asam_tri_solve_noalloc")
        return x
    if kind == "ensemble":
        state["batch"].ros_step([c.data_ptr() for c in state["states"]], 2.0, nsteps=case["steps"])
        return state["states"]
    if kind == "blockcycle":
        x = torch.zeros_like(state["b"])
        _lib.check(lib.asam_tri_tb_hier_vcycle(state["hier"].h, _ptr(state["b"]), _ptr(x), 1, 1, 1, 1),
                   "asam_tri_tb_hier_vcycle")
        return x
    blk = state["block"]
    if kind == "flux":
        _lib.check(lib.asam_fcn(blk.h, _ptr(state["c"]), _ptr(state["f"])), "asam_fcn")
        return state["f"]
    if kind == "transport":
        blk.ros_step_device(state["c"].data_ptr(), 2.0)
        return state["c"]
    if kind in ("bubble", "dynamics"):
        it, ps, rs, pr = (C.c_int * 4)(), (C.c_int * 4)(), (C.c_double * 4)(), (C.c_double * 4)()
        _lib.check(lib.asam_ros_step_dyn(blk.h, _ptr(state["c"]), 1.0 if kind == "bubble" else 2.0, it, rs, ps, pr),
                   "asam_ros_step_dyn", allow=NOT_FAILED)
        _lib.check(lib.asam_get_velocity(blk.h, *[_ptr(v) for v in state["vel"]]), "asam_get_velocity")
        return [state["c"]] + state["vel"]
    if kind == "project":
        blk.JacAccGrav(0.435866521508459, 2.0)
        vel = [v.clone() for v in state["start"]]
        incr = torch.zeros(blk.state_shape, dtype=torch.float64, device="cuda")
        p = torch.empty(case["nz"], case["ny"], case["nx"], dtype=torch.float64, device="cuda")
        torch.cuda.current_stream().synchronize()  # the block works on a stream of its own
        steps, res = C.c_int(), C.c_double()
        _lib.check(lib.asam_project_vel_face(blk.h, *[_ptr(v) for v in vel], _ptr(incr), None, -1, -1,
                                             (C.c_int * 1)(), 0, _ptr(p), C.byref(steps), C.byref(res)),
                   "asam_project_vel_face", allow=NOT_FAILED)
        return vel + [p]
    comp = blk.ncomp - 1
    J = C.c_double()
    _lib.check(lib.asam_tracer_gradient(blk.h, _ptr(state["c"]), comp, case["steps"], 2.0, case["every"],
                                        _box(case["nx"], case["ny"], case["nz"]), TOL, C.byref(J),
                                        _ptr(state["grad"])), "asam_tracer_gradient", allow=NOT_FAILED)
    return [J.value, state["grad"]]


def work(case):
    """Bytes of the inputs and outputs; FP64 operations (FP32 ones of the
    mixed-precision mode counted alike) of one pass of the algorithm: per cell
    and component 60 for the flux, 14 a stage product, 14 a relaxation; three
    stages a step with one product and two Gauss-Seidel calls of six sweeps
    (four products and line solves in mixed precision); 520 per cell a V-cycle
    (relaxations of all levels), with the FGMRES steps such blocks take."""
    kind = case["kind"]
    if kind == "columns":
        n = case["ncol"] * case["n1"]
        return {"bytes": 40 * n, "flops": 8 * n}
    if kind == "blockcycle":
        n = case["n3"] * case["n2"] * case["n1"]
        return {"bytes": 8 * n * (7 * 4 + 4), "flops": 3000 * n}
    if kind == "ensemble":
        cells = sum(a * b * c for a, b, c in _member_sizes(case)) * case["steps"]
        return {"bytes": 8 * 10 * 2 * cells, "flops": 10 * cells * _transport_flops(case["precision"])}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "flux":
        return {"bytes": 8 * cells * (2 * 10 + 7), "flops": 60 * 10 * cells}
    if kind == "transport":
        return {"bytes": 8 * cells * (2 * 10 + 7), "flops": 10 * cells * _transport_flops(case["precision"])}
    if kind in ("bubble", "dynamics"):
        ncomp, refined = (8 if kind == "bubble" else 10), case["precision"] != "fp64"
        cycles = 3 * 9 if refined else 3 * 3 * 10
        return {"bytes": 8 * cells * (2 * ncomp + 10),
                "flops": cells * (ncomp * _transport_flops(case["precision"]) + 520 * cycles)}
    if kind == "project":
        return {"bytes": 8 * cells * (3 * 2 + 8 + 1 + 4), "flops": cells * 520 * 10}
    return {"bytes": 8 * cells * (3 + 7 + 1), "flops": cells * 3 * case["steps"] * _transport_flops("fp64")}


def _transport_flops(precision):
    return 3 * (60 + (2 * (14 + 6 * 14) if precision == "fp64" else 4 * 28))


def exact(case, seed):
    """Column solves and the advection right-hand side in plain torch; the whole
    steps, solves and cycles (Krylov solutions to a tolerance, sweeps in a
    prescribed order) have no such value within seconds."""
    if case["kind"] == "columns":
        d, u, lo, b = _columns(case, seed)
        n1 = case["n1"]
        piv, y = [d[:, 0]], [b[:, 0]]
        for i in range(1, n1):
            m = lo[:, i - 1] / piv[-1]
            piv.append(d[:, i] - m * u[:, i - 1])
            y.append(b[:, i] - m * y[-1])
        x = [None] * n1
        x[n1 - 1] = y[-1] / piv[-1]
        for i in range(n1 - 2, -1, -1):
            x[i] = (y[i] - u[:, i] * x[i + 1]) / piv[i]
        return torch.stack(x, 1)
    if case["kind"] == "flux":
        geo, vel, st = G.hill_case(case["nx"], case["ny"], case["nz"], seed=seed)
        return _advection(geo, vel, _cuda(st.c))
    return None


def _advection(geo, vel, c):
    """Upwind fluxes with the Koren-limited correction on non-uniform cut cells,
    periodic in x and y, gathered into the padded cells and divided by volume."""
    eps = 1e-30
    V = _cuda(geo.volc)
    phi = c / (c[0] + eps)
    total = torch.zeros_like(c)
    for dim, F, u, periodic in ((3, geo.fu, vel[0], True), (2, geo.fv, vel[1], True), (1, geo.fw, vel[2], False)):
        own = [q for q in (1, 2, 3) if q != dim]  # interior range of the other two axes

        def along(a):  # (components, faces or cells of the axis last)
            a = a if a.dim() == 4 else a[None]
            return a.movedim(dim, -1)

        def interior(a):
            for q in own:
                if a.shape[q] > 1:
                    a = a.narrow(q, 1, a.shape[q] - 2)
            return a

        ph, vol = along(interior(phi)), along(interior(V[None]))
        F, u = along(_cuda(F)), along(_cuda(u))
        n = ph.shape[-1] - 2

        def upwind(ph, vol, F, u):  # flux of face s from cell s, s = 1 .. n
            cL, cC, cR = ph[..., :n], ph[..., 1:n + 1], ph[..., 2:]
            VL, VC, VR = vol[..., :n], vol[..., 1:n + 1], vol[..., 2:]
            FL, FR = F[..., 1:n + 1], F[..., 2:n + 2]  # faces of cell s: native index of face f is f + 1
            if dim == 3:
                cL = torch.where(VL < VC, ((VC - VL) * cC + VL * cL) / VC, cL)
                cR = torch.where(VR < VC, ((VC - VR) * cC + VR * cR) / VC, cR)
            cL = torch.where(FL < FR, ((FR - FL) * cC + FL * cL) / FR, cL)
            cR = torch.where(FR < FL, ((FL - FR) * cC + FR * cR) / FL, cR)
            k1 = (VC / (VC + VR + eps)) * ((VL + VC) / (VL + VC + VR + eps))
            k2 = (VC / (VL + VC + eps)) * (VR / (VL + VC + VR + eps))
            r = (cR - cC + eps) / ((cC - cL) + eps)
            lim = torch.clamp(torch.minimum(r, torch.clamp(k1 * r + k2, max=1.0)), min=0.0)
            flux = 0.5 * (u.abs() + u) * FR * (cC + FL / (FL + eps) * lim * (cC - cL))
            return torch.where(u > 0, flux, torch.zeros_like(flux))

        net = torch.zeros(ph.shape[:-1] + (n + 1,), dtype=torch.float64, device="cuda")
        net[..., 1:] += upwind(ph, vol, F, u[..., 1:])
        mirror = [q.flip(-1) for q in (ph, vol, F)]
        net[..., :n] -= upwind(*mirror, -u.flip(-1)[..., 1:]).flip(-1)
        halo_lo, halo_hi = -net[..., 0], net[..., n].clone()  # what leaves over the two sides
        if periodic:
            sides = net[..., 0] + net[..., n]
            net[..., 0] = sides
            net[..., n] = sides
        get = torch.zeros(ph.shape, dtype=torch.float64, device="cuda")
        get[..., 1:n + 1] = net[..., :n] - net[..., 1:]
        get[..., 0], get[..., n + 1] = halo_lo, halo_hi
        target = total
        for q in own:
            target = target.narrow(q, 1, target.shape[q] - 2)
        target += get.movedim(-1, dim)
    return total * V / (V + eps) / (V + eps)
