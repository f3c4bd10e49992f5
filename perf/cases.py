"""The work that users of this library have it do, as cases that can be timed and checked.

Four kinds, all through the Python binding of the C ABI:

``residual``  one second-order (or first-order) residual evaluation of a host state, from pinned host memory
              and back (``Euler3DGPU.residual_step``): what an outer driver that owns the state calls.
``spmv``      one block SpMV with the stored implicit system on device vectors (``spmv_device``).
``ilu``       one application of the block-multicolour ILU(0) on device vectors (``precond_apply_device``).
``steady``    implicit iterations of ``solve_steady`` from a given state: residual, Jacobian, linear solve, update.

Meshes are tet-split boxes in blocked RCM numbering, built once per size (a user's mesh file); the states,
vectors and everything made from them come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cfdsolutions_b200 import Euler3DGPU, box_mesh, capi, default_params, perturbed_freestream, to_rup
from cfdsolutions_b200.mesh import NUMBERING_PATCH_RCM

GAMMA, ALPHA, VENKAT_K = 1.4, 1.25, 5.0
FLUX = {"roe": capi.FLUX_ROE, "hllc": capi.FLUX_HLLC, "ausm": capi.FLUX_AUSM, "turkel": capi.FLUX_ROE_PRECOND}
GRAD = {"gg": capi.GRAD_GG, "lsq": capi.GRAD_LSQ}
# the precision of the stored system: FP64, or a low-precision matrix alone
PREC = {"fp64": capi.PREC_FP64, "fp32": capi.PREC_FP32 | capi.PREC_LOW_ONLY, "bf16": capi.PREC_BF16 | capi.PREC_LOW_ONLY}
BLOCK_BYTES = {"fp64": 200, "fp32": 100, "bf16": 50}
# stiffened-gas water at 10 m/s (c = 1625 m/s): the low-Mach channel
WATER = dict(gamma=4.4, pinf=6000.0, mach=0.0062)


def listed():
    return [
        # smallest call: a design-study cube; launches and copies of a few microseconds each
        dict(name="residual-roe-16", kind="residual", nx=16, ny=16, nz=16, flux="roe", grad="gg", order=2, mach=0.8),
        # the reference's own gradient (least squares) on a ragged box of the size its CPU path is sampled at
        dict(name="residual-lsq-hllc-47x52x41", kind="residual", nx=47, ny=52, nz=41, flux="hllc", grad="lsq", order=2,
             mach=0.6),
        # the headline workload: 2.1 M nodes, Green-Gauss + Venkatakrishnan + Roe, copies and kernels pipelined
        dict(name="residual-roe-128", kind="residual", nx=128, ny=128, nz=128, flux="roe", grad="gg", order=2, mach=0.8),
        # a caller's own Krylov loop on the mixed-precision system: operator and preconditioner
        dict(name="spmv-fp32-96", kind="spmv", nx=96, ny=96, nz=96, prec="fp32", mach=0.8),
        dict(name="ilu-fp32-96", kind="ilu", nx=96, ny=96, nz=96, prec="fp32", mach=0.8),
        # the same preconditioner in FP64 on a small ragged box
        dict(name="ilu-fp64-47x52x33", kind="ilu", nx=47, ny=52, nz=33, prec="fp64", mach=0.7),
        # the opening iterations of the large steady solve, mixed precision (the served and benched form)
        dict(name="steady-fp32-128", kind="steady", nx=128, ny=128, nz=128, flux="roe", grad="gg", prec="fp32",
             linear="gmres", iters=12, mach=0.8),
        # the plain FP64 solve of an ordinary size
        dict(name="steady-fp64-64", kind="steady", nx=64, ny=64, nz=64, flux="roe", grad="gg", prec="fp64",
             linear="gmres", iters=12, mach=0.8),
        # BF16 Jacobian storage, another flux, a ragged box
        dict(name="steady-bf16-ausm-55x47x60", kind="steady", nx=55, ny=47, nz=60, flux="ausm", grad="gg", prec="bf16",
             linear="gmres", iters=10, mach=0.5),
        # a whole solve to the 1e-8 drop at the size of a small served request: many short launches
        dict(name="solve-fp32-24", kind="steady", nx=24, ny=24, nz=24, flux="roe", grad="gg", prec="fp32",
             linear="gmres", iters=800, mach=0.6),
        # low-Mach liquid channel in (rho, u, v, w, p), Turkel preconditioning, least squares, FP64, walls and inflow
        dict(name="channel-rup-fp64-96x24x24", kind="steady", nx=96, ny=24, nz=24, flux="turkel", grad="lsq",
             prec="fp64", linear="gmres", iters=10, mach=WATER["mach"]),
        # the reference's stock implicit iteration: ten block Gauss-Seidel sweeps
        dict(name="steady-gs-20", kind="steady", nx=20, ny=20, nz=20, flux="roe", grad="lsq", prec="fp64", linear="gs",
             iters=4, mach=0.5),
    ]


def _box(rng, lo, hi, most):
    """Three sides, log-uniform in [lo, hi], with at most ``most`` hexes."""
    while True:
        n = [round(math.exp(rng.uniform(math.log(lo), math.log(hi)))) for _ in range(3)]
        if n[0] * n[1] * n[2] <= most:
            return dict(nx=n[0], ny=n[1], nz=n[2])


def draw(rng):
    kind = rng.choice(["residual", "spmv", "ilu", "steady", "steady"])
    mach = round(rng.uniform(0.3, 0.85), 3)
    if kind == "residual":
        return dict(_box(rng, 12, 128, 128 ** 3), kind=kind, flux=rng.choice(["roe", "hllc", "ausm"]),
                    grad=rng.choice(["gg", "lsq"]), order=rng.choice([2, 2, 2, 1]), mach=mach)
    if kind in ("spmv", "ilu"):
        return dict(_box(rng, 12, 96, 96 ** 3), kind=kind, prec=rng.choice(["fp64", "fp32", "bf16"]), mach=mach)
    sub = rng.choice(["gmres", "gmres", "gmres", "channel", "gs", "solve"])
    if sub == "gs":
        return dict(_box(rng, 10, 22, 20 ** 3), kind="steady", flux="roe", grad="lsq", prec="fp64", linear="gs", iters=4,
                    mach=mach)
    if sub == "solve":
        return dict(_box(rng, 12, 26, 24 ** 3), kind="steady", flux="roe", grad="gg", prec="fp32", linear="gmres",
                    iters=800, mach=mach)
    if sub == "channel":
        ny = rng.randint(8, 24)
        return dict(nx=4 * ny, ny=ny, nz=rng.randint(8, 24), kind="steady", flux="turkel", grad="lsq", prec="fp64",
                    linear="gmres", iters=10, mach=WATER["mach"])
    return dict(_box(rng, 16, 96, 72 ** 3), kind="steady", flux=rng.choice(["roe", "hllc", "ausm"]),
                grad=rng.choice(["gg", "lsq"]), prec=rng.choice(["fp64", "fp32", "bf16"]), linear="gmres", iters=10,
                mach=mach)


# ----------------------------------------------------------------- inputs
_mesh_cache: dict = {}


def _mesh(case):
    """The case's mesh (the last one is kept: a user reads a mesh once and runs many states on it)."""
    channel = case.get("flux") == "turkel"
    key = (case["nx"], case["ny"], case["nz"], channel)
    if key not in _mesh_cache:
        _mesh_cache.clear()
        size = key[:3]
        h = max(size)
        kw = (dict(lengths=(4.0, 1.0, 1.0), jitter=0.1, face_bc=(2, 3, 0, 0, 0, 0)) if channel
              else dict(lengths=tuple(s / h for s in size), jitter=0.15))
        _mesh_cache[key] = box_mesh(size, seed=1234, rcm=NUMBERING_PATCH_RCM, **kw)
    return _mesh_cache[key]


def _params(case):
    kw = dict(flux_scheme=FLUX[case.get("flux", "roe")], order=case.get("order", 2) - 1, limiter=1, limiter_order=0,
              gradient=GRAD[case.get("grad", "gg")], venkat_k=VENKAT_K, gamma=GAMMA, mach=case["mach"],
              mach_min=case["mach"], alpha_deg=ALPHA, cfl_min=10.0, cfl_max=10.0)
    if case.get("flux") == "turkel":
        kw.update(precond_method=capi.PRECOND_TURKEL, precond_type=capi.PRECOND_LOCAL, precond_mach=case["mach"],
                  gamma=WATER["gamma"], pinf=WATER["pinf"], alpha_deg=0.0, variables=capi.VARS_RUP, cfl_max=1e4,
                  cfl_ramp=20)
    elif case["kind"] == "steady" and case["linear"] == "gmres":
        kw.update(cfl_max=1000.0, cfl_ramp=20)
    elif case["kind"] in ("spmv", "ilu"):
        kw.update(cfl_min=200.0, cfl_max=200.0)
    return default_params(**kw)


def _initial(case, mesh, seed):
    if case.get("flux") == "turkel":
        Q = perturbed_freestream(mesh, WATER["gamma"], case["mach"], 0.0, noise=(0.0, 0.02, 0.0), seed=seed,
                                 pinf=WATER["pinf"])
        return to_rup(Q, WATER["gamma"], WATER["pinf"])
    return perturbed_freestream(mesh, GAMMA, case["mach"], ALPHA, noise=0.01, seed=seed)


def _vector(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn((n, 5), dtype=torch.float64, device="cuda", generator=g)


class _DeviceArray:
    """A solver's device memory as an array that torch can wrap without a copy; the tensor keeps the solver alive."""

    def __init__(self, solver, ptr, shape, strides):
        self.solver = solver
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, strides=strides, typestr="<f8", version=3)


def _state_view(solver):
    """The solver's resident state [5, nnode + nghost] as a torch tensor on its own memory."""
    p, ld = capi.P(), capi.I64()
    capi.check(capi.lib.cfd_state_device_ptr(solver.handle, p, ld), "cfd_state_device_ptr")
    n = solver.mesh.nnode + solver.mesh.nghost
    return torch.as_tensor(_DeviceArray(solver, p.value, (5, n), (ld.value * 8, 8)), device="cuda")


def prepare(case, seed):
    mesh = _mesh(case)
    stream = torch.cuda.Stream()
    solver = Euler3DGPU(mesh, _params(case), device=torch.cuda.current_device(), stream=stream.cuda_stream)
    Q = _initial(case, mesh, seed)
    s = dict(kind=case["kind"], solver=solver, stream=stream)
    if case["kind"] == "residual":
        host = lambda shape: torch.empty(shape, dtype=torch.float64, pin_memory=True)  # noqa: E731
        s["Q"], s["conv"], s["diss"] = host(Q.shape), host((5, mesh.nnode)), host((5, mesh.nnode))
        s["Q"].copy_(torch.from_numpy(Q))
        return s
    if case["kind"] == "steady":
        s["view"] = _state_view(solver)
        s["Q0"] = torch.from_numpy(Q).cuda()
        prec = PREC[case["prec"]]
        # GMRES(30) to a 0.1 relative residual, ILU(0) refreshed every 15 implicit iterations (5 in the channel)
        s["gmres"] = capi.GmresOpts(30, 30, 0.1, capi.PC_ILU0_MC, prec, 1)
        s["opts"] = dict(max_iterations=case["iters"], drop=1e-8, include_diss=1,
                         linear_solver=1 if case["linear"] == "gmres" else 0, linear_iters=10,
                         precond_update=5 if case["flux"] == "turkel" else 15)
        if case["linear"] == "gmres":
            capi.check(capi.lib.cfd_ilu_mc_order(solver.handle, None, None), "cfd_ilu_mc_order")
        return s
    prec = PREC[case["prec"]]
    solver.set_state(Q)
    solver.residual_step(0)
    solver.Compute_Jacobian(1, 0, include_diss=1, precision=prec)
    if case["kind"] == "ilu":
        solver.solve_gmres(restart=30, max_iters=2, rtol=1e-12, precond=capi.PC_ILU0_MC, precision=prec,
                           allow_not_converged=True)
    solver.synchronize()
    s["prec"] = prec & ~capi.PREC_LOW_ONLY
    s["x"] = _vector(mesh.nnode, seed)
    s["y"] = torch.empty_like(s["x"])
    return s


def run(state):
    solver = state["solver"]
    if state["kind"] == "residual":
        conv, diss = state["conv"].numpy(), state["diss"].numpy()
        solver.residual_step(0, state["Q"].numpy(), out=(conv, diss))
        return {"conv": state["conv"], "diss": state["diss"]}
    if state["kind"] == "spmv":
        solver.spmv_device(state["x"].data_ptr(), state["y"].data_ptr(), state["prec"])
        return state["y"]
    if state["kind"] == "ilu":
        solver.precond_apply_device(state["x"].data_ptr(), state["y"].data_ptr())
        return state["y"]
    view = _state_view(solver)  # tells the library that the state is written
    with torch.cuda.stream(state["stream"]):
        view.copy_(state["Q0"])
    st = solver.solve_steady(gmres=state["gmres"], **state["opts"])
    return {"state": view, "rms": [st.rms_first, st.rms_last]}


# ------------------------------------------------------------------ work
def _sizes(case):
    x, y, z = case["nx"], case["ny"], case["nz"]
    faces = x * y + y * z + x * z
    n = (x + 1) * (y + 1) * (z + 1)
    axis = x * (y + 1) * (z + 1) + (x + 1) * y * (z + 1) + (x + 1) * (y + 1) * z
    diag = x * y * (z + 1) + x * (y + 1) * z + (x + 1) * y * z
    return n, axis + diag + x * y * z, 12 * faces  # nodes, edges (6 tets per hex), ghosts


def work(case):
    n, e, g = _sizes(case)
    nnzb = n + 2 * e
    # Q in, faces and boundary faces (area vector + nodes), coordinates and volumes, both residuals out
    residual = 40 * (n + g) + 40 * (e + g) + 32 * n + 80 * n
    rflops = 300 * e + (250 * e if case.get("order", 2) == 2 else 0)
    if case["kind"] == "residual":
        return {"bytes": residual, "flops": rflops}
    matrix = BLOCK_BYTES[case["prec"]] * nnzb + 4 * nnzb + 4 * (n + 1)
    factors = max(BLOCK_BYTES[case["prec"]], 100) * nnzb + 4 * nnzb + 4 * (n + 1)  # BF16 systems keep FP32 factors
    if case["kind"] == "spmv":
        return {"bytes": matrix + 80 * n, "flops": 50 * nnzb}
    if case["kind"] == "ilu":
        return {"bytes": factors + 80 * n, "flops": 50 * nnzb}
    iters = case["iters"] if case["iters"] < 100 else 100  # a whole solve takes about 100 implicit iterations
    if case["linear"] == "gs":
        return {"bytes": iters * (residual + matrix + 10 * (matrix + 80 * n)), "flops": iters * (rflops + 10 * 50 * nnzb)}
    krylov = 4 * (matrix + factors + 3 * 40 * n)  # about four Krylov iterations per implicit one
    return {"bytes": iters * (residual + matrix + 80 * n + krylov), "flops": iters * (rflops + 600 * e + 400 * nnzb)}


# ----------------------------------------------------------------- exact
def exact(case, seed):
    """Residuals and block products in 64 bits with plain torch.  None for the ILU(0) and the implicit iterations:
    their sequential block elimination takes minutes in torch or numpy at these sizes."""
    if case["kind"] not in ("residual", "spmv") or case.get("flux") == "turkel":
        return None
    mesh = _mesh(case)
    E = _Exact(case, mesh, torch.from_numpy(_initial(case, mesh, seed)).cuda())
    conv, diss, dtsum = E.residual()
    if case["kind"] == "residual":
        return {"conv": conv, "diss": diss}
    return E.product(_vector(mesh.nnode, seed), dtsum / 200.0)


class _Exact:
    """The residual and the first-order Roe Jacobian's product, an edge at a time over whole arrays."""

    CHUNK = 1 << 20

    def __init__(self, case, mesh, Q):
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.case, self.n = case, mesh.nnode
        self.L, self.R = (dev(mesh.edge_nodes[:, k]).long() for k in (0, 1))
        self.S = dev(mesh.edge_areav)
        self.bL, self.bR = (dev(mesh.bedge_nodes[:, k]).long() for k in (0, 1))
        self.bS = dev(mesh.bedge_areav)
        self.x, self.vol = dev(mesh.coords), dev(mesh.cvol)
        self.Q = Q
        m, a = case["mach"], math.radians(ALPHA)
        self.inf = (m * math.sqrt(GAMMA) * math.cos(a), m * math.sqrt(GAMMA) * math.sin(a), 0.0)
        self._farfield()

    @staticmethod
    def _unit(S):
        area = S.norm(dim=1)
        return (S / area[:, None]).T, area

    @staticmethod
    def _prim(q, n):
        rho, u, v, w = q[0], q[1] / q[0], q[2] / q[0], q[3] / q[0]
        p = (GAMMA - 1) * (q[4] - 0.5 * rho * (u * u + v * v + w * w))
        return rho, u, v, w, p, (q[4] + p) / rho, u * n[0] + v * n[1] + w * n[2]

    def _farfield(self):
        """Characteristic far-field ghost states (rho = p = 1, c = sqrt(gamma) outside)."""
        n, _ = self._unit(self.bS)
        qi, qg = self.Q[:, self.bL], self.Q[:, self.bR]
        rho, u, v, w, p, _, ub = self._prim(qi, n)
        ro, _, _, _, po, _, l1 = self._prim(0.5 * (qi + qg), n)
        c = torch.sqrt(GAMMA * po / ro)
        rc, c2 = ro * c, c * c
        iu, iv, iw = self.inf
        t = n[0] * (iu - u) + n[1] * (iv - v) + n[2] * (iw - w)
        inflow, sub = l1 < 0, l1.abs() < c
        one = torch.ones_like(p)
        pb = torch.where(inflow, 0.5 * (1.0 + p - rc * t), one)
        base = [torch.where(inflow, o, i) for o, i in zip((one, iu * one, iv * one, iw * one, one), (rho, u, v, w, p))]
        dp = torch.where(inflow, pb - 1.0, pb - p)
        sg = torch.where(inflow, 1.0, -1.0)
        b = [base[0] + dp / c2] + [base[1 + k] + sg * n[k] * dp / rc for k in range(3)] + [pb]
        b = [torch.where(sub, x, y) for x, y in zip(b, base)]
        et = b[4] / ((GAMMA - 1) * b[0]) + 0.5 * (b[1] ** 2 + b[2] ** 2 + b[3] ** 2)
        self.Q[:, self.bR] = torch.stack([b[0], b[0] * b[1], b[0] * b[2], b[0] * b[3], b[0] * et])

    def _average(self, A, B):
        rho = torch.sqrt(A[0] * B[0])
        s = rho / (A[0] + rho)
        u, v, w, ht = (A[k] + s * (B[k] - A[k]) for k in (1, 2, 3, 5))
        return rho, u, v, w, ht, torch.sqrt((GAMMA - 1) * (ht - 0.5 * (u * u + v * v + w * w)))

    @staticmethod
    def _physical(F, n):
        m = F[0] * F[6]
        return torch.stack([m, F[1] * m + F[4] * n[0], F[2] * m + F[4] * n[1], F[3] * m + F[4] * n[2], F[5] * m])

    def _flux(self, qL, qR, S):
        n, area = self._unit(S)
        A, B = self._prim(qL, n), self._prim(qR, n)
        rho, u, v, w, ht, c = self._average(A, B)
        ub = u * n[0] + v * n[1] + w * n[2]
        lam = ub.abs() + c
        zero = torch.zeros_like(qL)
        if self.case.get("flux", "roe") == "roe":
            conv = 0.5 * area * (self._physical(A, n) + self._physical(B, n))
            d = [B[k] - A[k] for k in range(5)]
            dU = d[1] * n[0] + d[2] * n[1] + d[3] * n[2]
            a1 = (d[4] - rho * c * dU) / (2 * c * c) * (ub - c).abs()
            a5 = (d[4] + rho * c * dU) / (2 * c * c) * (ub + c).abs()
            a2 = (d[0] - d[4] / (c * c)) * ub.abs()
            q2 = 0.5 * (u * u + v * v + w * w)
            vel, out = (u, v, w), [a1 + a2 + a5]
            sh = [rho * ub.abs() * (d[1 + k] - dU * n[k]) for k in range(3)]
            out += [a1 * (vel[k] - c * n[k]) + a5 * (vel[k] + c * n[k]) + a2 * vel[k] + sh[k] for k in range(3)]
            out += [a1 * (ht - c * ub) + a5 * (ht + c * ub) + a2 * q2 + sum(vel[k] * sh[k] for k in range(3))]
            return conv, -0.5 * area * torch.stack(out), area * lam
        if self.case["flux"] == "hllc":
            cA, cB = torch.sqrt(GAMMA * A[4] / A[0]), torch.sqrt(GAMMA * B[4] / B[0])
            SL, SR = torch.minimum(A[6] - cA, ub - c), torch.maximum(B[6] + cB, ub + c)
            SM = ((B[0] * B[6] * (SR - B[6]) - A[0] * A[6] * (SL - A[6]) + A[4] - B[4])
                  / (B[0] * (SR - B[6]) - A[0] * (SL - A[6])))

            def star(F, q, Sk):
                ps = F[4] + F[0] * (F[6] - Sk) * (F[6] - SM)
                r = [F[0] * (Sk - F[6])] + [q[1 + k] * (Sk - F[6]) + (ps - F[4]) * n[k] for k in range(3)]
                r += [(Sk - F[6]) * q[4] - F[4] * F[6] + ps * SM]
                qs = torch.stack(r) / (Sk - SM)
                return qs * SM + torch.stack([0 * ps, ps * n[0], ps * n[1], ps * n[2], ps * SM])

            F = torch.where(SM > 0, star(A, qL, SL), star(B, qR, SR))
            F = torch.where(SL > 0, self._physical(A, n), torch.where(SR < 0, self._physical(B, n), F))
            return area * F, zero, area * lam
        k = 2 * (GAMMA - 1) / (GAMMA + 1)  # AUSM+
        cL, cR = torch.sqrt(k * A[5]), torch.sqrt(k * B[5])
        ch = torch.minimum(cL * cL / torch.maximum(cL, A[6]), cR * cR / torch.maximum(cR, -B[6]))
        M, N = A[6] / ch, B[6] / ch
        b, d = M * M - 1, N * N - 1
        Mp = torch.where(M.abs() >= 1, 0.5 * (M + M.abs()), 0.25 * (M + 1) ** 2 + b * b / 8)
        Pp = torch.where(M.abs() >= 1, (M > 0).double(), 0.25 * (M + 1) ** 2 * (2 - M) + 3 / 16 * M * b * b)
        Nm = torch.where(N.abs() >= 1, 0.5 * (N - N.abs()), -0.25 * (N - 1) ** 2 - d * d / 8)
        Pm = torch.where(N.abs() >= 1, (N < 0).double(), 0.25 * (N - 1) ** 2 * (2 + N) - 3 / 16 * N * d * d)
        m, p = Mp + Nm, Pp * A[4] + Pm * B[4]
        mL, mR = ch * m.clamp(min=0) * A[0], ch * m.clamp(max=0) * B[0]
        one = torch.ones_like(p)
        F = torch.stack([mL * a + mR * e for a, e in zip((one, *A[1:4], A[5]), (one, *B[1:4], B[5]))])
        return area * (F + torch.stack([0 * p, p * n[0], p * n[1], p * n[2], 0 * p])), zero, area * lam

    def _edges(self):
        for lo in range(0, len(self.L), self.CHUNK):
            yield slice(lo, lo + self.CHUNK)

    def _gradients(self):
        n, Q = self.n, self.Q
        if self.case.get("grad", "gg") == "gg":
            g = torch.zeros((5, n, 3), dtype=torch.float64, device="cuda")
            for e in self._edges():
                t = 0.5 * (Q[:, self.R[e]] - Q[:, self.L[e]])[:, :, None] * self.S[e]
                g.index_add_(1, self.L[e], t)
                g.index_add_(1, self.R[e], t)
            return g / self.vol[:, None]
        G = torch.zeros((n, 3, 3), dtype=torch.float64, device="cuda")
        r = torch.zeros((n, 3, 5), dtype=torch.float64, device="cuda")
        for e in self._edges():
            d = self.x[self.R[e]] - self.x[self.L[e]]
            dq = (Q[:, self.R[e]] - Q[:, self.L[e]]).T
            for side in (self.L[e], self.R[e]):
                G.index_add_(0, side, d[:, :, None] * d[:, None, :])
                r.index_add_(0, side, d[:, :, None] * dq[:, None, :])
        return torch.linalg.solve(G, r).permute(2, 0, 1).contiguous()

    def _limited(self):
        """Venkatakrishnan limiters times the gradients."""
        n, Q, g = self.n, self.Q, self._gradients()
        own = Q[:, :n]
        mx, mn = own.clone(), own.clone()
        for e in self._edges():
            for i, j in ((self.L[e], self.R[e]), (self.R[e], self.L[e])):
                mx.scatter_reduce_(1, i.expand(5, -1), Q[:, j], "amax")
                mn.scatter_reduce_(1, i.expand(5, -1), Q[:, j], "amin")
        mx, mn = mx - own, mn - own
        eps2 = 6.0 * VENKAT_K ** 3 * self.vol / math.pi
        phi = torch.ones_like(own)
        for e in self._edges():
            for i, j in ((self.L[e], self.R[e]), (self.R[e], self.L[e])):
                dm = (g[:, i] * (0.5 * (self.x[j] - self.x[i]))).sum(-1)
                dp = torch.where(dm > 0, mx[:, i], mn[:, i])
                f = (dp * dp + eps2[i] + 2 * dm * dp) / (dp * dp + 2 * dm * dm + dm * dp + eps2[i])
                phi.scatter_reduce_(1, i.expand(5, -1), torch.where(dm == 0, 1.0, f), "amin")
        return phi[:, :, None] * g

    def residual(self):
        n, Q = self.n, self.Q
        second = self.case.get("order", 2) == 2
        lg = self._limited() if second else None
        conv, diss = (torch.zeros((5, n), dtype=torch.float64, device="cuda") for _ in range(2))
        dtsum = torch.zeros(n, dtype=torch.float64, device="cuda")
        for e in self._edges():
            L, R = self.L[e], self.R[e]
            qL, qR = Q[:, L], Q[:, R]
            if second:
                r = 0.5 * (self.x[R] - self.x[L])
                qL, qR = qL + (lg[:, L] * r).sum(-1), qR - (lg[:, R] * r).sum(-1)
            c, d, lam = self._flux(qL, qR, self.S[e])
            for out, f in ((conv, c), (diss, d)):
                out.index_add_(1, L, f)
                out.index_add_(1, R, -f)
            dtsum.index_add_(0, L, lam)
            dtsum.index_add_(0, R, lam)
        c, d, lam = self._flux(Q[:, self.bL], Q[:, self.bR], self.bS)
        conv.index_add_(1, self.bL, c)
        diss.index_add_(1, self.bL, d)
        dtsum.index_add_(0, self.bL, lam)
        return conv, diss, dtsum

    def _matrices(self, qL, qR, S):
        """area * |A| at the Roe average, and area * dF/dQ at both states."""
        n, area = self._unit(S)
        rho, u, v, w, ht, c = self._average(self._prim(qL, n), self._prim(qR, n))
        ub = u * n[0] + v * n[1] + w * n[2]
        J = self._jacobian((u, v, w), ht, ub, n)
        eye = torch.eye(5, dtype=torch.float64, device="cuda")
        # |A| as a quadratic in A: eigenvalues ub (three times), ub + c, ub - c
        f0, fp, fm = ub.abs(), (ub + c).abs(), (ub - c).abs()
        d1, d2 = (fp - fm) / (2 * c), (fp + fm - 2 * f0) / (2 * c * c)
        D = J - ub[:, None, None] * eye
        absA = f0[:, None, None] * eye + d1[:, None, None] * D + d2[:, None, None] * (D @ D)
        both = []
        for q in (qL, qR):
            r, uu, vv, ww, _, h, b = self._prim(q, n)
            both.append(self._jacobian((uu, vv, ww), h, b, n) * area[:, None, None])
        return absA * area[:, None, None], both[0], both[1]

    @staticmethod
    def _jacobian(vel, ht, ub, n):
        g1 = GAMMA - 1
        ek = 0.5 * sum(x * x for x in vel)
        rows = [[0 * ub, n[0], n[1], n[2], 0 * ub]]
        for k in range(3):
            row = [g1 * ek * n[k] - vel[k] * ub]
            row += [vel[k] * n[j] - g1 * vel[j] * n[k] + (ub if j == k else 0) for j in range(3)]
            rows.append(row + [g1 * n[k]])
        rows.append([(g1 * ek - ht) * ub] + [ht * n[j] - g1 * vel[j] * ub for j in range(3)] + [GAMMA * ub])
        return torch.stack([torch.stack(r, -1) for r in rows], -2)

    def product(self, x, time_term):
        """A x with A[L,R] = (J_R - |A|)/2, A[R,L] = -(J_L + |A|)/2, the diagonal less its column's
        off-diagonal blocks, plus the boundary faces' (J_L + |A|)/2 and the time term."""
        Q, y = self.Q, time_term[:, None] * x
        act = lambda M, z: (M @ z[:, :, None])[:, :, 0]  # noqa: E731
        for lo in range(0, len(self.L), self.CHUNK // 2):
            e = slice(lo, lo + self.CHUNK // 2)
            L, R = self.L[e], self.R[e]
            A, JL, JR = self._matrices(Q[:, L], Q[:, R], self.S[e])
            up, down = 0.5 * (JR - A), -0.5 * (JL + A)
            y.index_add_(0, L, act(up, x[R]) - act(down, x[L]))
            y.index_add_(0, R, act(down, x[L]) - act(up, x[R]))
        A, JL, _ = self._matrices(Q[:, self.bL], Q[:, self.bR], self.bS)
        y.index_add_(0, self.bL, act(0.5 * (JL + A), x[self.bL]))
        return y
