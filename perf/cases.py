"""The work that programs on this library have it do, as measurable cases.

A case is a dict of plain values; `listed()` names the fixed ones, `draw(rng)`
gives another one of the same ranges:

  box       one RK4 call of a 3D case with its state resident on the device
            (the loop of a driver: dg_rk4_steps, `steps` steps a call), orders
            1..5, FP64 or mixed precision, both numerical fluxes, uniform
            periodic boxes from a few hundred to a quarter of a million
            hexahedra, even and odd, optionally with randomly turned element
            numberings (as mesh generators deliver them); Taylor-Green runs
            also take the kinetic energy, as their history needs it every call
  bent      the same on non-affine (trilinear) hexahedra
  ensemble  many small independent cases of different order and size advanced
            together, their states fetched at the end
  quad      the 2D path: steps on a quadrilateral box, the state fetched
  roundtrip a host program's use of the path: its state goes up from pinned
            host memory, is advanced, and comes back, with the L2 error taken

Every input (vortex strength, centre and free stream, Mach number, turning of
the elements, bend of the mesh) comes from the seed.  Time steps follow the CFL
number of the case and a bound of its wave speeds: 0.1 in FP64; in mixed
precision a step far below the stability limit, at which the state stays as
near to the FP64 one as an FP64 array is worth comparing (the FP32 residual's
rounding enters the state times the step).  A step costs the same at any size.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dg-mpi_b200"))
import dg_b200  # noqa: E402

GAMMA = 1.4
LENGTH = 10.0
TGV_LENGTH = 2.0 * math.pi
FP64, MIXED = "fp64", "mixed_fp32"
LF, HLLC = "LaxFriedrichs", "HLLC"


def _box(name, n, order, precision, flux, steps, flow="vortex", turned=False):
    nx, ny, nz = n
    return {"name": name, "kind": "box", "nx": nx, "ny": ny, "nz": nz, "order": order, "precision": precision,
            "flux": flux, "steps": steps, "flow": flow, "turned": turned}


def listed():
    return [
        # the regression deck's mesh, order and flux, one step a call: a driver's
        # loop on the smallest problem, all launches and latency
        _box("cube4_p3_hllc", (4, 4, 4), 3, FP64, HLLC, 1),
        # the CPU-runnable vortex deck: 8^3, p = 2, ten steps between outputs
        _box("cube8_p2", (8, 8, 8), 2, FP64, LF, 10),
        # an odd box as a mesh file holds it (elements turned at random), low order, mixed
        _box("odd21_p1_mixed_turned", (21, 17, 19), 1, MIXED, HLLC, 4, turned=True),
        # the at-scale FP64 configuration: 64^3, p = 3, Lax-Friedrichs
        _box("cube64_p3", (64, 64, 64), 3, FP64, LF, 1),
        # the same in mixed precision
        _box("cube64_p3_mixed", (64, 64, 64), 3, MIXED, LF, 1),
        # high order, mixed (the precision configuration at a size that is quick to set up)
        _box("cube36_p5_mixed", (36, 36, 36), 5, MIXED, LF, 1),
        # high order, FP64, the other flux, an odd box
        _box("odd27_p5_hllc", (27, 25, 29), 5, FP64, HLLC, 1),
        # low-Mach Taylor-Green at p = 4, mixed, kinetic energy after the step
        _box("taylor_green48_p4_mixed", (48, 48, 48), 4, MIXED, LF, 1, flow="taylor_green"),
        # bent hexahedra: per-point metric terms and dense inverse mass matrices
        {"name": "bent18_p3", "kind": "bent", "nx": 18, "ny": 17, "nz": 18, "order": 3, "precision": FP64, "flux": LF,
         "steps": 2},
        # a parameter study: 20 vortices of orders 1..5 on 8^3..16^3 boxes
        {"name": "ensemble20_mixed", "kind": "ensemble", "cases": 20, "nmin": 8, "nmax": 16, "precision": MIXED,
         "flux": LF, "steps": 8},
        # the reference's 2D vortex deck, refined: 256^2, p = 3, 60 steps
        {"name": "quad256_p3", "kind": "quad", "nx": 256, "ny": 256, "order": 3, "flux": HLLC, "steps": 60},
        # a solver that keeps its state on the host calls the path for a few steps
        {"name": "roundtrip32_p3", "kind": "roundtrip", "nx": 32, "ny": 32, "nz": 32, "order": 3, "precision": FP64,
         "flux": LF, "steps": 2},
    ]


def _cost(nelem, order, steps):
    return nelem * (order + 1) ** 3 * 5 * steps


MOST_COST = _cost(64 ** 3, 3, 1)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, nelem, lo=3):
    """Three sides of about nelem cells in all, none alike by rule."""
    side = nelem ** (1.0 / 3.0)
    a, b = rng.uniform(0.75, 1.33), rng.uniform(0.75, 1.33)
    return [max(lo, int(round(side * f))) for f in (a, b, 1.0 / (a * b))]


def draw(rng):
    kind = rng.choices(["box", "bent", "ensemble", "quad", "roundtrip"], [62, 9, 9, 9, 11])[0]
    precision, flux = rng.choice([FP64, MIXED]), rng.choice([LF, LF, HLLC])
    if kind == "ensemble":
        return {"kind": kind, "cases": rng.randint(6, 20), "nmin": rng.choice([6, 8]), "nmax": rng.choice([11, 12, 16]),
                "precision": precision, "flux": flux, "steps": rng.randint(2, 8)}
    order = rng.randint(1, 5)
    if kind == "quad":
        order = rng.randint(1, 4)
        return {"kind": kind, "nx": _log_int(rng, 16, 300), "ny": _log_int(rng, 16, 300), "order": order, "flux": flux,
                "steps": rng.randint(10, 60)}
    nb = (order + 1) ** 3
    if kind == "bent":
        n = _sides(rng, _log_int(rng, 200, max(400, 350000 // nb)))
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "precision": precision, "flux": flux,
                "steps": rng.randint(1, 3)}
    if kind == "roundtrip":
        n = _sides(rng, _log_int(rng, 64, 2500000 // nb))
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "precision": precision, "flux": flux,
                "steps": rng.randint(1, 4)}
    nelem = _log_int(rng, 64, 0.8 * MOST_COST / (5 * nb))
    n = _sides(rng, nelem)
    while _cost(n[0] * n[1] * n[2], order, 1) > MOST_COST:
        n[rng.randrange(3)] -= 1
    steps = max(1, min(rng.randint(1, 8), MOST_COST // _cost(n[0] * n[1] * n[2], order, 1)))
    if precision == MIXED:
        steps = min(steps, 4)
    return {"kind": "box", "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "precision": precision, "flux": flux,
            "steps": steps, "flow": rng.choice(["vortex", "vortex", "taylor_green"]), "turned": rng.random() < 0.3}


# ---------------------------------------------------------------------------
# inputs

def _vortex(rng):
    """rho, u, v, p, strength, centre, periods of the x-y vortex."""
    return [1.0, rng.uniform(0.5, 1.5), rng.uniform(0.5, 1.5), 1.0, rng.uniform(1.0, 5.0), rng.uniform(3.0, 7.0),
            rng.uniform(3.0, 7.0), LENGTH, LENGTH]


def _time_step(precision, order, h, speed):
    cfl = 0.1 if precision == FP64 else 0.0002
    return cfl * h / ((2 * order + 1) * speed)


def _vortex_speed(d):
    return math.hypot(d[1], d[2]) + d[4] / (2 * math.pi) + math.sqrt(GAMMA)


def _setup(case, seed):
    """Mesh, flow family and data, time step of a 3D case."""
    rng = random.Random(int(seed) * 7919 + 17)
    n = (case["nx"], case["ny"], case["nz"])
    flow = case.get("flow", "vortex")
    if flow == "taylor_green":
        length, name, data = TGV_LENGTH, "TaylorGreen", [rng.uniform(0.08, 0.16)]
        speed = 1.0 + 1.0 / data[0]
    else:
        length, name, data = LENGTH, "IsentropicVortexXY", _vortex(rng)
        speed = _vortex_speed(data)
    turn = rng.randrange(1, 1 << 20) if case.get("turned") else 0
    mesh = dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (length,) * 3, rotate_seed=turn)
    if case["kind"] == "bent":
        x = mesh.node_coords
        k, amp = 2 * math.pi / length, rng.uniform(0.02, 0.05)
        s = np.sin(k * x)
        bend = amp * np.stack([s[:, 1] * s[:, 2], s[:, 0] * s[:, 2], s[:, 0] * s[:, 1]], 1) * (length / np.array(n))
        mesh = dg_b200.Mesh(np.ascontiguousarray(x + bend), mesh.elem_to_node_ids, mesh.interior_faces)
    dt = _time_step(case["precision"], case["order"], length / max(n), speed)
    return mesh, length, name, data, dt


class _DeviceState:
    """A case's device state as something torch takes without a copy; the tensor
    made of it keeps the case, and with it the memory, alive."""

    def __init__(self, case):
        self.case = case
        self.__cuda_array_interface__ = {"shape": (case.ne, 5, case.nb), "typestr": "<f8",
                                         "data": (case.device_state_ptr(), False), "version": 3}


def _ensemble_cases(case, seed):
    """(cells per side, order, vortex data) of each member: sizes, orders and flows in turn."""
    rng = random.Random(int(seed) * 104729 + 5)
    out = []
    lo, hi = case["nmin"], case["nmax"]
    for i in range(case["cases"]):
        n = lo + (i * 5) % (hi - lo + 1)
        out.append((n, 1 + i % 5, _vortex(rng)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        spec = _ensemble_cases(case, seed)
        boxes = {n: dg_b200.periodic_box((n, n, n), (0.0, 0.0, 0.0), (LENGTH,) * 3) for n in {s[0] for s in spec}}
        batch = dg_b200.Batch([(boxes[n], p) for n, p, _ in spec], flux=case["flux"], gas_constant=1.0,
                              precision=case["precision"])
        for i, (n, p, data) in enumerate(spec):
            batch.project_ic(i, "IsentropicVortexXY", data)
            batch.set_time_step(i, _time_step(case["precision"], p, LENGTH / n, _vortex_speed(data)))
        return {"kind": kind, "batch": batch, "steps": case["steps"]}
    if kind == "quad":
        rng = random.Random(int(seed) * 7919 + 29)
        n = (case["nx"], case["ny"])
        data = _vortex(rng)
        mesh = dg_b200.periodic_box_2d(n, (0.0, 0.0), (LENGTH, LENGTH))
        c = dg_b200.Case2D(mesh, case["order"], flux=case["flux"], gas_constant=1.0)
        c.project_ic("IsentropicVortexXY", data)
        return {"kind": kind, "case": c, "steps": case["steps"],
                "dt": _time_step(FP64, case["order"], LENGTH / max(n), _vortex_speed(data))}
    mesh, _, name, data, dt = _setup(case, seed)
    c = dg_b200.Case(mesh, case["order"], flux=case["flux"], gas_constant=1.0, precision=case["precision"])
    state = {"kind": kind, "case": c, "dt": dt, "steps": case["steps"], "energy": case.get("flow") == "taylor_green"}
    U0 = c.project_ic(name, data)
    if kind == "roundtrip":
        state["host_in"] = torch.from_numpy(U0).pin_memory()
        state["host_out"] = torch.empty_like(state["host_in"]).pin_memory()
        state["flow"] = (name, data, dt * case["steps"])
    else:
        state["U"] = torch.as_tensor(_DeviceState(c), device="cuda")
    return state


# ---------------------------------------------------------------------------
# one pass

def run(state):
    kind = state["kind"]
    if kind == "ensemble":
        batch = state["batch"]
        batch.rk4(state["steps"])
        return [batch.get_state(i) for i in range(len(batch))]
    c = state["case"]
    if kind == "quad":
        c.rk4(state["dt"], state["steps"])
        return c.get_state()
    if kind == "roundtrip":
        c.set_state_ptr(state["host_in"].data_ptr())
        c.rk4(state["dt"], state["steps"])
        c.get_state_ptr(state["host_out"].data_ptr())
        name, data, t = state["flow"]
        return {"U": state["host_out"], "l2_error": c.l2_error(name, data, t)}
    c.rk4(state["dt"], state["steps"])
    if state["energy"]:
        return {"U": state["U"], "kinetic_energy": c.kinetic_energy()}
    return {"U": state["U"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _flops_per_dof(p):
    """Sum-factorised arithmetic per DOF and RK stage (n = p+1 nodes, m = p+2 points a direction)."""
    n, m = p + 1, p + 2
    interp = 2 * (m * n ** 3 + m ** 2 * n ** 2 + m ** 3 * n)
    trace = 6 * 5 * 2 * (n ** 3 + m * n ** 2 + m ** 2 * n)
    total = 5 * interp + 15 * interp + 2 * trace + 5 * 3 * 2 * n ** 4 + 130 * m ** 3 + 600 * m ** 2 + 20 * n ** 3
    return total / (5 * n ** 3)


def work(case):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        dof = flops = 0
        for n, p, _ in _ensemble_cases(case, 0):
            d = n ** 3 * (p + 1) ** 3 * 5
            dof += d
            flops += d * _flops_per_dof(p) * 4 * steps
        return {"bytes": 16 * dof, "flops": flops}
    p = case["order"]
    if kind == "quad":
        n, m = p + 1, p + 2
        ne = case["nx"] * case["ny"]
        per = 4 * 2 * (m * n * n + m * m * n) * 3 + 70 * m * m + 4 * n * 4 * 2 * n * 2 + 4 * n * 120 + 4 * 2 * 2 * n ** 3
        return {"bytes": 16 * ne * n * n * 4, "flops": ne * per * 4 * steps}
    ne = case["nx"] * case["ny"] * case["nz"]
    nb = (p + 1) ** 3
    dof = ne * nb * 5
    per_elem = 8 * (nb * nb + 9 * (p + 2) ** 3 + 24 * (p + 2) ** 2) if kind == "bent" else 0  # inverse mass, metric terms
    flops = dof * _flops_per_dof(p) * 4 * steps + (ne * nb * nb * 10 * 4 * steps if kind == "bent" else 0)
    return {"bytes": 16 * dof + ne * per_elem, "flops": flops}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits, from the definition of the scheme on uniform
# boxes: nodal Lagrange basis on equidistant points, Gauss-Legendre
# quadrature, classical Runge-Kutta; states are [variable, cells..., nodes...]
# with the slowest axis first

def _lagrange(nodes, x):
    """Values and derivatives [len(x), len(nodes)] of the Lagrange polynomials."""
    n = len(nodes)
    val, der = np.ones((len(x), n)), np.zeros((len(x), n))
    for j in range(n):
        for k in range(n):
            if k != j:
                val[:, j] *= (x - nodes[k]) / (nodes[j] - nodes[k])
        for i in range(n):
            if i != j:
                t = np.full(len(x), 1.0 / (nodes[j] - nodes[i]))
                for k in range(n):
                    if k not in (i, j):
                        t = t * (x - nodes[k]) / (nodes[j] - nodes[k])
                der[:, j] += t
    return val, der


class _Scheme:
    def __init__(self, p, h, flux, face_points, device):
        self.dim, self.h, self.flux = len(h), h, flux
        self.nodes = np.linspace(-1.0, 1.0, p + 1)
        self.p = p
        self.dev = device
        xq, wq = np.polynomial.legendre.leggauss(p + 2)
        B, D = _lagrange(self.nodes, xq)
        minv = np.linalg.inv(B.T @ (wq[:, None] * B))
        self.B, self.D, self.w, self.minv = (self._t(a) for a in (B, D, wq, minv))
        xf, wf = np.polynomial.legendre.leggauss(face_points)
        self.Bf, self.wf = self._t(_lagrange(self.nodes, xf)[0]), self._t(wf)

    def _t(self, a):
        return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)

    @staticmethod
    def along(M, T, axis):
        """M applied to axis `axis` of T."""
        return torch.movedim(torch.tensordot(T, M, dims=([axis], [1])), -1, axis)

    def axes(self, d):
        """(cell axis, node axis) of direction d (0 = x, the fastest) in a state array."""
        return 1 + self.dim - 1 - d, 1 + 2 * self.dim - 1 - d

    def project(self, fcn, counts):
        xe, we = np.polynomial.legendre.leggauss(2 * max(self.p, 1) + 2)
        Be = self._t(_lagrange(self.nodes, xe)[0])
        xe, we = self._t(xe), self._t(we)
        x, nd = [], 2 * self.dim
        for d in range(self.dim):
            ca, na = self.axes(d)
            shape_c, shape_n = [1] * nd, [1] * nd
            shape_c[ca - 1], shape_n[na - 1] = counts[d], len(xe)
            cell = torch.arange(counts[d], dtype=torch.float64, device=self.dev).reshape(shape_c)
            x.append((cell + 0.5 + 0.5 * xe.reshape(shape_n)) * self.h[d])
        shape = [counts[d] for d in reversed(range(self.dim))] + [len(xe)] * self.dim
        U = fcn(*[v.expand(shape) for v in x])
        P = self.minv @ (Be.T * we)
        for d in range(self.dim):
            U = self.along(P, U, self.axes(d)[1])
        return U

    def pressure(self, U):
        m2 = sum(U[1 + d] ** 2 for d in range(self.dim))
        return (GAMMA - 1.0) * (U[-1] - 0.5 * m2 / U[0]), m2

    def normal_flux(self, U, d, P):
        u = U[1 + d] / U[0]
        F = U * u
        F[1 + d] += P
        F[-1] += P * u
        return F

    def numerical(self, UL, UR, d):
        (PL, mL), (PR, mR) = self.pressure(UL), self.pressure(UR)
        FL, FR = self.normal_flux(UL, d, PL), self.normal_flux(UR, d, PR)
        aL, aR = torch.sqrt(GAMMA * PL / UL[0]), torch.sqrt(GAMMA * PR / UR[0])
        if self.flux == LF:
            a = torch.maximum(torch.sqrt(mL) / UL[0] + aL, torch.sqrt(mR) / UR[0] + aR)
            return 0.5 * (FL + FR) - 0.5 * a * (UR - UL)
        rL, rR, uL, uR = UL[0], UR[0], UL[1 + d] / UL[0], UR[1 + d] / UR[0]
        pst = torch.clamp(0.5 * (PL + PR - (uR - uL) * 0.25 * (rL + rR) * (aL + aR)), min=0.0)
        g = (GAMMA + 1.0) / (2.0 * GAMMA)
        qL = torch.sqrt(1.0 + g * torch.clamp(pst / PL - 1.0, min=0.0))
        qR = torch.sqrt(1.0 + g * torch.clamp(pst / PR - 1.0, min=0.0))
        sL, sR = uL - aL * qL, uR + aR * qR
        sM = (PR - PL + rL * uL * (sL - uL) - rR * uR * (sR - uR)) / (rL * (sL - uL) - rR * (sR - uR))

        def starred(U, F, u, P, s):
            c = U[0] * (s - u) / (s - sM)
            V = U / U[0]
            V[0] = 1.0
            V[1 + d] = sM
            V[-1] = U[-1] / U[0] + (sM - u) * (sM + P / (U[0] * (s - u)))
            return F + s * (c * V - U)

        F = torch.where(sM >= 0.0, starred(UL, FL, uL, PL, sL), starred(UR, FR, uR, PR, sR))
        F = torch.where(sL >= 0.0, FL, F)
        return torch.where(sR <= 0.0, FR, F)

    def rate(self, U):
        """dU/dt."""
        dim, vol = self.dim, math.prod(0.5 * v for v in self.h)
        Q = U
        for d in range(dim):
            Q = self.along(self.B, Q, self.axes(d)[1])
        P, _ = self.pressure(Q)
        R = torch.zeros_like(U)
        for d in range(dim):
            G = self.normal_flux(Q, d, P)
            for a in range(dim):
                na = self.axes(a)[1]
                M = self.D if a == d else self.B
                G = self.along((M * self.w[:, None]).T.contiguous(), G, na)
            R += G * (vol * 2.0 / self.h[d])
        del Q, P, G
        for d in range(dim):
            ca, na = self.axes(d)
            left, right = U.select(na, self.p), torch.roll(U.select(na, 0), -1, ca)
            # node axes left of the face, in the array without axis na
            rest = [self.axes(a)[1] - (1 if self.axes(a)[1] > na else 0) for a in range(dim) if a != d]
            for ax in rest:
                left, right = self.along(self.Bf, left, ax), self.along(self.Bf, right, ax)
            F = self.numerical(left, right, d) * (vol * 2.0 / self.h[d])
            for ax in rest:
                F = self.along((self.Bf * self.wf[:, None]).T.contiguous(), F, ax)
            R.select(na, self.p).sub_(F)
            R.select(na, 0).add_(torch.roll(F, 1, ca))
        for d in range(dim):
            R = self.along(self.minv, R, self.axes(d)[1])
        return R / vol

    def rk4(self, U, dt, steps):
        for _ in range(steps):
            k = self.rate(U) * dt
            total = k
            k = self.rate(U + 0.5 * k) * dt
            total = total + 2.0 * k
            k = self.rate(U + 0.5 * k) * dt
            total = total + 2.0 * k
            k = self.rate(U + k) * dt
            U = U + (total + k) / 6.0
        return U


def _vortex_fcn(data, dim, t=0.0):
    _, ub, vb, _, beta, xc, yc, lx, ly = data

    def fcn(x, y, z=None):
        xr, yr = x - xc - ub * t, y - yc - vb * t
        xr = xr - lx * torch.floor(xr / lx + 0.5)
        yr = yr - ly * torch.floor(yr / ly + 0.5)
        r2 = xr * xr + yr * yr
        s = beta / (2 * math.pi) * torch.exp(0.5 * (1.0 - r2))
        T = 1.0 - (GAMMA - 1.0) * beta ** 2 / (8 * GAMMA * math.pi ** 2) * torch.exp(1.0 - r2)
        u, v = ub - s * yr, vb + s * xr
        rho = T ** (1.0 / (GAMMA - 1.0))
        E = rho * T / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)
        mom = [rho * u, rho * v] + ([torch.zeros_like(rho)] if dim == 3 else [])
        return torch.stack([rho] + mom + [E])
    return fcn


def _taylor_green_fcn(mach):
    def fcn(x, y, z):
        u, v = torch.sin(x) * torch.cos(y) * torch.cos(z), -torch.cos(x) * torch.sin(y) * torch.cos(z)
        P = 1.0 / (GAMMA * mach ** 2) + (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0) / 16.0
        return torch.stack([torch.ones_like(u), u, v, torch.zeros_like(u), P / (GAMMA - 1.0) + 0.5 * (u * u + v * v)])
    return fcn


def _by_element(U, mesh, n, h, p):
    """[variable, cells, nodes] of a box as [element, variable, node] of a mesh of it:
    each element's cell from its nodes, each of its basis nodes from its own axes."""
    dim = len(n)
    X = mesh.node_coords[mesh.elem_to_node_ids.astype(np.int64)]
    h = np.asarray(h)
    lo = X.min(1)
    cell = np.rint(lo / h).astype(np.int64)
    edge = np.stack([X[:, 1 << a] - X[:, 0] for a in range(dim)], 1)
    idx = np.indices((p + 1,) * dim)[::-1].reshape(dim, -1).T / p  # x fastest
    pos = np.rint((X[:, :1] + np.einsum("ia,ead->eid", idx, edge) - lo[:, None]) / h * p).astype(np.int64)
    node = np.zeros(pos.shape[:2], np.int64)
    at = np.zeros(len(cell), np.int64)
    for d in reversed(range(dim)):
        node = node * (p + 1) + pos[:, :, d]
        at = at * n[d] + cell[:, d]
    nb = (p + 1) ** dim
    flat = U.reshape(U.shape[0], -1, nb)[:, torch.from_numpy(at).to(U.device)].transpose(0, 1)
    return torch.gather(flat, 2, torch.from_numpy(node).to(U.device)[:, None].expand(-1, U.shape[0], -1))


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "bent":
        return None
    if kind == "ensemble":
        out = []
        for n, p, data in _ensemble_cases(case, seed):
            h = (LENGTH / n,) * 3
            s = _Scheme(p, h, case["flux"], p + 2, dev)
            dt = _time_step(case["precision"], p, LENGTH / n, _vortex_speed(data))
            U = s.rk4(s.project(_vortex_fcn(data, 3), (n, n, n)), dt, case["steps"])
            mesh = dg_b200.periodic_box((n, n, n), (0.0, 0.0, 0.0), (LENGTH,) * 3)
            out.append(_by_element(U, mesh, (n, n, n), h, p).transpose(1, 2).contiguous())
        return out
    if kind == "quad":
        rng = random.Random(int(seed) * 7919 + 29)
        n, p, data = (case["nx"], case["ny"]), case["order"], _vortex(rng)
        h = tuple(LENGTH / v for v in n)
        s = _Scheme(p, h, case["flux"], p + 1, dev)
        U = s.rk4(s.project(_vortex_fcn(data, 2), n), _time_step(FP64, p, LENGTH / max(n), _vortex_speed(data)),
                  case["steps"])
        mesh = dg_b200.periodic_box_2d(n, (0.0, 0.0), (LENGTH, LENGTH))
        return _by_element(U, mesh, n, h, p).transpose(1, 2).contiguous()
    mesh, length, name, data, dt = _setup(case, seed)
    n, p = (case["nx"], case["ny"], case["nz"]), case["order"]
    h = tuple(length / v for v in n)
    s = _Scheme(p, h, case["flux"], p + 2, dev)
    fcn = _taylor_green_fcn(data[0]) if name == "TaylorGreen" else _vortex_fcn(data, 3)
    U = s.rk4(s.project(fcn, n), dt, case["steps"])
    state = _by_element(U, mesh, n, h, p)
    if kind == "roundtrip":
        return {"U": state.transpose(1, 2).contiguous(), "l2_error": None}
    if name == "TaylorGreen":
        return {"U": state, "kinetic_energy": None}
    return {"U": state}
