"""Workloads of the D3Q19 time step, its diagnostics and its adjoint, for timing.

A case is a lattice with its boundary flags, body, storage precision and what a program
does with it in one pass:

  run          `steps` time steps, then the force history of these steps and the whole state
  monitored    as run, but one step per call and the force read after each
  restart      a state uploaded from page-locked host memory, then as monitored
  production   `steps` time steps, then what a long run writes out: the force history, the
               monitor, probes, and the profiles of plane means along every axis (the state
               itself would be 9 to 20 GB per pass)
  diagnostics  every reader of a state once: monitor, plane means, lines, control-volume
               drag, region sums, probes
  adjoint      `steps` partial-bounce-back steps and their checkpointed discrete adjoint

`prepare` makes the solver and its inputs, `run` one pass, `exact` the same outputs from an
independent FP64 formulation in plain torch.
"""
import math

import numpy as np
import torch

import euplectella_hpc_b200 as eup
from euplectella_hpc_b200 import workloads

U_IN = 0.05

# Boundary flags (front, rear, right, left, up, down).
BC = {
    "channel": (5, 4, 3, 3, 0, 0),   # inflow/outflow, free-slip y, periodic z
    "tunnel": (5, 4, 3, 3, 3, 3),    # inflow/outflow, free-slip y and z
    "cavity": (1, 1, 1, 1, 2, 1),    # closed box under a moving lid
    "duct": (0, 0, 3, 3, 1, 1),      # periodic x with a body force, free-slip y, no-slip z
    "couette": (0, 0, 0, 0, 2, 1),   # periodic x and y under a moving lid
}
PRECISION = {"fp32": eup.FP32, "fp64": eup.FP64, "fp16": eup.FP16_DEV, "bf16": eup.BF16_DEV}
STORE_BYTES = {"fp32": 4, "fp64": 8, "fp16": 2, "bf16": 2}


def _case(name, kind, size, bc, body, precision, steps, svisc, d, **more):
    lx, ly, lz = size
    return {"name": name, "kind": kind, "lx": lx, "ly": ly, "lz": lz, "bc": bc, "body": body,
            "precision": precision, "steps": steps, "svisc": svisc, "d": float(d), **more}


def listed():
    return [
        # first contact and unit checks: a 16k-node channel, one step per call, the force watched
        _case("monitored_64x32x8_fp32", "monitored", (64, 32, 8), "channel", "cylinder", "fp32", 20, 0.004, 8),
        # the cylinder channel at Re 100 of the parity runs and precision studies, in the
        # reference's precision, in 16-bit storage, and as the FP64 run both are held to
        _case("channel_256x128x64_fp32", "run", (256, 128, 64), "channel", "cylinder", "fp32", 200, 0.01, 20),
        _case("channel_256x128x64_fp16", "run", (256, 128, 64), "channel", "cylinder", "fp16", 400, 0.01, 20),
        _case("channel_256x128x64_fp64", "run", (256, 128, 64), "channel", "cylinder", "fp64", 100, 0.01, 20),
        # lid-driven cavity with nodes at the centre lines: odd row length, walls all round
        _case("cavity_127_fp32", "run", (127, 127, 127), "cavity", "none", "fp32", 100, 0.02, 16),
        # half-scale reticular shell: an ordinary study run that writes its state
        _case("shell_384x192x192_fp32", "run", (384, 192, 192), "tunnel", "shell", "fp32", 100, 0.0048, 48),
        # the production lattices
        _case("shell_768x384x384_fp32", "production", (768, 384, 384), "tunnel", "shell", "fp32", 100, 0.0024, 96),
        _case("ridged_1024x512x512_fp16", "production", (1024, 512, 512), "tunnel", "ridged", "fp16", 60, 0.0024, 96),
        # a restarted half-scale run: state in, 20 watched steps, state out
        _case("restart_384x192x192_fp32", "restart", (384, 192, 192), "tunnel", "shell", "fp32", 20, 0.0048, 48),
        # one diagnostics interval of a run
        _case("diagnostics_384x192x192_fp32", "diagnostics", (384, 192, 192), "tunnel", "shell", "fp32", 1, 0.0048, 48),
        # drag gradient for every voxel: a design step, and the size gradients are checked at
        _case("adjoint_192x96x96_fp32", "adjoint", (192, 96, 96), "channel", "fraction", "fp32", 400, 0.012, 24,
              avg=100, checkpoints=16),
        _case("adjoint_48x24x12_fp64", "adjoint", (48, 24, 12), "channel", "fraction", "fp64", 150, 0.004, 8,
              avg=50, checkpoints=8),
    ]


def draw(rng):
    kind = rng.choice(["run"] * 5 + ["monitored", "restart", "diagnostics", "adjoint", "adjoint"])
    precision = rng.choice(["fp32", "fp32", "fp64", "fp16", "bf16"])
    top = {"monitored": 2e5, "adjoint": 2e6, "run": 1.4e7}.get(kind, 1e7)
    low = {"adjoint": 1.4e4}.get(kind, 1.6e4)
    n = math.exp(rng.uniform(math.log(low), math.log(top)))
    ay, az = rng.uniform(0.3, 1.0), rng.uniform(0.15, 1.0)
    lx = max(24, int(round((n / (ay * az)) ** (1 / 3))))
    ly, lz = max(12, int(round(lx * ay))), max(8, int(round(lx * az)))
    if rng.random() < 0.5:  # a row length that pairs and vectors fit
        lx = (lx + 15) // 16 * 16
    bc = "channel" if kind == "adjoint" else rng.choice(["channel", "channel", "tunnel", "cavity", "duct", "couette"])
    body = {"channel": "cylinder", "tunnel": rng.choice(["cylinder", "block"]), "duct": "block"}.get(bc, "none")
    if kind == "adjoint":
        body = "fraction"
    d = max(6.0, round(0.2 * ly, 1))
    nodes = lx * ly * lz
    steps = int(min(400, max(10, 6e8 / nodes)))
    more = {}
    if kind == "adjoint":
        steps = int(min(300, max(20, 2e8 / nodes)))
        more = {"avg": max(1, steps // 4), "checkpoints": rng.choice([4, 8, 16])}
    elif kind in ("monitored", "restart"):
        steps = 20
    elif kind == "diagnostics":
        steps = 1
    svisc = round(math.exp(rng.uniform(math.log(0.008), math.log(0.05))), 4)
    c = _case("", kind, (lx, ly, lz), bc, body, precision, steps, svisc, d, **more)
    del c["name"]
    return c


# ---- inputs --------------------------------------------------------------------------

def _dtype(case):
    return torch.float64 if case["precision"] == "fp64" else torch.float32


def _body_force_u0(case):
    return 0.05 if case["bc"] == "duct" else 0.0


def _centre(case):
    return case["lx"] / 4.0, (case["ly"] + 1) / 2.0, (case["lz"] + 1) / 2.0


def _config(case):
    open_x = case["bc"] in ("channel", "tunnel")
    return eup.Config(case["lx"], case["ly"], case["lz"], bc=BC[case["bc"]], svisc=case["svisc"],
                      u0=_body_force_u0(case), u_inflow=U_IN if open_x else 0.0,
                      u00=0.1 if BC[case["bc"]][4] == eup.LID else 0.0, precision=PRECISION[case["precision"]],
                      cd_uref=U_IN, cd_length=case["d"], cd_span=float(case["lz"]))


def _geometry(case):
    xc, yc, zc = _centre(case)
    if case["body"] == "cylinder":
        return eup.Geometry.cylinder_z(xc, yc, 0.5 * case["d"])
    s = case["d"] / 96.0  # the shells' lengths scale with their diameter
    if case["body"] == "shell":
        return eup.Geometry.reticular_shell(xc, 256.0 * s, yc, zc, 96.0 * s, 4.0 * s, 16.0 * s, 2024)
    if case["body"] == "ridged":
        return eup.Geometry.ridged_shell(xc, 256.0 * s, yc, zc, 96.0 * s, 4.0 * s, 16.0 * s, 8.0 * s, 4.0 * s,
                                         4.0 * s, 10.0 * s, 2025)
    return None


def _block(case):
    l, m, n = case["lx"], case["ly"], case["lz"]
    obs = np.zeros((n, m, l), np.int32)
    w = max(2, int(case["d"]) // 2)
    x0 = l // 3
    obs[n // 3:2 * n // 3, m // 3:2 * m // 3, x0:x0 + w] = 1
    return obs


# D3Q19 velocities and weights in the order of the populations a01 .. a19.
_C = ((1, -1, 0), (1, 0, -1), (1, 1, 0), (1, 0, 1), (1, 0, 0), (0, 0, 1), (0, 1, 1), (0, 1, 0), (0, 1, -1),
      (-1, -1, 0), (-1, 0, -1), (-1, 1, 0), (-1, 0, 1), (-1, 0, 0), (0, 0, -1), (0, -1, -1), (0, -1, 0), (0, -1, 1),
      (0, 0, 0))
_W = tuple(1 / 3 if not any(c) else (1 / 18 if sum(map(abs, c)) == 1 else 1 / 36) for c in _C)
_OPP = tuple(_C.index((-c[0], -c[1], -c[2])) for c in _C)


def _initial(case, seed):
    """Equilibrium at rho near 1 about the inlet velocity, a random 1e-4 on each component,
    halo included, in the precision a program hands over; on the GPU."""
    shape = (case["lz"] + 2, case["ly"] + 2, case["lx"] + 2)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = _dtype(case)
    u = [torch.rand(shape, generator=gen, device="cuda", dtype=dt).mul_(2e-4).sub_(1e-4) for _ in range(3)]
    if case["bc"] in ("channel", "tunnel"):
        u[0] += U_IN
    usq = (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]).mul_(1.5)
    out = torch.empty((19, *shape), device="cuda", dtype=dt)
    for q, (c, w) in enumerate(zip(_C, _W)):
        cu = sum(c[d] * u[d] for d in range(3) if c[d]) if any(c) else torch.zeros((), device="cuda", dtype=dt)
        out[q] = w * (1 + 3 * cu + 4.5 * cu * cu - usq)
    return out


def _solid_fraction(case, seed):
    xc, yc, _ = _centre(case)
    return workloads.solid_fraction_cylinder(case["lx"], case["ly"], case["lz"], case["d"], xc, yc, 0.05, int(seed))


def _probe_points(case):
    xc, yc, zc = (int(v) for v in _centre(case))
    return [(1 + (xc * (t + 1)) % case["lx"], 1 + (yc + t) % case["ly"], 1 + (zc + t) % case["lz"]) for t in range(3)]


def _cv_box(case):
    l, m, n = case["lx"], case["ly"], case["lz"]
    return (l // 8 + 1, l - l // 8, m // 8 + 1, m - m // 8, 1, n)


def _cavity(case):
    _, yc, zc = _centre(case)
    j, k = np.meshgrid(np.arange(1, case["ly"] + 1), np.arange(1, case["lz"] + 1))
    disc = (j - yc) ** 2 + (k - zc) ** 2 < (0.4 * case["d"]) ** 2
    return np.ascontiguousarray(np.broadcast_to(disc[:, :, None], (case["lz"], case["ly"], case["lx"])))


def _pointers(t):
    return [t[q].data_ptr() for q in range(19)]


def prepare(case, seed):
    s = eup.Solver(_config(case))
    st = {"case": case, "solver": s, "elem": 8 if case["precision"] == "fp64" else 4}
    if case["body"] == "block":
        s.set_obstacles(_block(case))
    elif case["body"] == "fraction":
        s.set_solid_fraction(_solid_fraction(case, seed))
    elif case["body"] != "none":
        s.build_obstacles(_geometry(case))
    if case["kind"] == "production":
        s.init_state(U_IN, 1e-4, int(seed))
        return st
    shape = (19, case["lz"] + 2, case["ly"] + 2, case["lx"] + 2)
    host = torch.empty(shape, dtype=_dtype(case), pin_memory=True)
    host.copy_(_initial(case, seed))
    s.upload_ptrs(_pointers(host), st["elem"])
    st["host"] = host
    if case["kind"] == "restart":
        st["out"] = torch.empty(shape, dtype=_dtype(case), pin_memory=True)
    if case["kind"] == "diagnostics":
        st["region"] = _cavity(case)
    return st


def _state_to_host(st, buf):
    st["solver"].download_ptrs(_pointers(buf), st["elem"])
    return buf


def run(st):
    case, s = st["case"], st["solver"]
    kind, steps = case["kind"], case["steps"]
    if kind == "run":
        s.step(steps)
        return {"force": s.force_series(s.itime - steps, steps + 1), "state": _state_to_host(st, st["host"])}
    if kind in ("monitored", "restart"):
        if kind == "restart":
            s.upload_ptrs(_pointers(st["host"]), st["elem"])
        force = np.empty((steps, 3))
        for t in range(steps):
            s.step(1)
            force[t] = s.forces()
        return {"force": force, "state": _state_to_host(st, st["out"] if kind == "restart" else st["host"])}
    if kind == "production":
        s.step(steps)
        return {"force": s.force_series(s.itime - steps, steps + 1), "monitor": s.monitor(),
                "probes": s.probes(_probe_points(case)), "planes": [s.plane_means(axis) for axis in range(3)]}
    if kind == "diagnostics":
        l, m, n = case["lx"], case["ly"], case["lz"]
        return {"monitor": s.monitor(), "planes": [s.plane_means(axis) for axis in range(3)],
                "lines": [s.line(0, (m + 1) // 2, (n + 1) // 2), s.line(1, (l + 1) // 2, (n + 1) // 2),
                          s.line(2, (l + 1) // 2, (m + 1) // 2)],
                "cv_drag": s.cv_drag(_cv_box(case)), "region": s.region_sums(st["region"]),
                "probes": s.probes(_probe_points(case))}
    objective, grad, _ = s.adjoint(steps, case["avg"], case["checkpoints"])
    return {"objective": objective, "gradient": grad}


def work(case):
    """Bytes and operations of one pass: each step reads and writes every population once; an
    adjoint step reads the state, the adjoint field and the solid fraction and updates the
    adjoint field and the gradient.  About 260 operations per node and step, 700 per node of
    an adjoint step."""
    nodes = case["lx"] * case["ly"] * case["lz"]
    haloed = (case["lx"] + 2) * (case["ly"] + 2) * (case["lz"] + 2)
    sb = STORE_BYTES[case["precision"]]
    rb = 8 if case["precision"] == "fp64" else 4
    kind, steps = case["kind"], case["steps"]
    step_bytes, transfer = 2 * 19 * sb * nodes, 19 * haloed * rb
    if kind in ("run", "monitored"):
        return {"bytes": steps * step_bytes + transfer, "flops": 260.0 * nodes * steps}
    if kind == "restart":
        return {"bytes": steps * step_bytes + 2 * transfer, "flops": 260.0 * nodes * steps}
    if kind == "production":
        return {"bytes": steps * step_bytes + 19 * sb * nodes, "flops": 260.0 * nodes * steps}
    if kind == "diagnostics":
        return {"bytes": 19 * sb * nodes + nodes, "flops": 4 * 60.0 * nodes}
    adjoint = (19 * sb + 2 * 19 * rb + rb + 16) * nodes
    return {"bytes": steps * (step_bytes + adjoint), "flops": 960.0 * nodes * steps}


# ---- the same in 64 bits ---------------------------------------------------------------
# The reference's step on one array of haloed populations f[q][k][j][i].

class _Lattice:
    def __init__(self, case, f, solid=None, ns=None):
        self.case, self.f, self.ns = case, f, ns
        self.l, self.m, self.n = case["lx"], case["ly"], case["lz"]
        self.bc = BC[case["bc"]]
        self.u_in = U_IN if case["bc"] in ("channel", "tunnel") else 0.0
        self.lid = (0.1 if self.bc[4] == eup.LID else 0.0) / 6.0
        sv = case["svisc"]
        self.omega = 2.0 / (6.0 * sv + 1.0)
        self.fgrad = 4.0 * _body_force_u0(case) * sv / (5.0 * self.n * self.n)
        self.links = []  # per q: solid nodes with fluid or halo beyond, and the momentum-exchange links
        if solid is not None and bool(solid.any()):
            n, m, l = solid.shape
            hal = torch.zeros((n + 2, m + 2, l + 2), dtype=torch.bool, device=f.device)
            hal[1:-1, 1:-1, 1:-1] = solid
            wrap = hal.clone()  # the solids seen across periodic axes; walls count as solid
            wrap[:, :, 0], wrap[:, :, -1] = (wrap[:, :, -2], wrap[:, :, 1]) if self.bc[0] == 0 else (True, True)
            wrap[:, 0], wrap[:, -1] = (wrap[:, -2], wrap[:, 1]) if self.bc[2] == 0 else (True, True)
            wrap[0], wrap[-1] = (wrap[-2], wrap[1]) if self.bc[4] == 0 else (True, True)
            for q in range(18):
                cx, cy, cz = _C[q]
                k, j, i = torch.nonzero(solid, as_tuple=True)
                k, j, i = k + 1, j + 1, i + 1
                open_ = ~hal[k + cz, j + cy, i + cx]
                fluid = ~wrap[k + cz, j + cy, i + cx]
                here = (k[open_], j[open_], i[open_])
                there = (k[open_] + cz, j[open_] + cy, i[open_] + cx)
                fk, fj, fi = k[fluid] + cz, j[fluid] + cy, i[fluid] + cx
                inside = ((fk - 1) % n + 1, (fj - 1) % m + 1, (fi - 1) % l + 1)
                self.links.append((q, here, there, inside))

    def force(self):
        out = torch.zeros(3, dtype=torch.float64, device=self.f.device)
        for q, _, _, inside in self.links:
            s = self.f[_OPP[q]][inside].sum()
            out -= 2.0 * s * torch.tensor(_C[q], dtype=torch.float64, device=self.f.device)
        return out

    def bounce(self):
        for q, here, there, _ in self.links:
            self.f[q][here] = self.f[_OPP[q]][there]

    def halo(self):
        """The halo blocks in the reference's order (populations 1-based as in its source)."""
        f, l, m, n, bc = self.f, self.l, self.m, self.n, self.bc
        J, K, I = slice(1, m + 1), slice(1, n + 1), slice(1, l + 1)

        def a(q, k, j, i):
            return f[q - 1][k, j, i]

        def put(q, k, j, i, v):
            f[q - 1][k, j, i] = v

        def sh(s, d):
            return slice(s.start + d, s.stop + d)

        if bc[0] == 0:
            put(12, K, 0, l + 1, a(12, K, m, 1).clone())
            for q in range(10, 15):
                put(q, K, J, l + 1, a(q, K, J, 1))
        elif bc[0] == 1:
            for q, src, dk, dj in ((12, 1, 0, -1), (13, 2, -1, 0), (10, 3, 0, 1), (11, 4, 1, 0), (14, 5, 0, 0)):
                put(q, sh(K, dk), sh(J, dj), l + 1, a(src, K, J, l))
        else:
            col = f[:18, 1:n + 1, 1:m + 1, l]
            j = [sum(_C[q][d] * col[q] for q in range(18) if _C[q][d]) for d in range(3)]
            jj = j[0] ** 2 + j[1] ** 2 + j[2] ** 2
            for q in range(9, 14):
                cj = sum(_C[q][d] * j[d] for d in range(3) if _C[q][d])
                put(q + 1, K, J, l + 1, _W[q] * (1 + 3 * cj + 1.5 * (3 * cj * cj - jj)))
                put(q + 1, 0, J, l + 1, a(q + 1, 1, J, l + 1).clone())
                put(q + 1, n + 1, J, l + 1, a(q + 1, n, J, l + 1).clone())
                put(q + 1, K, 0, l + 1, a(q + 1, K, 1, l + 1).clone())
                put(q + 1, K, m + 1, l + 1, a(q + 1, K, m, l + 1).clone())
        if bc[1] == 0:
            put(1, K, m + 1, 0, a(1, K, 1, l).clone())
            for q in range(1, 6):
                put(q, K, J, 0, a(q, K, J, l))
        elif bc[1] == 1:
            for q, src, dk, dj in ((3, 10, 0, -1), (4, 11, -1, 0), (1, 12, 0, 1), (2, 13, 1, 0), (5, 14, 0, 0)):
                put(q, sh(K, dk), sh(J, dj), 0, a(src, K, J, 1))
        else:
            for q in range(5):
                cu = _C[q][0] * self.u_in
                f[q][:, :, 0] = _W[q] * (1 + 3 * cu + 1.5 * (3 * cu * cu - self.u_in ** 2))
        if bc[4] == 0:
            for q in (2, 9, 11, 15, 16):
                put(q, n + 1, J, I, a(q, 1, J, I))
        elif bc[4] in (1, 2):
            for q, src, dj, di, sgn in ((15, 6, 0, 0, 0), (2, 13, 0, -1, 1), (9, 18, -1, 0, 0), (11, 4, 0, 1, -1),
                                        (16, 7, 1, 0, 0)):
                put(q, n + 1, sh(J, dj), sh(I, di), a(src, n, J, I) + (sgn * self.lid if bc[4] == 2 else 0.0))
        else:
            for q, src in ((15, 6), (11, 13), (16, 18), (2, 4), (9, 7)):
                f[q - 1][n + 1] = f[src - 1][n].clone()
        if bc[5] == 0:
            for q in (4, 6, 7, 13, 18):
                put(q, 0, J, I, a(q, n, J, I))
        elif bc[5] == 1:
            for q, src, dj, di in ((6, 15, 0, 0), (4, 11, 0, -1), (7, 16, -1, 0), (13, 2, 0, 1), (18, 9, 1, 0)):
                put(q, 0, sh(J, dj), sh(I, di), a(src, 1, J, I))
        else:
            for q, src in ((6, 15), (13, 11), (18, 16), (4, 2), (7, 9)):
                put(q, 0, J, I, a(src, 1, J, I))
        if bc[3] == 0:
            put(3, K, 0, 0, a(3, K, m, l).clone())
            for q in (3, 7, 8, 9, 12):
                put(q, K, 0, I, a(q, K, m, I))
        elif bc[3] == 1:
            for q, src, dk, di in ((8, 17, 0, 0), (12, 1, 0, 1), (3, 10, 0, -1), (7, 16, -1, 0), (9, 18, 1, 0)):
                put(q, sh(K, dk), 0, sh(I, di), a(src, K, 1, I))
        else:
            for q, src in ((8, 17), (3, 1), (12, 10), (9, 16), (7, 18)):
                put(q, K, 0, I, a(src, K, 1, I))
        if bc[2] == 0:
            put(10, K, m + 1, l + 1, a(10, K, 1, 1).clone())
            for q in (1, 10, 16, 17, 18):
                put(q, K, m + 1, I, a(q, K, 1, I))
        elif bc[2] == 1:
            for q, src, dk, di in ((10, 3, 0, 1), (16, 7, 1, 0), (17, 8, 0, 0), (18, 9, -1, 0), (1, 12, 0, -1)):
                put(q, sh(K, dk), m + 1, sh(I, di), a(src, K, m, I))
        else:
            for q, src in ((1, 3), (18, 7), (17, 8), (16, 9), (10, 12)):
                put(q, K, m + 1, I, a(src, K, m, I))
        if bc[3] == 3 and bc[4] == 3:
            put(9, n + 1, 0, I, a(18, n, 1, I))
        if bc[2] == 3 and bc[4] == 3:
            put(16, n + 1, m + 1, I, a(7, n, m, I))
        if bc[2] == 3 and bc[5] == 3:
            put(18, 0, m + 1, I, a(9, 1, m, I))
        if bc[3] == 3 and bc[5] == 3:
            put(7, 0, 0, I, a(16, 1, 1, I))

    def pulled(self):
        n, m, l = self.n, self.m, self.l
        return [self.f[q][1 - c[2]:n + 1 - c[2], 1 - c[1]:m + 1 - c[1], 1 - c[0]:l + 1 - c[0]]
                for q, c in enumerate(_C)]

    def collided(self, p):
        rho = sum(p)
        u = [sum(_C[q][d] * p[q] for q in range(18) if _C[q][d]) / rho for d in range(3)]
        usq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
        out = []
        for q in range(19):
            cu = sum(_C[q][d] * u[d] for d in range(3) if _C[q][d]) if q < 18 else 0.0 * rho
            feq = rho * _W[q] * (1 + 3 * cu + 4.5 * cu * cu - usq)
            out.append((1 - self.omega) * p[q] + self.omega * feq + _C[q][0] * self.fgrad * rho)
        return out

    def step(self):
        """One step in place; with a solid fraction returns the force its voxels take."""
        force = None
        if self.ns is None:
            self.bounce()
        self.halo()
        p = [v.clone() for v in self.pulled()]
        new = self.collided(p)
        if self.ns is not None:
            force = torch.stack([(2.0 * self.ns * sum(_C[q][d] * p[q] for q in range(18) if _C[q][d])).sum()
                                 for d in range(3)])
            new = [(1 - self.ns) * new[q] + self.ns * p[_OPP[q]] for q in range(19)]
        for q in range(19):
            self.f[q][1:-1, 1:-1, 1:-1] = new[q]
        return force


def _solid(case):
    l, m, n = case["lx"], case["ly"], case["lz"]
    if case["body"] == "block":
        return torch.from_numpy(_block(case)).cuda().bool()
    xc, yc, _ = _centre(case)
    x = torch.arange(1, l + 1, device="cuda", dtype=torch.float64)[None, None, :] - xc
    y = torch.arange(1, m + 1, device="cuda", dtype=torch.float64)[None, :, None] - yc
    return (x * x + y * y <= (0.5 * case["d"]) ** 2).expand(n, m, l).contiguous()


def _macro(f):
    rho = f.sum(0)
    u = [sum(_C[q][d] * f[q] for q in range(18) if _C[q][d]) / rho for d in range(3)]
    return rho, u


def _exact_diagnostics(case, f):
    rho, u = _macro(f[:, 1:-1, 1:-1, 1:-1])
    rows = torch.stack([u[0], u[1], u[2], rho], -1).cpu().numpy()  # [k][j][i][4]
    l, m, n = case["lx"], case["ly"], case["lz"]
    planes = [rows.mean((0, 1)), rows.mean((0, 2)), rows.mean((1, 2))]
    cj, ck, ci = (m + 1) // 2 - 1, (n + 1) // 2 - 1, (l + 1) // 2 - 1
    probes = np.stack([np.concatenate([rows[k - 1, j - 1, i - 1, 3:], rows[k - 1, j - 1, i - 1, :3]])
                       for i, j, k in _probe_points(case)])
    return {"monitor": None, "planes": planes, "lines": [rows[ck, cj], rows[ck, :, ci], rows[:, cj, ci]],
            "cv_drag": None, "region": None, "probes": probes}


def _exact_adjoint(case, f, ns):
    ns = ns.clone().requires_grad_(True)
    total = torch.zeros((), dtype=torch.float64, device=f.device)
    for t in range(case["steps"]):
        lat = _Lattice(case, f.clone(), ns=ns)
        # the halo is written into a copy, the interior into another: autograd sees no overwrite
        lat.halo()
        p = lat.pulled()
        new = lat.collided(p)
        jx = sum(_C[q][0] * p[q] for q in range(18) if _C[q][0])
        if t >= case["steps"] - case["avg"]:
            total = total + (2.0 * ns * jx).sum()
        inner = torch.stack([(1 - ns) * new[q] + ns * p[_OPP[q]] for q in range(19)])
        f = lat.f.clone()
        f[:, 1:-1, 1:-1, 1:-1] = inner
    norm = 0.5 * U_IN * U_IN * case["d"] * case["lz"]
    objective = total / (case["avg"] * norm)
    (grad,) = torch.autograd.grad(objective, ns)
    return {"objective": float(objective), "gradient": grad.cpu().numpy()}


def exact(case, seed):
    nodes = case["lx"] * case["ly"] * case["lz"]
    if case["kind"] == "production":
        return None
    if case["kind"] == "diagnostics":
        return _exact_diagnostics(case, _initial(case, seed).double())
    if case["body"] in ("shell", "ridged") or nodes * case["steps"] > 1.5e9:
        return None
    if case["kind"] == "adjoint":
        if nodes * case["steps"] > 4e6:  # every step's tensors are kept for the way back
            return None
        return _exact_adjoint(case, _initial(case, seed).double(),
                              torch.from_numpy(_solid_fraction(case, seed)).cuda())
    with torch.no_grad():
        lat = _Lattice(case, _initial(case, seed).double(), None if case["body"] == "none" else _solid(case))
        force = [lat.force()]
        for _ in range(case["steps"]):
            lat.step()
            force.append(lat.force())
        if case["kind"] != "run":
            force = force[1:]
        return {"force": torch.stack(force).cpu().numpy(), "state": lat.f.cpu()}
