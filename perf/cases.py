"""Cases by which the speed of this framework is measured, and their values in 64 bits.

A case is one call of the public interface (flame3d_mhd_gb300.solver.Flame3D) on one flow:

  op "step"  the solver's main loop on a state U: Q and ghosts from it (q_from_u), then `steps`
             SSP-RK3 steps (time_step) on a side stream, as run.py does after a restart
  op "rhs"   one right-hand side from a ghost-filled Q (rhs)
  op "vjp"   the reverse of one SSP-RK3 step (rk3_step_vjp), the unit of every gradient

The flows are those of the benchmark and of the configurations it names, generated on the GPU:

  "sod"     shock tube on a sinusoidally perturbed grid: zero-gradient x, periodic y, z, inviscid
  "vortex"  Taylor-Green vortex with drift and smooth variations, periodic
  "ramp"    Mach 2.9 viscous flow over a 24-degree compression ramp with its oblique shock:
            profile inflow, isothermal wall, Dirichlet far field, periodic span
  "plate"   the default boundary conditions (inlet, outlet, adiabatic wall, far field, periodic
            span): a boundary layer with a pressure pulse

exact() evaluates the same schemes with plain torch in 64 bits.
"""
from __future__ import annotations

import math
import random
from fractions import Fraction

import torch

NG = 4
GAMMA, RG, PR = 1.4, 287.0, 0.72
GM1 = GAMMA - 1.0
LIN = [c / 420.0 for c in (-3.0, 25.0, -101.0, 319.0, 214.0, -38.0, 4.0)]


# ---- the cases ----------------------------------------------------------------------------
def _case(op, flow, n, name=None, **kw):
    c = {"op": op, "flow": flow, "nx": n[0], "ny": n[1], "nz": n[2], "precision": "fp64", "scheme": "fdm",
         "split": "SW", "character": True, "viscous": flow in ("ramp", "plate"), "les": 0, "weno5": False,
         "steps": 1 if op == "step" else 0}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a test-sized evaluation: one RHS of a tiny vortex, five launches of latency
        _case("rhs", "vortex", (16, 16, 16), "rhs_fp64_vortex_16"),
        # the smallest time loop: a coarse tube while a set-up is tried out
        _case("step", "sod", (32, 16, 16), "step_fp64_sod_32x16x16", steps=4),
        # the benchmark's workload in its four forms: the FP64 drop-in, mixed precision, the
        # reference's own Float32 arrays, and its default finite-volume scheme
        _case("step", "sod", (256, 64, 64), "step_fp64_sod_256x64x64", steps=2),
        _case("step", "sod", (256, 64, 64), "step_mixed_sod_256x64x64", precision="mixed", steps=4),
        _case("step", "sod", (256, 64, 64), "step_ref32_sod_256x64x64", precision="ref32", steps=4),
        _case("step", "sod", (256, 64, 64), "step_fvm_sod_256x64x64", scheme="fvm_eigen"),
        # WENO5 at every face, component-wise: the first configuration's vortex
        _case("step", "vortex", (64, 64, 64), "step_fp64_weno5_vortex_64", character=False, weno5=True, steps=2),
        # sizes that divide no tile, default boundary conditions, another splitting
        _case("step", "plate", (125, 61, 37), "step_fp64_plate_125x61x37", split="AUSM", character=False),
        # the compression ramp at its configuration's size: the largest FP64 and mixed runs
        _case("step", "ramp", (512, 256, 128), "step_fp64_ramp_512x256x128"),
        _case("step", "ramp", (512, 256, 128), "step_mixed_ramp_512x256x128", precision="mixed"),
        # gradients: the viscous vortex's component-wise reverse, the tube's characteristic one
        _case("vjp", "vortex", (128, 128, 128), "vjp_vortex_viscous_128", character=False, viscous=True),
        _case("vjp", "sod", (256, 64, 64), "vjp_sod_256x64x64"),
    ]


def draw(rng: random.Random):
    op = rng.choice(["step", "step", "step", "rhs", "vjp"])
    flow = rng.choice(["sod", "sod", "vortex", "ramp", "plate"])
    precision = "fp64" if op == "vjp" else rng.choice(["fp64", "fp64", "mixed", "ref32"])
    if flow == "ramp" and precision == "ref32":  # profile inflow has no Float32 form
        precision = "mixed"
    scheme = "fdm"
    if flow == "sod" and precision == "fp64" and op != "vjp" and rng.random() < 0.4:
        scheme = rng.choice(["fvm_eigen", "fvm_cons"])
    most = {"vjp": 1.0e6, "step": 4.0e6, "rhs": 8.0e6}[op] * (2.0 if precision != "fp64" else 1.0)
    cells = math.exp(rng.uniform(math.log(4096.0), math.log(most)))
    # aspect ratios of the flows: tubes and ramps are longer than they are wide
    ax, ay = (rng.uniform(2.0, 5.0), rng.uniform(0.8, 1.25)) if flow != "vortex" else (1.0, rng.uniform(0.7, 1.4))
    base = (cells / (ax * ay)) ** (1.0 / 3.0)
    n = [max(8, int(round(base * f))) for f in (ax, ay, 1.0)]
    if rng.random() < 0.5:  # sizes of real grids are often multiples of 8
        n = [max(8, v // 8 * 8) for v in n]
    kw = {"precision": precision, "scheme": scheme, "character": rng.random() < 0.6,
          "split": rng.choice(["SW", "SW", "SW", "LF", "VL", "AUSM"])}
    if flow == "vortex":
        kw["viscous"] = rng.random() < 0.5
        kw["weno5"] = not kw["viscous"] and rng.random() < 0.4
    if flow == "plate" and op != "vjp" and rng.random() < 0.3:
        kw["les"] = 1
    if op == "step":
        kw["steps"] = 1 if cells > 1e6 else rng.choice([1, 2, 3])
    return _case(op, flow, n, **kw)


# ---- grids, gas, boundary conditions and initial states -------------------------------------
def _axis(n, h, origin=0.0):
    return origin + (torch.arange(n + 2 * NG, dtype=torch.float64, device="cuda") - NG + 0.5) * h


def _stretch_beta(n, first):
    """beta of s(eta) = 1 - tanh(beta (1 - eta)) / tanh(beta) with s(1/n) = first."""
    lo, hi = 1e-6, 50.0
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        if 1.0 - math.tanh(mid * (1.0 - 1.0 / n)) / math.tanh(mid) > first:
            lo = mid
        else:
            hi = mid
    return 0.5 * (lo + hi)


def _ramp_wall(x, angle, r=0.5):
    return math.tan(angle) * r * torch.logaddexp(torch.zeros_like(x), x / r)


def _flow(case, seed):
    """Gas constants, boundary conditions, coordinates (ghosts included), the primitive state
    (its interior is used), the time step and, for a profile inflow, its state."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    r = random.Random(int(seed))
    f = {"c_s": 1.458e-6, "t_s": 110.4, "phi": (0.05, 1.0, 10.0), "profile": None}
    per, zg = {"kind": "periodic"}, {"kind": "zero_gradient"}

    def noise(shape):
        return 2.0 * torch.rand(shape, generator=g, dtype=torch.float64, device="cuda") - 1.0

    def mesh(ax, ay, az):
        z, y, x = torch.meshgrid(az, ay, ax, indexing="ij")
        return x, y, z

    tp = 2.0 * math.pi
    if case["flow"] == "sod":
        X, E, Z = mesh(_axis(nx, 1.0 / nx), _axis(ny, 1.0 / ny), _axis(nz, 1.0 / nz))
        amp = 0.02
        x = X + amp * torch.sin(tp * E) * torch.sin(tp * Z)
        y = E + amp * torch.sin(tp * Z) * torch.sin(tp * X)
        z = Z + amp * torch.sin(tp * X) * torch.sin(tp * E)
        # the finite-volume scheme has no positivity limit: its diaphragm spans a few cells
        at = 0.5 + 0.02 * (r.random() - 0.5)
        left = (x < at).double() if case["scheme"] == "fdm" else 0.5 + 0.5 * torch.tanh((at - x) * (nx / 1.5))
        rho = 0.125 + 0.875 * left + 1e-3 * noise(x.shape)
        p = 0.1 + 0.9 * left
        # at rest at first; a gradient is taken along a trajectory, of a tube in motion
        u = [torch.full_like(x, a if case["op"] == "vjp" else 0.0) for a in (0.05, 0.03, -0.02)]
        f["bc"] = [zg, zg, per, per, per, per]
        f["dt"] = 0.5 * (1.0 - 2.0 * amp * tp) / max(nx, ny, nz) / math.sqrt(GAMMA / (1.0 - 1e-3))
    elif case["flow"] == "vortex":
        X, Y, Z = mesh(_axis(nx, tp / nx), _axis(ny, tp / ny), _axis(nz, tp / nz))
        amp = 0.05 if case["viscous"] else 0.0
        x = X + amp * torch.sin(Y) * torch.sin(Z)
        y = Y + amp * torch.sin(Z) * torch.sin(X)
        z = Z + amp * torch.sin(X) * torch.sin(Y)
        u0, a = 0.1, [r.uniform(0.0, tp) for _ in range(3)]
        rho = 1.0 + 0.05 * torch.sin(X + 2 * Y + 3 * Z + a[0])
        u = [u0 * torch.sin(X) * torch.cos(Y) * torch.cos(Z) + 0.03,
             -u0 * torch.cos(X) * torch.sin(Y) * torch.cos(Z) + 0.02,
             0.05 + 0.02 * torch.cos(2 * X - Y + Z + a[1])]
        p = (1.0 / GAMMA + u0 ** 2 / 16.0 * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0))
        p = p * (1.0 + 0.03 * torch.cos(3 * X + Y - 2 * Z + a[2]))
        t0 = 1.0 / (GAMMA * RG)
        f["c_s"] = u0 / 1600.0 * (t0 + f["t_s"]) / t0 ** 1.5
        f["bc"] = [per] * 6
        f["dt"] = 0.4 * (1.0 - 2.0 * amp) * tp / max(nx, ny, nz) / 1.2
        if case["weno5"]:
            f["phi"] = (0.0, 0.0, float("inf"))
    elif case["flow"] == "ramp":
        angle, mach, height, span, re, c_inf = math.radians(24.0), 2.9, 10.0, 4.0, 1e5, 1.0
        beta = _stretch_beta(ny, 1e-3 / height)
        xs, et, zs = _axis(nx, 16.0 / nx, -8.0), _axis(ny, 1.0 / ny), _axis(nz, span / nz)
        s = 1.0 - torch.tanh(beta * (1.0 - et)) / math.tanh(beta)
        x, S, z = mesh(xs, s, zs)
        yw = _ramp_wall(x, angle)
        y = yw + (height - yw) * S
        p_inf, u_inf, t_inf = 1.0 / GAMMA, mach * c_inf, 1.0 / (GAMMA * RG)
        f["t_s"] = t_inf * 110.4 / 108.1
        f["c_s"] = u_inf / re * (t_inf + f["t_s"]) / t_inf ** 1.5
        t_w = t_inf * (1.0 + PR ** (1.0 / 3.0) * 0.5 * GM1 * mach ** 2)

        def layer(d):
            q = d.clamp(0.0, 1.0) ** (1.0 / 7.0)
            return t_w + (t_w - t_inf) * q - (t_w - t_inf) * q * q, q

        # the oblique shock of the ramp's angle: theta-beta-M relation, then its jump
        b = angle + 1e-3
        while math.tan(angle) > 2.0 / math.tan(b) * ((mach * math.sin(b)) ** 2 - 1.0) / (
                mach ** 2 * (GAMMA + math.cos(2 * b)) + 2.0):
            b += 1e-4
        m2 = (mach * math.sin(b)) ** 2
        pj = 1.0 + 2.0 * GAMMA / (GAMMA + 1.0) * (m2 - 1.0)
        rj = (GAMMA + 1.0) * m2 / (GM1 * m2 + 2.0)
        vj = math.sqrt(math.cos(b) ** 2 + (math.sin(b) / rj) ** 2)
        w = 0.5 * (1.0 + torch.tanh((x * math.sin(b) - y * math.cos(b)) / (8.0 / nx)))
        T, q = layer(y - yw)
        p = p_inf * (1.0 + w * (pj - 1.0))
        # behind the shock the gas is hotter, down to the wall's temperature at the wall
        rho = p / (RG * T * (1.0 + w * (pj / rj - 1.0) * q * q)) * (1.0 + 1e-3 * noise(x.shape))
        ul = u_inf * q
        u = [ul * (1.0 - w + w * vj * math.cos(angle)), ul * w * vj * math.sin(angle), torch.zeros_like(x)]
        u = [a + 1e-3 * ul * noise(x.shape) for a in u]
        T, q = layer((y - yw)[:, :, NG])
        zero = torch.zeros_like(q)
        f["profile"] = torch.stack([p_inf / (RG * T), u_inf * q, zero, zero, zero + p_inf]).contiguous()
        f["bc"] = [{"kind": "profile"}, zg, {"kind": "isothermal", "t_wall": t_w},
                   {"kind": "dirichlet", "rho": 1.0, "u": u_inf, "v": 0.0, "w": 0.0, "p": p_inf}, per, per]
        first = float(s[NG + 1] - s[NG]) * (height - float(_ramp_wall(xs[-NG - 1], angle)))
        f["dt"] = 0.5 * min(16.0 / nx, first * math.cos(angle), span / nz) / (u_inf + math.sqrt(t_w / t_inf))
    else:  # plate
        X, E, Z = mesh(_axis(nx, 4.0 / nx), _axis(ny, 1.0 / ny), _axis(nz, 1.0 / nz))
        amp = 0.01
        x = X + amp * torch.sin(math.pi * E) * torch.sin(tp * Z)
        y = E + amp * torch.sin(tp * Z) * torch.sin(tp * X)
        z = Z + amp * torch.sin(tp * X) * torch.sin(math.pi * E)
        t0 = 1.0 / (GAMMA * RG)
        f["c_s"] = 0.5 / 1e4 * (t0 + f["t_s"]) / t0 ** 1.5
        cx = [r.uniform(1.2, 2.8), r.uniform(0.3, 0.7), r.uniform(0.3, 0.7)]
        pulse = ((X - cx[0]) ** 2 + (E - cx[1]) ** 2 + (Z - cx[2]) ** 2) < 0.04
        rho = 1.0 + 1e-3 * noise(x.shape)
        p = torch.where(pulse, 1.6, 1.0).double() / GAMMA
        u = 0.5 * (E / 0.2).clamp(0.0, 1.0) ** (1.0 / 7.0)
        u = [u * (a + 1e-2 * noise(x.shape)) for a in (1.0, 0.0, 0.0)]
        fs = {"kind": "dirichlet", "rho": 1.0, "u": 0.5, "v": 0.0, "w": 0.0, "p": 1.0 / 1.4}
        f["bc"] = [fs, zg, {"kind": "adiabatic"}, fs, per, per]
        f["dt"] = 0.3 * min(4.0 / nx, 1.0 / ny, 1.0 / nz) * 0.9 / 2.0
    f["xyz"] = [a.contiguous() for a in (x, y, z)]
    q = torch.zeros((6, *x.shape), dtype=torch.float64, device="cuda")
    body = torch.stack([rho, *u, p, p / (rho * RG)])
    I = (slice(None), *(slice(NG, -NG),) * 3)
    q[I] = body[I]
    f["Q"] = q
    return f


def _prim2c(q):
    e = q[4] / GM1 + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)
    return torch.stack([q[0], q[1] * q[0], q[2] * q[0], q[3] * q[0], e])


def _cotangent(case, seed, U):
    """A seeded cotangent of the final state, smooth and noisy parts, interior cells."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    b = torch.zeros_like(U)
    I = (slice(None), *(slice(NG, -NG),) * 3)
    b[I] = 1.0 + 0.1 * torch.rand(U[I].shape, generator=g, dtype=torch.float64, device="cuda")
    return b


# ---- the framework's side -------------------------------------------------------------------
def prepare(case, seed):
    from flame3d_mhd_gb300 import abi
    from flame3d_mhd_gb300.solver import Flame3D

    f = _flow(case, seed)
    kinds = {"periodic": abi.BC_PERIODIC, "dirichlet": abi.BC_DIRICHLET, "zero_gradient": abi.BC_ZERO_GRADIENT,
             "adiabatic": abi.BC_WALL_ADIABATIC, "isothermal": abi.BC_WALL_ISOTHERMAL,
             "profile": abi.BC_INFLOW_PROFILE}
    ref32 = case["precision"] == "ref32"
    kw = {"gamma": GAMMA, "rg": RG, "pr": PR, "c_s": f["c_s"], "t_s": f["t_s"], "phi1": f["phi"][0],
          "phi2": f["phi"][1], "phi3": f["phi"][2], "character": int(case["character"]),
          "viscous": int(case["viscous"]), "split": case["split"], "les": case["les"],
          "scheme": {"fdm": abi.SCHEME_FDM, "fvm_eigen": abi.SCHEME_FVM_EIGEN,
                     "fvm_cons": abi.SCHEME_FVM_CONS}[case["scheme"]],
          "bc": [dict(b, kind=kinds[b["kind"]]) for b in f["bc"]]}
    n = (case["nx"], case["ny"], case["nz"])
    # metrics from coordinates, on the device and in FP64 as a set-up does
    first = Flame3D(abi.make_params(*n, **kw))
    ms, J = first.compute_metrics(*f["xyz"])
    if case["precision"] == "fp64":
        s = first
    else:
        first.close()
        s = Flame3D(abi.make_params(*n, precision=abi.PREC_REF32 if ref32 else abi.PREC_MIXED, **kw))
    if ref32:
        ms, J = [m.float() for m in ms], J.float()
    s.set_metrics(ms, J)
    if case["scheme"] != "fdm":
        s.set_coordinates(*f["xyz"])
    if f["profile"] is not None:
        s.set_inflow_profile(0, f["profile"])
    U0 = _prim2c(f["Q"]).to(s.dtype).contiguous()
    st = {"case": case, "solver": s, "U0": U0, "U": U0.clone(), "Q": s.field(6), "dt": f["dt"]}
    s.q_from_u(st["U"], st["Q"])
    if case["op"] == "step":
        st["Un"] = s.field(5)
        st["stream"] = torch.cuda.Stream()
    elif case["op"] == "rhs":
        st["out"] = s.field(5)
    else:
        st["bar"] = _cotangent(case, seed, U0)
        st["out"] = s.field(5)
    return st


def run(st):
    from flame3d_mhd_gb300.solver import side_stream

    s, case = st["solver"], st["case"]
    if case["op"] == "rhs":
        return {"L": s.rhs(st["Q"], st["out"])}
    if case["op"] == "vjp":
        return {"U_bar": s.rk3_step_vjp(st["dt"], st["U"], st["bar"], st["out"])}
    st["U"].copy_(st["U0"])
    with side_stream(st["stream"]):
        s.q_from_u(st["U"], st["Q"])
        s.time_step(st["U"], st["Un"], st["Q"], st["dt"], case["steps"])
    return {"U": st["U"], "Q": st["Q"]}


def work(case):
    """Bytes: the state, nine metrics and J (and, finite-volume, coordinates) read once, the
    results written once. Flops per cell and RHS: operation counts of the formulas, adds,
    multiplications, divisions and roots each as one, for the usual branch mix of the flow."""
    cells = case["nx"] * case["ny"] * case["nz"]
    size = 4 if case["precision"] == "ref32" else 8
    arrays = {"rhs": 6 + 10 + 5, "step": 5 + 10 + 5 + 6, "vjp": 5 + 5 + 10 + 5}[case["op"]]
    arrays += 3 if case["scheme"] != "fdm" else 0
    flops = 1700.0 if case["weno5"] else 1100.0 if case["scheme"] == "fdm" else 1500.0
    flops += 400.0 if case["viscous"] else 0.0
    times = {"rhs": 1.0, "step": 3.0 * case["steps"], "vjp": 2.0 + 3.0 * 2.0}[case["op"]]
    return {"bytes": float(cells * size * arrays), "flops": float(cells) * flops * times}


# ---- the schemes in plain torch, 64 bits ------------------------------------------------------
def _weno7_forms():
    """The WENO7 smoothness indicators (expanded quadratic forms of four values) as weighted
    sums of squares of first differences: LDL^T of the 3 x 3 form, in exact fractions."""
    expanded = [
        [(0, 0, 547), (0, 1, -3882), (0, 2, 4642), (0, 3, -1854), (1, 1, 7043), (1, 2, -17246), (1, 3, 7042),
         (2, 2, 11003), (2, 3, -9402), (3, 3, 2107)],
        [(0, 0, 267), (0, 1, -1642), (0, 2, 1602), (0, 3, -494), (1, 1, 2843), (1, 2, -5966), (1, 3, 1922),
         (2, 2, 3443), (2, 3, -2522), (3, 3, 547)],
        [(0, 0, 547), (0, 1, -2522), (0, 2, 1922), (0, 3, -494), (1, 1, 3443), (1, 2, -5966), (1, 3, 1602),
         (2, 2, 2843), (2, 3, -1642), (3, 3, 267)],
        [(0, 0, 2107), (0, 1, -9402), (0, 2, 7042), (0, 3, -1854), (1, 1, 11003), (1, 2, -17246), (1, 3, 4642),
         (2, 2, 7043), (2, 3, -3882), (3, 3, 547)]]
    forms = []
    for terms in expanded:
        V = [[Fraction(0)] * 4 for _ in range(4)]
        for a, b, c in terms:
            V[a][b] += Fraction(c, 2)
            V[b][a] += Fraction(c, 2)
        # value j = value 0 + the first j differences
        M = [[sum(V[a][b] for a in range(i + 1, 4) for b in range(j + 1, 4)) for j in range(3)] for i in range(3)]
        D, L = [], []
        for i in range(3):
            d = M[i][i]
            row = [M[i][j] / d for j in range(i + 1, 3)]
            D.append(float(d))
            L.append([float(v) for v in row])
            for a in range(i + 1, 3):
                for b in range(i + 1, 3):
                    M[a][b] -= row[a - i - 1] * d * row[b - i - 1]
        forms.append((D, L))
    return forms


_W7 = _weno7_forms()


def _weno7(v, s0, eps):
    d = [v[k + 1] - v[k] for k in range(6)]
    num, den = 0.0, 0.0
    q = (-3 * v[0] + 13 * v[1] - 23 * v[2] + 25 * v[3], v[1] - 5 * v[2] + 13 * v[3] + 3 * v[4],
         -v[2] + 7 * v[3] + 7 * v[4] - v[5], 3 * v[3] + 13 * v[4] - 5 * v[5] + v[6])
    for k, (D, L) in enumerate(_W7):
        y = (d[k] + L[0][0] * d[k + 1] + L[0][1] * d[k + 2], d[k + 1] + L[1][0] * d[k + 2], d[k + 2])
        t = eps + (D[0] * y[0] ** 2 + D[1] * y[1] ** 2 + D[2] * y[2] ** 2) * s0
        a = (1.0, 12.0, 18.0, 4.0)[k] / (t * t)
        num, den = num + a * q[k], den + a
    return num / den / 12.0


def _weno5(v, s0, eps):
    s = (13 * (v[0] - 2 * v[1] + v[2]) ** 2 + 3 * (v[0] - 4 * v[1] + 3 * v[2]) ** 2,
         13 * (v[1] - 2 * v[2] + v[3]) ** 2 + 3 * (v[1] - v[3]) ** 2,
         13 * (v[2] - 2 * v[3] + v[4]) ** 2 + 3 * (3 * v[2] - 4 * v[3] + v[4]) ** 2)
    q = (2 * v[0] - 7 * v[1] + 11 * v[2], -v[1] + 5 * v[2] + 2 * v[3], 2 * v[2] + 5 * v[3] - v[4])
    a = [c / (eps + x * s0) ** 2 for c, x in zip((1.0, 6.0, 3.0), s)]
    return (a[0] * q[0] + a[1] * q[1] + a[2] * q[2]) / (a[0] + a[1] + a[2]) / 6.0


def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a.abs() > b.abs(), b, a), torch.zeros_like(a))


def _split(method, q, A):
    """Fp, Fm of every cell for the metric row A."""
    rho, u, v, w, p, T = q
    S = torch.sqrt(A[0] ** 2 + A[1] ** 2 + A[2] ** 2)
    un = A[0] * u + A[1] * v + A[2] * w
    kin = u * u + v * v + w * w
    if method == "SW":
        c = torch.sqrt(GAMMA * RG * T)
        H = [a / S for a in A]
        e = (un, un - c * S, un + c * S)
        vel = ((u - c * H[0], v - c * H[1], w - c * H[2]), (u + c * H[0], v + c * H[1], w + c * H[2]))
        w2 = (3.0 - GAMMA) / (2.0 * GM1) * c * c
        out = []
        for sign in (1.0, -1.0):
            e1, e2, e3 = (0.5 * (x + sign * x.abs()) for x in e)
            F = [2 * GM1 * e1 + e2 + e3]
            for k, x in enumerate((u, v, w)):
                F.append(2 * GM1 * e1 * x + e2 * vel[0][k] + e3 * vel[1][k])
            k2, k3 = (0.5 * (x[0] ** 2 + x[1] ** 2 + x[2] ** 2) for x in vel)
            F.append(GM1 * e1 * kin + e2 * k2 + e3 * k3 + w2 * (e2 + e3))
            out.append(torch.stack(F) * (rho / (2.0 * GAMMA)))
        return out
    c = torch.sqrt(GAMMA * p / rho)
    E = p / GM1 + 0.5 * rho * kin
    U = torch.stack([rho, rho * u, rho * v, rho * w, E])
    P = torch.stack([torch.zeros_like(p), A[0] * p, A[1] * p, A[2] * p, p * un])
    F = U * un + P
    if method == "LF":
        lam = un.abs() + c * S
        return 0.5 * (F + lam * U), 0.5 * (F - lam * U)
    M = un / (c * S)
    if method == "VL":
        unn = un / S

        def side(sg):
            m = sg * 0.25 * rho * c * (M + sg) ** 2 * S
            t = (-unn + sg * 2 * c) / (GAMMA * S)
            en = (GM1 * unn + sg * 2 * c) ** 2 / (2.0 * (GAMMA ** 2 - 1.0)) + 0.5 * (kin - unn ** 2)
            return torch.stack([m, m * (A[0] * t + u), m * (A[1] * t + v), m * (A[2] * t + w), m * en])
    else:  # AUSM
        h = GAMMA * p / (rho * GM1) + 0.5 * kin

        def side(sg):
            m = sg * 0.25 * (M + sg) ** 2 * rho * c * S
            pp = p * 0.25 * (M + sg) ** 2 * (2.0 - sg * M)
            return torch.stack([m, m * u + A[0] * pp, m * v + A[1] * pp, m * w + A[2] * pp, m * h])
    zero = torch.zeros_like(F)
    fp = torch.where(M >= 1, F, torch.where(M <= -1, zero, side(1.0)))
    fm = torch.where(M <= -1, F, torch.where(M >= 1, zero, side(-1.0)))
    return fp, fm


def _tangents(n, eps):
    """Two tangents of the unit normal n; eps is added under the root."""
    nx, ny, nz = n
    flat = nz.abs() <= ny.abs()
    one = torch.ones_like(nx)
    ra = 1.0 / torch.sqrt(torch.where(flat, nx * nx + ny * ny, one) + eps)
    rb = 1.0 / torch.sqrt(torch.where(flat, one, nx * nx + nz * nz) + eps)
    zero = torch.zeros_like(nx)
    l = (torch.where(flat, -ny * ra, -nz * rb), torch.where(flat, nx * ra, zero), torch.where(flat, zero, nx * rb))
    m = (ny * l[2] - nz * l[1], nz * l[0] - nx * l[2], nx * l[1] - ny * l[0])
    return l, m


def _eigen(u, c, H, n, l, m):
    """Rows of the left and columns of the right eigenvectors, fields in the order
    u - c, entropy, u + c, shear, shear."""
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
    q2 = 0.5 * dot(u, u)
    K = GM1 / (c * c)
    qn, ql, qm = dot(u, n), dot(u, l), dot(u, m)
    one, zero = torch.ones_like(c), torch.zeros_like(c)

    def acoustic(sg):
        left = [0.5 * (K * q2 + sg * qn / c)] + [-0.5 * (K * u[k] + sg * n[k] / c) for k in range(3)] + [0.5 * K]
        right = [one] + [u[k] - sg * c * n[k] for k in range(3)] + [H - sg * c * qn]
        return left, right
    fields = [acoustic(1.0), ([one - K * q2] + [K * u[k] for k in range(3)] + [-K], [one, *u, q2]), acoustic(-1.0),
              ([-ql, *l, zero], [zero, *l, ql]), ([-qm, *m, zero], [zero, *m, qm])]
    return fields


def _along(a, d):
    """The sweep's view: transverse interior, direction d (0 = x) last, full extent along it."""
    s = [slice(NG, -NG)] * 3
    s[2 - d] = slice(None)
    return a[(..., *s)].movedim(-1 - d, -1)


def _faces_fdm(case, phi_t, d, q, A, phi):
    fp, fm = _split(case["split"], [_along(x, d) for x in q], [_along(a, d) for a in A])
    N = fp.shape[-1] - 2 * NG
    P = [fp[..., k:k + N + 1] for k in range(8)]
    M = [fm[..., k:k + N + 1] for k in range(8)]
    ph = _along(phi, d)
    top = torch.stack([ph[..., k:k + N + 1] for k in range(1, 7)]).amax(0)
    F = sum(LIN[k] * (P[k] + M[7 - k]) for k in range(7))
    br = torch.where(top < phi_t[0], 0, torch.where(top < phi_t[1], 1, torch.where(top < phi_t[2], 2, 3)))
    S = torch.sqrt(sum(_along(a, d) ** 2 for a in A))
    s0 = 2.0 / (S[..., 3:N + 4] + S[..., 4:N + 5])
    for b in (1, 2, 3):
        at = br == b
        if not bool(at.any()):
            continue
        p, m = [x[:, at] for x in P], [x[:, at] for x in M]
        if b == 3:
            val = p[3] + 0.5 * _minmod(p[4] - p[3], p[3] - p[2]) + m[4] - 0.5 * _minmod(m[5] - m[4], m[4] - m[3])
        else:
            w = s0[at]
            rec = _weno7 if b == 1 else _weno5
            eps = 1e-20 if b == 1 else 1e-16
            side = (lambda x: x) if b == 1 else (lambda x: x[1:6])
            if not case["character"]:
                val = rec(side(p[:7]), w, eps) + rec(side(m[:0:-1]), w, eps)
            else:
                mean = lambda x: (0.5 * (_along(x, d)[..., 3:N + 4] + _along(x, d)[..., 4:N + 5]))[at]  # noqa: E731
                u, T = [mean(q[k]) for k in (1, 2, 3)], mean(q[5])
                n = [mean(a) * w for a in A]
                l, t = _tangents(n, 0.0)
                c = torch.sqrt(GAMMA * RG * T)
                H = c * c / GM1 + 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
                val = 0.0
                for left, right in _eigen(u, c, H, n, l, t):
                    proj = lambda x: sum(left[k] * x[k] for k in range(5))  # noqa: E731
                    f = rec(side([proj(x) for x in p[:7]]), w, eps) + rec(side([proj(x) for x in m[:0:-1]]), w, eps)
                    val = val + torch.stack([right[k] * f for k in range(5)])
        F = F.clone()
        F[:, at] = val
    return F


def _face_geometry(xyz, d):
    """Unit normals and areas of the faces of direction d from cell centres."""
    ta, tb = [(1, 2), (0, 2), (0, 1)][d]
    nd = xyz[0].shape[2 - d] - 2 * NG

    def at(a, side, pa, pb):
        s = [slice(NG, -NG)] * 3
        s[2 - d] = slice(NG - 1 + side, NG + side + nd)
        for ax, o in ((ta, pa), (tb, pb)):
            k = 2 - ax
            s[k] = slice(NG + o, xyz[0].shape[k] - NG + o)
        return a[tuple(s)]

    def diag(a, pa, pb):
        v = 0.0
        for side in (0, 1):
            v = v + at(a, side, pa, 0) + at(a, side, 0, pb) + at(a, side, pa, pb)
            v = v - at(a, side, -pa, 0) - at(a, side, 0, -pb) - at(a, side, -pa, -pb)
        return 0.125 * v
    e, g = [diag(a, 1, 1) for a in xyz], [diag(a, -1, 1) for a in xyz]
    sg = -0.5 if d == 1 else 0.5
    n = [sg * (e[1] * g[2] - e[2] * g[1]), sg * (e[2] * g[0] - e[0] * g[2]), sg * (e[0] * g[1] - e[1] * g[0])]
    area = torch.sqrt(n[0] ** 2 + n[1] ** 2 + n[2] ** 2 + 1e-20)
    return [(x / area).movedim(-1 - d, -1) for x in n], area.movedim(-1 - d, -1)


def _hllc(L, R, n):
    def side(U):
        r, v = U[0], [U[k] / U[0] for k in (1, 2, 3)]
        p = GM1 * (U[4] - 0.5 * r * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2))
        return r, v, p, torch.sqrt((GAMMA * p / r).abs()), sum(a * b for a, b in zip(v, n)), U[4]
    l, r = side(L), side(R)
    sl, sr = torch.sqrt(l[0]), torch.sqrt(r[0])
    roe = lambda a, b: (sl * a + sr * b) / (sl + sr)  # noqa: E731
    v = [roe(a, b) for a, b in zip(l[1], r[1])]
    H = roe((l[5] + l[2]) / l[0], (r[5] + r[2]) / r[0])
    c = torch.sqrt((GM1 * (H - 0.5 * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2))).abs())
    qn = sum(a * b for a, b in zip(v, n))
    SL, SR = torch.minimum(l[4] - l[3], qn - c), torch.maximum(r[4] + r[3], qn + c)
    Ss = (r[2] - l[2] + l[0] * l[4] * (SL - l[4]) - r[0] * r[4] * (SR - r[4])) / (
        l[0] * (SL - l[4]) - r[0] * (SR - r[4]) + 1e-12)

    def flux(x, U, S):
        rho, vel, p, _, q, E = x
        F = torch.stack([rho * q, *(rho * a * q + p * b for a, b in zip(vel, n)), (E + p) * q])
        f = rho * (S - q) / (S - Ss)
        star = torch.stack([f, *(f * (a + (Ss - q) * b) for a, b in zip(vel, n)),
                            f * (E / rho + (Ss - q) * (Ss + p / (rho * (S - q))))])
        return F, F + S * (star - U)
    fl, fls = flux(l, L, SL)
    fr, frs = flux(r, R, SR)
    return torch.where(SL >= 0, fl, torch.where(SR <= 0, fr, torch.where(Ss >= 0, fls, frs)))


def _faces_fvm(case, phi_t, d, q, A, phi, U, xyz):
    u = _along(U, d)
    N = u.shape[-1] - 2 * NG
    V = [u[..., k:k + N + 1] for k in range(8)]
    n, area = _face_geometry(xyz, d)
    ph = _along(phi, d)
    top = torch.stack([ph[..., k:k + N + 1] for k in range(1, 7)]).amax(0)
    S = torch.sqrt(sum(_along(a, d) ** 2 for a in A))
    s0 = 2.0 / (S[..., 3:N + 4] + S[..., 4:N + 5])
    UL = sum(LIN[k] * V[k] for k in range(7))
    UR = sum(LIN[k] * V[7 - k] for k in range(7))

    def rec(b, right, v, w):
        if b == 1:
            return _weno7(v, w, 1e-10)
        if b == 2:
            return _weno5(v[1:6], w, 1e-8)
        return v[3] - 0.5 * _minmod(v[3] - v[2], v[3] - v[4]) if right else v[3] + 0.5 * _minmod(v[3] - v[2],
                                                                                                v[4] - v[3])
    for b in (1, 2, 3):
        at = (top >= (phi_t[b - 1])) & ((top < phi_t[b]) if b < 3 else torch.ones_like(top, dtype=torch.bool))
        if not bool(at.any()):
            continue
        v, w = [x[:, at] for x in V], s0[at]
        if case["scheme"] == "fvm_cons":
            l, r = rec(b, False, v[:7], w), rec(b, True, v[:0:-1], w)
        else:
            a = [_along(x, d)[..., 3:N + 4][at] for x in q]
            z = [_along(x, d)[..., 4:N + 5][at] for x in q]
            ra, rz = torch.sqrt(a[0]), torch.sqrt(z[0])
            roe = lambda x, y: (ra * x + rz * y) / (ra + rz)  # noqa: E731
            vel = [roe(a[k], z[k]) for k in (1, 2, 3)]
            hof = lambda x: GAMMA / GM1 * x[4] / x[0] + 0.5 * (x[1] ** 2 + x[2] ** 2 + x[3] ** 2)  # noqa: E731
            H = roe(hof(a), hof(z))
            c = torch.sqrt(GM1 * (H - 0.5 * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)))
            nn = [x[at] for x in n]
            tl, tm = _tangents(nn, 1e-12)
            l = r = 0.0
            for left, right in _eigen(vel, c, H, nn, tl, tm):
                proj = lambda x: sum(left[k] * x[k] for k in range(5))  # noqa: E731
                pv = [proj(x) for x in v]
                col = torch.stack([x + torch.zeros_like(c) for x in right])
                l, r = l + col * rec(b, False, pv[:7], w), r + col * rec(b, True, pv[:0:-1], w)
        UL, UR = UL.clone(), UR.clone()
        UL[:, at], UR[:, at] = l, r
    return _hllc(UL, UR, n) * area


def _viscous(case, f, q, m, J):
    """Fv of the three directions at full cells 2 .. Nt-3, (4, ...) each."""
    box = slice(2, -2)
    core = lambda a: a[(..., box, box, box)]  # noqa: E731

    def d4(a, d):
        k = a.dim() - 1 - d
        n = a.shape[k]
        s = lambda o: core(a.roll(-o, k)) if n else None  # noqa: E731
        return (s(-2) - s(2)) / 12.0 - (s(-1) - s(1)) * (2.0 / 3.0)
    M = [core(x) for x in m]
    Jc = core(J)
    T = core(q[5])
    mu = f["c_s"] * T * torch.sqrt(T) / (T + f["t_s"])
    cp = RG * GAMMA / GM1
    lam = mu * (cp / PR)
    grad = []
    for k in (1, 2, 3, 5):
        g = [d4(q[k], d) for d in range(3)]
        grad.append([(g[0] * M[x] + g[1] * M[3 + x] + g[2] * M[6 + x]) * Jc for x in range(3)])
    du, gT = grad[:3], grad[3]
    div = du[0][0] + du[1][1] + du[2][2]
    if case["les"] == 1:  # Smagorinsky
        sii = du[0][0] ** 2 + du[1][1] ** 2 + du[2][2] ** 2
        sij = sum((0.5 * (du[a][b] + du[b][a])) ** 2 for a, b in ((0, 1), (0, 2), (1, 2)))
        mut = core(q[0]) * (0.1 * Jc ** (-1.0 / 3.0)) ** 2 * torch.sqrt(2.0 * (sii + 2.0 * sij))
        mut = torch.minimum(mut, 2.0 * mu)
        mu, lam = mu + mut, lam + cp * mut / 0.9
    tau = [[mu * (du[a][b] + du[b][a]) if a != b else mu * (2.0 * du[a][a] - 2.0 / 3.0 * div) for b in range(3)]
           for a in range(3)]
    vel = [core(q[k]) for k in (1, 2, 3)]
    E = [sum(vel[b] * tau[b][a] for b in range(3)) + lam * gT[a] for a in range(3)]
    return [torch.stack([sum(M[3 * d + a] * tau[a][n] for a in range(3)) for n in range(3)]
                        + [sum(M[3 * d + a] * E[a] for a in range(3))]) for d in range(3)]


def _rhs(case, f, q, m, J, xyz, U=None):
    """dU/dt at interior cells from the ghost-filled primitive state."""
    p = q[4].detach()
    phi = 0.0
    for k in range(3):
        lo, hi = p.roll(1, k), p.roll(-1, k)
        phi = phi + (2.0 * p - lo - hi).abs() / (lo + 2.0 * p + hi)
    fv = _viscous(case, f, q, m, J) if case["viscous"] else None
    out = 0.0
    for d in range(3):
        A = m[3 * d:3 * d + 3]
        if case["scheme"] == "fdm":
            F = _faces_fdm(case, f["phi"], d, q, A, phi)
        else:
            F = _faces_fvm(case, f["phi"], d, q, A, phi, U if U is not None else _prim2c(q), xyz)
        D = F[..., :-1] - F[..., 1:]
        if fv is not None:
            s = [slice(2, -2)] * 3
            s[2 - d] = slice(None)
            v = fv[d][(..., *s)].movedim(-1 - d, -1)
            N = v.shape[-1] - 4
            w = lambda o: v[..., 2 + o:2 + o + N]  # noqa: E731
            dv = (w(-2) - w(2)) / 12.0 - (w(-1) - w(1)) * (2.0 / 3.0)
            D = D + torch.cat([torch.zeros_like(dv[:1]), dv])
        out = out + D.movedim(-1, -1 - d)
    return out * J[(slice(NG, -NG),) * 3]


def _fill(f, qi):
    """The ghost-filled primitive state from its interior: x, then y, then z faces."""
    q = qi
    for d in range(3):
        k = 3 - d
        n = q.shape[k]
        sides = []
        for hi in (0, 1):
            b = f["bc"][2 * d + hi]
            inner = lambda a, c: q.narrow(k, a, c)  # noqa: E731
            if b["kind"] == "periodic":
                g = inner(0, NG) if hi else inner(n - NG, NG)
            elif b["kind"] == "zero_gradient":
                g = torch.cat([inner(n - 1 if hi else 0, 1)] * NG, k)
            elif b["kind"] in ("adiabatic", "isothermal"):
                g = (inner(n - NG, NG) if hi else inner(0, NG)).flip(k)
                if b["kind"] == "isothermal":
                    T = 2.0 * b["t_wall"] - g[5]
                    g = torch.stack([g[4] / (RG * T), -g[1], -g[2], -g[3], g[4], T])
                else:
                    g = torch.stack([g[0], -g[1], -g[2], -g[3], g[4], g[5]])
            else:
                shape = list(q.shape[1:])
                shape[k - 1] = NG
                if b["kind"] == "dirichlet":
                    v = [torch.full(shape, b[x], dtype=q.dtype, device=q.device) for x in ("rho", "u", "v", "w", "p")]
                else:  # the profile of an x- face
                    v = [x[NG:-NG, NG:-NG, None].expand(shape) for x in f["profile"]]
                g = torch.stack([*v, v[4] / (v[0] * RG)])
            sides.append(g)
        q = torch.cat([sides[0], q, sides[1]], k)
    return q


def _c2prim(U):
    eps = 2.0 ** -23
    rho = U[0].clamp(min=eps)
    v = [U[k] / rho for k in (1, 2, 3)]
    p = GM1 * (U[4] - 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)).clamp(min=eps)
    return torch.stack([rho, *v, p, p / (rho * RG)])


def _metrics(xyz):
    def diff(a, k):
        n = a.shape[k]
        s = lambda o: a.roll(-o, k)  # noqa: E731
        mid = (s(3) - s(-3)) / 60.0 - (s(2) - s(-2)) * (3.0 / 20.0) + (s(1) - s(-1)) * 0.75
        low = 2.0 * s(1) - 0.5 * s(2) - 1.5 * a
        high = -2.0 * s(-1) + 0.5 * s(-2) + 1.5 * a
        return torch.cat([low.narrow(k, 0, 3), mid.narrow(k, 3, n - 6), high.narrow(k, n - 3, 3)], k)
    (xa, xb, xc), (ya, yb, yc), (za, zb, zc) = [[diff(a, k) for k in (2, 1, 0)] for a in xyz]
    m = [yb * zc - yc * zb, xc * zb - xb * zc, xb * yc - xc * yb, yc * za - ya * zc, xa * zc - xc * za,
         xc * ya - xa * yc, ya * zb - yb * za, xb * za - xa * zb, xa * yb - xb * ya]
    return m, 1.0 / (xa * m[0] + xb * m[3] + xc * m[6])


def exact(case, seed):
    f = _flow(case, seed)
    m, J = _metrics(f["xyz"])
    U0 = _prim2c(f["Q"])
    if case["precision"] == "ref32":  # the Float32 inputs, held in 64 bits
        U0, m, J = U0.float().double(), [a.float().double() for a in m], J.float().double()
    I = (slice(None), *(slice(NG, -NG),) * 3)
    dt = f["dt"]

    def full(a, like):
        b = torch.zeros((a.shape[0], *like.shape[1:]), dtype=torch.float64, device="cuda")
        b[I] = a
        return b

    def L(u):
        q = _fill(f, _c2prim(u))
        return _rhs(case, f, q, m, J, f["xyz"])

    u0 = U0[I]
    if case["op"] == "rhs":
        return {"L": full(L(u0), U0)}
    if case["op"] == "step":
        u = u0
        for _ in range(case["steps"]):
            a = u + dt * L(u)
            b = 0.25 * (a + dt * L(a)) + 0.75 * u
            u = 2.0 / 3.0 * (b + dt * L(b)) + u / 3.0
        q = _fill(f, _c2prim(u))
        U = _prim2c(q)
        U[I] = u
        return {"U": U, "Q": q}

    def back(u, bar):
        x = u.detach().requires_grad_(True)
        return torch.autograd.grad(L(x), x, bar)[0]
    with torch.no_grad():
        u1 = u0 + dt * L(u0)
        u2 = 0.25 * (u1 + dt * L(u1)) + 0.75 * u0
    top = _cotangent(case, seed, U0)[I]
    w = 2.0 / 3.0 * top
    b2 = w + dt * back(u2, w)
    w = 0.25 * b2
    b1 = w + dt * back(u1, w)
    return {"U_bar": full(top / 3.0 + 0.75 * b2 + b1 + dt * back(u0, b1), U0)}
