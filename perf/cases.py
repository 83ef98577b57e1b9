"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is one call sequence through the public entry points over planar Couette domains: explicit
second-order steps (on a `Solver`, operator by operator as a host driver calls them, and on the caller's own
device arrays), the two implicit methods' pseudo-steps, the explicit high-order S2CN2 step, a batch of S2CN2
instances and a gradient through S2CN2 steps.  Inputs are made from a seed: the gas (Knudsen number, wall
speed, wall temperature) and a smooth non-equilibrium state near the uniform one a run starts from.

`exact` restates the explicit second-order step and the S2CN2 step in plain 64-bit torch."""
import ctypes
import functools
import math

import numpy as np
import torch

from ugks2d_high_order_b200 import capi
from ugks2d_high_order_b200.adjoint import wall_outputs
from ugks2d_high_order_b200.batch import Batch
from ugks2d_high_order_b200.case import CouetteCase, batched_cases, velocity_table
from ugks2d_high_order_b200.solver import Solver

METHOD = {"noalloc": "Explicit", "explicit": "Explicit", "operators": "Explicit", "implicit": "ImplicitSteady",
          "high_order": "HighOrderImplicit", "s2cn2": "S2CN2", "batch": "S2CN2", "gradient": "S2CN2"}


def listed():
    return [
        # one step on the caller's own device arrays, the smallest domain of the tests: the latency of a call
        {"name": "noalloc_8x8_v16", "kind": "noalloc", "nx": 8, "ny": 8, "nv": 16, "steps": 1},
        # a host driver that replaces its own routines one by one: four calls a step, small domain, 24^2 table
        {"name": "operators_8x32_v24", "kind": "operators", "nx": 8, "ny": 32, "nv": 24, "steps": 10},
        # the throughput variant of the delivered explicit case (CFL 0.5, omega 0.81), between two outputs
        {"name": "explicit_8x64_v32", "kind": "explicit", "nx": 8, "ny": 64, "nv": 32, "steps": 200},
        # an odd domain with a table above 1024 velocities, where the kernels take their other shapes
        {"name": "explicit_13x51_v48", "kind": "explicit", "nx": 13, "ny": 51, "nv": 48, "steps": 100},
        # the delivered implicit case (8x64 cells, 32^2 velocities, 8 slabs): part of a solve to steady state
        {"name": "implicit_8x64_v32", "kind": "implicit", "nx": 8, "ny": 64, "nv": 32, "nslab": 8, "steps": 200},
        # the delivered high-order implicit case
        {"name": "high_order_8x64_v32", "kind": "high_order", "nx": 8, "ny": 64, "nv": 32, "nslab": 8, "steps": 64},
        # its refined variant, the largest single domain of the benchmark
        {"name": "high_order_16x128_v48", "kind": "high_order", "nx": 16, "ny": 128, "nv": 48, "nslab": 8, "steps": 24},
        # the delivered explicit high-order case
        {"name": "s2cn2_8x64_v32", "kind": "s2cn2", "nx": 8, "ny": 64, "nv": 32, "steps": 64},
        # the same method on a small odd domain and a 20^2 table (no multiple of 32 velocities)
        {"name": "s2cn2_7x21_v20", "kind": "s2cn2", "nx": 7, "ny": 21, "nv": 20, "steps": 25},
        # a parameter sweep: instances of the benchmark's batched distribution (8x{32,64,128} cells, 24^2 to
        # 48^2 velocities), a few steps of each between two outputs
        {"name": "batch_16", "kind": "batch", "instances": 16, "streams": 8, "steps": 10},
        # gradients of the wall outputs of two cases of that distribution at 8x64 cells, 32^2 velocities
        {"name": "gradient_2x8x64_v32", "kind": "gradient", "instances": 2, "ny": 64, "nv": 32, "steps": 40, "every": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(sorted(METHOD))
    nv = 2 * rng.randint(7, 25)                 # 14^2 .. 50^2 velocities
    nx, ny = _log(rng, 4, 20), _log(rng, 9, 140)
    if kind == "batch":
        return {"kind": kind, "instances": rng.randint(2, 15), "streams": rng.randint(1, 8), "steps": rng.randint(2, 10)}
    if kind == "gradient":
        ny, nv = _log(rng, 16, 64), 2 * rng.randint(10, 16)
        return {"kind": kind, "instances": rng.randint(1, 2), "ny": ny, "nv": nv, "steps": rng.randint(4, 40),
                "every": rng.randint(4, 20)}
    if kind == "noalloc":                       # the 36 MiB working set of that entry bounds nx ny nv^2
        ny = min(ny, max(9, int(500000 / (nx * nv * nv)) - 2))
    c = {"kind": kind, "nx": nx, "ny": ny, "nv": nv}
    if kind in ("implicit", "high_order"):
        c["nslab"] = rng.choice((1, 2, 4, 8))
        rows = max(1, min(ny // c["nslab"], 384 // nx))
        rows = max(rows, -(-9 // c["nslab"]))
        c["ny"] = rows * c["nslab"]
    n = nx * c["ny"] * nv * nv
    most = {"noalloc": 2e7, "operators": 2e7, "explicit": 8e7, "implicit": 6e7, "high_order": 3e7, "s2cn2": 3e7}[kind]
    c["steps"] = rng.randint(1, max(1, min(100, int(most / n))))
    return c


@functools.lru_cache(maxsize=None)
def _table(nv):
    return tuple(np.ascontiguousarray(a) for a in velocity_table(nv))


def _couette(case, rng):
    """A gas and walls of the batched distribution's ranges around the delivered case."""
    kn = 10.0 ** rng.uniform(-1.5, -0.5)
    tw = 2.0 * rng.uniform(0.9, 1.1)
    ux = rng.uniform(1.0, 3.0) * math.sqrt(5.0 / 3.0 * 0.5 * tw)
    c = CouetteCase(nx=case["nx"], ny=case["ny"], dx=1.0 / case["nx"], dy=1.0 / case["ny"], mu_ref=kn / math.sqrt(math.pi),
                    wall_ux=(-ux, ux), wall_tnative=(tw, tw), method=METHOD[case["kind"]], nslab=case.get("nslab", 8))
    if case["kind"] in ("noalloc", "explicit", "operators"):
        c = c.with_(cfl=0.5, omega=0.81)
    if case["kind"] in ("implicit", "high_order"):
        c = c.with_(mass_rescale=True, residual_tol=0.0)     # every pass takes all its pseudo-steps
    return c


def _state(c, table, rng):
    """h, b [ny][nx][nvel] and their moments W [ny][nx][4]: a smooth state near the uniform one at rest."""
    u, v, w = table
    x = 2 * np.pi * (np.arange(c.nx) + 0.5)[None, :] / c.nx + rng.uniform(0, 6.28)
    y = np.pi * (np.arange(c.ny) + 0.5)[:, None] / c.ny
    a = rng.uniform(0.01, 0.03, size=4)
    rho = 1.0 + a[0] * np.sin(x) * np.sin(y)
    U, V = a[1] * np.cos(x) * np.sin(2 * y) - 0.05 * np.cos(y), a[2] * np.sin(x) * np.sin(y)
    T = 2.0 * (1.0 + a[3] * np.cos(x) * np.cos(y))
    cx, cy = u - U[..., None], v - V[..., None]
    h = (rho / (np.pi * T))[..., None] * np.exp(-(cx * cx + cy * cy) / T[..., None])
    h *= 1.0 + 0.05 * cx * cy / (1.0 + cx * cx * cy * cy)
    b = 0.5 * c.ck * T[..., None] * h * (1.0 + 0.02 * cy / (1.0 + cy * cy))
    W = np.stack([h @ w, h @ (w * u), h @ (w * v), 0.5 * (h @ (w * (u * u + v * v)) + b @ w)], axis=-1)
    return h, b, W


def _batch_cases(case, seed):
    """The first instances' grids and tables of the benchmark's distribution, with gases and walls by the seed."""
    return [(c.with_(ny=size.ny, dy=size.dy), n) for (c, _), (size, n) in
            zip(batched_cases(case["instances"], seed=1000 + seed), batched_cases(case["instances"]))]


def _gradient_cases(case, seed):
    out = [c.with_(ny=case["ny"], dy=1.0 / case["ny"]) for c, _ in batched_cases(case["instances"], seed=1000 + seed)]
    # the parameters of a case: wall speed, wall temperature, scale of its viscosity
    p = [(c.wall_ux[1], c.wall_tnative[0], 1.0) for c in out]
    return out, torch.tensor(p, dtype=torch.float64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = Batch([(c, _table(n)) for c, n in _batch_cases(case, seed)], max_streams=case["streams"])
        b.set_streams(case["streams"])
        return {"kind": kind, "batch": b, "steps": case["steps"], "rho": 1.0 + 1e-3 * (seed % 97)}
    if kind == "gradient":
        cases, p = _gradient_cases(case, seed)
        return {"kind": kind, "cases": [(c, _table(case["nv"])) for c in cases], "p": p.cuda(),
                "seed": _gradient_seed(case, seed).cuda(), "steps": case["steps"], "every": case["every"]}
    rng = np.random.default_rng(seed)
    c, table = _couette(case, rng), _table(case["nv"])
    state = _state(c, table, rng)
    if kind == "noalloc":
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in table + state]
        return {"kind": kind, "params": Solver.params_for(c, len(table[0])), "dev": dev, "steps": case["steps"], "L": capi.load()}
    lap = _lap(kind)
    into = [_with_halo(np.zeros_like(a), lap) for a in state[:2]] + [np.zeros_like(state[2])]
    state = [_with_halo(a, lap) for a in state[:2]] + [state[2]]
    return {"kind": kind, "solver": Solver(c, *table), "state": state, "into": into, "lap": lap, "steps": case["steps"]}


def _lap(kind):
    """A host driver keeps its distributions with a halo of two cells; other programs without one."""
    return 2 if kind == "operators" else 0


def _with_halo(a, lap):
    return np.pad(a, ((lap, lap), (lap, lap), (0, 0)))


def _gradient_seed(case, seed):
    return torch.from_numpy(np.random.default_rng(seed).uniform(0.5, 1.5, size=(case["instances"], 2, 2)))


def run(s):
    kind, n = s["kind"], s["steps"]
    if kind == "noalloc":
        dt, res = ctypes.c_double(), (ctypes.c_double * 4)()
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in s["dev"]]
        capi.check(s["L"], None, s["L"].ugks_step_explicit_noalloc(
            ctypes.byref(s["params"]), *ptr, n, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
            ctypes.byref(dt), res), "noalloc step")
        return {"h": s["dev"][3], "b": s["dev"][4], "W": s["dev"][5], "dt": dt.value}
    if kind == "batch":
        b = s["batch"]
        b.init_freestream(rho=s["rho"])
        b.run(n)
        return {"state": [b.download(i) for i in range(b.n)], "wall": np.concatenate([b.wall_aero(i) for i in range(b.n)])}
    if kind == "gradient":
        p = s["p"].clone().requires_grad_(True)
        out = wall_outputs(p, s["cases"], n, every=s["every"])
        out.backward(s["seed"])
        return {"wall": out.detach(), "grad": p.grad}
    v = s["solver"]
    v.upload_halo(*s["state"], lap=s["lap"])
    if kind == "explicit":
        v.step_explicit(n)
    elif kind == "operators":
        for _ in range(n):
            v.time_step()
            v.evolution()
            v.compute_residual()
            v.apply_explicit_update()
    elif kind == "s2cn2":
        v.s2cn2_init()
        v.step_s2cn2(n)
    else:
        v.implicit_init()
        v.step_implicit(n)
    h, b, W = s["into"]
    v.download_halo(h, b, W, lap=s["lap"])
    return {"h": h, "b": b, "W": W, "wall": v.wall_aero(), "fields": v.macro_fields()}


def work(case):
    """The state read once and written once a pass; the operations of an update of the plain algorithms, with
    every velocity sum over a tensor table taken factor by factor (about 900 for a second-order step, 2000 for an
    implicit pseudo-step, 6000 for a high-order step, three times that for its transpose)."""
    if case["kind"] == "batch":
        n = sum(c.nx * c.ny * nv * nv for c, nv in _batch_cases(case, 0))
    elif case["kind"] == "gradient":
        n = case["instances"] * 8 * case["ny"] * case["nv"] ** 2
    else:
        n = case["nx"] * case["ny"] * case["nv"] ** 2
    ops = {"implicit": 2000, "high_order": 7000, "s2cn2": 6000, "batch": 6000, "gradient": 18000}.get(case["kind"], 900)
    return {"bytes": 32.0 * n, "flops": float(ops) * n * case["steps"]}


# ----------------------------------------------------------------------------------------------------
# plain 64-bit restatement


def exact(case, seed):
    """The explicit second-order cases and the S2CN2 cases.  None for the implicit methods, whose relaxation
    sweeps go cell by cell (a minute and more a pass in plain torch); no value for the gradient itself."""
    kind, n = case["kind"], case["steps"]
    if kind in ("implicit", "high_order"):
        return None
    if kind == "batch":
        out = [_Plain(c, _table(nv)).s2cn2(*_uniform(c, _table(nv), 1.0 + 1e-3 * (seed % 97)), n)
               for c, nv in _batch_cases(case, seed)]
        return {"state": [tuple(o[:3]) for o in out], "wall": torch.cat([o[3] for o in out])}
    if kind == "gradient":
        cases, _ = _gradient_cases(case, seed)
        wall = []
        for c in cases:
            # the sweep's walls move at -U and +U and share one temperature, as the cases have them
            aero = _Plain(c, _table(case["nv"])).s2cn2(*_uniform(c, _table(case["nv"]), 1.0), n)[3]
            wall.append(aero[:, :, 1:].mean(dim=1))
        return {"wall": torch.stack(wall), "grad": None}
    rng = np.random.default_rng(seed)
    c, table = _couette(case, rng), _table(case["nv"])
    p = _Plain(c, table)
    h, b, W, wall = (p.s2cn2 if kind == "s2cn2" else p.explicit)(*_state(c, table, rng), n)
    if kind == "noalloc":
        return {"h": h, "b": b, "W": W, "dt": float(p.last_dt)}
    fields, lap = p.fields(h, b, W), _lap(kind)
    h, b = (torch.nn.functional.pad(a, (0, 0, lap, lap, lap, lap)) for a in (h, b))
    return {"h": h, "b": b, "W": W, "wall": wall, "fields": fields}


def _uniform(c, table, rho):
    """The uniform state a high-order run starts from: the discrete Maxwellian of W."""
    W = np.zeros((c.ny, c.nx, 4))
    W[..., 0], W[..., 3] = rho, rho * c.tinf * (c.ck + 2) / 4
    p = _Plain(c, table)
    th, _ = p.closure(torch.from_numpy(W[0, 0]).to(p.dev)[None])
    h, b = p.maxwellian(th)[:2]
    return h.expand(c.ny, c.nx, -1), b.expand(c.ny, c.nx, -1), W


SMV, EPS = 1.1754943508222875e-38, np.finfo(np.float64).eps
GAUSS_W = (5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0)
GAUSS_X = (-0.5 * math.sqrt(0.6), 0.0, 0.5 * math.sqrt(0.6))


def _cell_average_map(offsets):
    """[sample][power]: the polynomial whose averages over the cells at `offsets` are the samples."""
    n = len(offsets)
    A = np.array([[((o + 0.5) ** (d + 1) - (o - 0.5) ** (d + 1)) / (d + 1) for d in range(n)] for o in offsets])
    return np.linalg.inv(A).T


def _point_weights():
    """E, D [point][candidate][sample]: value and derivative of a candidate at -1/2, 1/2 and the Gauss nodes."""
    E, D = np.zeros((5, 4, 5)), np.zeros((5, 4, 5))
    for c, off in enumerate(((-2, -1, 0), (-1, 0, 1), (0, 1, 2), (-2, -1, 0, 1, 2))):
        m = _cell_average_map(off)
        for p, x in enumerate((-0.5, 0.5) + GAUSS_X):
            for k, o in enumerate(off):
                E[p, c, o + 2] = sum(m[k, d] * x ** d for d in range(len(off)))
                D[p, c, o + 2] = sum(d * m[k, d] * x ** (d - 1) for d in range(1, len(off)))
    return E, D


_E, _D = _point_weights()


def _weno_weights(q):
    """Final weights of the four candidates of the WENO-AO(5,3) stencil q (five tensors)."""
    a, b, c, d, e = q
    beta = [13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
            13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
            13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2,
            (231153 * c * c + 104963 * (b * b + d * d) + 6908 * (a * a + e * e) - 38947 * a * d
             + b * (-51001 * a + 179098 * d - 38947 * e) - 3 * c * (99692 * b - 22641 * a + 99692 * d - 22641 * e)
             + 8209 * a * e - 51001 * d * e) / 5040]
    tau = ((beta[3] - beta[0]).abs() + (beta[3] - beta[1]).abs() + (beta[3] - beta[2]).abs()) / 3
    gam = (0.01125, 0.1275, 0.01125, 0.85)
    al = [g * (1 + (tau / (bt + 1e-8)) ** 2) for g, bt in zip(gam, beta)]
    s = al[0] + al[1] + al[2] + al[3]
    f3 = al[3] / s / 0.85
    return [al[k] / s - f3 * gam[k] for k in range(3)] + [f3]


def _combine(f, q, T):
    out = 0.0
    for c in range(4):
        out = out + f[c] * sum(T[c, k] * q[k] for k in range(5) if T[c, k] != 0.0)
    return out


def _side(q, der, xi, hi):
    """The one-sided quartic through the five rows next to a wall, at xi of row `der`'s cell."""
    off = tuple(r - hi for r in range(5))
    m = _cell_average_map(off)
    val = sum(q[k] * sum(m[k, d] * xi ** d for d in range(5)) for k in range(5))
    return (val, sum(q[k] * sum(d * m[k, d] * xi ** (d - 1) for d in range(1, 5)) for k in range(5))) if der else val


class _Plain:
    def __init__(self, c, table):
        self.c, self.dev = c, "cuda" if torch.cuda.is_available() else "cpu"
        self.u, self.v, self.w = (torch.from_numpy(a).to(self.dev) for a in table)
        self.gm1 = (c.ck + 4) / (c.ck + 2) - 1.0
        self.last_dt = None

    # ---- moments and equilibria (mod_Tools.f90, mod_ImplicitCommon.f90)
    def primitive(self, W):
        r = W[..., 0]
        e = W[..., 3] - 0.5 * (W[..., 1] ** 2 + W[..., 2] ** 2) / r
        return torch.stack([r, W[..., 1] / r, W[..., 2] / r, 0.5 * r / (self.gm1 * e)], -1)

    def conserved(self, p):
        r, U, V, L = p.unbind(-1)
        return torch.stack([r, r * U, r * V, 0.5 * r / (L * self.gm1) + 0.5 * r * (U * U + V * V)], -1)

    def tau(self, p):
        return self.c.mu_ref * (1 / p[..., 3]) ** self.c.omega / (0.5 * p[..., 0] / p[..., 3])

    def moments(self, h, b, u, v):
        w = self.w
        return torch.stack([h @ w, h @ (w * u), h @ (w * v), 0.5 * (h @ (w * (u * u + v * v)) + b @ w)], -1)

    def heat(self, U, V, h, b, u, v):
        cx, cy = u - U[..., None], v - V[..., None]
        t = 0.5 * self.w * ((cx * cx + cy * cy) * h + b)
        return (t * cx).sum(-1), (t * cy).sum(-1)

    def timestep(self, W):
        c, p = self.c, self.primitive(W)
        s = (0.5 * (self.gm1 + 1) / p[..., 3]).sqrt()
        a, b = (p[..., 1].abs() + s).clamp(min=self.u.max().item()), (p[..., 2].abs() + s).clamp(min=self.v.max().item())
        return (c.cfl * c.dx * c.dy / (c.dy * a + c.dx * b)).min()

    def gauss(self, p, u, v):
        cx, cy = u - p[..., 1, None], v - p[..., 2, None]
        H = (p[..., 0] * p[..., 3] / math.pi)[..., None] * torch.exp(-p[..., 3, None] * (cx * cx + cy * cy))
        return H, H * (self.c.ck / (2 * p[..., 3]))[..., None], cx, cy

    def project(self, H, B, u, v, target, WH=None, WB=None):
        """Minimum-change correction of (H, B) to the conserved moments `target`."""
        WH, WB = (H if WH is None else WH).abs(), (B if WB is None else WB).abs()
        wh = torch.maximum(WH, EPS * WH.amax(-1, keepdim=True).clamp(min=1.0))
        wb = torch.maximum(WB, EPS * WB.amax(-1, keepdim=True).clamp(min=1.0))
        k = torch.stack([torch.ones_like(u), u, v, 0.5 * (u * u + v * v)])
        G = torch.einsum("...k,ak,bk->...ab", wh * self.w, k, k)
        G[..., 3, 3] += 0.25 * (wb @ self.w)
        lam = torch.linalg.solve(G, (target - self.moments(H, B, u, v))[..., None])[..., 0]
        return H + wh * (lam @ k), B + 0.5 * wb * lam[..., 3, None]

    def micro_slope(self, p, s):
        ck2, (r, U, V, L) = self.c.ck + 2.0, p.unbind(-1)
        a3 = 4 * L * L / (ck2 * r) * (2 * s[..., 3] - 2 * U * s[..., 1] - 2 * V * s[..., 2]
                                      + s[..., 0] * (U * U + V * V - 0.5 * ck2 / L))
        a2 = 2 * L / r * (s[..., 2] - V * s[..., 0]) - V * a3
        a1 = 2 * L / r * (s[..., 1] - U * s[..., 0]) - U * a3
        a0 = s[..., 0] / r - U * a1 - V * a2 - 0.5 * (U * U + V * V + 0.5 * ck2 / L) * a3
        return torch.stack([a0, a1, a2, a3], -1)

    def moment_tables(self, p):
        r, U, V, L = p.unbind(-1)
        e = 0.5 * torch.exp(-L * U * U) / (math.pi * L).sqrt()
        lo = [0.5 * torch.erfc(-L.sqrt() * U)]
        hi = [0.5 * torch.erfc(L.sqrt() * U)]
        lo.append(U * lo[0] + e)
        hi.append(U * hi[0] - e)
        t = [torch.ones_like(V), V]
        for i in range(2, 7):
            lo.append(U * lo[-1] + 0.5 * (i - 1) * lo[-2] / L)
            hi.append(U * hi[-1] + 0.5 * (i - 1) * hi[-2] / L)
            t.append(V * t[-1] + 0.5 * (i - 1) * t[-2] / L)
        ck = self.c.ck
        return [x + y for x, y in zip(lo, hi)], lo, hi, t, [torch.ones_like(L), 0.5 * ck / L, ck * (ck + 2) / (4 * L * L)]

    @staticmethod
    def slope_moments(a, Mu, Mv, Mx, al, be):
        def m(i, j, d):
            return torch.stack([Mu[i] * Mv[j] * Mx[d], Mu[i + 1] * Mv[j] * Mx[d], Mu[i] * Mv[j + 1] * Mx[d],
                                0.5 * (Mu[i + 2] * Mv[j] * Mx[d] + Mu[i] * Mv[j + 2] * Mx[d] + Mu[i] * Mv[j] * Mx[d + 1])], -1)
        return (a[..., 0, None] * m(al, be, 0) + a[..., 1, None] * m(al + 1, be, 0) + a[..., 2, None] * m(al, be + 1, 0)
                + 0.5 * a[..., 3, None] * (m(al + 2, be, 0) + m(al, be + 2, 0) + m(al, be, 1)))

    @staticmethod
    def time_coefficients(dt, tau):
        """The integrals over the step by their series where dt / tau is small (the closed forms cancel there)."""
        x = dt / tau
        small = x < 0.1
        e = torch.exp(-x)
        m3 = tau * (1 - e)
        m4 = -tau * dt * e + tau * m3
        m0 = dt - m3
        closed = [m0, -tau * m0 + m4, 0.5 * dt * dt - tau * m0, m3, m4]
        ser = [torch.zeros_like(tau) for _ in range(5)]
        t = torch.ones_like(tau)
        for n in range(1, 25):
            t = t * (-x) / n
            ser[3] = ser[3] - tau * t
            if n >= 2:
                ser[0], ser[4] = ser[0] + tau * t, ser[4] + tau * tau * (n - 1) * t
            if n >= 3:
                ser[1], ser[2] = ser[1] + tau * tau * (n - 2) * t, ser[2] - tau * tau * t
        return [torch.where(small, a, b) for a, b in zip(ser, closed)]

    @staticmethod
    def kinetic(a, vn, vt, H, B, mxi2):
        """The microscopic slope a applied to (H, B)."""
        lin = a[..., 0, None] + a[..., 1, None] * vn + a[..., 2, None] * vt
        v2, c = vn * vn + vt * vt, 0.5 * a[..., 3, None]
        return lin * H + c * (v2 * H + B), lin * B + c * (v2 * B + mxi2[..., None] * H)

    # ---- the second-order step (mod_Interpolation.f90, mod_Evolution.f90, mod_Residual.f90, mod_TimeIntegrator.f90)
    @staticmethod
    def limited(a, b):
        return (torch.sign(a) + torch.sign(b)) * a.abs() * b.abs() / (a.abs() + b.abs() + SMV)

    def slopes(self, f):
        c = self.c
        sx = self.limited((f - f.roll(1, 1)) / c.dx, (f.roll(-1, 1) - f) / c.dx)
        d = (f[1:] - f[:-1]) / c.dy
        return sx, torch.cat([d[:1], self.limited(d[:-1], d[1:]), d[-1:]])

    def rotated(self, W, axis):
        return W if axis == 0 else torch.stack([W[..., 0], W[..., 2], -W[..., 1], W[..., 3]], -1)

    def shakhov(self, p, H, B, cx, cy, q):
        k = (0.8 * (1 - self.c.pr) * p[..., 3] ** 2 / p[..., 0])[..., None]
        qd = cx * q[0][..., None] + cy * q[1][..., None]
        s = 2 * p[..., 3, None] * (cx * cx + cy * cy) - 4
        return k * qd * s * H, k * qd * (s + 2.0 / self.c.ck) * B

    def face(self, axis, L, R, dt):
        """L, R: (h, b, normal and tangential slopes of h and b, W) of the cells beside the faces."""
        c = self.c
        vn, vt = (self.u, self.v) if axis == 0 else (self.v, -self.u)
        hl, length = 0.5 * (c.dx if axis == 0 else c.dy), c.dy if axis == 0 else c.dx
        sg = 1.0 if axis == 0 else -1.0
        up = vn > 0
        h, b, nh, th, nb, tb = (torch.where(up, x, y) for x, y in zip(L[:6], R[:6]))
        h, b, th, tb = h + torch.where(up, hl * nh, -hl * nh), b + torch.where(up, hl * nb, -hl * nb), sg * th, sg * tb
        cv, st = self.moments(h, b, vn, vt), self.moments(th, tb, vn, vt)
        p = self.primitive(cv)
        WL, WR = self.rotated(L[6], axis), self.rotated(R[6], axis)
        aL, aR, aT = self.micro_slope(p, (cv - WL) / hl), self.micro_slope(p, (WR - cv) / hl), self.micro_slope(p, st)
        Mu, Ml, Mr, Mv, Mx = self.moment_tables(p)
        s = (self.slope_moments(aL, Ml, Mv, Mx, 1, 0) + self.slope_moments(aR, Mr, Mv, Mx, 1, 0)
             + self.slope_moments(aT, Mu, Mv, Mx, 0, 1))
        A = self.micro_slope(p, -p[..., 0, None] * s)
        mt = [x[..., None] for x in self.time_coefficients(dt, self.tau(p))]
        H, B, cx, cy = self.gauss(p, vn, vt)
        q = self.heat(p[..., 1], p[..., 2], h, b, vn, vt)
        H, B = self.project(H, B, vn, vt, self.conserved(p))
        Hp, Bp = self.shakhov(p, H, B, cx, cy, q)
        kl, kr, kt, kA = (self.kinetic(a, vn, vt, H, B, Mx[2]) for a in (aL, aR, aT, A))
        out = [length * vn * (mt[0] * (f + fp) + mt[1] * (vn * torch.where(up, kl[i], kr[i]) + vt * kt[i]) + mt[2] * kA[i]
                              + mt[3] * fr - mt[4] * (vn * n + vt * t))
               for i, (f, fp, fr, n, t) in enumerate(((H, Hp, h, nh, th), (B, Bp, b, nb, tb)))]
        return out[0], out[1], self.moments(out[0], out[1], self.u, self.v)

    def wall(self, side, h, b, sx, sy, sxb, syb, W, dt):
        """The moving diffuse wall below row 0 (side -1) or above the last row (+1)."""
        c, iw = self.c, 0 if side < 0 else 1
        vn, vt = self.v, -self.u
        pc = self.primitive(W)
        lam = 1.0 / c.wall_tnative[iw]
        pg = torch.stack([pc[..., 0] / pc[..., 3] * lam, torch.zeros_like(pc[..., 0]),
                          torch.full_like(pc[..., 0], -c.wall_ux[iw]), torch.full_like(pc[..., 0], lam)], -1)
        mt = [x[..., None] for x in self.time_coefficients(dt, self.tau(pg))]
        th, tb = -sx, -sxb
        h, b = h + side * 0.5 * c.dy * sy, b + side * 0.5 * c.dy * syb
        q = self.heat(pg[..., 1], pg[..., 2], h, b, vn, vt)
        an = self.micro_slope(pg, (self.conserved(pg) - self.rotated(W, 1)) / (side * 0.5 * c.dy))
        at = self.micro_slope(pg, self.moments(th, tb, vn, vt))
        Mu, _, _, Mv, Mx = self.moment_tables(pg)
        A = self.micro_slope(pg, -pg[..., 0, None] * (self.slope_moments(an, Mu, Mv, Mx, 1, 0)
                                                      + self.slope_moments(at, Mu, Mv, Mx, 0, 1)))
        pw = torch.cat([torch.ones_like(pg[..., :1]), pg[..., 1:]], -1)
        Hg, Bg, cx, cy = self.gauss(pg, vn, vt)
        Hg, Bg = self.project(Hg, Bg, vn, vt, self.conserved(pg))
        Hw, Bw = self.gauss(pw, vn, vt)[:2]
        Hw, Bw = self.project(Hw, Bw, vn, vt, self.conserved(pw))
        Hp, Bp = self.shakhov(pg, Hg, Bg, cx, cy, q)
        kn, kt, kA = (self.kinetic(a, vn, vt, Hg, Bg, Mx[2]) for a in (an, at, A))
        inc = [mt[0] * (f + fp) + mt[1] * (vn * kn[i] + vt * kt[i]) + mt[2] * kA[i] + mt[3] * fr - mt[4] * (vn * n + vt * t)
               for i, (f, fp, fr, n, t) in enumerate(((Hg, Hp, h, sy, th), (Bg, Bp, b, syb, tb)))]
        toward = side * vn > 0                       # the gas that meets the wall
        rho = -(torch.where(toward, inc[0], 0 * inc[0]) @ (self.w * vn)) / (
            dt * (torch.where(toward, 0 * Hw, Hw) @ (self.w * vn)))
        f = [vn * torch.where(toward, i, dt * rho[..., None] * x) for i, x in ((inc[0], Hw), (inc[1], Bw))]
        m = self.moments(f[0], f[1], vn, vt)
        aero = torch.stack([m[..., 1] / dt, m[..., 2] / dt, m[..., 3] / dt + c.wall_ux[iw] * m[..., 2] / dt], -1)
        return (c.dx * f[0], c.dx * f[1], c.dx * torch.stack([m[..., 0], -m[..., 2], m[..., 1], m[..., 3]], -1)), aero

    def explicit(self, h, b, W, steps):
        c = self.c
        h, b, W = (torch.as_tensor(np.ascontiguousarray(a) if isinstance(a, np.ndarray) else a).to(self.dev) for a in (h, b, W))
        area = c.dx * c.dy
        for _ in range(steps):
            dt = self.last_dt = self.timestep(W)
            (sx, sy), (sxb, syb) = self.slopes(h), self.slopes(b)
            R = (h, b, sx, sy, sxb, syb, W)
            fx = self.face(0, tuple(a.roll(1, 1) for a in R), R, dt)
            T = (h, b, sy, sx, syb, sxb, W)
            fy = self.face(1, tuple(a[:-1] for a in T), tuple(a[1:] for a in T), dt)
            lo, alo = self.wall(-1, h[0], b[0], sx[0], sy[0], sxb[0], syb[0], W[0], dt)
            hi, ahi = self.wall(1, h[-1], b[-1], sx[-1], sy[-1], sxb[-1], syb[-1], W[-1], dt)
            fy = [torch.cat([x[None], y, z[None]]) for x, y, z in zip(lo, fy, hi)]
            dh, db, dW = ((x - x.roll(-1, 1) + y[:-1] - y[1:]) / area for x, y in zip(fx, fy))
            rh, rb = self.project(dh / dt, db / dt, self.u, self.v, dW / dt, h, b)
            po, Wn = self.primitive(W), W + dW
            pn = self.primitive(Wn)
            q = self.heat(po[..., 1], po[..., 2], h, b, self.u, self.v)
            eq = []
            for p, tgt in ((po, self.conserved(po)), (pn, Wn)):
                H, B, cx, cy = self.gauss(p, self.u, self.v)
                Hp, Bp = self.shakhov(p, H, B, cx, cy, q)
                eq.append(self.project(H + Hp, B + Bp, self.u, self.v, tgt))
            to, tn = self.tau(po)[..., None], self.tau(pn)[..., None]
            h, b = ((f + r * dt + 0.5 * dt * (en / tn + (eo - f) / to)) / (1 + 0.5 * dt / tn)
                    for f, r, en, eo in ((h, rh, eq[1][0], eq[0][0]), (b, rb, eq[1][1], eq[0][1])))
            W = Wn
        return h, b, W, torch.stack([alo, ahi])

    # ---- the high-order step (mod_S2D1.f90, mod_S2D1Reconstruction.f90, mod_CorrectedWF2DClosure.f90)
    def maxwellian(self, th):
        """The closure Maxwellian of th = (rho, u, v, T) and its logarithmic derivatives by th."""
        r, U, V, T = (x[..., None] for x in th.unbind(-1))
        cx, cy = self.u - U, self.v - V
        c2 = cx * cx + cy * cy
        qh = r / (math.pi * T) * torch.exp(-c2 / T)
        one = torch.ones_like(qh)
        ld = [one / r, 2 * cx / T, 2 * cy / T, -one / T + c2 / (T * T)]
        return qh, 0.5 * self.c.ck * T * qh, ld, ld[:3] + [ld[3] + one / T]

    def closure(self, W):
        """theta whose discrete Maxwellian has the moments W, and the moments' Jacobian there."""
        r = W[..., 0]
        U, V = W[..., 1] / r, W[..., 2] / r
        th = torch.stack([r, U, V, 4 * (W[..., 3] / r - 0.5 * (U * U + V * V)) / (self.c.ck + 2)], -1)
        for it in range(12):
            qh, qb, ld, ldb = self.maxwellian(th)
            J = torch.stack([self.moments(qh * x, qb * y, self.u, self.v) for x, y in zip(ld, ldb)], -1)
            step = torch.linalg.solve(J, (W - self.moments(qh, qb, self.u, self.v))[..., None])[..., 0]
            if it and step.abs().max() < 1e-14:
                break
            th = th + step
        return th, J

    def direction(self, q, t):
        qh, qb, ld, ldb = q
        return (sum(qh * l * t[..., i, None] for i, l in enumerate(ld)), sum(qb * l * t[..., i, None] for i, l in enumerate(ldb)))

    def gas(self, W):
        r = W[..., 0]
        U, V = W[..., 1] / r, W[..., 2] / r
        theta = 2.0 / (self.c.ck + 2) * (W[..., 3] / r - 0.5 * (U * U + V * V))
        return torch.stack([r, U, V, 0.5 / theta], -1)

    def equilibrium(self, W):
        """M, K_x, K_y (each h and b) of W, its Maxwellian and the Jacobian."""
        th, J = self.closure(W)
        q = self.maxwellian(th)
        p = self.gas(W)
        cx, cy = self.u - p[..., 1, None], self.v - p[..., 2, None]
        s = 2 * p[..., 3, None] * (cx * cx + cy * cy) - 4
        k = (0.8 * (1 - self.c.pr) * p[..., 3] ** 2 / p[..., 0])[..., None]
        out = [q[0], q[1]]
        for cc in (cx, cy):
            kh, kb = k * cc * s * q[0], k * cc * (s + 2.0 / self.c.ck) * q[1]
            d = self.direction(q, torch.linalg.solve(J, self.moments(kh, kb, self.u, self.v)[..., None])[..., 0])
            out += [kh - d[0], kb - d[1]]
        return out, q, J, p

    def reconstruct(self, F):
        """F [ny][nx][*] -> face [4][3], normal and tangential derivatives [4][3] (sides x-, x+, y-, y+; Gauss
        nodes), volume nodes [3][3], with one-sided quartics in the three rows next to each wall."""
        ny = F.shape[0]
        fx = _weno_weights([F.roll(-s, 1) for s in range(-2, 3)])
        qx = [F.roll(-s, 1) for s in range(-2, 3)]
        X = [_combine(fx, qx, t) for t in (_E[0], _D[0], _E[1], _D[1], _E[2], _E[3], _E[4])]
        rows = slice(3, ny - 3)
        inner = lambda A: [A[3 + s:ny - 3 + s] for s in range(-2, 3)]  # noqa: E731
        wallrows = [(j, 0, j) for j in range(3)] + [(j, ny - 5, j - (ny - 5)) for j in range(ny - 3, ny)]
        face, dn, dt = ([[torch.empty_like(F) for _ in range(3)] for _ in range(4)] for _ in range(3))
        vol = [[torch.empty_like(F) for _ in range(3)] for _ in range(3)]
        for s in range(2):
            A, Dv = X[2 * s], X[2 * s + 1]
            q, comp = inner(A), inner(Dv)
            f = _weno_weights(q)
            Y, YD = torch.empty_like(F), torch.empty_like(F)
            qy = inner(F)
            fy = _weno_weights(qy)
            Y[rows], YD[rows] = _combine(fy, qy, _E[s]), _combine(fy, qy, _D[s])
            for a in range(3):
                face[s][a][rows], dt[s][a][rows], dn[s][a][rows] = (
                    _combine(f, q, _E[2 + a]), _combine(f, q, _D[2 + a]), _combine(f, comp, _E[2 + a]))
                for j, first, hi in wallrows:
                    face[s][a][j], dt[s][a][j] = _side([A[first + r] for r in range(5)], True, GAUSS_X[a], hi)
                    dn[s][a][j] = _side([Dv[first + r] for r in range(5)], False, GAUSS_X[a], hi)
            for j, first, hi in wallrows:
                Y[j], YD[j] = _side([F[first + r] for r in range(5)], True, (-0.5, 0.5)[s], hi)
            q, comp = ([B.roll(-r, 1) for r in range(-2, 3)] for B in (Y, YD))
            f = _weno_weights(q)
            for a in range(3):
                face[2 + s][a], dt[2 + s][a], dn[2 + s][a] = (
                    _combine(f, q, _E[2 + a]), _combine(f, q, _D[2 + a]), _combine(f, comp, _E[2 + a]))
        for a in range(3):
            A = X[4 + a]
            q = inner(A)
            f = _weno_weights(q)
            for g in range(3):
                vol[a][g][rows] = _combine(f, q, _E[2 + g])
                for j, first, hi in wallrows:
                    vol[a][g][j] = _side([A[first + r] for r in range(5)], False, GAUSS_X[g], hi)
        return face, dn, dt, vol

    def limit(self, h, b):
        """Face values and derivatives per cell size of h and b under the common positivity factor."""
        c, margin = self.c, 64 * EPS
        rec = [self.reconstruct(f) for f in (h, b)]
        theta = torch.ones_like(h)
        for m, (face, _, _, vol) in zip((h, b), rec):
            for x in [y for side in face for y in side] + [y for row in vol for y in row]:
                theta = torch.where(x < 0, torch.minimum(theta, (1 - margin) * m / (m - x)), theta)
        theta = torch.where((h <= 0) | (b <= 0), torch.zeros_like(theta), theta.clamp(0, 1))
        return [[[(m + theta * (face[s][a] - m), theta * dn[s][a] / (c.dx if s < 2 else c.dy),
                   theta * dt[s][a] / (c.dy if s < 2 else c.dx)) for a in range(3)] for s in range(4)]
                for m, (face, dn, dt, _) in zip((h, b), rec)]

    def high_node(self, axis, L, R, nl, nr, tg, dt):
        """The flux at one Gauss node: L, R = ((value, normal, tangential) of h, of b) of the two sides."""
        vn, vt = (self.u, self.v) if axis == 0 else (self.v, self.u)
        up = vn >= 0
        (fh, nh, th), (fb, nb, tb) = (tuple(torch.where(up, x, y) for x, y in zip(L[i], R[i])) for i in range(2))
        W = self.moments(fh, fb, self.u, self.v)
        (mh, mb, kxh, kxb, kyh, kyb), q, J, p = self.equilibrium(W)
        g = torch.stack([p[..., 0], p[..., 1], p[..., 2], p[..., 3]], -1)
        eh, eb = self.gauss(g, self.u, self.v)[:2]
        qx, qy = (x[..., None] for x in self.heat(p[..., 1], p[..., 2], fh - eh, fb - eb, self.u, self.v))
        solve = lambda m: self.direction(q, torch.linalg.solve(J, m[..., None])[..., 0])  # noqa: E731
        dl, dr, dg = solve(nl), solve(nr), solve(tg)
        s = [vn * torch.where(up, x, y) + vt * z for x, y, z in zip(dl, dr, dg)]
        dm = solve(-self.moments(s[0], s[1], self.u, self.v))
        mt = [x[..., None] for x in self.time_coefficients(dt, self.tau(p))]
        F = [vn * (mt[0] * (m + kx * qx + ky * qy) + mt[1] * s[i] + mt[2] * dm[i] + mt[3] * f - mt[4] * (vn * n + vt * t))
             for i, (m, kx, ky, f, n, t) in enumerate(((mh, kxh, kyh, fh, nh, th), (mb, kxb, kyb, fb, nb, tb)))]
        return F[0], F[1], self.moments(F[0], F[1], self.u, self.v)

    def high_wall(self, top, rh, rb, W, dt):
        """The multiscale diffuse wall at one Gauss node; rh, rb = (value, normal, tangential) at the wall."""
        c, side, iw = self.c, 1.0 if top else -1.0, 1 if top else 0
        ux, lam = c.wall_ux[iw], 1.0 / c.wall_tnative[iw]
        theta = 0.5 / lam
        pressure = 2.0 / (c.ck + 2) * (W[..., 3] - 0.5 * (W[..., 1] ** 2 + W[..., 2] ** 2) / W[..., 0])
        r, zero = pressure / theta, torch.zeros_like(pressure)
        pg = torch.stack([r, zero, zero - ux, zero + lam], -1)
        wg = torch.stack([r, zero, -r * ux, r * ((c.ck + 2) / (4 * lam) + 0.5 * ux * ux)], -1)
        ww = torch.stack([r, r * ux, zero, r * ((c.ck + 2) * theta / 2 + ux * ux / 2)], -1)
        th, _ = self.closure(ww)
        mh, mb = self.maxwellian(th)[:2]
        vn, vt = self.v, -self.u
        an = self.micro_slope(pg, (wg - self.rotated(W, 1)) / (side * 0.5 * c.dy))
        at = self.micro_slope(pg, self.moments(-rh[2], -rb[2], vn, vt))
        Mu, _, _, Mv, Mx = self.moment_tables(pg)
        A = self.micro_slope(pg, -r[..., None] * (self.slope_moments(an, Mu, Mv, Mx, 1, 0) + self.slope_moments(at, Mu, Mv, Mx, 0, 1)))
        q = self.heat(zero, zero - ux, rh[0], rb[0], vn, vt)
        mt = [x[..., None] for x in self.time_coefficients(dt, self.tau(pg))]
        ch, cb = self.shakhov(pg, mh, mb, vn, vt + ux, q)
        kn, kt, kA = (self.kinetic(a, vn, vt, mh, mb, Mx[2]) for a in (an, at, A))
        inc = [mt[0] * (m + k) + mt[1] * (vn * kn[i] + vt * kt[i]) + mt[2] * kA[i] + mt[3] * f[0]
               - mt[4] * (vn * f[1] + self.u * f[2]) for i, (m, k, f) in enumerate(((mh, ch, rh), (mb, cb, rb)))]
        toward = side * self.v > 0
        hw, bw = mh / r[..., None], mb / r[..., None]
        rho = -(torch.where(toward, inc[0], 0 * inc[0]) @ (self.w * self.v)) / (
            dt * (torch.where(toward, 0 * hw, hw) @ (self.w * self.v)))
        f = [self.v * torch.where(toward, x, dt * rho[..., None] * y) for x, y in ((inc[0], hw), (inc[1], bw))]
        return f[0], f[1], self.moments(f[0], f[1], self.u, self.v)

    def gauss_sum(self, nodes, length):
        return [length * sum(g * n[i] for g, n in zip(GAUSS_W, nodes)) for i in range(3)]

    def targets(self, W):
        vol = self.reconstruct(W)[3]
        mean = sum(GAUSS_W[a] * GAUSS_W[g] * vol[a][g] for a in range(3) for g in range(3))
        out = None
        for a in range(3):
            for g in range(3):
                e = self.equilibrium(vol[a][g] + W - mean)[0]
                k = GAUSS_W[a] * GAUSS_W[g]
                out = [k * x for x in e] if out is None else [o + k * x for o, x in zip(out, e)]
        return out

    def s2cn2(self, h, b, W, steps):
        c = self.c
        h, b, W = (torch.as_tensor(np.ascontiguousarray(a) if isinstance(a, np.ndarray) else a).to(self.dev) for a in (h, b, W))
        T = self.targets(W)
        for _ in range(steps):
            dt = self.last_dt = self.timestep(W)
            rec = self.limit(h, b)
            _, dn, dtg, _ = self.reconstruct(W)
            at = lambda s, a, f: tuple(tuple(f(x) for x in rec[i][s][a]) for i in range(2))  # noqa: E731
            nxt, lo, hi = (lambda x: x.roll(-1, 1)), (lambda x: x[:-1]), (lambda x: x[1:])
            fx = self.gauss_sum([self.high_node(0, at(1, a, lambda x: x), at(0, a, nxt), dn[1][a] / c.dx, nxt(dn[0][a]) / c.dx,
                                                0.5 * (dtg[1][a] + nxt(dtg[0][a])) / c.dy, dt) for a in range(3)], c.dy)
            fy = self.gauss_sum([self.high_node(1, at(3, a, lo), at(2, a, hi), lo(dn[3][a]) / c.dy, hi(dn[2][a]) / c.dy,
                                                0.5 * (lo(dtg[3][a]) + hi(dtg[2][a])) / c.dx, dt) for a in range(3)], c.dx)
            bot = self.gauss_sum([self.high_wall(False, *at(2, a, lambda x: x[0]), W[0], dt) for a in range(3)], c.dx)
            top = self.gauss_sum([self.high_wall(True, *at(3, a, lambda x: x[-1]), W[-1], dt) for a in range(3)], c.dx)
            wall = []
            for iw, f in enumerate((bot, top)):
                r = f[2] / (dt * c.dx)
                wall.append(torch.stack([r[..., 2], -r[..., 1], r[..., 3] - c.wall_ux[iw] * r[..., 1]], -1))
            fy = [torch.cat([x[None], y, z[None]]) for x, y, z in zip(bot, fy, top)]
            dh, db, dW = ((x.roll(1, 1) - x + y[:-1] - y[1:]) / (c.dx * c.dy) for x, y in zip(fx, fy))
            p, Wn = self.gas(W), W + dW
            pn = self.gas(Wn)
            q0, q1 = (x[..., None] for x in self.heat(p[..., 1], p[..., 2], h - T[0], b - T[1], self.u, self.v))
            old, beta = (dt / (2 * self.tau(x))[..., None] for x in (p, pn))
            rh = h + dh + old * (T[0] + T[2] * q0 + T[4] * q1 - h)
            rb = b + db + old * (T[1] + T[3] * q0 + T[5] * q1 - b)
            T = self.targets(Wn)
            hq = lambda f, g: self.heat(pn[..., 1], pn[..., 2], f, g, self.u, self.v)  # noqa: E731
            r, m, kx, ky, bb = hq(rh, rb), hq(T[0], T[1]), hq(T[2], T[3]), hq(T[4], T[5]), beta[..., 0]
            a11, a12, a21, a22 = 1 + bb - bb * kx[0], -bb * ky[0], -bb * kx[1], 1 + bb - bb * ky[1]
            det, s0, s1 = a11 * a22 - a12 * a21, r[0] - m[0], r[1] - m[1]
            n0, n1 = ((s0 * a22 - a12 * s1) / det)[..., None], ((a11 * s1 - s0 * a21) / det)[..., None]
            h = (rh + beta * (T[0] + T[2] * n0 + T[4] * n1)) / (1 + beta)
            b = (rb + beta * (T[1] + T[3] * n0 + T[5] * n1)) / (1 + beta)
            W = Wn
        return h, b, W, torch.stack(wall)

    def fields(self, h, b, W):
        """Density, velocity, temperature, pressure, stress and heat flux of every cell (mod_Output.f90)."""
        p = self.primitive(W)
        cx, cy, w = self.u - p[..., 1, None], self.v - p[..., 2, None], self.w
        pr = ((w * (cx * cx + cy * cy) * h).sum(-1) + b @ w) / (self.c.ck + 2)
        q = self.heat(p[..., 1], p[..., 2], h, b, self.u, self.v)
        T = 1 / p[..., 3]
        return torch.stack([p[..., 0], p[..., 1], p[..., 2], T, 0.5 * p[..., 0] * T, (w * cx * cx * h).sum(-1) - pr,
                            (w * cx * cy * h).sum(-1), (w * cy * cy * h).sum(-1) - pr, q[0], q[1]], -1)
