"""What is timed: the calls a user of this framework makes, over their range.

Each case is one pass through a public entry point: a field set on a solver,
advanced a number of levels and read back (Engine), a differentiable solve with
its gradients (heat_solve), or a batch of independent fields (Batch).  Sizes are
those of the reference's study (160 to 1120 squared, blocksizes 8 to 32), of this
repository's benchmark (heat at 8192 squared, Euler at 1024 and 4096 squared, the
adjoint at 2048 squared) and ragged ones between them.
"""
import math

import numpy as np
import torch

from pysweep_b200 import Batch, Engine, plugin_constants
from pysweep_b200.adjoint import heat_solve

GAMMA = 1.4

# The heat equation as a user's plugin: the __device__ step of the reference's
# plugin format, compiled when the solver is made.
HOOK = """
__device__ __constant__ double DT;
__device__ __constant__ double DX;
__device__ __constant__ double ALPHA;

__device__ void step(double *s, int idx, int globalTimeStep)
{
    const double courant = ALPHA * DT / DX / DX;
    const double c = s[idx];
    const double sx = courant * ((s[idx + SY] - 2 * c) + s[idx - SY]);
    const double sy = courant * ((s[idx + 1] - 2 * c) + s[idx - 1]);
    s[idx + TIMES] = (sx + sy) + c;
}
"""

# operations of one cell update: heat's two second differences and their sum;
# Euler's two faces, one pressure and the update of four variables
HEAT_FLOPS, EULER_FLOPS = 10, 295


def _field(eq, nx, ny, bs, levels, mode="swept", its=1, dtype="float64", frame_every=0):
    return {"kind": "field", "eq": eq, "mode": mode, "nx": nx, "ny": ny, "bs": bs, "its": its,
            "levels": levels, "dtype": dtype, "frame_every": frame_every}


def listed():
    return [
        # the smallest run of the reference's study: launches and latency
        dict(_field("heat", 160, 160, 8, 500), name="heat_160"),
        # the run the reference's logs quote: heat, GPU share 1, 1120 squared, 500 steps
        dict(_field("heat", 1120, 1120, 16, 500), name="heat_1120"),
        # the benchmark's grid: fields far larger than L2
        dict(_field("heat", 8192, 8192, 32, 480), name="heat_8192"),
        # two-stage Runge-Kutta on a ragged grid, a frame kept every 50 steps
        dict(_field("heat", 1000, 1400, 8, 500, its=2, frame_every=50), name="heat_rk2_frames"),
        # the standard decomposition the swept one is compared with
        dict(_field("heat", 1120, 1120, 16, 500, mode="standard"), name="heat_standard_1120"),
        # float32 fields (the yaml key dtype)
        dict(_field("heat", 2048, 2048, 32, 480, dtype="float32"), name="heat_f32_2048"),
        # the compressible vortex at the size the reference's logs quote
        dict(_field("euler", 1120, 1120, 16, 100, its=2), name="euler_1120"),
        # the benchmark's large vortex through the standard decomposition
        dict(_field("euler", 4096, 4096, 16, 40, mode="standard", its=2),
             name="euler_standard_4096"),
        # a gradient with respect to the initial field and the diffusivity
        {"name": "adjoint_2048", "kind": "solve", "nx": 2048, "ny": 2048, "levels": 256,
         "every": 64, "swept": False},
        # the same through the swept engines, on a grid that is not square
        {"name": "adjoint_swept", "kind": "solve", "nx": 1024, "ny": 1536, "levels": 256,
         "every": 64, "swept": True},
        # a parameter study: independent fields of many sizes advanced together
        {"name": "batch_heat", "kind": "batch", "count": 32, "lo": 128, "hi": 512, "bs": 32,
         "levels": 2000, "sizes": 5},
        # a user's own plugin
        {"name": "hook_1024", "kind": "hook", "nx": 1024, "ny": 1024, "bs": 16, "levels": 200},
    ]


def _size(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi // step, max(-(-lo // step), round(n / step)))) * step


def draw(rng):
    kind = rng.choice(["heat", "heat", "heat", "rk2", "standard", "f32", "euler", "euler",
                       "euler_standard", "solve", "swept", "batch", "hook"])
    bs = rng.choice([8, 16, 32])
    if kind == "heat":
        nx, ny = _size(rng, 160, 8192, bs), _size(rng, 160, 8192, bs)
        levels = rng.randint(100, 480)
        return _field("heat", nx, ny, bs, levels, frame_every=rng.choice([0, 0, 0, 40]) if nx * ny < 3e6 else 0)
    if kind == "rk2":
        nx, ny = _size(rng, 160, 3000, bs), _size(rng, 160, 3000, bs)
        return _field("heat", nx, ny, bs, 2 * rng.randint(50, 250), its=2,
                      frame_every=rng.choice([0, 50]))
    if kind == "standard":
        nx, ny = _size(rng, 160, 4096, bs), _size(rng, 160, 4096, bs)
        return _field("heat", nx, ny, bs, rng.randint(100, 480), mode="standard")
    if kind == "f32":
        bs = rng.choice([16, 32])
        nx, ny = _size(rng, 160, 4096, bs), _size(rng, 160, 4096, 32)
        return _field("heat", nx, ny, bs, rng.randint(100, 480), dtype="float32")
    if kind == "euler":
        nx, ny = _size(rng, 160, 2048, bs), _size(rng, 160, 2048, bs)
        return _field("euler", nx, ny, bs, 2 * rng.randint(20, 50), its=2)
    if kind == "euler_standard":
        nx, ny = _size(rng, 160, 2048, bs), _size(rng, 160, 2048, bs)
        return _field("euler", nx, ny, bs, 2 * rng.randint(10, 30), mode="standard", its=2)
    if kind == "solve":
        return {"kind": "solve", "nx": _size(rng, 200, 2048, 1), "ny": _size(rng, 256, 2048, 64),
                "levels": rng.randint(60, 256), "every": rng.choice([32, 64]), "swept": False}
    if kind == "swept":
        return {"kind": "solve", "nx": _size(rng, 256, 2048, 32), "ny": _size(rng, 256, 2048, 64),
                "levels": rng.randint(60, 256), "every": rng.choice([32, 64]), "swept": True}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(8, 48), "lo": 128, "hi": rng.choice([384, 512, 768]),
                "bs": rng.choice([16, 32]), "levels": rng.randint(500, 1500),
                "sizes": rng.randint(0, 1000)}
    return {"kind": "hook", "nx": _size(rng, 160, 2048, bs), "ny": _size(rng, 160, 2048, bs),
            "bs": bs, "levels": rng.randint(60, 200)}


# ------------------------------------------------------------------ inputs ---
def _heat_globals(n, alpha=1.0):
    dx = 1.0 / n
    return [0.0, 1.0, 0.2 * dx * dx / alpha, dx, dx, alpha, True]


def _fourier(nx, ny, seed, device="cuda"):
    """A smooth periodic field: eight Fourier modes of random phase."""
    rng = np.random.default_rng(seed)
    f64 = dict(dtype=torch.float64, device=device)
    x = torch.arange(nx, **f64)[:, None] / nx
    y = torch.arange(ny, **f64)[None, :] / ny
    u = torch.zeros((nx, ny), **f64)
    for _ in range(8):
        kx, ky = (int(k) for k in rng.integers(1, 9, 2))
        px, py, a = (float(v) for v in rng.random(3))
        u += (0.2 + a) * (torch.sin(2 * math.pi * (kx * x + px)) * torch.cos(2 * math.pi * (ky * y + py)))
    return u


def _vortex(nx, ny, seed, device="cuda"):
    """An isentropic vortex on [-5, 5]^2: rho, rho u, rho v, E; strength,
    heading and centre from the seed."""
    rng = np.random.default_rng(seed)
    strength, heading = float(rng.uniform(4.0, 5.5)), float(rng.uniform(0, 2 * math.pi))
    cx, cy = (float(v) for v in rng.uniform(-1, 1, 2))
    f64 = dict(dtype=torch.float64, device=device)
    x = (-5 + 10 * torch.arange(nx, **f64) / nx)[:, None] - cx
    y = (-5 + 10 * torch.arange(ny, **f64) / ny)[None, :] - cy
    mach = math.sqrt(2 / GAMMA)
    beta = mach * strength * math.sqrt(2) / 4 / math.pi * math.exp(0.5)
    c = math.sqrt(GAMMA)
    om = beta * torch.exp(-0.5 * (x * x + y * y))
    u = mach * c * math.cos(heading) - y * om
    v = mach * c * math.sin(heading) + x * om
    t = 1 - (GAMMA - 1) * om * om / 2
    rho = t ** (1 / (GAMMA - 1))
    p = t ** (GAMMA / (GAMMA - 1)) / GAMMA
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)])


def _diffusivity(nx, ny, seed):
    return 1.0 + 0.4 * _fourier(nx, ny, seed + 1) / 8


def _batch_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    lo, hi = case["lo"] // 32, case["hi"] // 32
    return [(32 * int(a), 32 * int(b)) for a, b in rng.integers(lo, hi + 1, (case["count"], 2))]


def _constants(case):
    if case.get("eq") == "euler":
        dx = 10.0 / case["nx"]
        return [0.0, 1.0, 0.1 * dx, dx, dx, GAMMA]
    g = _heat_globals(case["nx"])
    if case.get("its") == 2:
        g[-1] = False
    return g


# -------------------------------------------------------------------- pass ---
def prepare(case, seed):
    kind = case["kind"]
    nx, ny = case.get("nx"), case.get("ny")
    if kind == "solve":
        state = {"u0": _fourier(nx, ny, seed).requires_grad_(),
                 "alpha": _diffusivity(nx, ny, seed).requires_grad_(),
                 "w": _fourier(nx, ny, seed + 2)}
    elif kind == "batch":
        sizes = _batch_sizes(case)
        b = Batch("heat", sizes, its=1, blocksize=case["bs"])
        for i, (n, _) in enumerate(sizes):
            b.set_constants(i, plugin_constants("heat", _heat_globals(n)))
        state = {"batch": b, "u0": [_fourier(*s, seed + i) for i, s in enumerate(sizes)]}
    elif kind == "hook":
        e = Engine("heat_plugin", nx, ny, nv=1, ops=1, its=1, blocksize=case["bs"], hook_source=HOOK)
        g = _heat_globals(nx)
        for k, v in (("DT", g[2]), ("DX", g[3]), ("ALPHA", g[5])):
            e.set_global(k, v)
        state = {"engine": e, "u0": _fourier(nx, ny, seed)[None]}
        state["out"] = [torch.empty_like(state["u0"])]
    else:
        e = Engine(case["eq"], nx, ny, its=case["its"], blocksize=case["bs"], dtype=case["dtype"])
        for k, v in plugin_constants(case["eq"], _constants(case)).items():
            e.set_global(k, v)
        u0 = _vortex(nx, ny, seed) if case["eq"] == "euler" else _fourier(nx, ny, seed)[None]
        u0 = u0.to(getattr(torch, case["dtype"]))
        state = {"engine": e, "u0": u0, "out": [torch.empty_like(u0) for _ in range(case["its"])]}
        if case["frame_every"]:
            k = case["levels"] // case["its"] // case["frame_every"]
            state["frames"] = torch.empty((k,) + tuple(u0.shape), dtype=u0.dtype, device="cuda")
    state["case"] = case
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        u0, alpha = state["u0"], state["alpha"]
        n = case["nx"]
        uT = heat_solve(u0, alpha, case["levels"], 0.15 / (n * n), 1.0 / n, every=case["every"],
                        swept=case["swept"])
        g0, ga = torch.autograd.grad(uT, (u0, alpha), state["w"])
        return uT.detach(), g0, ga
    if case["kind"] == "batch":
        b = state["batch"]
        for i, u in enumerate(state["u0"]):
            b.set_state(i, u)
        b.run(case["levels"])
        return [b.get_state(i) for i in range(len(b))]
    e = state["engine"]
    e.set_state(state["u0"])
    if "frames" in state:
        e.run(case["levels"], mode=case["mode"], frames=state["frames"],
              frame_every=case["frame_every"])
    else:
        e.run(case["levels"], mode=case.get("mode", "swept"))
    for level, out in enumerate(state["out"]):
        e.get_state(level, out=out)
    return state["out"] + ([state["frames"]] if "frames" in state else [])


def work(case):
    if case["kind"] == "batch":
        cells = sum(a * b for a, b in _batch_sizes(case))
        return {"bytes": 16 * cells, "flops": HEAT_FLOPS * cells * case["levels"]}
    cells, levels = case["nx"] * case["ny"], case["levels"]
    if case["kind"] == "solve":
        # in: the field, the diffusivity, the output's gradient; out: the field, two gradients.
        # forward 10, the adjoint level 11 and the old level's Laplacian with its product 8
        return {"bytes": 48 * cells, "flops": 29 * cells * levels}
    if case["kind"] == "hook":
        return {"bytes": 16 * cells, "flops": HEAT_FLOPS * cells * levels}
    size = 4 if case["dtype"] == "float32" else 8
    nv, per = (4, EULER_FLOPS) if case["eq"] == "euler" else (1, HEAT_FLOPS)
    frames = levels // case["its"] // case["frame_every"] if case["frame_every"] else 0
    return {"bytes": size * nv * cells * (1 + case["its"] + frames), "flops": per * cells * levels}


# ------------------------------------------------------------------- exact ---
def _second(u):
    return ((torch.roll(u, -1, -2) - 2 * u) + torch.roll(u, 1, -2),
            (torch.roll(u, -1, -1) - 2 * u) + torch.roll(u, 1, -1))


def _heat_change(u, c):
    xx, yy = _second(u)
    return c * xx + c * yy


def _pressure(gm1, q):
    return gm1 * (q[3] - (q[1] * q[1] + q[2] * q[2]) / (2.0 * q[0]))


def _limited(a, b, num, den):
    r = num / den
    r = torch.where(torch.isfinite(r) & (r <= 1e6) & (r >= 0), r, torch.zeros_like(r))
    h = torch.clamp(r, max=1.0) * 0.5
    return a + h * (b - a)


def _euler_change(q, axis, gm1):
    """The flux difference along axis 1 (rows) or 2 (columns)."""
    A, B = axis, 3 - axis
    up = lambda t: torch.roll(t, -1, axis - 3)  # noqa: E731  the next cell's
    P = _pressure(gm1, q)
    d = up(P) - P
    L = _limited(q, up(q), d, torch.roll(d, 1, axis - 3))
    R = _limited(up(q), q, d, up(d))
    pl, pr = _pressure(gm1, L), _pressure(gm1, R)
    f = torch.empty_like(q)
    f[0] = L[A] + R[A]
    f[A] = ((L[A] * L[A] / L[0] + pl) + R[A] * R[A] / R[0]) + pr
    f[B] = L[1] * L[2] / L[0] + R[1] * R[2] / R[0]
    f[3] = (L[3] + pl) * L[A] / L[0] + (R[3] + pr) * R[A] / R[0]
    rl, rr = torch.sqrt(L[0]), torch.sqrt(R[0])
    inv = 1.0 / (rl + rr)
    m = rl * rr
    v = [(rl * (L[k] / L[0]) + rr * (R[k] / R[0])) * inv for k in (1, 2, 3)]
    p = _pressure(gm1, [m, m * v[0], m * v[1], m * v[2]])
    rad = torch.sqrt(GAMMA * p / m) + torch.abs(v[A - 1])
    rad = torch.where(torch.isnan(rad), torch.zeros_like(rad), rad)
    s = rad * (L - R)
    lo = lambda t: torch.roll(t, 1, axis - 3)  # noqa: E731  the lower face's
    return (((lo(f) + lo(s)) - f) - s) * 0.5


def _advance(case, u, c):
    """All levels from u; (newest, the one before, frames)."""
    prev, frames, its, every = u, [], case.get("its", 1), case.get("frame_every", 0)
    euler = case.get("eq") == "euler"
    for level in range(1, case["levels"] + 1):
        if euler:
            dtdx = 0.1 * (10.0 / case["nx"]) / (10.0 / case["nx"])
            d = _euler_change(u, 1, GAMMA - 1) * dtdx + _euler_change(u, 2, GAMMA - 1) * dtdx
        else:
            d = _heat_change(u, c)
        if its == 1:
            new = d + u
        else:
            new = prev + d if level % 2 == 0 else u + 0.5 * d
        prev, u = u, new
        if every and level % its == 0 and (level // its) % every == 0:
            frames.append(u)
    return u, prev, frames


def exact(case, seed):
    nx, ny = case.get("nx"), case.get("ny")
    if case["kind"] == "batch":
        out = []
        for i, (a, b) in enumerate(_batch_sizes(case)):
            g = _heat_globals(a)
            one = {"levels": case["levels"]}
            out.append(_advance(one, _fourier(a, b, seed + i)[None], g[5] * g[2] / g[3] / g[3])[0].cpu().numpy())
        return out
    if case["kind"] == "solve":
        u, alpha, w = _fourier(nx, ny, seed), _diffusivity(nx, ny, seed), _fourier(nx, ny, seed + 2)
        dt, dx = 0.15 / (nx * nx), 1.0 / nx
        c = alpha * dt / dx / dx
        states = []
        for _ in range(case["levels"]):
            states.append(u)
            u = _heat_change(u, c) + u
        lam, gc = w, torch.zeros_like(w)
        for old in reversed(states):
            xx, yy = _second(old)
            gc = gc + lam * (xx + yy)
            xx, yy = _second(c * lam)
            lam = lam + (xx + yy)
        return u, lam, gc * (dt / dx / dx)
    dtype = getattr(torch, case.get("dtype", "float64"))
    if case.get("eq") == "euler":
        u, c = _vortex(nx, ny, seed), None
    else:
        g = _heat_globals(nx)
        u, c = _fourier(nx, ny, seed)[None].to(dtype).double(), g[5] * g[2] / g[3] / g[3]
    new, old, frames = _advance(case, u, c)
    out = [new, old][:case.get("its", 1)]
    return out + ([torch.stack(frames)] if frames else [])
