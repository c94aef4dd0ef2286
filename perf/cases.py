"""Performance cases of the channel-flow library: what is timed, on which inputs, and what
the results have to agree with.

Every case goes through the package's public entry points, as a program that uses the
library does:

* ``step``     -- Channel.step(n): n RK2 projection steps on device-resident fields, the
                  work of a DNS run.  FP64 and mixed precision, Thomas and PDD.
* ``solve``    -- DevicePoissonSolver.solve on a device array: the Poisson operator inside
                  another program's step.
* ``hostsolve``-- PoissonSolver.execute on the ghosted host array: the reference solver's
                  call sequence, linked in place of its C solver.
* ``adjoint``  -- Channel.adjoint_ke_gradient: forward sweep, recomputed segments and the
                  reverse sweep (the backward direction of the step).
* ``monitors`` -- a step whose results a run reports (diagnostics, skin friction, bulk
                  velocity, kinetic energy, a probe).

``exact`` states the same results with torch in 64 bits, independently of the package: the
momentum equations in flux form, complex FFTs, and the wall-normal systems solved by
elimination, with the reference's truncated PDD where partitions are asked for.
"""
import math

import numpy as np
import torch

import powerllel_channel_b200 as plb

LX, LY, LZ = 2.0 * math.pi, math.pi, 2.0
DT = 1e-4


def _case(kind, name, nx, ny, nz, precision="fp64", parts=0, re_tau=180.0, stretch=1.5, noise=0.1, u_crf=0.0, steps=1,
          every=1):
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "parts": parts,
            "re_tau": re_tau, "stretch": stretch, "noise": noise, "u_crf": u_crf, "steps": steps, "every": every}


def listed():
    return [
        # a single step of the smallest benchmark channel: latency and launches
        _case("step", "step_64x64x64_fp64", 64, 64, 64),
        # the same channel in mixed precision, ten steps between two outputs
        _case("step", "step_64x64x64_mixed", 64, 64, 64, "mixed", steps=10),
        # an ordinary run over four wall-normal partitions (PDD), both precisions
        _case("step", "step_256x192x128_pdd4_fp64", 256, 192, 128, parts=4, re_tau=550.0, stretch=1.8, noise=0.05,
              steps=3),
        _case("step", "step_256x192x128_pdd4_mixed", 256, 192, 128, "mixed", 4, 550.0, 1.8, 0.05, steps=3),
        # the headline channel, both precisions (three steps: the mixed path's third one is
        # its first incremental projection)
        _case("step", "step_512x384x256_fp64", 512, 384, 256, re_tau=1000.0, stretch=2.0, steps=3),
        _case("step", "step_512x384x256_mixed", 512, 384, 256, "mixed", 0, 1000.0, 2.0, steps=3),
        # the largest benchmark channel
        _case("step", "step_1024x768x512_pdd8_mixed", 1024, 768, 512, "mixed", 8, 2000.0, 2.0, steps=2),
        # a grid chosen for its resolution alone: lengths 2 * 3^a, planes that no tile divides
        _case("step", "step_324x162x150_fp64", 324, 162, 150, re_tau=395.0, stretch=1.7, steps=2),
        # the Poisson solve on its own, in another program's step
        _case("solve", "solve_512x384x256_mixed", 512, 384, 256, "mixed", 0, 1000.0, 2.0),
        # the reference's call sequence on a host array
        _case("hostsolve", "hostsolve_128x96x64_pdd4", 128, 96, 64, parts=4),
        # gradient of the kinetic energy at the adjoint's benchmark grid
        _case("adjoint", "adjoint_256x192x128", 256, 192, 128, re_tau=550.0, stretch=1.8, noise=0.05, steps=6, every=3),
        # a step that a run reports on: the monitors' reductions follow it
        _case("monitors", "monitors_256x192x128", 256, 192, 128, parts=4, re_tau=550.0, stretch=1.8, noise=0.05),
    ]


# even lengths 2^a 3^b, what the transforms take
_LENGTHS = sorted(2 ** a * 3 ** b for a in range(1, 10) for b in range(0, 6) if 16 <= 2 ** a * 3 ** b <= 512)


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["solve"] * 2 + ["hostsolve", "adjoint", "monitors"])
    most = {"step": 512 * 384 * 256, "solve": 512 * 384 * 256, "hostsolve": 1 << 20, "adjoint": 256 * 192 * 64,
            "monitors": 512 * 384 * 128}[kind]
    while True:
        # sizes even over their logarithm
        nx, ny = rng.choice(_LENGTHS), rng.choice(_LENGTHS)
        nz = 2 * round(math.exp(rng.uniform(math.log(8.0), math.log(192.0))))
        if 32768 <= nx * ny * nz <= most:
            break
    parts = rng.choice([p for p in (3, 4, 5, 6, 8) if nz // p >= 4]) if rng.random() < 0.4 else 0
    precision = rng.choice(["fp64", "mixed"])
    if kind in ("hostsolve", "adjoint", "monitors"):
        precision = "fp64"
    if kind == "adjoint":
        parts = 0  # the adjoint is defined for the Thomas solve
    if kind in ("hostsolve", "monitors") or (kind == "solve" and precision == "fp64"):
        # with Thomas in FP64 the pressure's free constant is round-off over round-off (as in
        # the reference), so a bare solve is compared over partitions, where it is determined;
        # likewise the divergence left by the projection, which the monitors report
        parts = parts or rng.choice([p for p in (3, 4, 5, 6, 8) if nz // p >= 4])
    if kind == "solve" and precision == "mixed":
        parts = 0
    steps = 1
    if kind == "step":
        steps = rng.choice([1, 2, 3, 5])
        while steps * nx * ny * nz > 100_000_000:
            steps -= 1
    every = 1
    if kind == "adjoint":
        steps = rng.choice([2, 3, 4])
        every = rng.choice([1, 2, 3])
    case = _case(kind, "", nx, ny, nz, precision, parts, rng.choice([180.0, 395.0, 550.0]),
                 rng.choice([0.0, 1.5, 2.0]), 0.1, rng.choice([0.0, 0.0, 0.3]) if kind == "step" else 0.0, steps, every)
    del case["name"]
    return case


def work(case):
    """Bytes and operations of one pass that the method cannot do without: per step the velocity
    read and written once (and, mixed, the two old pressures read and the new one written); the
    arithmetic of two momentum evaluations (about 150 operations a point in flux form), of the
    four real transforms and of the wall-normal solves."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = float(nx) * ny * nz
    solve_flops = n * (5.0 * (math.log2(nx) + math.log2(ny)) + 8.0)
    step_flops = n * (300.0 + 20.0) + solve_flops
    step_bytes = n * (48.0 + (12.0 if case["precision"] == "mixed" and case["parts"] == 0 else 0.0))
    kind = case["kind"]
    if kind == "step":
        return {"bytes": case["steps"] * step_bytes, "flops": case["steps"] * step_flops}
    if kind == "solve":
        return {"bytes": n * (16.0 if case["precision"] == "fp64" else 8.0), "flops": solve_flops}
    if kind == "hostsolve":
        return {"bytes": n * 16.0, "flops": solve_flops}
    if kind == "adjoint":
        # forward steps, segments recomputed but for their last step, and the reverse steps
        # (state and adjoint read, adjoint written; two transposed stencils and the stage-1
        # field, about three momentum evaluations)
        segments = -(-case["steps"] // case["every"])
        forward = 2 * case["steps"] - segments
        return {"bytes": forward * n * 48.0 + case["steps"] * n * 72.0,
                "flops": forward * step_flops + case["steps"] * (n * 550.0 + solve_flops)}
    return {"bytes": step_bytes, "flops": step_flops + n * 40.0}  # the monitors can ride on the step's passes


def tolerance(case):
    """About four times the largest difference between the library and the FP64 torch statement
    below, over the listed cases and a few dozen drawn ones.  Mixed: the FP32 stencils and
    transforms; the first projection of a noisy field, a full pressure solve, leaves 4e-7 in
    v and w at most grids (6e-7 at the worst drawn one), and the (0,0) mode's FP32 transform 2e-6 in a bare solve.  FP64: rounding; the
    adjoint's dJ/df and the monitors' divergence are sums and differences that cancel."""
    if case["precision"] == "mixed":
        return {"rel": 2.5e-6, "max": 2e-5} if case["kind"] == "step" else {"rel": 1e-5, "max": 4e-5}
    if case["kind"] in ("adjoint", "monitors"):
        return {"rel": 4e-11, "max": 1e-10}
    return {"rel": 2e-13, "max": 2e-12}


# ---------------------------------------------------------------------------
# inputs and passes
# ---------------------------------------------------------------------------
class _DeviceArray:
    """A device array of the library, for torch.as_tensor (no copy)."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f8", "version": 2}


def _field(state, which):
    ch = state["channel"]
    ptr = ch.field_ptr(which)
    if ptr not in state["views"]:  # the step alternates between two sets of arrays
        c = ch.cfg
        state["views"][ptr] = torch.as_tensor(_DeviceArray(ch, ptr, (c.nz + 2, c.ny, c.nx)), device="cuda")
    return state["views"][ptr]


def _spacing(case):
    """dzf[0 .. nz+1] of the tanh-stretched grid (uniform for stretch 0)."""
    nz, s = case["nz"], case["stretch"]
    if s == 0.0:
        return np.full(nz + 2, LZ / nz)
    zf = 0.5 * (1.0 + np.tanh((np.arange(nz + 1) / nz - 0.5) * s) / math.tanh(s / 2.0))
    zf[0] = 0.0
    d = LZ * np.diff(zf)
    return np.concatenate([d[:1], d, d[-1:]])


def _right_hand_side(case, seed):
    """Divergence of a random velocity field that vanishes at the walls: what a projection
    hands to the solve, and consistent with the walls' Neumann condition."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    dzf = torch.tensor(_spacing(case)[1:-1], device="cuda")[:, None, None]
    q = torch.randn((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64)
    r = (q - q.roll(1, 2)) * (nx / LX)
    q = torch.randn((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64)
    r += (q - q.roll(1, 1)) * (ny / LY)
    q = torch.randn((nz, ny, nx), generator=g, device="cuda", dtype=torch.float64)
    q[-1] = 0.0
    r[0] += q[0] / dzf[0]
    r[1:] += (q[1:] - q[:-1]) / dzf[1:]
    return r


def _channel(case):
    return plb.Channel(plb.ChannelConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], stretch_ratio=case["stretch"],
                                         re_tau=case["re_tau"], dt=DT, u_crf=case["u_crf"], trid_parts=case["parts"],
                                         precision=plb.PL_MIXED if case["precision"] == "mixed" else plb.PL_FP64))


_HOST_SOLVER = {}  # the reference's solver is one per process


def _host_solver(case):
    key = (case["nx"], case["ny"], case["nz"], case["stretch"], case["parts"])
    if key not in _HOST_SOLVER:
        for old in list(_HOST_SOLVER):
            _HOST_SOLVER.pop(old).free()
        _HOST_SOLVER[key] = plb.PoissonSolver(case["nx"], case["ny"], case["nz"], LX / case["nx"], LY / case["ny"],
                                              _spacing(case), nparts=case["parts"])
    return _HOST_SOLVER[key]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        fp64 = case["precision"] == "fp64"
        solver = plb.DevicePoissonSolver(case["nx"], case["ny"], case["nz"], LX / case["nx"], LY / case["ny"],
                                         _spacing(case), nparts=case["parts"],
                                         precision=plb.PL_FP64 if fp64 else plb.PL_MIXED)
        rhs = _right_hand_side(case, seed).to(torch.float64 if fp64 else torch.float32)
        return {"kind": kind, "solver": solver, "rhs": rhs, "x": torch.empty_like(rhs)}
    if kind == "hostsolve":
        rhs = np.zeros((case["nz"] + 2, case["ny"] + 2, case["nx"] + 2))
        rhs[1:-1, 1:-1, 1:-1] = _right_hand_side(case, seed).cpu().numpy()
        return {"kind": kind, "solver": _host_solver(case), "rhs": rhs, "x": np.empty_like(rhs)}
    ch = _channel(case)
    ch.init_flow(int(seed), case["noise"])
    state = {"kind": kind, "channel": ch, "views": {}, "steps": case["steps"], "every": case["every"]}
    if kind == "adjoint":
        shape = (case["nz"] + 2, case["ny"], case["nx"])
        state["grad"] = [torch.empty(shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    if kind == "monitors":
        state["probe"] = (case["nx"] // 3, case["ny"] // 2, case["nz"] // 4)
    return state


def run(state):
    kind = state["kind"]
    if kind == "solve":
        # the solve is in place: the program's new right-hand side goes into its array first
        state["x"].copy_(state["rhs"])
        state["solver"].solve(state["x"], stream=torch.cuda.current_stream())
        return state["x"]
    if kind == "hostsolve":
        np.copyto(state["x"], state["rhs"])
        state["solver"].execute(state["x"])
        return state["x"]
    ch = state["channel"]
    if kind == "step":
        ch.step(state["steps"])
        # the pressure is not carried on (FP64 solves for it anew) or enters the next steps'
        # velocities (mixed), and its constant is arbitrary: the velocity is the state
        return [_field(state, q) for q in range(3)]
    if kind == "adjoint":
        ke, gf = ch.adjoint_ke_gradient(state["steps"], state["every"], *state["grad"])
        return {"ke": ke, "gf": gf, "grad": state["grad"]}
    ch.step(1)
    d = ch.diagnostics()
    return {"fields": [_field(state, q) for q in range(3)], "div_max": d["div_max"], "cfl_max": d["cfl_max"], "nan_count": d["nan_count"], "cfl_ijk": list(d["cfl_ijk"]),
            "skin": [list(ch.skin_friction(wall)) for wall in (0, 1)], "means": ch.forcing_means(),
            "ke": ch.kinetic_energy(), "probe": ch.probe(*state["probe"])}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
class _Grid:
    def __init__(self, case):
        self.nx, self.ny, self.nz, self.parts = case["nx"], case["ny"], case["nz"], case["parts"]
        self.dx, self.dy = LX / self.nx, LY / self.ny
        self.re_inv = 1.0 / (case["re_tau"] / 0.09) ** (1.0 / 0.88)
        self.u_crf = case["u_crf"]
        f = _spacing(case)
        c = 0.5 * (f[:-1] + f[1:])
        c = np.append(c, c[-1])
        self.f_np, self.c_np = f, c
        col = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)[:, None, None]  # noqa: E731
        self.f, self.c = col(f), col(c)

    # wall-normal operator d/dz (1/dzc) d/dz, Neumann at both walls
    def rows(self):
        f, nz = self.f_np, self.nz
        lo = 2.0 / (f[1:nz + 1] * (f[:nz] + f[1:nz + 1]))
        up = 2.0 / (f[1:nz + 1] * (f[2:] + f[1:nz + 1]))
        di = -lo - up
        di[0] += lo[0]
        di[-1] += up[-1]
        lo[0] = up[-1] = 0.0
        return lo, di, up

    def eigenvalues(self):
        w = lambda n, h: 2.0 * (torch.cos(2.0 * math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n) - 1.0) / h ** 2  # noqa: E731
        return w(self.ny, self.dy)[:, None] + w(self.nx, self.dx)[None, :self.nx // 2 + 1]


def _eliminate(lo, di, up, lam, r):
    """Thomas elimination over dim 0 of r (complex), real rows; di + lam is the diagonal."""
    n = len(di)
    piv, x = di[0] + lam, [r[0]]
    pivots = [piv]
    for k in range(1, n):
        m = lo[k] / piv
        piv = di[k] + lam - m * up[k - 1]
        x.append(r[k] - m * x[-1])
        pivots.append(piv)
    for k in range(n - 1, -1, -1):
        x[k] = (x[k] if k == n - 1 else x[k] - up[k] * x[k + 1]) / pivots[k]
    return torch.stack(x)


def _partitions(nz, parts):
    size, extra = divmod(nz, parts)
    sizes = [size + (1 if m >= parts - extra else 0) for m in range(parts)]
    starts = [sum(sizes[:m]) for m in range(parts)]
    return list(zip(starts, sizes))


def _wall_normal(g, spectrum, transpose=False):
    """The systems of all wavenumber pairs: Thomas with the (0,0) system's free constant fixed
    at the last row, or the truncated PDD over g.parts partitions."""
    lo, di, up = (list(map(float, a)) for a in g.rows())
    lam = g.eigenvalues()
    if g.parts == 0:
        if transpose:
            lo, up = [0.0] + up[:-1], lo[1:] + [0.0]
        # the free constant: the last diagonal of the singular system is moved off its value,
        # so that x[nz-1] is the (vanishing) inconsistency of the right-hand side
        last = torch.full_like(lam, di[-1])
        last[0, 0] = 2.0 * di[-1] - 1.0
        return _eliminate(lo, di[:-1] + [last], up, lam, spectrum)
    blocks = []
    for k0, n in _partitions(g.nz, g.parts):
        s = slice(k0, k0 + n)
        a, b, c = lo[s], di[s], up[s]
        zero = torch.zeros((n,) + lam.shape, device="cuda", dtype=torch.float64)
        v, w = zero.clone(), zero
        v[0], w[-1] = a[0], c[-1]
        blocks.append([_eliminate(a, b, c, lam, spectrum[s]), _eliminate(a, b, c, lam, v), _eliminate(a, b, c, lam, w)])
    below = [None] * g.parts  # value under a partition's first row, over its last row
    above = [None] * g.parts
    for m in range(g.parts - 1):
        (x0, _, w0), (x1, v1, _) = blocks[m], blocks[m + 1]
        det = 1.0 - w0[-1] * v1[0]
        below[m + 1] = (x0[-1] - w0[-1] * x1[0]) / det
        above[m] = (x1[0] - v1[0] * x0[-1]) / det
    out = []
    for (x, v, w), lower, upper in zip(blocks, below, above):
        if lower is not None:
            x = x - v * lower
        if upper is not None:
            x = x - w * upper
        out.append(x)
    return torch.cat(out)


class _Poisson(torch.autograd.Function):
    """p with L p = r over (nz, ny, nx); the gradient is the transposed solve."""

    @staticmethod
    def forward(ctx, r, g, transpose):
        ctx.g, ctx.transpose = g, transpose
        return torch.fft.irfft2(_wall_normal(g, torch.fft.rfft2(r), transpose), s=r.shape[1:])

    @staticmethod
    def backward(ctx, grad):
        return _Poisson.apply(grad, ctx.g, not ctx.transpose), None, None


def _east(a):
    return a.roll(-1, 2)


def _west(a):
    return a.roll(1, 2)


def _north(a):
    return a.roll(-1, 1)


def _south(a):
    return a.roll(1, 1)


def _walls(g, u, v, w):
    """Interior levels (w: up to nz-1 used) to levels 0 .. nz+1 with the no-slip walls."""
    zero = torch.zeros_like(w[:1])
    return (torch.cat([-2.0 * g.u_crf - u[:1], u, -2.0 * g.u_crf - u[-1:]]), torch.cat([-v[:1], v, -v[-1:]]),
            torch.cat([zero, w[:-1], zero, zero]))


def _momentum(g, q, which):
    """Viscous minus convective terms of one component on levels 1..nz."""
    u, v, w = q
    dxi, dyi = 1.0 / g.dx, 1.0 / g.dy
    own = q[which]
    mid = own[1:-1]
    if which == 0:
        fx = (mid + _east(mid)) ** 2
        fy = (mid + _north(mid)) * (v[1:-1] + _east(v[1:-1]))
    elif which == 1:
        fx = (u[1:-1] + _north(u[1:-1])) * (mid + _east(mid))
        fy = (mid + _north(mid)) ** 2
    else:
        fx = (u[1:-1] * g.f[2:] + u[2:] * g.f[1:-1]) / g.c[1:-1] * (mid + _east(mid))
        fy = (v[1:-1] * g.f[2:] + v[2:] * g.f[1:-1]) / g.c[1:-1] * (mid + _north(mid))
    out = -0.25 * ((fx - _west(fx)) * dxi + (fy - _south(fy)) * dyi)
    del fx, fy
    if which == 2:
        fz = (own[:-1] + own[1:]) ** 2
        out = out - 0.25 * (fz[1:] - fz[:-1]) / g.c[1:-1]
        visc = (own[1:] - own[:-1]) / g.f[1:]
        visc = (visc[1:] - visc[:-1]) / g.c[1:-1]
    else:
        side = _east if which == 0 else _north
        fz = (own[:-1] * g.f[1:] + own[1:] * g.f[:-1]) / g.c[:-1] * (w[:-1] + side(w[:-1]))
        out = out - 0.25 * (fz[1:] - fz[:-1]) / g.f[1:-1]
        visc = (own[1:] - own[:-1]) / g.c[:-1]
        visc = (visc[1:] - visc[:-1]) / g.f[1:-1]
    del fz
    if g.u_crf != 0.0:
        out = out - 0.5 * g.u_crf * dxi * (_east(mid) - _west(mid))
    visc = visc + (_east(mid) - 2.0 * mid + _west(mid)) * dxi ** 2
    visc = visc + (_north(mid) - 2.0 * mid + _south(mid)) * dyi ** 2
    return out + g.re_inv * visc


def _step(g, q, force=None):
    q1 = [q[c][1:-1] + DT * (_momentum(g, q, c) if force is None else _momentum(g, q, c) + force[c]) for c in range(3)]
    q1 = _walls(g, *q1)
    q = [0.5 * (q1[c][1:-1] + DT * (_momentum(g, q1, c) if force is None else _momentum(g, q1, c) + force[c]) +
                q[c][1:-1]) for c in range(3)]
    del q1
    u, v, w = q
    w = torch.cat([w[:-1], torch.zeros_like(w[:1])])
    below = torch.cat([torch.zeros_like(w[:1]), w[:-1]])
    r = ((u - _west(u)) / g.dx + (v - _south(v)) / g.dy + (w - below) / g.f[1:-1]) / DT
    del below
    p = _Poisson.apply(r, g, False)
    g.p = p.detach()
    del r
    u = u - DT / g.dx * (_east(p) - p)
    v = v - DT / g.dy * (_north(p) - p)
    w = torch.cat([w[:-1] - DT * (p[1:] - p[:-1]) / g.c[1:-2], w[-1:]])
    u = u + (1.0 - (u * g.f[1:-1]).sum() / (LZ * g.nx * g.ny))
    return _walls(g, u, v, w)


def _initial(g, seed, noise):
    """Poiseuille profile with SplitMix64 noise, unit bulk velocity, in the moving frame."""
    def uniform(start, count):
        z = torch.arange(start + 1, start + 1 + count, device="cuda", dtype=torch.int64)
        z = z * (0x9E3779B97F4A7C15 - (1 << 64)) + int(seed)
        z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * (0xBF58476D1CE4E5B9 - (1 << 64))
        z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * (0x94D049BB133111EB - (1 << 64))
        z = z ^ ((z >> 31) & ((1 << 33) - 1))
        return ((z >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53
    n = g.nx * g.ny * g.nz
    parts = [(2.0 * (uniform(c * n, n) - 0.5) * noise).view(g.nz, g.ny, g.nx) for c in range(3)]
    z = np.concatenate([[-0.5 * g.f_np[0]], 0.5 * (g.f_np[:-1] + g.f_np[1:])]).cumsum()[1:-1] / LZ
    u = parts[0] + torch.tensor(6.0 * (1.0 - z) * z, device="cuda")[:, None, None]
    mean = (u * g.f[1:-1]).sum() / (LZ * g.nx * g.ny)
    return u / mean - g.u_crf, parts[1], parts[2]


def _energy(g, q):
    u, v, w = q
    return 0.5 * g.dx * g.dy * ((g.f[1:-1] * (u[1:-1] ** 2 + v[1:-1] ** 2)).sum() + (g.c[1:-2] * w[1:-2] ** 2).sum())


def exact(case, seed):
    g = _Grid(case)
    kind = case["kind"]
    if kind in ("solve", "hostsolve"):
        r = _right_hand_side(case, seed)
        if case["precision"] == "mixed":
            r = r.float().double()
        p = _Poisson.apply(r, g, False)
        if case["precision"] == "mixed":
            # the mixed solve's free constant: zero plane mean at the middle row where the column
            # is swept from both walls, at the last row otherwise
            nz = g.nz
            p = p - p[nz // 2 if nz % 16 == 0 and 16 <= nz <= 256 else nz - 1].mean()
        if kind == "solve":
            return p
        out = np.zeros((g.nz + 2, g.ny + 2, g.nx + 2))
        out[1:-1, 1:-1, 1:-1] = p.cpu().numpy()
        return out
    start = _initial(g, seed, case["noise"])
    if kind == "step":
        q = _walls(g, *start)
        for _ in range(case["steps"]):
            q = _step(g, q)
        return list(q)
    if kind == "adjoint":
        x = [a.clone().requires_grad_(True) for a in start]
        force = torch.zeros(3, device="cuda", dtype=torch.float64, requires_grad=True)
        q = _walls(g, *x)
        for _ in range(case["steps"]):
            q = _step(g, q, force)
        ke = _energy(g, q)
        ke.backward()
        pad = lambda a: torch.cat([torch.zeros_like(a[:1]), a, torch.zeros_like(a[:1])])  # noqa: E731
        return {"ke": float(ke.detach()), "gf": force.grad.cpu().numpy(), "grad": [pad(a.grad) for a in x]}
    q = _step(g, _walls(g, *start))
    u, v, w = (a[1:-1] for a in q)
    div = (u - _west(u)) / g.dx + (v - _south(v)) / g.dy + (w - q[2][:-2]) / g.f[1:-1]
    cfl = 0.5 * ((u + _west(u)).abs() / g.dx + (v + _south(v)).abs() / g.dy + (w + q[2][:-2]).abs() / g.f[1:-1])
    skin = []
    for level in (1, g.nz):
        tau = float(q[0][level].mean()) * g.re_inv / (0.5 * g.f_np[level])
        skin.append([math.sqrt(tau), 2.0 * tau])
    i, j, k = case["nx"] // 3 - 1, case["ny"] // 2 - 1, case["nz"] // 4
    return {"fields": list(q), "div_max": float(div.abs().max()), "cfl_max": float(cfl.max()) * DT, "nan_count": None, "cfl_ijk": None,
            "skin": skin, "means": np.array([float((u * g.f[1:-1]).sum()) / (LZ * g.nx * g.ny), 0.0, 0.0]),
            "ke": float(_energy(g, q)), "probe": np.array([float(a[k, j, i]) for a in q] + [float(g.p[k - 1, j, i])])}
