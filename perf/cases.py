"""The calls that the performance of this framework is judged by, and how to run one pass of each.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges.  ``prepare`` makes what a
program holds before the call (a plan, positions, charges), ``run`` is one pass through the public
entry points, ``exact`` the same result in 64 bits from plain torch, ``work`` the bytes and
operations that a pass cannot do without.

Kinds of case:

solve   one system on one plan, device buffers (``SpectralEwald.solve``), optionally replayed from
        a CUDA graph as a time-stepping program does
host    the same through pinned host arrays (``SpectralEwald.solve_host``)
batch   many systems of uneven size in one launch set (``BatchSolver.solve``)
real    the short-range and self parts of the Ewald sum (``real_space``, ``self_term``)
steps   the reference's own step calls on device arrays (``SE_FGG_expand_all`` ... ``SE_FGG_int``)

FP64 results are returned as they come.  A program that chooses FP32 gridding (results good to
about 1e-6) holds its potentials and forces in single precision, so those cases end with the
conversion into its float32 array.
"""
import ctypes
import math
import random

import torch

from se_fast_gridding_b200 import fgg, solver

# grid sizes of the configurations and tests (whole 16^3 tiles), and FFT-friendly sizes between them
TILED = (32, 48, 64, 80, 96, 112, 128, 144, 160, 192, 208, 224, 240, 256)
RAGGED = (36, 40, 45, 50, 54, 60, 72, 75, 90, 100, 108, 120, 135, 150, 180, 200, 216, 250)


def listed():
    return [
        # a small molecule-sized system in full precision: launches and latency only
        {"name": "tiny_fp64", "kind": "solve", "N": 100, "M": 32, "P": 21, "L": 1.0, "xi": 8.0,
         "mode": "potential", "precision": "fp64", "graph": False, "clusters": 0},
        # the small end of a request stream
        {"name": "small_fp32", "kind": "solve", "N": 1501, "M": 64, "P": 8, "L": 1.0, "xi": 8.0,
         "mode": "force", "precision": "fp32", "graph": False, "clusters": 0},
        # the headline system, stepped in time from a graph
        {"name": "force_fp32", "kind": "solve", "N": 100_000, "M": 128, "P": 16, "L": 1.0, "xi": 20.0,
         "mode": "force", "precision": "fp32", "graph": True, "clusters": 0},
        # the same in full precision, called directly
        {"name": "force_fp64", "kind": "solve", "N": 100_000, "M": 128, "P": 16, "L": 1.0, "xi": 20.0,
         "mode": "force", "precision": "fp64", "graph": False, "clusters": 0},
        # a large request of a stream, potentials only, FFTs in FP32 too
        {"name": "pot_fft32", "kind": "solve", "N": 777_777, "M": 224, "P": 12, "L": 1.0, "xi": 28.0,
         "mode": "potential", "precision": "fp32-fft32", "graph": False, "clusters": 0},
        # a grid that is not cut into whole tiles and a stencil above 16
        {"name": "ragged_fp64", "kind": "solve", "N": 20_011, "M": 100, "P": 20, "L": 2.0, "xi": 9.0,
         "mode": "force", "precision": "fp64", "graph": False, "clusters": 0},
        # clustered particles: crowded tiles beside empty ones
        {"name": "clustered_fp32", "kind": "solve", "N": 2_000_000, "M": 256, "P": 12, "L": 1.0,
         "xi": 30.0, "mode": "force", "precision": "fp32", "graph": False, "clusters": 64},
        # the largest system
        {"name": "large_fp32", "kind": "solve", "N": 16_000_000, "M": 512, "P": 12, "L": 1.0,
         "xi": 60.0, "mode": "force", "precision": "fp32", "graph": False, "clusters": 64},
        # 256 systems of 1,000 to 64,000 particles and three stencils in one launch set
        {"name": "batch_fp32", "kind": "batch", "systems": 256, "n_min": 1000, "n_max": 64_000,
         "M": 64, "mode": "potential", "precision": "fp32", "graph": False, "mix": 3},
        # host arrays in and out: the drop-in for one call of the reference's solver
        {"name": "host_fp64", "kind": "host", "N": 250_001, "M": 192, "P": 12, "L": 1.0, "xi": 24.0,
         "mode": "potential", "precision": "fp64", "clusters": 0},
        # the short-range part that completes the sum: about 100 neighbours each
        {"name": "real_fp64", "kind": "real", "N": 50_000, "L": 1.0, "rc": 0.078, "xi": 50.0,
         "mode": "force"},
        # a program written for the reference's step calls, its arrays on the GPU
        {"name": "steps_fp64", "kind": "steps", "N": 30_011, "M": 64, "P": 16, "L": 1.0, "xi": 8.0,
         "mode": "force"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(("solve", "batch", "host", "real", "steps"), (62, 12, 9, 9, 8))[0]
    mode = rng.choice(("potential", "force"))
    L = round(_log(rng, 1.0, 4.0), 3)
    if kind == "batch":
        systems = int(round(_log(rng, 4, 128)))
        return {"kind": kind, "systems": systems, "n_min": 500,
                "n_max": int(_log(rng, 4000, 64_000)), "M": rng.choice((32, 48, 64, 96)),
                "mode": mode, "precision": rng.choice(("fp32", "fp32", "fp64")),
                "graph": rng.random() < 0.25, "mix": rng.randrange(1 << 20)}
    if kind == "real":
        N = int(_log(rng, 1000, 60_000))
        near = _log(rng, 40, 300)   # particles inside the cutoff
        rc = min(0.3, (near / N * 3 / (4 * math.pi)) ** (1 / 3)) * L
        return {"kind": kind, "N": N, "L": L, "rc": round(rc, 5),
                "xi": round(rng.uniform(3.0, 4.5) / rc, 4), "mode": mode}
    N = int(_log(rng, 100, 60_000 if kind == "steps" else 2_000_000))
    want = min(256.0, max(32.0, (N * _log(rng, 2.5, 60.0)) ** (1 / 3)))
    sizes = TILED if rng.random() < 0.7 else RAGGED
    if kind == "steps":
        sizes = tuple(m for m in sizes if m <= 128)
    M = min(sizes, key=lambda m: abs(m - want))
    P = rng.choice((8, 8, 12, 12, 16, 16, 16, 10, 14, 15, 20, 21))
    case = {"kind": kind, "N": N, "M": M, "P": P, "L": L, "xi": round(rng.uniform(0.11, 0.25) * M / L, 4),
            "mode": mode}
    if kind == "steps":
        return case
    case["precision"] = rng.choice(("fp32", "fp32", "fp32-fft32", "fp64", "fp64"))
    case["clusters"] = 64 if rng.random() < 0.15 else 0
    if kind == "solve":
        case["graph"] = rng.random() < 0.25
    return case


# ------------------------------------------------------------------ inputs --

def _particles(N, L, clusters, seed, charges="uniform"):
    """Positions in [0, L)^3 as x[n], x[n+N], x[n+2N] and charges of zero sum, uniform in [-1, 1] or
    +-1; clustered: Gaussians of width 0.02 L around uniform centres, wrapped into the box."""
    g = torch.Generator("cuda").manual_seed(seed)
    kw = dict(device="cuda", dtype=torch.float64, generator=g)
    if clusters:
        centres = torch.rand(3, clusters, **kw) * L
        which = torch.randint(0, clusters, (N,), device="cuda", generator=g)
        x = torch.randn(3, N, **kw).mul_(0.02 * L).add_(centres[:, which]).remainder_(L)
        x[x >= L] = 0.0
    else:
        x = torch.rand(3, N, **kw) * L
    if charges == "pm1":
        q = torch.ones(N, device="cuda", dtype=torch.float64)
        q[N // 2:] = -1.0
        q = q[torch.randperm(N, device="cuda", generator=g)]
    else:
        q = torch.rand(N, **kw) * 2 - 1
        q -= q.mean()
    return x.reshape(-1).contiguous(), q.contiguous()


def _systems(case):
    """The batch's systems: N log-uniform, L uniform in [1, 4], P from {8, 12, 16}, xi = M / (8 L)."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["systems"]):
        N, L, P = int(_log(rng, case["n_min"], case["n_max"])), rng.uniform(1.0, 4.0), rng.choice((8, 12, 16))
        out.append(solver.System(N=N, M=case["M"], P=P, L=L, xi=case["M"] / (8.0 * L), mode=case["mode"]))
    return out


def _batch_inputs(case, seed):
    parts = [_particles(s.N, s.L, 0, seed * 1000 + i, "pm1") for i, s in enumerate(_systems(case))]
    return torch.cat([x for x, _ in parts]), torch.cat([q for _, q in parts])


def _inputs(case, seed):
    return _particles(case["N"], case["L"], case.get("clusters", 0), seed)


def _field(case, seed):
    """A smooth periodic field on the M^3 grid, as the steps after the FFTs meet it (a few waves)."""
    g = torch.Generator("cuda").manual_seed(seed + 77)
    M = case["M"]
    spec = torch.zeros(M, M, M // 2 + 1, dtype=torch.complex128, device="cuda")
    n = max(2, M // 8)
    spec[:n, :n, :n] = torch.randn(n, n, n, dtype=torch.complex128, device="cuda", generator=g)
    return torch.fft.irfftn(spec, s=(M, M, M)) * M ** 1.5


def prepare(case, seed):
    kind, state = case["kind"], {"case": case}
    if kind == "batch":
        systems = _systems(case)
        state["batch"] = solver.BatchSolver(systems, case["precision"])
        if case["graph"]:
            state["batch"].set_graph(True)
        state["x"], state["q"] = _batch_inputs(case, seed)
        state["out"] = torch.empty(sum(s.N * s.out_width for s in systems), dtype=torch.float64, device="cuda")
        state["stream"] = torch.cuda.Stream() if case["graph"] else None
        return state
    x, q = _inputs(case, seed)
    if kind == "real":
        return state | {"x": x, "q": q}
    if kind == "steps":
        N, M, P = case["N"], case["M"], case["P"]
        _, p = fgg.fcn_params(M, P, case["L"], case["xi"], solver.default_m(P), N)
        work = fgg.Work(p, force=case["mode"] == "force", where="cuda")
        fgg.call("SE_FGG_base_gaussian", ctypes.byref(work.s), ctypes.byref(p))
        width = 3 if case["mode"] == "force" else 1
        # the reference's periodic arrays are column-major
        field = _field(case, seed).permute(2, 1, 0).contiguous().reshape(-1)
        return state | {"x": x, "q": q, "p": p, "work": work, "field": field,
                        "grid": torch.empty(M ** 3, dtype=torch.float64, device="cuda"),
                        "out": torch.empty(width * N, dtype=torch.float64, device="cuda")}
    plan = solver.SpectralEwald(case["M"], case["P"], case["L"], case["xi"], mode=case["mode"],
                                precision=case["precision"], max_particles=case["N"])
    state["plan"] = plan
    if kind == "host":
        x, q = x.cpu().pin_memory(), q.cpu().pin_memory()
        out = torch.empty(plan.out_width * case["N"], dtype=torch.float64).pin_memory()
        return state | {"x": x.numpy(), "q": q.numpy(), "out": out.numpy()}
    if case["graph"]:
        plan.set_graph(True)
    state |= {"x": x, "q": q, "stream": torch.cuda.Stream() if case["graph"] else None,
              "out": torch.empty(plan.out_width * case["N"], dtype=torch.float64, device="cuda")}
    return state


# ------------------------------------------------------------------- a pass --

def _solve(state, solve):
    """One solve on the caller's stream, or on the program's own stream where it replays a graph
    (solves on the default stream always run directly)."""
    s = state["stream"]
    if s is None:
        return solve(state["x"], state["q"], state["out"])
    s.wait_stream(torch.cuda.current_stream())
    out = solve(state["x"], state["q"], state["out"], stream=s)
    torch.cuda.current_stream().wait_stream(s)
    return out


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "steps":
        return _run_steps(state)
    if kind == "real":
        phi, force = solver.real_space(state["x"], state["q"], case["L"], case["xi"], 1, case["rc"],
                                       want_force=case["mode"] == "force")
        solver.self_term(state["q"], case["xi"], phi)
        return [phi] if force is None else [phi, force]
    if kind == "host":
        out = state["plan"].solve_host(state["x"], state["q"], state["out"])
        return out if case["precision"] == "fp64" else out.astype("float32")
    out = _solve(state, state["batch"].solve if kind == "batch" else state["plan"].solve)
    return out if case["precision"] == "fp64" else out.to(torch.float32)


def _run_steps(state):
    """Particles to the periodic grid, and a field back to the particles."""
    case, p, work = state["case"], state["p"], state["work"]
    w, pp = ctypes.byref(work.s), ctypes.byref(p)
    padded = p.npdims[0] * p.npdims[1] * p.npdims[2]
    st = fgg.state(state["x"], state["q"])
    force = case["mode"] == "force"
    fgg.call("SE_FGG_expand_all_SSE_force" if force else "SE_FGG_expand_all", w, ctypes.byref(st), pp)
    fgg.call("SE_fp_set_zero", work.s.H, padded)
    fgg.call("SE_FGG_grid_split_AVX_dispatch_force" if force else "SE_FGG_grid_split", w, ctypes.byref(st), pp)
    grid, out = fgg.dptr(state["grid"]), fgg.dptr(state["out"])
    fgg.call("SE_fp_set_zero", grid, state["grid"].numel())
    fgg.call("SE_FGG_wrap_fcn", grid, w, pp)
    fgg.call("SE_FGG_extend_fcn", w, fgg.dptr(state["field"]), pp)
    if force:
        fgg.call("SE_FGG_int_split_AVX_dispatch_force", out, ctypes.byref(st), w, pp)
    else:
        fgg.call("SE_FGG_int_split", out, w, pp)
    return {"grid": state["grid"], "out": state["out"]}


# --------------------------------------------------------------------- work --

def work(case):
    kind = case["kind"]
    if kind == "real":
        pairs = case["N"] ** 2 * min(1.0, 4 / 3 * math.pi * (case["rc"] / case["L"]) ** 3)
        width = 4 if case["mode"] == "force" else 1
        return {"bytes": (32 + 8 * width) * case["N"], "flops": (40 if width == 4 else 30) * pairs}
    if kind == "batch":
        parts = [(s.N, s.M, s.P) for s in _systems(case)]
    else:
        parts = [(case["N"], case["M"], case["P"])]
    force = case["mode"] == "force"
    width, out = 3 if force else 1, 8 if case.get("precision", "fp64") == "fp64" else 4
    nbytes = flops = 0.0
    for N, M, P in parts:
        nbytes += 32.0 * N + out * width * N
        flops += N * P ** 3 * (2.0 + (4.0 if force else 2.0))   # spread, interpolation
        if kind == "steps":
            nbytes += 16.0 * M ** 3   # the field in, the grid out
        else:
            flops += 2 * 2.5 * M ** 3 * math.log2(M ** 3)       # two real transforms
    return {"bytes": nbytes, "flops": flops}


# -------------------------------------------------------------------- exact --

class _Gaussian:
    """The truncated Gaussian window of one system and its sums over the P^3 stencils, in 64 bits."""

    def __init__(self, x, N, M, P, L, xi):
        self.N, self.M, self.P, self.L, self.xi = N, M, P, L, xi
        h = L / M
        m = 0.94 * math.sqrt(math.pi * P)
        self.eta = (2.0 * (P * h / 2) * xi / m) ** 2
        self.c = 2.0 * xi * xi / self.eta
        self.d = (self.c / math.pi) ** 1.5
        self.h = h
        lo = -((P - 1) // 2)
        # (a tensor divisor: a plain number is turned into a multiplication, which may round into the next cell)
        cell = torch.floor(x.view(3, N) / torch.full_like(x[:1], h) + (0.5 if P % 2 else 0.0))
        steps = lo + torch.arange(P, device=x.device)
        u = (x.view(3, N) - cell * h)[..., None] - steps.double() * h
        self.index = (cell.long()[..., None] + steps) % M
        self.weight = torch.exp(-self.c * u * u)
        self.slope = -self.c * u * self.weight

    def chunks(self):
        n = max(1, (1 << 25) // self.P ** 3)
        for a in range(0, self.N, n):
            s = slice(a, a + n)
            ix, iy, iz = (self.index[k, s] for k in range(3))
            at = ((ix[:, :, None, None] * self.M + iy[:, None, :, None]) * self.M + iz[:, None, None, :])
            yield s, at

    def spread(self, q):
        grid = torch.zeros(self.M ** 3, dtype=torch.float64, device=q.device)
        for s, at in self.chunks():
            wx, wy, wz = (self.weight[k, s] for k in range(3))
            v = (q[s] * self.d)[:, None, None, None] * wx[:, :, None, None] * wy[:, None, :, None] * wz[:, None, None, :]
            grid.index_add_(0, at.reshape(-1), v.reshape(-1))
        return grid.view(self.M, self.M, self.M)

    def kspace(self, grid):
        n = torch.arange(self.M, dtype=torch.float64, device=grid.device)
        k2 = (torch.where(n < (self.M + 1) // 2, n, n - self.M) * (2 * math.pi / self.L)) ** 2
        K2 = k2[:, None, None] + k2[None, :, None] + k2[None, None, : self.M // 2 + 1]
        K2[0, 0, 0] = 1.0
        Z = torch.exp(-(1.0 - self.eta) / (4 * self.xi * self.xi) * K2) / K2 * (4 * math.pi)
        Z[0, 0, 0] = 0.0
        return torch.fft.irfftn(torch.fft.rfftn(grid) * Z, s=grid.shape)

    def interpolate(self, field, q, force):
        flat, out = field.reshape(-1), torch.empty(3 if force else 1, self.N, dtype=torch.float64, device=q.device)
        for s, at in self.chunks():
            (wx, wy, wz), (fx, fy, fz) = ([v[k, s] for k in range(3)] for v in (self.weight, self.slope))
            H = flat[at]
            if not force:
                out[0, s] = torch.einsum("nxyz,nx,ny,nz->n", H, wx, wy, wz) * (self.h ** 3 * self.d)
                continue
            scale = self.h ** 3 * self.d * q[s]
            for k, (a, b, c) in enumerate(((fx, wy, wz), (wx, fy, wz), (wx, wy, fz))):
                out[k, s] = torch.einsum("nxyz,nx,ny,nz->n", H, a, b, c) * scale
        return out.reshape(-1)


def _exact_solve(x, q, N, M, P, L, xi, mode):
    g = _Gaussian(x, N, M, P, L, xi)
    return g.interpolate(g.kspace(g.spread(q)), q, mode == "force")


def _exact_real(case, x, q):
    N, L, xi, rc = case["N"], case["L"], case["xi"], case["rc"]
    r, a = x.view(3, N), 2.0 * xi / math.sqrt(math.pi)
    phi, force = -a * q, torch.zeros(3, N, dtype=torch.float64, device=q.device)
    n = max(1, (1 << 26) // N)
    for s in range(0, N, n):
        d = r[:, s:s + n, None] - r[:, None, :]
        d -= L * torch.round(d / L)
        r2 = (d * d).sum(0)
        m, k = torch.nonzero((r2 <= rc * rc) & (r2 > 0), as_tuple=True)
        dist = r2[m, k].sqrt()
        v = q[k] * torch.erfc(xi * dist) / dist
        phi.index_add_(0, m + s, v)
        f = (v + q[k] * a * torch.exp(-(xi * dist) ** 2)) / dist ** 2 * q[m + s]
        for c in range(3):
            force[c].index_add_(0, m + s, f * d[c, m, k])
    return [phi] if case["mode"] != "force" else [phi, force.reshape(-1)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        x, q = _batch_inputs(case, seed)
        out, at = [], 0
        for s in _systems(case):
            out.append(_exact_solve(x[3 * at:3 * (at + s.N)], q[at:at + s.N], s.N, s.M, s.P, s.L, s.xi, case["mode"]))
            at += s.N
        return torch.cat(out)
    if kind == "real":
        return _exact_real(case, *_inputs(case, seed))
    if case["N"] * case["P"] ** 3 > 1e10:   # minutes in plain torch
        return None
    x, q = _inputs(case, seed)
    if kind == "steps":
        g = _Gaussian(x, case["N"], case["M"], case["P"], case["L"], case["xi"])
        # grid_split weights by the charges, wrap gives the column-major periodic grid
        grid = g.spread(q).permute(2, 1, 0).reshape(-1)
        return {"grid": grid, "out": g.interpolate(_field(case, seed), q, case["mode"] == "force")}
    out = _exact_solve(x, q, case["N"], case["M"], case["P"], case["L"], case["xi"], case["mode"])
    return out.cpu().numpy() if kind == "host" else out
