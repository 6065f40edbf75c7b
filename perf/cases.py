"""Performance cases of the stencil and multigrid framework: what its users run, through the
package's public entry points, on seeded synthetic inputs.

A case is a plain dict with a ``kind``:

* ``layers``     the frozen Conv3D / restriction / prolongation layer objects;
* ``twogrid``    the two-grid step of a cycle from the stateless operators: two weighted-Jacobi
                 sweeps, then (even extents) the fused residual + restriction and the fused
                 prolongation + correction + sweep, or (odd extents) the residual;
* ``momentum``   the two stages of the flow solver's momentum update;
* ``sawtooth``   ten cycles of the reference multigrid;
* ``pcg``        float32 conjugate gradients preconditioned by one V-cycle, to 1e-6;
* ``serve``      a stream of requests of mixed sizes through the continuous-batching server
                 (bf16 cycles inside float64 refinement);
* ``ns``         one whole time step of the obstacle-flow stepper;
* ``kolmogorov`` 102 steps of the 2D periodic flow;
* ``tomography`` the misfit and its gradient (forward and adjoint solves).

``exact`` restates each of them in float64 with plain torch.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()
ops, multigrid, serving, ns = pkg.ops, pkg.multigrid, pkg.serving, pkg.ns
kolmogorov, tomography, weights, L = pkg.kolmogorov, pkg.tomography, pkg.weights, pkg._lib

OMEGA = 2.0 / 3.0
STEPS_2D = 102  # two graph replays of 50 steps and two more


def listed():
    return [
        # the smallest calls: the frozen layers on a coarse grid, where launches count
        {"name": "layers_32", "kind": "layers", "B": 1, "Z": 32, "Y": 32, "X": 32},
        # the frozen layers at the reference notebooks' own grid
        {"name": "layers_128", "kind": "layers", "B": 1, "Z": 128, "Y": 128, "X": 128},
        # a ragged batch: odd extents, rows that are no multiple of a vector
        {"name": "smooth_ragged", "kind": "twogrid", "op": "sigma7", "B": 4, "Z": 75, "Y": 90, "X": 101},
        # variable conductivities at the precision workload's grid (float32)
        {"name": "twogrid_sigma_256", "kind": "twogrid", "op": "sigma7", "B": 1, "Z": 256, "Y": 256, "X": 256},
        # the flow solver's 27-point pressure operator on its grid
        {"name": "twogrid_pressure", "kind": "twogrid", "op": "k27", "B": 1, "Z": 64, "Y": 128, "X": 128},
        # the flow solver's momentum update on its grid
        {"name": "momentum_flow", "kind": "momentum", "Z": 64, "Y": 128, "X": 128, "diffusion": "7"},
        # the reference's 128^3 anisotropic run, ten cycles of it
        {"name": "sawtooth_128", "kind": "sawtooth", "op": "const7", "Z": 128, "Y": 128, "X": 128},
        # the plain method: one 64^3 anisotropic potential solve, float32
        {"name": "pcg_64", "kind": "pcg", "slots": 1, "Z": 64, "Y": 64, "X": 64, "log_std": 1.0},
        # the server: requests of all five edges, solved to the precision workload's tolerance
        {"name": "serve_mixed", "kind": "serve", "count": 48},
        # one time step of the obstacle flow
        {"name": "ns_step", "kind": "ns", "Z": 64, "Y": 128, "X": 128, "pressure": "fcycle"},
        # the 2D flow at its configured size
        {"name": "kolmogorov_512", "kind": "kolmogorov", "n": 512, "storage": "f32"},
        # forward and backward of the tomography misfit
        {"name": "tomography_48", "kind": "tomography", "n": 48, "sources": 8, "receivers": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layers", "layers", "twogrid", "twogrid", "twogrid", "momentum", "sawtooth", "pcg",
                       "serve", "ns", "kolmogorov", "tomography"])
    if kind == "layers":
        return {"kind": kind, "B": rng.choice([1, 1, 2, 5]), "Z": _log_int(rng, 16, 128),
                "Y": _log_int(rng, 16, 128), "X": _log_int(rng, 16, 160)}
    if kind == "twogrid":
        op = rng.choice(["sigma7", "sigma7", "k27", "const7"])
        z, y, x = _log_int(rng, 12, 160), _log_int(rng, 12, 160), _log_int(rng, 12, 256)
        if rng.random() < 0.7:  # the grids of a hierarchy are even
            z, y, x = 2 * (z // 2), 2 * (y // 2), rng.choice([2, 4, 8]) * (x // 8) or 2
        return {"kind": kind, "op": op, "B": rng.choice([1, 1, 3]), "Z": z, "Y": y, "X": x}
    if kind == "momentum":
        return {"kind": kind, "Z": _log_int(rng, 16, 64), "Y": _log_int(rng, 24, 128),
                "X": _log_int(rng, 24, 128), "diffusion": rng.choice(["7", "27"])}
    if kind == "sawtooth":
        e = rng.choice([32, 64, 128])
        return {"kind": kind, "op": rng.choice(["const7", "k27"]), "Z": e * rng.choice([1, 1, 2]) if e < 128 else e,
                "Y": e, "X": e}
    if kind == "pcg":
        return {"kind": kind, "slots": rng.choice([1, 2, 3]), "Z": 8 * rng.randint(4, 9), "Y": 8 * rng.randint(4, 9),
                "X": 8 * rng.randint(4, 9), "log_std": round(rng.uniform(0.5, 1.5), 2)}
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(6, 48)}
    if kind == "ns":
        if rng.random() < 0.3:
            return {"kind": kind, "Z": rng.choice([32, 64]), "Y": rng.choice([64, 128]), "X": rng.choice([64, 128]),
                    "pressure": "reference"}
        return {"kind": kind, "Z": rng.choice([32, 48, 64]), "Y": 16 * rng.randint(4, 8), "X": 16 * rng.randint(4, 8),
                "pressure": "fcycle"}
    if kind == "kolmogorov":
        return {"kind": kind, "n": rng.choice([96, 128, 160, 192, 224, 256, 320, 384, 448, 512]),
                "storage": rng.choice(["f32", "bf16"])}
    return {"kind": "tomography", "n": 8 * rng.randint(4, 6), "sources": rng.randint(2, 8),
            "receivers": rng.choice([16, 33, 64])}


# ------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _sigma(shape, seed, log_std):
    """Log-normal conductivities (..., 3, Z, Y, X), smoothed by a 5^3 box filter."""
    g = torch.randn((shape[0] * 3, 1) + tuple(shape[1:]), device="cuda", generator=_gen(seed))
    g = torch.nn.functional.pad(g, (2,) * 6, mode="replicate")
    g = torch.nn.functional.avg_pool3d(g, 5, stride=1)[:, 0]
    g = g - g.mean(dim=(1, 2, 3), keepdim=True)
    g = g / (g.std(dim=(1, 2, 3), keepdim=True) + 1e-30) * log_std
    return torch.exp(g).view((shape[0], 3) + tuple(shape[1:]))


def _dipoles(shape, seed):
    rng = np.random.default_rng(seed)
    f = torch.zeros(shape, device="cuda")
    for b in range(shape[0]):
        p = q = None
        while p == q:
            p, q = (tuple(int(rng.integers(4, n - 4)) for n in shape[1:]) for _ in range(2))
        f[(b,) + p] = 1.0
        f[(b,) + q] = -1.0
    return f


def _twogrid_inputs(c, seed):
    shape = (c["B"], c["Z"], c["Y"], c["X"])
    g = _gen(seed)
    phi = torch.randn(shape, device="cuda", generator=g)
    f = torch.randn(shape, device="cuda", generator=g)
    w = torch.randn((c["B"], c["Z"] // 2, c["Y"] // 2, c["X"] // 2), device="cuda", generator=g)
    sig = _sigma(shape, seed + 1, 1.0).transpose(0, 1).contiguous() if c["op"] == "sigma7" else None
    return phi, f, w, sig


def _requests(c, seed):
    """Backlogged requests, every edge in turn, each with its own conductivities and dipole."""
    rng = np.random.default_rng(seed)
    gen, out = _gen(seed), []
    for i in range(c["count"]):
        n, log_std = serving.EDGES[i % len(serving.EDGES)], float(rng.uniform(0.5, 2.0))
        out.append(serving.SolveRequest(i, n, 0.0, serving.sigma_field(n, gen, log_std, "cuda"),
                                        serving.dipole_field(n, rng, "cuda"), log_std))
    return out


def _even(c):
    return not (c["Z"] | c["Y"] | c["X"]) & 1


def _flow_inputs(c, seed):
    """A sheared flow with eddies: velocities of order one, as the stepper meets them."""
    g = _gen(seed)
    shape = (c["Z"], c["Y"], c["X"])
    e = torch.randn((3, 1) + shape, device="cuda", generator=g)
    e = torch.nn.functional.avg_pool3d(torch.nn.functional.pad(e, (2,) * 6, mode="replicate"), 5, stride=1)[:, 0]
    u, v, w = (2.0 * e[k] for k in range(3))
    return (u + 1.0).contiguous(), v.contiguous(), w.contiguous()


def _flow_kernels(c):
    dt, nu = 0.5, 0.05
    K = ns.laplacian7(dt * nu) if c["diffusion"] == "7" else weights.diffusion27(dt, nu, 1.0)
    return (K,) + weights.advection(dt, 1.0, 1.0)


def _sawtooth_inputs(c, seed):
    """The reference's box of sources, moved and weighted by the seed."""
    shape = (c["Z"], c["Y"], c["X"])
    rng = np.random.default_rng(seed)
    f = pkg.problems.reference_box_source(shape)
    f = np.roll(f, tuple(int(v) for v in rng.integers(-2, 3, 3)), (0, 1, 2)) * np.float32(rng.uniform(0.5, 1.5))
    return torch.from_numpy(np.ascontiguousarray(f)).cuda()


def _tomography_inputs(c, seed):
    survey = tomography.make_survey(n=c["n"], n_src=c["sources"], n_rec=c["receivers"], seed=seed)
    truth = tomography.true_sigma(c["n"], seed=seed)
    u = _solve64(truth.double(), survey.q.double(), 1e-12)
    d_obs = u.view(c["sources"], -1)[:, survey.receivers]
    return survey, d_obs


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = {"case": c}
    if kind == "layers":
        st["x"] = torch.randn((c["B"], c["Z"], c["Y"], c["X"]), device="cuda", generator=_gen(seed))
        st["layers"] = (ops.Conv3DSame(weights.pressure27()), ops.Restriction(), ops.Prolongation())
    elif kind == "twogrid":
        st["phi"], st["f"], st["w"], sig = _twogrid_inputs(c, seed)
        if c["op"] == "sigma7":
            st["op"] = ops.Sigma7(sig[0], sig[1], sig[2])
        elif c["op"] == "k27":
            st["op"] = ops.Stencil27(weights.pressure27())
        else:
            st["op"] = ops.Const7(0.5, 1.0, 2.0)
    elif kind == "momentum":
        st["vel"] = _flow_inputs(c, seed)
        st["K"] = _flow_kernels(c)
        st["b"] = tuple(torch.empty_like(t) for t in st["vel"])
        st["out"] = tuple(torch.empty_like(t) for t in st["vel"])
    elif kind == "sawtooth":
        st["f"] = _sawtooth_inputs(c, seed)
        shape = (c["Z"], c["Y"], c["X"])
        cfg = multigrid.SolverConfig.reference(n_levels=int(math.log2(min(shape))) + 1, cycles=10 ** 9)
        if c["op"] == "const7":
            op = ops.Const7(50.0, 100.0, 200.0)
        else:
            op = ops.Stencil27(weights.pressure27())
        st["mg"] = multigrid.Multigrid(shape, op.kind, cfg, slots=1)
        st["mg"].set_operator(op)
    elif kind == "pcg":
        shape = (c["slots"], c["Z"], c["Y"], c["X"])
        sig = _sigma(shape, seed, c["log_std"]).transpose(0, 1).contiguous()
        st["f"] = _dipoles(shape, seed)
        cfg = multigrid.SolverConfig(cycle="V", accel="cg", tol=1e-6, max_cycles=500)
        st["mg"] = multigrid.Multigrid(shape[1:], L.OP_SIGMA7, cfg, slots=c["slots"])
        st["mg"].set_operator(ops.Sigma7(sig[0], sig[1], sig[2]))
    elif kind == "serve":
        st["requests"] = _requests(c, seed)
        cfg = multigrid.SolverConfig(cycle="V", accel="ir", storage="bf16", tol=1e-10, max_cycles=2000,
                                     inner_tol=1e-3)
        st["server"] = serving.SolveServer(cfg=cfg, slots=64, keep_solutions=True)
    elif kind == "ns":
        cfg = ns.NSConfig(dt=0.5, dx=1.0, Re=0.05, ub=1.0, diffusion="7", pressure=c["pressure"], p_tol=1e-5)
        shape = (c["Z"], c["Y"], c["X"])
        s = st["stepper"] = ns.NSStepper(shape, cfg, sigma=ns.obstacle_mask(shape, seed=seed))
        for _ in range(2):  # the flow round the boxes has begun
            s.step()
        st["fields"] = [t.clone() for t in (s.u, s.v, s.w, s.p)]
    elif kind == "kolmogorov":
        st["flow"] = kolmogorov.KolmogorovFlow(n=c["n"], storage=c["storage"], seed=seed)
    elif kind == "tomography":
        st["survey"], st["d_obs"] = _tomography_inputs(c, seed)
        st["solver"] = tomography.ForwardSolver(c["n"], group=c["sources"], tol=1e-10)
        st["logs"] = torch.zeros((3,) + (c["n"],) * 3, device="cuda")
    else:
        raise ValueError(kind)
    return st


# ------------------------------------------------------------------------------- one pass
def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "layers":
        conv, res, prol = state["layers"]
        y = conv(state["x"])
        r = res(y)
        return y, r, prol(r)
    if kind == "twogrid":
        op, f = state["op"], state["f"]
        phi = ops.jacobi(op, state["phi"], f, omega=OMEGA, sweeps=2)
        if not _even(c):
            return phi, ops.residual(op, phi, f)
        rc = ops.residual_restrict(op, phi, f)
        return phi, rc, ops.prolong_correct_smooth(op, phi, state["w"], f, omega=OMEGA)
    if kind == "momentum":
        vel, b, out = state["vel"], state["b"], state["out"]
        ns.momentum_stage(vel, vel, b, *state["K"], 0.5)
        ns.momentum_stage(b, vel, out, *state["K"], 1.0)
        return b, out
    if kind == "sawtooth":
        mg = state["mg"]
        mg.load(0, state["f"], state["f"])
        mg.run(10)
        return mg.fetch(0)
    if kind == "pcg":
        return state["mg"].solve(state["f"])[0]
    if kind == "serve":
        done = state["server"].serve(state["requests"], realtime=False)
        return [r.phi for r in sorted(done, key=lambda r: r.rid)]
    if kind == "ns":
        s = state["stepper"]  # restored from a checkpoint, then one step
        for a, b in zip((s.u, s.v, s.w, s.p), state["fields"]):
            a.copy_(b)
        s.step()
        return s.u, s.v, s.w, s.p
    if kind == "kolmogorov":
        state["flow"].run(STEPS_2D)
        return state["flow"].u, state["flow"].v, state["flow"].p
    logs = state["logs"].detach().requires_grad_(True)
    J = tomography.misfit(logs, state["survey"], state["d_obs"], state["solver"])
    J.backward()
    return J.detach().float(), logs.grad


# ------------------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; operations of the path's own arithmetic."""
    c, kind = case, case["kind"]
    if kind == "kolmogorov":
        n2 = c["n"] ** 2
        return {"bytes": 4.0 * 6 * n2, "flops": STEPS_2D * n2 * (2 * 40 + 10 + 3 * (4 / 3 * 5 * 12 + 12) + 10)}
    if kind == "tomography":
        n3 = c["n"] ** 3
        return {"bytes": n3 * (4.0 * 3 + 4.0 * c["sources"] + 4.0 * 3), "flops": 2.0 * c["sources"] * n3 * 40 * 150}
    if kind == "serve":
        n3 = c["count"] * sum(e ** 3 for e in serving.EDGES) / len(serving.EDGES)
        return {"bytes": n3 * (4.0 * 4 + 8.0), "flops": n3 * 70 * 150}
    n = float(c["Z"] * c["Y"] * c["X"])
    if kind == "layers":
        n *= c["B"]
        return {"bytes": n * (4 + 4 + 0.5 + 4), "flops": n * (54 + 1)}
    if kind == "twogrid":
        n *= c["B"]
        coef = 12.0 if c["op"] == "sigma7" else 0.0
        per = 54.0 if c["op"] == "k27" else 30.0
        if _even(c):
            return {"bytes": n * (8 + 0.5 + coef + 4 + 0.5 + 4), "flops": 4 * n * per}
        return {"bytes": n * (8 + coef + 8), "flops": 3 * n * per}
    if kind == "momentum":
        return {"bytes": n * 4 * 9, "flops": n * 2 * 3 * (7 + 18 + 18 + 18) * 2}
    if kind == "sawtooth":
        return {"bytes": n * 12, "flops": 10 * n * (3 + 1 / 7) * (54 if c["op"] == "k27" else 16)}
    if kind == "pcg":
        n *= c["slots"]
        return {"bytes": n * 20, "flops": n * 25 * 180}
    return {"bytes": n * 4 * 9, "flops": n * (2 * 3 * 61 * 2 + 20 * 5 * 8 / 7 * 54)}  # ns


# ------------------------------------------------------------------------------- float64
def _pad(x):
    return torch.nn.functional.pad(x, (1,) * 6)


def _conv64(x, K):
    """Cross-correlation with a 3x3x3 kernel, zero padding, float64."""
    K = np.asarray(K, np.float64).reshape(3, 3, 3)
    Z, Y, X = x.shape[-3:]
    p = _pad(x)
    out = torch.zeros_like(x)
    for a in range(3):
        for b in range(3):
            for d in range(3):
                if K[a, b, d]:
                    out += float(K[a, b, d]) * p[..., a:a + Z, b:b + Y, d:d + X]
    return out


def _restrict64(x):
    Z, Y, X = (2 * (n // 2) for n in x.shape[-3:])
    x = x[..., :Z, :Y, :X]
    x = x[..., 0::2, :, :] + x[..., 1::2, :, :]
    x = x[..., 0::2, :] + x[..., 1::2, :]
    return 0.125 * (x[..., 0::2] + x[..., 1::2])


def _prolong64(x):
    return x.repeat_interleave(2, -1).repeat_interleave(2, -2).repeat_interleave(2, -3)


class _Faces64:
    """The 7-point operator from conductivities (sx, sy, sz): face means, wall faces of the
    cell's own conductivity, zero outside."""

    def __init__(self, sx, sy, sz):
        self.f = []
        for s, ax in ((sx, -1), (sy, -2), (sz, -3)):
            n = s.shape[ax]
            self.f.append((ax, torch.cat([s.narrow(ax, 0, 1), 0.5 * (s.narrow(ax, 0, n - 1) + s.narrow(ax, 1, n - 1)),
                                          s.narrow(ax, n - 1, 1)], ax)))
        self.diag = sum(f.narrow(ax, 0, f.shape[ax] - 1) + f.narrow(ax, 1, f.shape[ax] - 1) for ax, f in self.f)

    def apply(self, x):
        out = self.diag * x
        for ax, f in self.f:
            n = x.shape[ax]
            inner = f.narrow(ax, 1, n - 1)
            out.narrow(ax, 0, n - 1).sub_(inner * x.narrow(ax, 1, n - 1))
            out.narrow(ax, 1, n - 1).sub_(inner * x.narrow(ax, 0, n - 1))
        return out


class _Kernel64:
    def __init__(self, K):
        self.K = np.asarray(K, np.float64).reshape(3, 3, 3)
        self.diag = float(self.K[1, 1, 1])

    def apply(self, x):
        return _conv64(x, self.K)


def _const7_kernel(kz, ky, kx):
    K = np.zeros((3, 3, 3))
    K[1, 1, 1] = 2 * (kz + ky + kx)
    K[0, 1, 1] = K[2, 1, 1] = -kz
    K[1, 0, 1] = K[1, 2, 1] = -ky
    K[1, 1, 0] = K[1, 1, 2] = -kx
    return K


def _solve64(sig, f, tol):
    """A(sigma) x = f by diagonally preconditioned conjugate gradients; sig (3, [B,] Z, Y, X),
    f (B, Z, Y, X), all float64."""
    op = _Faces64(sig[0], sig[1], sig[2])
    dot = lambda a, b: (a * b).sum(dim=(-3, -2, -1), keepdim=True)
    x = torch.zeros_like(f)
    r = f.clone()
    z = r / op.diag
    p, rz, stop = z, dot(r, z), dot(f, f) * tol ** 2
    for it in range(20000):
        q = op.apply(p)
        alpha = rz / dot(p, q).clamp_min(1e-300)
        x += alpha * p
        r -= alpha * q
        if it % 16 == 15 and bool((dot(r, r) <= stop).all()):
            break
        z = r / op.diag
        new = dot(r, z)
        p = z + (new / rz.clamp_min(1e-300)) * p
        rz = new
    return x


def _jacobi64(op, phi, f, omega):
    return phi + omega * (f - op.apply(phi)) / op.diag


def _exact_kolmogorov(c, seed):
    n, nu, dt, fk = c["n"], 1.0 / 40.0, 1e-3, 4.0
    h = 2 * math.pi / n
    flow = kolmogorov.KolmogorovFlow(n=n, storage="f32", seed=seed)  # its initial fields alone
    u, v, p = (t.double() for t in (flow.u, flow.v, flow.p))
    sh = lambda a, dy, dx: torch.roll(a, (-dy, -dx), (0, 1))
    lap = lambda a: sh(a, 0, -1) + sh(a, 0, 1) + sh(a, -1, 0) + sh(a, 1, 0) - 4 * a
    ddx = lambda a: (sh(a, 0, 1) - sh(a, 0, -1)) / (2 * h)
    ddy = lambda a: (sh(a, 1, 0) - sh(a, -1, 0)) / (2 * h)
    force = torch.sin(fk * h * torch.arange(n, device="cuda", dtype=torch.float64))[:, None]
    nlev, m = 1, n
    while m // 2 >= 4:
        m, nlev = m // 2, nlev + 1
    d = [4 / h ** 2 * 0.25 ** l for l in range(nlev)]
    A = lambda l, a: -lap(a) * (d[l] / 4)

    def stage(a, b, bu, bv, k):
        ou = bu + k * dt * (nu * lap(a) / h ** 2 - a * ddx(a) - b * ddy(a) + force)
        return ou, bv + k * dt * (nu * lap(b) / h ** 2 - a * ddx(b) - b * ddy(b))

    def cycle(l, f):
        w = 0.8 * f / d[l]
        sweeps = 31 if l == nlev - 1 else 1
        for _ in range(sweeps):
            w = w + 0.8 * (f - A(l, w)) / d[l]
        if l == nlev - 1:
            return w
        r = A(l, w) - f
        r = 0.25 * (r[0::2, 0::2] + r[0::2, 1::2] + r[1::2, 0::2] + r[1::2, 1::2])
        w = w - cycle(l + 1, r).repeat_interleave(2, 0).repeat_interleave(2, 1)
        for _ in range(2):
            w = w + 0.8 * (f - A(l, w)) / d[l]
        return w

    for _ in range(STEPS_2D):
        bu, bv = stage(u, v, u, v, 0.5)
        u1, v1 = stage(bu, bv, u, v, 1.0)
        f = -(ddx(u1) + ddy(v1)) / dt
        for _ in range(3):
            p = p - cycle(0, A(0, p) - f)
        p = p - p.mean()
        u, v = u1 - dt * ddx(p), v1 - dt * ddy(p)
    return u, v, p


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "layers":
        x = torch.randn((c["B"], c["Z"], c["Y"], c["X"]), device="cuda", generator=_gen(seed)).double()
        y = _conv64(x, weights.pressure27())
        r = _restrict64(y)
        return y, r, _prolong64(r)
    if kind == "twogrid":
        phi, f, w, sig = (None if t is None else t.double() for t in _twogrid_inputs(c, seed))
        op = (_Faces64(sig[0], sig[1], sig[2]) if c["op"] == "sigma7" else
              _Kernel64(weights.pressure27() if c["op"] == "k27" else _const7_kernel(0.5, 1.0, 2.0)))
        for _ in range(2):
            phi = _jacobi64(op, phi, f, OMEGA)
        if not _even(c):
            return phi, op.apply(phi) - f
        return phi, _restrict64(op.apply(phi) - f), _jacobi64(op, phi - _prolong64(w), f, OMEGA)
    if kind == "momentum":
        vel = [t.double() for t in _flow_inputs(c, seed)]
        Kd, Kx, Ky, Kz = _flow_kernels(c)
        conv = lambda a, K: _conv64(a, K)
        rhs = lambda g, a: conv(g, Kd) - a[0] * conv(g, Kx) - a[1] * conv(g, Ky) - a[2] * conv(g, Kz)
        b = tuple(g + 0.5 * rhs(g, vel) for g in vel)
        return b, tuple(base + rhs(g, b) for base, g in zip(vel, b))
    if kind == "sawtooth":
        f = _sawtooth_inputs(c, seed).double()
        op = _Kernel64(_const7_kernel(50.0, 100.0, 200.0) if c["op"] == "const7" else weights.pressure27())
        phi = f
        for _ in range(10):
            r = [op.apply(phi) - f]
            while min(r[-1].shape) > 1:
                r.append(_restrict64(r[-1]))
            w = r[-1] / op.diag
            for rl in reversed(r[:-1]):
                w = _jacobi64(op, _prolong64(w), rl, 1.0)
            phi = _jacobi64(op, phi - w, f, 1.0)
        return phi
    if kind == "pcg":
        shape = (c["slots"], c["Z"], c["Y"], c["X"])
        sig = _sigma(shape, seed, c["log_std"]).transpose(0, 1).double()
        return _solve64(sig, _dipoles(shape, seed).double(), 1e-12)
    if kind == "serve":
        out, requests = {}, _requests(c, seed)
        for e in serving.EDGES:
            group = [r for r in requests if r.n == e]
            if group:
                sig = torch.stack([r.sigma.double() for r in group], 1)
                x = _solve64(sig, torch.stack([r.rhs.double() for r in group]), 1e-13)
                out.update({r.rid: x[k] for k, r in enumerate(group)})
        return [out[rid] for rid in sorted(out)]
    if kind == "ns":
        return None  # the pressure is an iterate stopped at its tolerance
    if kind == "kolmogorov":
        return _exact_kolmogorov(c, seed)
    survey, d_obs = _tomography_inputs(c, seed)
    n, S = c["n"], c["sources"]
    one = torch.ones((3, n, n, n), device="cuda", dtype=torch.float64)
    u = _solve64(one, survey.q.double(), 1e-13)
    res = u.view(S, -1)[:, survey.receivers] - d_obs
    back = torch.zeros((S, n ** 3), device="cuda", dtype=torch.float64)
    back[:, survey.receivers] = res
    lam = _solve64(one, back.view(S, n, n, n), 1e-13)
    grad = []
    for ax in (-1, -2, -3):  # sigma_x, sigma_y, sigma_z
        du, dl = (torch.diff(t, dim=ax) for t in (u, lam))
        face = (du * dl).sum(0)
        g = torch.zeros((n, n, n), device="cuda", dtype=torch.float64)
        g.narrow(ax, 0, n - 1).add_(0.5 * face)
        g.narrow(ax, 1, n - 1).add_(0.5 * face)
        wall = (u * lam).sum(0)
        for at in (0, n - 1):
            g.narrow(ax, at, 1).add_(wall.narrow(ax, at, 1))
        grad.append(-g)
    return 0.5 * (res * res).sum(), torch.stack(grad)
