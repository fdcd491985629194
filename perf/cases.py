"""The work a user of this framework gives it, as cases that can be timed and compared.

`listed()` are the standing cases and `draw(rng)` one more of the same ranges.  A case names a kind:

  reconstruct  samples on the host -> context, build, solve, result: what the command line does
  solve        the solve of a system that is already built, and its result read back
  build        new samples into a context and its build: sampling, density, frames, stencils
  sweeps       paired Gauss-Seidel sweeps of one level of a caller's own system (epr_gs)
  operators    energy, gradient and Gauss-Newton product of one level of a caller's own system
  batch        a lockstep batch of small reconstructions, solved from their built systems

Precisions: "fp64" is the library's and the command line's default; "mixed" is the benchmark's
configuration (FP32 relaxation, levels 0-3 in double-float, FP64 energies); "fp32" (sweeps,
operators) is the FP32 relaxation alone.  `radius` is the adaptive indexer's (-1: regular grid).
Results of FP32 relaxation are kept as FP32 values.

Whole mixed-precision solves take inputs without spot outliers: around outliers the schedule ends far
from convergence, and there the last bit of one sweep's rounding shows in the third digit of the
result.  The FP64 solves and the builds take outliers too.
"""
import math

import numpy as np
import torch

import exteriorpoissonrecon_gb300 as epr

MIXED = dict(precision="fp32", fp64_from=0, fp64_levels=4, band_precision="df")


# ---------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------
def _shape(name, a=0.0, b=0.0, sigma=0.0, angle=0.0, spots=0.0):
    return dict(shape=name, a=a, b=b, sigma=sigma, angle=angle, spots=spots)


def listed():
    spots = _shape("link", sigma=0.005, angle=5.0, spots=0.1)
    link = _shape("link", sigma=0.005, angle=5.0)
    knot = _shape("knot", 2.0, 3.0)
    torus = _shape("clifford", sigma=0.002, angle=2.0)
    return [
        # the reference command line's defaults (depth 5, adaptive radius 3, FP64) on a small clean curve
        dict(name="knot5_reconstruct_adaptive_fp64", kind="reconstruct", dim=3, depth=5, samples=4096, radius=3, precision="fp64", **knot),
        # the plain method: a clean curve on the regular grid, FP64, depth 5
        dict(name="knot5_solve_fp64", kind="solve", dim=3, depth=5, samples=4096, radius=-1, precision="fp64", **knot),
        # a noisy scan at a fine depth in the default precision
        dict(name="link7_solve_fp64", kind="solve", dim=3, depth=7, samples=200000, radius=-1, precision="fp64", **spots),
        # the command line with --precision fp32 on a noisy scan (its default indexer)
        dict(name="helix7_reconstruct_adaptive_mixed", kind="reconstruct", dim=3, depth=7, samples=200000, radius=3, precision="mixed",
             **_shape("helix", 4.3, sigma=0.004, angle=5.0)),
        # the benchmark's solve: depth 8, 1M samples, mixed precision
        dict(name="link8_solve_mixed", kind="solve", dim=3, depth=8, samples=1000000, radius=-1, precision="mixed", **link),
        # the same input end to end, from host buffers to the finest grid
        dict(name="link8_reconstruct_mixed", kind="reconstruct", dim=3, depth=8, samples=1000000, radius=-1, precision="mixed", **link),
        # the build alone: new samples into a kept context
        dict(name="link7_build", kind="build", dim=3, depth=7, samples=250000, radius=-1, precision="mixed", **spots),
        # a surface in 4D in the default precision
        dict(name="torus4_solve_fp64", kind="solve", dim=4, depth=4, samples=60000, radius=-1, precision="fp64", **torus),
        # 4D relaxation in FP32: the kernel that carries the depth-6 4D reconstruction, one level down
        dict(name="torus5_sweeps_fp32", kind="sweeps", dim=4, level=5, iters=2, precision="fp32"),
        # 3D relaxation in FP32 by a program that drives its own schedule
        dict(name="grid6_sweeps_fp32", kind="sweeps", dim=3, level=6, iters=4, precision="fp32"),
        # the energy hooks in FP64 (line searches, convergence checks of an outer solver)
        dict(name="grid6_operators_fp64", kind="operators", dim=3, level=6, precision="fp64"),
        # many small inputs at once
        dict(name="batch24_mixed", kind="batch", count=24, lo=5, hi=6, precision="mixed"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_shape(rng, dim, outliers):
    noise = dict(sigma=round(rng.uniform(0.0, 0.008), 4), angle=round(rng.uniform(0.0, 8.0), 2), spots=rng.choice([0.0, 0.05, 0.1]) if outliers else 0.0)
    if dim == 4:
        return _shape("clifford", sigma=round(rng.uniform(0.0, 0.004), 4), angle=round(rng.uniform(0.0, 4.0), 2))
    s = rng.choice(["knot", "link", "helix"])
    if s == "knot":
        p, q = rng.choice([(2, 3), (3, 2), (2, 5), (3, 4), (5, 2)])
        return _shape("knot", float(p), float(q), **noise)
    if s == "helix":
        return _shape("helix", round(rng.uniform(1.0, 6.0), 2), **noise)
    return _shape("link", **noise)


def draw(rng):
    kind = rng.choice(["reconstruct", "reconstruct", "solve", "solve", "build", "sweeps", "operators", "batch"])
    if kind == "sweeps":
        dim = rng.choice([3, 4])
        return dict(kind=kind, dim=dim, level=rng.randint(2, 6) if dim == 3 else rng.randint(2, 4), iters=rng.randint(1, 6),
                    precision=rng.choice(["fp32", "fp64"]))
    if kind == "operators":
        dim = rng.choice([3, 3, 4])
        return dict(kind=kind, dim=dim, level=rng.randint(2, 6) if dim == 3 else rng.randint(2, 4), precision=rng.choice(["fp32", "fp64"]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 32), lo=rng.choice([4, 5]), hi=rng.choice([5, 6]), precision="mixed")
    if rng.random() < 0.2:
        return dict(kind=kind, dim=4, depth=3, samples=_log_uniform(rng, 5000, 100000), radius=rng.choice([-1, 1]), precision="fp64",
                    **_draw_shape(rng, 4, False))
    depth, precision = rng.randint(4, 7), rng.choice(["fp64", "mixed"])
    return dict(kind=kind, dim=3, depth=depth, samples=_log_uniform(rng, 1000 << (depth - 3), 8000 << (depth - 2)), radius=rng.choice([-1, -1, 3, 1]),
                precision=precision, **_draw_shape(rng, 3, kind == "build" or precision == "fp64"))


# ---------------------------------------------------------------------------------------------
# what a user's program has in hand
# ---------------------------------------------------------------------------------------------
def _sampler(c, seed):
    return epr.sampler(c["shape"], c["a"], c["b"], pos_sigma=c["sigma"], angle_deg=c["angle"], spot_frac=c["spots"], seed=seed)


def _solver(c):
    return dict(MIXED if c["precision"] == "mixed" else {}, aRadius=c["radius"])


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        rng = np.random.default_rng(seed)
        recons = []
        for k in range(c["count"]):
            depth = c["lo"] + k % (c["hi"] - c["lo"] + 1)
            s = dict(sigma=float(rng.uniform(0.0, 0.008)), angle=float(rng.uniform(0.0, 8.0)))
            shape = _shape("knot", 2.0, 3.0, **s) if k % 2 else _shape("helix", float(rng.uniform(1.0, 5.0)), **s)
            r = epr.Reconstructor(3, depth, build=False, **MIXED)
            r.set_generated_samples(_sampler(shape, seed * 64 + k), int(math.exp(rng.uniform(math.log(2000), math.log(64000)))))
            recons.append(r)
        batch = epr.LockstepBatch(recons)
        batch.run(build=True)
        return dict(case=c, batch=batch)
    if kind in ("sweeps", "operators"):
        R, B, const, x, y = (v.cpu().numpy() if torch.is_tensor(v) else v for v in _system(c["dim"], c["level"], seed))
        r = epr.Reconstructor(c["dim"], c["level"], build=False, precision=c["precision"])
        r.set_level_system(c["level"], R, B, const)
        st = dict(case=c, r=r, x=x, y=y)
        if kind == "operators":
            st["dx"], st["dy"] = (v.cpu().numpy() for v in _fields(c["dim"], c["level"], seed + 1))
        return st
    if kind == "solve":
        r = epr.Reconstructor(c["dim"], c["depth"], build=False, **_solver(c))
        r.set_generated_samples(_sampler(c, seed), c["samples"])
        r.build()
        return dict(case=c, r=r)
    pos, skew = epr.generate_samples(_sampler(c, seed), c["samples"])
    pos, _ = epr.unit_cube(pos)
    st = dict(case=c, pos=pos, skew=skew)
    if kind == "build":
        st["r"] = epr.Reconstructor(c["dim"], c["depth"], build=False, **_solver(c))
    return st


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _result(r, c):
    """The solve's result: in FP64 every level's hierarchical coefficients (Reconstructor::x, y), of
    FP32 relaxation the finest grid's coefficients, kept as FP32 values."""
    if c["precision"] == "fp64":
        return r.solution()
    return [v.astype(np.float32) for v in r.coefficients(r.depth)]


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "reconstruct":
        r = epr.Reconstructor(c["dim"], c["depth"], state["pos"], state["skew"], **_solver(c))
        r.solve()
        out = _result(r, c)
        r.close()
        return out
    if kind == "solve":
        state["r"].solve()
        return _result(state["r"], c)
    if kind == "build":
        r = state["r"]
        r.set_samples(state["pos"], state["skew"])
        r.build()
        coarse = min(c["depth"] - 1, 4 if c["dim"] == 3 else 2)
        return {"c": r.get("c"), "frames": r.get("S"), "measure": r.get("measure"), "noise": r.get("noise"), "depth": r.get("depth"),
                "R": r.get("R", coarse), "B": r.get("B", coarse)}
    if kind == "sweeps":
        out = state["r"].gs(c["level"], state["x"], state["y"], c["iters"])
        return [v.astype(np.float32) for v in out] if c["precision"] == "fp32" else out
    if kind == "operators":
        r, l = state["r"], c["level"]
        e = r.energy(l, state["x"], state["y"])
        out = [e, *r.gradient(l), *r.gn_matvec(l, state["dx"], state["dy"])]
        return [e] + [v.astype(np.float32) for v in out[1:]] if c["precision"] == "fp32" else out
    state["batch"].run()
    return [[v.astype(np.float32) for v in r.coefficients(r.depth)] for r in state["batch"].recons]


# ---------------------------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _nodes(dim, level):
    return (2 ** level + 1) ** dim


def _update_flops(dim):
    """A node's quadratic model: the 2^dim incident elements' five wedge integrals (28 x 6 products in
    3D through the 21 minors of the corner differences, 105 minors in 4D) and its stencil columns."""
    return 2 ** dim * (450 if dim == 3 else 4200) + 8 * 3 ** dim


def _solve_work(dim, depth, samples, real):
    sweeps = [math.ceil(2.0 ** (depth - l) * 10) for l in range(depth + 1)]
    flops = sum(s * _nodes(dim, l) for l, s in enumerate(sweeps)) * _update_flops(dim)
    read = sum(_nodes(dim, l) for l in range(depth + 1)) * 2 * 3 ** dim * real
    return read + 16 * _nodes(dim, depth), flops


def work(case):
    c, kind = case, case["kind"]
    real = 8 if c["precision"] == "fp64" else 4
    if kind == "batch":
        b, f = (v * c["count"] for v in _solve_work(3, (c["lo"] + c["hi"]) // 2, 0, real))
        return {"bytes": b, "flops": f}
    if kind in ("sweeps", "operators"):
        n = _nodes(c["dim"], c["level"])
        if kind == "sweeps":
            return {"bytes": n * (2 * 3 ** c["dim"] * real + 32), "flops": n * c["iters"] * _update_flops(c["dim"])}
        return {"bytes": n * (2 * 3 ** c["dim"] * real + 64), "flops": n * 3 * _update_flops(c["dim"]) // 2}
    n, d = _nodes(c["dim"], c["depth"]), c["dim"]
    in_bytes = c["samples"] * 8 * (d + d * (d - 1) // 2)
    # build: samples in, the frame field and the two stencils of every level out
    stencils = sum(_nodes(d, l) for l in range(c["depth"] + 1)) * 2 * 3 ** d * 8
    build = (in_bytes + stencils + n * 8 * d * (d - 1) // 2, n * 2 * 3 ** d * 3 ** d // 2)
    if kind == "build":
        return {"bytes": build[0], "flops": build[1]}
    b, f = _solve_work(d, c["depth"], c["samples"], real)
    if kind == "reconstruct":
        b, f = b + build[0], f + build[1]
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------------
# a caller's own system on one level, and the operators on it in 64 bits
# ---------------------------------------------------------------------------------------------
DEV = "cuda" if torch.cuda.is_available() else "cpu"
D_WEIGHT = 0.00625  # the library's default Dirichlet weight


def _corner_bits(dim):
    return torch.tensor([[(k >> (dim - 1 - d)) & 1 for d in range(dim)] for k in range(2 ** dim)], device=DEV)


def _hat_and_slopes(dim, pts):
    """Hat functions of the unit element's corners at pts (n x dim) and their derivatives (n x dim x corners)."""
    bits = _corner_bits(dim)
    f = [torch.where(bits[:, d] > 0, pts[:, d:d + 1], 1 - pts[:, d:d + 1]) for d in range(dim)]
    s = [torch.where(bits[:, d] > 0, 1.0, -1.0).to(pts).expand_as(f[d]) for d in range(dim)]
    hat = torch.stack(f).prod(0)
    slopes = torch.stack([torch.stack([s[k] if k == d else f[k] for k in range(dim)]).prod(0) for d in range(dim)], 1)
    return hat, slopes


def _gauss(dim):
    """3-point Gauss rule on every axis of the unit element: points (3^dim x dim), weights."""
    p = torch.tensor([0.5 - math.sqrt(0.15), 0.5, 0.5 + math.sqrt(0.15)], dtype=torch.float64, device=DEV)
    w = torch.tensor([5 / 18, 8 / 18, 5 / 18], dtype=torch.float64, device=DEV)
    idx = torch.cartesian_prod(*[torch.arange(3, device=DEV)] * dim)
    return p[idx], w[idx].prod(1)


def _fields(dim, level, seed):
    """Smooth (x, y) with a little noise, as the schedule's prolonged iterates are."""
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    n = 2 ** level + 1
    axes = torch.meshgrid(*[torch.linspace(0, 1, n, dtype=torch.float64, device=DEV)] * dim, indexing="ij")
    out = []
    for _ in range(2):
        v = 0.01 * (torch.rand(n ** dim, generator=g, dtype=torch.float64).to(DEV).reshape([n] * dim) - 0.5)
        for _ in range(3):
            k = torch.randint(-2, 3, (dim,), generator=g)
            ph, a = 2 * math.pi * float(torch.rand(1, generator=g)), 0.1 + 0.2 * float(torch.rand(1, generator=g))
            v = v + a * torch.sin(ph + math.pi * sum(float(k[d]) * axes[d] for d in range(dim)))
        out.append(v.reshape(-1))
    return out


def _scatter(n, index, values):
    """Sums of values by index, in one order (on the host: sums on the GPU come in any order)."""
    out = torch.zeros(n, dtype=torch.float64)
    return out.index_add_(0, index.reshape(-1).cpu(), values.reshape(-1).cpu()).to(DEV)


def _system(dim, level, seed):
    """Column stencils of a screening term of samples along a random closed curve (R, weight 100) and
    of a frame term of random frames in the elements they fall into (B), the constant c, and (x, y)."""
    g = torch.Generator(device="cpu").manual_seed(int(seed) + 7)
    r, S = 2 ** level, 3 ** dim
    n1 = r + 1
    bits = _corner_bits(dim)
    m = 64 * r
    t = 2 * math.pi * torch.rand(m, generator=g, dtype=torch.float64)
    a = torch.randn(2, 2, dim, generator=g, dtype=torch.float64) / torch.tensor([1.0, 2.0], dtype=torch.float64)[:, None, None]
    pos = sum(torch.cos((k + 1) * t)[:, None] * a[k, 0] + torch.sin((k + 1) * t)[:, None] * a[k, 1] for k in range(2))
    pos = (0.5 + 0.4 * pos / pos.abs().max()).to(DEV)
    cell = (pos * r).floor().clamp(0, r - 1).long()
    stride = torch.tensor([n1 ** (dim - 1 - d) for d in range(dim)], device=DEV)
    three = torch.tensor([3 ** (dim - 1 - d) for d in range(dim)], device=DEV)
    node = (cell[:, None, :] + bits[None]).mul(stride).sum(-1)                       # samples x corners
    off = ((bits[None, :, :] - bits[:, None, :] + 1) * three).sum(-1)                # [a, b]: offset of b from a
    hat, _ = _hat_and_slopes(dim, pos * r - cell)
    R = _scatter(n1 ** dim * S, node[:, :, None] * S + off[None], 100.0 / m * hat[:, :, None] * hat[:, None, :])
    # frames: one per occupied element
    occ = torch.unique(cell, dim=0)
    frame = torch.randn(dim, dim, generator=g, dtype=torch.float64).to(DEV) + 0.3 * torch.randn(
        occ.shape[0], dim, dim, generator=g, dtype=torch.float64).to(DEV)
    frame = 20.0 * (frame - frame.transpose(1, 2))
    pts, w = _gauss(dim)
    _, sl = _hat_and_slopes(dim, pts)
    mix = torch.einsum("p,pxa,pyb->xyab", w, sl, sl) * float(r) ** (2 - dim)         # int d_x phi_a d_y phi_b
    el = torch.einsum("exy,xyab->eab", frame, mix)                                   # antisymmetric in (a, b)
    enode = (occ[:, None, :] + bits[None]).mul(stride).sum(-1)
    B = _scatter(n1 ** dim * S, enode[:, :, None] * S + off[None], el)
    const = float((frame ** 2).sum()) / r ** dim
    return (R.reshape(-1, S), B.reshape(-1, S), const, *_fields(dim, level, seed))


def _dirichlet(dim, level):
    """Column stencil of int grad phi_i . grad phi_j on the level's grid (N x 3^dim)."""
    r = 2 ** level
    h = 1.0 / r
    mass = torch.zeros(r + 1, 3, dtype=torch.float64, device=DEV)
    stiff = torch.zeros_like(mass)
    for o, (mv, sv) in enumerate([(h / 6, -1 / h), (2 * h / 3, 2 / h), (h / 6, -1 / h)]):
        mass[:, o], stiff[:, o] = mv, sv
    for row, gone in ((0, 0), (r, 2)):
        mass[row, 1], stiff[row, 1] = h / 3, 1 / h
        mass[row, gone] = stiff[row, gone] = 0
    total = 0
    for k in range(dim):
        v = torch.ones(1, 1, dtype=torch.float64, device=DEV)
        for d in range(dim):
            f = stiff if d == k else mass
            v = torch.einsum("ns,mt->nmst", v, f).reshape(v.shape[0] * f.shape[0], v.shape[1] * 3)
        total = total + v
    return total


class _Level:
    """The energy of one level in 64 bits: wedge integrals by a 3^dim-point Gauss rule per element."""

    def __init__(self, dim, level, R, B):
        self.dim, self.r, self.n = dim, 2 ** level, 2 ** level + 1
        self.A, self.B = R + D_WEIGHT * _dirichlet(dim, level), B
        self.pts, self.w = _gauss(dim)
        _, self.sl = _hat_and_slopes(dim, self.pts)
        self.scale = (float(self.r) if dim == 3 else 1.0) * 0.5
        self.axes = [(p, q) for p in range(dim) for q in range(p)]
        self.stride = torch.tensor([self.n ** (dim - 1 - d) for d in range(dim)], device=DEV)
        self.offs = torch.cartesian_prod(*[torch.tensor([-1, 0, 1], device=DEV)] * dim)

    def _slopes(self, f, corners):
        return torch.einsum("pdc,mc->pdm", self.sl, f[corners])

    def wedge_sums(self, nodes, x, y, dx=None, dy=None):
        """Sums over the elements at `nodes` (m x dim): (|U|^2, |V|^2, <U,V>, <Z,U>, <Z,V>) with U, V the
        derivatives of W(x, y) along the node's x and y and Z = W(x, y), or W(dx, y) + W(x, dy)."""
        tot = torch.zeros(5, nodes.shape[0], dtype=torch.float64, device=DEV)
        bits = _corner_bits(self.dim)
        for mirror in bits:
            el = nodes - mirror
            sel = ((el >= 0) & (el < self.r)).all(1).nonzero()[:, 0]
            if not sel.numel():
                continue
            for at in sel.split(max(1, 40_000_000 // (3 ** self.dim * self.dim * 4))):
                corners = ((el[at, None, :] + bits[None]) * self.stride).sum(-1)
                me = int((mirror * torch.tensor([1 << (self.dim - 1 - d) for d in range(self.dim)], device=DEV)).sum())
                ph = self.sl[:, :, me:me + 1]
                X, Y = self._slopes(x, corners), self._slopes(y, corners)
                if dx is not None:
                    DX, DY = self._slopes(dx, corners), self._slopes(dy, corners)
                for p, q in self.axes:
                    U = Y[:, p] * ph[:, q] - ph[:, p] * Y[:, q]
                    V = ph[:, p] * X[:, q] - X[:, p] * ph[:, q]
                    if dx is None:
                        Z = Y[:, p] * X[:, q] - X[:, p] * Y[:, q]
                    else:
                        Z = Y[:, p] * DX[:, q] - DX[:, p] * Y[:, q] + DY[:, p] * X[:, q] - X[:, p] * DY[:, q]
                    for k, v in enumerate((U * U, V * V, U * V, Z * U, Z * V)):
                        tot[k, at] += torch.einsum("p,pm->m", self.w, v)
        return tot * self.scale

    def column(self, M, nodes, f, centre=True):
        i = (nodes * self.stride).sum(1)
        s = torch.zeros(nodes.shape[0], dtype=torch.float64, device=DEV)
        for o, off in enumerate(self.offs):
            if not centre and not off.any():
                continue
            q = nodes + off
            ok = ((q >= 0) & (q < self.n)).all(1)
            s += torch.where(ok, M[i, o] * f[(q.clamp(0, self.n - 1) * self.stride).sum(1)], torch.zeros_like(s))
        return s

    def model(self, nodes, x, y):
        """(Q20, Q02, Q11, Q10, Q01) of E(x + s e_i, y + t e_i)."""
        h = self.wedge_sums(nodes, x, y)
        a = self.A[(nodes * self.stride).sum(1), 3 ** self.dim // 2]
        ax, ay = self.column(self.A, nodes, x), self.column(self.A, nodes, y)
        bx, by = self.column(self.B, nodes, x, False), self.column(self.B, nodes, y, False)
        return h[0] + a, h[1] + a, 2 * h[2], 2 * h[3] + 2 * ax - 2 * by, 2 * h[4] + 2 * ay + 2 * bx

    def nodes(self, colour=None):
        ax = [torch.arange(self.n, device=DEV) if colour is None else torch.arange((colour >> d) & 1, self.n, 2, device=DEV)
              for d in range(self.dim)]
        return torch.cartesian_prod(*ax)

    def sweep(self, x, y):
        x, y = x.clone(), y.clone()
        for colour in range(2 ** self.dim):
            nodes = self.nodes(colour)
            q20, q02, h01, g0, g1 = self.model(nodes, x, y)
            h00, h11 = 2 * q20, 2 * q02
            det = h00 * h11 - h01 * h01
            i = (nodes * self.stride).sum(1)
            ok = det.abs() > 1e-20
            x[i] += torch.where(ok, -(h11 * g0 - h01 * g1) / det / 2, torch.zeros_like(det))
            y[i] += torch.where(ok, -(h00 * g1 - h01 * g0) / det / 2, torch.zeros_like(det))
        return x, y

    def energy(self, x, y, const):
        e = torch.zeros((), dtype=torch.float64, device=DEV)
        el = torch.cartesian_prod(*[torch.arange(self.r, device=DEV)] * self.dim)
        for at in el.split(max(1, 40_000_000 // (3 ** self.dim * self.dim * 4))):
            corners = ((at[:, None, :] + _corner_bits(self.dim)[None]) * self.stride).sum(-1)
            X, Y = self._slopes(x, corners), self._slopes(y, corners)
            for p, q in self.axes:
                e += torch.einsum("p,pm->", self.w, (Y[:, p] * X[:, q] - X[:, p] * Y[:, q]) ** 2)
        nodes = self.nodes()
        quad = (x * self.column(self.A, nodes, x) + y * self.column(self.A, nodes, y)).sum()
        frame = (x * self.column(self.B, nodes, y)).sum()
        wedge = float(e) * self.scale
        return [wedge - 2 * float(frame) + const, float(quad), wedge]


def exact(case, seed):
    """What run() returns for a caller's own system, in 64 bits; whole solves and builds have no such value."""
    c = case
    if c["kind"] not in ("sweeps", "operators"):
        return None
    R, B, const, x, y = _system(c["dim"], c["level"], seed)
    lv = _Level(c["dim"], c["level"], R, B)
    if c["kind"] == "sweeps":
        for _ in range(c["iters"]):
            x, y = lv.sweep(x, y)
        return [x.cpu().numpy(), y.cpu().numpy()]
    dx, dy = _fields(c["dim"], c["level"], seed + 1)
    nodes = lv.nodes()
    q = lv.model(nodes, x, y)
    h = lv.wedge_sums(nodes, x, y, dx, dy)
    gn = [h[3] + lv.column(lv.A, nodes, dx), h[4] + lv.column(lv.A, nodes, dy)]
    return [np.array(lv.energy(x, y, const)), q[3].cpu().numpy(), q[4].cpu().numpy(), gn[0].cpu().numpy(), gn[1].cpu().numpy()]
