"""What a program built on this framework has it do, as cases that can be timed.

Each case is one call (or the few calls that belong together) through the
public entry points, with everything a program keeps between calls made in
``prepare``: the context or batch, the device buffers, the charges.

The charges are those of the framework's workloads: rigid neutral three-site
molecules (-0.834, +0.417, +0.417; 0.9572 A, 104.52 degrees) with uniform
centres and orientations at the density of water, and the two unit charges of
the pair test.  Boxes follow the named configurations (pair L 20 / M 20, water
23,559 / L 62.23 / M 64, 48,000 / L 78.4 / M 80, 262,143 / L 140 / M 144, the
256 uneven systems), a larger box of the same density, and an orthorhombic box
whose sides are not multiples of 16.

Programs on the mixed form hold their coordinates in FP32 and integrate or
train in FP32, so they take the energies, forces and gradients that the
library hands over in double arrays on in that type; ``run`` does the same.
Programs on the FP64 form keep the doubles.

``exact`` is the same mathematics in 64-bit PyTorch, without this
repository's code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

CCELEC = 332.0716
KAPPA = 0.4
LAMBDA = 3.0
DENSITY = 0.0978  # charges per cubic Angstrom


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def _box(kind, name, precision, n, m, length, sigma=2.0):
    if isinstance(m, int):
        m = (m, m, m)
    if not isinstance(length, tuple):
        length = (length, length, length)
    c = {"kind": kind, "precision": precision, "n": n, "mx": m[0], "my": m[1], "mz": m[2],
         "lx": length[0], "ly": length[1], "lz": length[2], "sigma": sigma}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call there is: two charges, FP64, as the pair test runs
        # them; launches and latency
        _box("forward", "pair_fp64", "fp64", 2, 20, 20.0, 2.121320344),
        # MD steps (energy and forces of the current positions, on the device):
        # a small protein-sized box, the headline box, and a large one
        _box("forward", "md_23k_mixed", "mixed", 23559, 64, 62.23),
        _box("forward", "md_262k_mixed", "mixed", 262143, 144, 140.0),
        _box("forward", "md_639k_mixed", "mixed", 639000, 192, 186.9),
        # the plain FP64 form of the headline box: reference forces
        _box("forward", "md_262k_fp64", "fp64", 262143, 144, 140.0),
        # a caller written against the reference's classes: host arrays, the
        # four calls one after the other, FP64 (the 48k box of its own driver)
        _box("classes", "classes_48k_fp64", "fp64", 48192, 80, 80.0, 2.1213),
        # constant-pressure MD in an orthorhombic box with sides that are not
        # multiples of 16: energy, forces and virial
        _box("pressure", "npt_90k_mixed", "mixed", 90210, (100, 90, 108), (97.5, 89.1, 106.2)),
        # training through the differentiable op: forward, loss, backward
        _box("train", "train_48k_mixed", "mixed", 48000, 80, 78.4),
        # the FP64 gradient a mixed-form program is checked against
        _box("gradient", "gradient_23k_fp64", "fp64", 23559, 64, 62.23),
        # 256 uneven systems, forward and reverse pass in one captured graph
        {"name": "batch_256_mixed", "kind": "batch", "precision": "mixed", "systems": 256,
         "n_min": 501, "n_max": 8001, "sigma": 2.0},
        # grid operations of the real-space variant on a 144^3 grid: on-grid
        # Gaussian spreading, field, dipole
        _box("grid", "grid_144_mixed", "mixed", 0, 144, 140.0),
        # the accuracy check of a box: the whole Ewald sum, host arrays
        _box("ewald", "ewald_23k_fp64", "fp64", 23559, 64, 62.23),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "forward", "classes", "pressure", "train",
                       "gradient", "batch", "grid", "ewald"])
    if kind == "batch":
        n_min = int(_log_uniform(rng, 300, 2000))
        return {"kind": "batch", "precision": "mixed", "systems": int(_log_uniform(rng, 8, 256)),
                "n_min": n_min, "n_max": int(n_min * rng.uniform(1.5, 4.0)), "sigma": 2.0}
    precision = {"forward": rng.choice(["mixed", "mixed", "fp64"]), "classes": "fp64",
                 "pressure": "mixed", "train": "mixed", "gradient": "fp64",
                 "grid": rng.choice(["mixed", "fp64"]), "ewald": "fp64"}[kind]
    top = {"forward": 192 if precision == "mixed" else 144, "classes": 80, "pressure": 144,
           "train": 96, "gradient": 64, "grid": 144, "ewald": 60}[kind]
    m = int(_log_uniform(rng, 20, top))
    if rng.random() < 0.5:  # sides that a program picks for the transform
        m = max(16, 16 * round(m / 16)) if rng.random() < 0.5 else m + m % 2
    m = (m, m, m)
    if kind == "pressure" or rng.random() < 0.3:
        m = tuple(min(top, max(20, int(v * rng.uniform(0.8, 1.2)))) for v in m)
    h = rng.uniform(0.9, 1.25)
    length = tuple(round(v * h, 3) for v in m)
    n = int(DENSITY * length[0] * length[1] * length[2] * rng.uniform(0.5, 1.0))
    n = 0 if kind == "grid" else min(n, {"ewald": 20000, "gradient": 23559}.get(kind, 639000))
    return _box(kind, None, precision, n, m, length)


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _boxes(c):
    return (c["mx"], c["my"], c["mz"]), (c["lx"], c["ly"], c["lz"])


def _molecules(rng, k, box):
    """k molecules with centres uniform in the box (3,) or (k, 3): (3k, 4) float32."""
    def unit(v):
        return v / np.linalg.norm(v, axis=1, keepdims=True)

    centre = rng.uniform(0.0, 1.0, (k, 3)) * np.asarray(box)
    a = unit(rng.standard_normal((k, 3)))
    b = rng.standard_normal((k, 3))
    b = unit(b - (a * b).sum(1, keepdims=True) * a)
    half = math.radians(104.52) / 2
    out = np.empty((k, 3, 4), dtype=np.float32)
    out[:, 0, :3] = centre
    out[:, 1, :3] = centre + 0.9572 * (math.cos(half) * a + math.sin(half) * b)
    out[:, 2, :3] = centre + 0.9572 * (math.cos(half) * a - math.sin(half) * b)
    out[:, 0, 3] = -0.834
    out[:, 1:, 3] = 0.417
    return out.reshape(-1, 4)


def _charges(c, seed):
    """(n, 4) host array in the case's type (FP32 values, widened for FP64)."""
    rng = np.random.default_rng(seed)
    n = c["n"]
    if n == 2:  # charges -1 (centre) and +1 at distance 1 along a random direction
        u = rng.standard_normal(3)
        x = np.zeros((2, 4), dtype=np.float64)
        x[0] = (c["lx"] / 2, c["ly"] / 2, c["lz"] / 2, -1.0)
        x[1, :3] = x[0, :3] + u / np.linalg.norm(u)
        x[1, 3] = 1.0
    else:
        x = _molecules(rng, (n + 2) // 3, (c["lx"], c["ly"], c["lz"]))[:n]
    return np.ascontiguousarray(x, dtype=np.float64 if c["precision"] == "fp64" else np.float32)


def _systems(c, seed):
    """Sizes, boxes and charges of an uneven batch: charges log-uniform, boxes at
    the density of water, grid sides the nearest multiple of 8 to the box."""
    size = np.random.default_rng(12345 + c["systems"])  # sizes belong to the case, not to the seed
    k = np.maximum(1, np.rint(np.exp(size.uniform(math.log(c["n_min"]), math.log(c["n_max"]),
                                                  c["systems"])) / 3)).astype(np.int64)
    length = np.cbrt(3 * k / DENSITY)
    m = np.maximum(16, 8 * np.rint(length / 8)).astype(np.int64)
    x = _molecules(np.random.default_rng(seed), int(k.sum()), np.repeat(length, k)[:, None])
    return [{"size": (int(v),) * 3, "box": (float(l),) * 3, "n": int(3 * j)}
            for v, l, j in zip(m, length, k)], x


def _upstream(n, seed):
    return np.random.default_rng([seed, 7]).standard_normal((3, n))


def _targets(c, seed):
    """What a training program fits: forces per charge and energy per charge."""
    rng = np.random.default_rng([seed, 9])
    return rng.standard_normal((c["n"], 3)).astype(np.float32), np.float32(rng.standard_normal())


def _grids(c, seed):
    """A charge density and a potential on the grid, in the case's type."""
    rng = np.random.default_rng(seed)
    t = np.float64 if c["precision"] == "fp64" else np.float32
    shape = (c["mz"], c["my"], c["mx"])
    return (rng.standard_normal(shape, dtype=np.float32).astype(t),
            rng.standard_normal(shape, dtype=np.float32).astype(t))


def _context(c):
    from gse_b200.gse import Context
    m, length = _boxes(c)
    return Context(*m, sigma=c["sigma"], kappa=KAPPA, lambdaSigma=LAMBDA, lambdaSigma1=LAMBDA,
                   boxx=length[0], boxy=length[1], boxz=length[2], ccelec=CCELEC,
                   precision=c["precision"])


def prepare(case, seed):
    c = case
    s = {"case": c}
    kind = c["kind"]
    if kind in ("forward", "pressure", "gradient"):
        n = c["n"]
        s["ctx"] = _context(c)
        s["x"] = torch.from_numpy(_charges(c, seed)).cuda()
        s["f"] = torch.empty(3, n, dtype=torch.float64, device="cuda")
        s["e"] = torch.empty(1, dtype=torch.float64, device="cuda")
        s["v"] = torch.empty(6, dtype=torch.float64, device="cuda")
        if kind == "gradient":
            s["g"] = torch.from_numpy(_upstream(n, seed)).cuda()
            s["d"] = torch.empty(4, n, dtype=torch.float64, device="cuda")
    elif kind == "classes":
        from gse_b200.gse import CpuGSEk
        m, length = _boxes(c)
        s["gse"] = CpuGSEk(*m, c["sigma"], KAPPA, LAMBDA, LAMBDA, *length, ccelec=CCELEC,
                           precision=c["precision"])
        s["x"] = _charges(c, seed)
        s["f"] = [np.zeros(c["n"]) for _ in range(3)]
    elif kind == "train":
        s["ctx"] = _context(c)
        x = _charges(c, seed)
        s["pos"] = torch.from_numpy(x[:, :3].copy()).cuda().requires_grad_()
        s["q"] = torch.from_numpy(x[:, 3].copy()).cuda().requires_grad_()
        f, e = _targets(c, seed)
        s["f"], s["e"] = torch.from_numpy(f).cuda(), torch.tensor(e, device="cuda")
    elif kind == "batch":
        from gse_b200.gse import Batch
        systems, x = _systems(c, seed)
        b = Batch(systems, sigma=c["sigma"], kappa=KAPPA, lambdaSigma1=LAMBDA, ccelec=CCELEC)
        s["batch"], s["buf"] = b, b.buffers()
        s["buf"]["xyzq"].copy_(torch.from_numpy(x))
        s["buf"]["dLdE"].fill_(1.0)
        s["buf"]["grad_forces"].copy_(torch.from_numpy(_upstream(x.shape[0], seed)))
        torch.cuda.synchronize()
        b.capture(with_adjoint=True)
    elif kind == "grid":
        s["ctx"] = _context(c)
        s["rho"], s["phi"] = (torch.from_numpy(a).cuda() for a in _grids(c, seed))
        s["out"] = [torch.empty_like(s["rho"]) for _ in range(4)]
        s["dip"] = torch.empty(3, dtype=torch.float64, device="cuda")
        s["sigma2"], s["rcut2"] = _second_spread(c)
    elif kind == "ewald":
        from gse_b200 import gse, workloads
        s["x"] = _charges(c, seed)
        s["box"] = _boxes(c)[1]
        s["kcut"] = gse.ewald_kcut(c["sigma"], s["box"])
        s["excl"] = workloads.triplet_exclusions(c["n"])
    else:
        raise ValueError(kind)
    return s


def _second_spread(c):
    """Width and cut-off of the real-space variant's second spreading."""
    sigma2 = c["sigma"] * math.sqrt(1.0 - 2.0 * KAPPA)
    return sigma2, LAMBDA * math.sqrt(2.0) * sigma2


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def run(state):
    s = state
    c = s["case"]
    kind, n = c["kind"], c.get("n", 0)
    if kind in ("forward", "pressure"):
        ctx, f = s["ctx"], s["f"]
        ctx.forward(n, s["x"], f[0], f[1], f[2], energy_out=s["e"])
        out = [s["e"], f]
        if kind == "pressure":
            out.append(ctx.virial(out=s["v"]))
        return out if c["precision"] == "fp64" else [t.float() for t in out]
    if kind == "gradient":
        g, d = s["g"], s["d"]
        s["ctx"].adjoint(n, s["x"], 1.0, g[0], g[1], g[2], d[0], d[1], d[2], d[3])
        return d
    if kind == "classes":
        gse, f = s["gse"], s["f"]
        gse.spreadCharge1(n, s["x"])
        gse.solvePoisson()
        e = gse.calculateEnergy()
        gse.interpolateForce(n, s["x"], f[0], f[1], f[2])
        return [e] + f
    if kind == "train":
        from gse_b200.torch_binding import gse_energy_forces
        E, F = gse_energy_forces(s["pos"], s["q"], s["ctx"])
        E, F = E.float(), F.float()
        loss = (F - s["f"]).square().mean() + (E / n - s["e"]).square()
        return [E.detach(), F.detach(), *torch.autograd.grad(loss, [s["pos"], s["q"]])]
    if kind == "batch":
        s["batch"].launch()
        b = s["buf"]
        return [b["energies"].float(), b["forces"].float(), b["grad_out"].float()]
    if kind == "grid":
        ctx, o = s["ctx"], s["out"]
        length = _boxes(c)[1]
        ctx.gauss_spread_on_grid(s["sigma2"], s["rcut2"], *length, s["rho"], o[0])
        ctx.gauss_efield_on_grid(*length, s["phi"], o[1], o[2], o[3])
        ctx.gauss_dipole_sum(*length, s["rho"], s["dip"])
        return o + [s["dip"]]
    if kind == "ewald":
        from gse_b200 import gse
        e1, f1 = gse.ewald_recip(c["sigma"], s["kcut"], s["box"], s["x"], CCELEC)
        e2, f2 = gse.ewald_direct(c["sigma"], 9.0, s["box"], s["x"], *s["excl"], CCELEC)
        return [e1, f1, e2, f2]
    raise ValueError(kind)


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _mesh_flops(n, m, length, sigma):
    """(spread and gather flops, flops of one solve) of one mesh evaluation."""
    s1 = sigma * math.sqrt(KAPPA)
    rcut = LAMBDA * math.sqrt(2.0) * s1
    h = [l / k for l, k in zip(length, m)]
    cube = math.prod(2 * math.ceil(rcut / v) + 1 for v in h)
    ball = 4.0 / 3.0 * math.pi * rcut ** 3 / math.prod(h)
    points = math.prod(m)
    return n * (2.0 * cube + 8.0 * ball), 5.0 * points * math.log2(points)


def work(case):
    c = case
    kind = c["kind"]
    if kind == "batch":
        systems, _ = _systems(c, 0)
        n = sum(v["n"] for v in systems)
        flops = 0.0
        for v in systems:
            a, f = _mesh_flops(v["n"], v["size"], v["box"], c["sigma"])
            flops += 3 * a + 2 * f
        # positions, cotangents in; forces and gradients out, handed on in FP32
        return {"bytes": n * (16.0 + 24 + 24 + 32) + 28.0 * n + 16.0 * len(systems), "flops": flops}
    m, length = _boxes(c)
    n = c["n"]
    w = 8 if c["precision"] == "fp64" else 4
    if kind == "grid":
        taps = [2 * math.ceil(_second_spread(c)[1] * k / l) + 1 for k, l in zip(m, length)]
        p = math.prod(m)
        return {"bytes": 6.0 * w * p, "flops": p * (2.0 * sum(taps) + 6 + 9)}
    if kind == "ewald":
        kcut = math.ceil(math.sqrt(2 * math.log(1e12)) / c["sigma"] * max(length) / (2 * math.pi))
        k = 2.0 / 3.0 * math.pi * kcut ** 3  # half of the sphere of k-vectors
        pairs = n * min(n, 4.0 / 3.0 * math.pi * 9.0 ** 3 * n / math.prod(length)) / 2
        return {"bytes": 2 * n * (32.0 + 24), "flops": n * k * 16 + pairs * 40}
    a, f = _mesh_flops(n, m, length, c["sigma"])
    if kind == "gradient":  # the grids again, the adjoint source, its solve, the reverse gather
        return {"bytes": n * (32.0 + 24 + 32), "flops": 3 * a + 2 * f}
    if kind == "train":
        return {"bytes": n * (16.0 + 24 + 12 + 16) + n * 16.0, "flops": 4 * a + 3 * f}
    return {"bytes": n * (4.0 * w + 24 + (12 if w == 4 else 0)), "flops": a + f}


# --------------------------------------------------------------------------
# The same in 64 bits, plain PyTorch
# --------------------------------------------------------------------------
class _Mesh:
    """The Gaussian-split mesh evaluation of one box in FP64."""

    def __init__(self, m, length, sigma):
        self.m, self.length = m, length
        self.h = [l / k for l, k in zip(length, m)]
        self.s1 = sigma * math.sqrt(KAPPA)
        self.s2 = sigma * math.sqrt(1.0 - 2.0 * KAPPA)
        self.sigma = sigma
        self.rcut = LAMBDA * math.sqrt(2.0) * self.s1
        self.nst = [math.ceil(self.rcut / v) for v in self.h]
        self.vol = math.prod(self.h)
        self.pref = (2 * math.pi * self.s1 ** 2) ** -1.5
        self.amp = (2 * math.pi) ** -1.5 * self.vol * self.s1 ** -5
        k = [2 * math.pi / l * torch.fft.fftfreq(v, 1.0 / v, dtype=torch.float64, device="cuda")
             for v, l in zip(m, length)]
        k[0] = 2 * math.pi / length[0] * torch.arange(m[0] // 2 + 1, dtype=torch.float64, device="cuda")
        self.k = (k[0][None, None, :], k[1][None, :, None], k[2][:, None, None])
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        self.green = 4 * math.pi * torch.exp(-0.5 * self.s2 ** 2 * self.k2) / self.k2
        self.green[0, 0, 0] = 0.0

    def chunks(self, x):
        """(slice, flat indices, offsets x - x_p per axis, exp factor) over the cubes."""
        w = [2 * n + 1 for n in self.nst]
        step = max(1, (48 << 20) // math.prod(w))
        for a in range(0, x.shape[0], step):
            sl = slice(a, min(a + step, x.shape[0]))
            idx, u = [], []
            for d in range(3):
                p = x[sl, d] / self.h[d]
                c = torch.sign(p) * torch.floor(p.abs() + 0.5)
                t = c[:, None] + torch.arange(-self.nst[d], self.nst[d] + 1, device=x.device)
                idx.append(torch.remainder(t, self.m[d]).long())
                u.append(x[sl, d, None] - t * self.h[d])
            flat = (idx[0][:, None, None, :] +
                    (idx[1][:, None, :, None] + idx[2][:, :, None, None] * self.m[1]) * self.m[0])
            u = (u[0][:, None, None, :], u[1][:, None, :, None], u[2][:, :, None, None])
            r2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
            yield sl, flat, u, r2, torch.exp(-0.5 / self.s1 ** 2 * r2)

    def _to_grid(self, grid, flat, val):
        grid.index_add_(0, flat.reshape(-1), val.reshape(-1))

    def spread(self, x):
        rho = torch.zeros(math.prod(self.m), dtype=torch.float64, device=x.device)
        for sl, flat, u, r2, e in self.chunks(x):
            self._to_grid(rho, flat, e * (self.pref * x[sl, 3])[:, None, None, None])
        return rho

    def solve(self, rho):
        r = torch.fft.rfftn(rho.view(self.m[2], self.m[1], self.m[0]))
        return torch.fft.irfftn(r * self.green, s=(self.m[2], self.m[1], self.m[0])).reshape(-1)

    def energy(self, rho, phi):
        return 0.5 * CCELEC * self.vol * (rho * phi).sum()

    def forces(self, x, phi):
        f = torch.empty(3, x.shape[0], dtype=torch.float64, device=x.device)
        for sl, flat, u, r2, e in self.chunks(x):
            t = torch.where(r2 < self.rcut ** 2, e, 0.0) * phi[flat]
            for d in range(3):
                f[d, sl] = CCELEC * self.amp * x[sl, 3] * (t * u[d]).sum((1, 2, 3))
        return f

    def virial(self, rho):
        r = torch.fft.rfftn(rho.view(self.m[2], self.m[1], self.m[0]))
        wgt = torch.full_like(self.k[0], 2.0)
        wgt[..., 0] = 1.0
        if self.m[0] % 2 == 0:
            wgt[..., -1] = 1.0
        ek = 0.5 * CCELEC * self.vol / math.prod(self.m) * wgt * self.green * (r.real ** 2 + r.imag ** 2)
        g = 1.0 / self.k2 + 0.5 * self.sigma ** 2
        g[0, 0, 0] = 0.0
        # a component with an odd power of a Nyquist k_x, k_y or k_z is what
        # the transform's sign convention (negative) gives it
        out = []
        for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
            t = -2.0 * self.k[a] * self.k[b] * g
            out.append((ek * (t + 1.0 if a == b else t)).sum())
        return torch.stack(out)

    def gradient(self, x, phi, dE, G):
        """(dL/dq, dL/dx, dL/dy, dL/dz) for dL/dE = dE and dL/dF = G (3, n)."""
        lam = torch.zeros_like(phi)
        for sl, flat, u, r2, e in self.chunks(x):
            gu = sum(G[d, sl, None, None, None] * u[d] for d in range(3))
            t = torch.where(r2 < self.rcut ** 2, e, 0.0) * gu
            self._to_grid(lam, flat, t * (CCELEC * self.amp * x[sl, 3])[:, None, None, None])
        psi = self.solve(lam) + dE * CCELEC * self.vol * phi
        out = torch.empty(4, x.shape[0], dtype=torch.float64, device=x.device)
        for sl, flat, u, r2, e in self.chunks(x):
            c = self.pref * e * psi[flat]
            t = CCELEC * self.amp * torch.where(r2 < self.rcut ** 2, e, 0.0) * phi[flat]
            gu = sum(G[d, sl, None, None, None] * u[d] for d in range(3))
            out[0, sl] = (c + t * gu).sum((1, 2, 3))
            for d in range(3):
                v = -(c + t * gu) * u[d] / self.s1 ** 2 + t * G[d, sl, None, None, None]
                out[1 + d, sl] = x[sl, 3] * v.sum((1, 2, 3))
        return out

    def forward(self, x):
        rho = self.spread(x)
        phi = self.solve(rho)
        return rho, phi, self.energy(rho, phi), self.forces(x, phi)


def _conv(a, sigma, rcut, m, length):
    """Periodic Gaussian convolution of a grid [mz, my, mx], tap by tap."""
    out = a
    for axis, (k, l) in zip((2, 1, 0), zip(m, length)):
        h = l / k
        n = math.ceil(rcut / h)
        out = sum(math.exp(-h * h * i * i / (2 * sigma ** 2)) * torch.roll(out, -i, axis)
                  for i in range(-n, n + 1))
    return out * (2 * math.pi * sigma ** 2) ** -1.5 * math.prod(l / k for k, l in zip(m, length))


def _ewald_recip(x, sigma, kcut, length):
    r = torch.arange(-kcut, kcut + 1, device=x.device, dtype=torch.float64)
    k = torch.cartesian_prod(r, r, r)
    k = k[(k.square().sum(1) <= kcut * kcut) &
          ((k[:, 0] > 0) | ((k[:, 0] == 0) & ((k[:, 1] > 0) | ((k[:, 1] == 0) & (k[:, 2] > 0)))))]
    k = k * (2 * math.pi / torch.tensor(length, dtype=torch.float64, device=x.device))
    q, pos = x[:, 3], x[:, :3]
    e = torch.zeros((), dtype=torch.float64, device=x.device)
    f = torch.zeros_like(pos)
    step = max(1, (64 << 20) // max(1, x.shape[0]))
    for a in range(0, k.shape[0], step):
        kk = k[a:a + step]
        k2 = kk.square().sum(1)
        w = 2 * 2 * math.pi / math.prod(length) * CCELEC * torch.exp(-0.5 * sigma ** 2 * k2) / k2
        p = kk @ pos.T
        c, s = torch.cos(p), torch.sin(p)
        C, S = c @ q, s @ q
        e += (w * (C * C + S * S)).sum()
        f += 2 * q[:, None] * ((s * (w * C)[:, None] - c * (w * S)[:, None]).T @ kk)
    return e, f


def _ewald_direct(x, sigma, rcut, length):
    box = torch.tensor(length, dtype=torch.float64, device=x.device)
    n = x.shape[0]
    mol = torch.arange(n, device=x.device) // 3
    mol[n - n % 3:] = -1 - torch.arange(n % 3, device=x.device)  # no whole molecule: no exclusions
    e = -CCELEC / math.sqrt(2 * math.pi * sigma ** 2) * x[:, 3].square().sum()
    f = torch.zeros(n, 3, dtype=torch.float64, device=x.device)
    step = max(1, (16 << 20) // n)
    for a in range(0, n, step):
        d = x[a:a + step, None, :3] - x[None, :, :3]
        d = d - box * torch.round(d / box)
        r2 = d.square().sum(2)
        i = torch.arange(a, min(a + step, n), device=x.device)
        ok = (r2 < rcut * rcut) & (mol[i][:, None] != mol[None, :])
        r = torch.where(ok, r2, 1.0).sqrt()
        qq = torch.where(ok, CCELEC * x[i, 3][:, None] * x[None, :, 3], 0.0)
        v = qq * torch.erfc(r / (math.sqrt(2) * sigma)) / r
        e += 0.5 * v.sum()
        de = -(v + qq * math.sqrt(2 / math.pi) / sigma * torch.exp(-r * r / (2 * sigma ** 2))) / r
        f[i] = ((de / r)[:, :, None] * d).sum(1)
    return e, f


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "batch":
        systems, x = _systems(c, seed)
        x = torch.from_numpy(x).cuda().double()
        G = torch.from_numpy(_upstream(x.shape[0], seed)).cuda()
        e, f, d, a = [], [], [], 0
        for v in systems:
            sl = slice(a, a + v["n"])
            mesh = _Mesh(v["size"], v["box"], c["sigma"])
            _, phi, ev, fv = mesh.forward(x[sl])
            e.append(ev)
            f.append(fv)
            d.append(mesh.gradient(x[sl], phi, 1.0, G[:, sl]))
            a += v["n"]
        return [torch.stack(e), torch.cat(f, 1), torch.cat(d, 1)]
    m, length = _boxes(c)
    if kind == "grid":
        rho, phi = (torch.from_numpy(a).cuda().double() for a in _grids(c, seed))
        sigma2, rcut2 = _second_spread(c)
        h = [l / k for l, k in zip(length, m)]
        out = [_conv(rho, sigma2, rcut2, m, length)]
        out += [-(torch.roll(phi, -1, axis) - phi) / hd for axis, hd in zip((2, 1, 0), h)]
        dip = []
        for d in range(3):
            i = torch.arange(m[d], device="cuda", dtype=torch.float64) * h[d]
            i = (i[None, None, :], i[None, :, None], i[:, None, None])[d]
            dip.append((rho * math.prod(h) * i).sum())
        return out + [torch.stack(dip)]
    x = torch.from_numpy(_charges(c, seed)).cuda().double()
    if kind == "ewald":
        kcut = math.ceil(math.sqrt(2 * math.log(1e12)) / c["sigma"] * max(length) / (2 * math.pi))
        return [*_ewald_recip(x, c["sigma"], kcut, length), *_ewald_direct(x, c["sigma"], 9.0, length)]
    mesh = _Mesh(m, length, c["sigma"])
    rho, phi, e, f = mesh.forward(x)
    if kind == "forward":
        return [e[None], f]
    if kind == "classes":
        return [e, *f]
    if kind == "pressure":
        return [e[None], f, mesh.virial(rho)]
    if kind == "gradient":
        return mesh.gradient(x, phi, 1.0, torch.from_numpy(_upstream(c["n"], seed)).cuda())
    if kind == "train":
        n = c["n"]
        tf, te = _targets(c, seed)
        dF = 2.0 / (3 * n) * (f - torch.from_numpy(tf).cuda().double().T)
        dE = 2.0 / n * (e / n - float(te))
        g = mesh.gradient(x, phi, dE, dF)
        return [e, f.T.contiguous(), g[1:].T.contiguous(), g[0]]
    raise ValueError(kind)
