"""Performance cases of npme_b200: the calls its users make, over the range of
sizes, kernels, splittings and precisions they make them with.

A case is a dict of plain values.  ``prepare`` builds what a program holds
before the call (inputs from a seed, a set-up solver, device buffers), ``run``
makes the call through the package's public entry points, ``exact`` computes
the same numbers in 64 bits with torch alone: the particle-mesh method itself
(B-spline spreading, zero-padded convolution, derivative-match or Ewald
split), so that a result is compared with what its own method gives and not
with another sum.

Kinds of cases
  step     CalcV of a set-up solver on device buffers, again and again with
           new charges in the same buffers (an iterative solver's matrix
           product, a Monte Carlo move of charges)
  direct   the short-range direct sum alone, on device buffers
  solve    a new geometry on an existing solver, then CalcV through host
           buffers (a step of molecular dynamics, a request of a service)
  batch    batched CalcV of many set-up systems of a serving stream
  exact    the O(N^2) sum a user checks errors with
"""
import math

import numpy as np
import torch

import npme_b200 as npme
from npme_b200 import api, autotune

KERNEL = {"laplace": {}, "ralpha": {"alpha": -0.5}, "helmholtz": {"k0": 0.5}}


# --- cases -------------------------------------------------------------------

def _case(kind, kernel, n, box, order, rdir, grid, precision="fp32", split="dm", nderiv=None,
          alpha=-0.5, k0=0.5, name=None):
    if nderiv is None:
        nderiv = 3 if order == 4 else (6 if order == 6 else 8)
    c = {"kind": kind, "kernel": kernel, "split": split, "n": n,
         "bx": float(box[0]), "by": float(box[1]), "bz": float(box[2]),
         "order": order, "nderiv": nderiv, "rdir": float(rdir),
         "n1": grid[0], "n2": grid[1], "n3": grid[2], "precision": precision,
         "alpha": alpha, "k0": k0}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest of the repository's workloads: launches and latency
        _case("step", "laplace", 4000, (20, 20, 20), 6, 8, (64, 64, 64), name="step_laplace_4k"),
        # a mid-size system of odd size in a flat box, order 8
        _case("step", "laplace", 30011, (61, 41, 12), 8, 7, (160, 120, 48),
              name="step_laplace_30k_flat"),
        # the headline workload
        _case("step", "laplace", 1000000, (100, 100, 100), 6, 8, (256, 256, 256),
              name="step_laplace_1m"),
        # r^-0.5 in a long box
        _case("step", "ralpha", 500000, (200, 100, 50), 8, 10, (384, 192, 96),
              name="step_ralpha_500k"),
        # complex charges
        _case("step", "helmholtz", 250000, (80, 80, 80), 6, 8, (192, 192, 192),
              name="step_helmholtz_250k"),
        # double precision: what the reference's users run, and the command line's default
        _case("step", "laplace", 1000000, (100, 100, 100), 6, 8, (256, 256, 256), "fp64",
              name="step_laplace_1m_fp64"),
        _case("step", "helmholtz", 62501, (50, 50, 25), 8, 8, (128, 128, 72), "fp64",
              name="step_helmholtz_62k_fp64"),
        # the original Ewald split on the reference's example box
        _case("step", "laplace", 100000, (50, 75, 100), 6, 6, (160, 240, 320), split="orig",
              name="step_ewald_100k"),
        # new geometries: a small request and a molecular-dynamics-sized one
        _case("solve", "laplace", 2003, (12.6, 12.6, 12.6), 8, 5, (48, 48, 48),
              name="solve_laplace_2k"),
        _case("solve", "ralpha", 200000, (58.5, 58.5, 58.5), 8, 6, (160, 160, 160),
              name="solve_ralpha_200k"),
        # the serving mix, log-uniform sizes, parameters from the autotuner
        {"kind": "batch", "count": 16, "nmin": 1000, "nmax": 120000, "precision": "fp32",
         "name": "batch_serving_16"},
        # error check of a small run
        _case("exact", "laplace", 40001, (40, 40, 25), 6, 8, (64, 64, 64), "fp64",
              name="exact_laplace_40k"),
    ]


def _fft_length(extent, order, rdir, h):
    """Smallest FFT length (multiple of 4, factors 2, 3, 5) with
    grid spacing <= h over the extent."""
    n = 4 * (order + 2)
    while True:
        m = n
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        a1 = 1.0 - 2.0 * (order + 1) / n
        a2 = 1.0 - 4.0 * (order + 1) / n
        x = max(extent, extent / a1 - rdir / 2.0 * a2 / a1)
        if m == 1 and 2.0 * (x + rdir) / n <= h:
            return n
        n += 4


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "direct", "solve", "solve", "batch", "exact"])
    if kind == "batch":
        nmin = int(math.exp(rng.uniform(math.log(500), math.log(5000))))
        return {"kind": "batch", "count": rng.randint(3, 20), "nmin": nmin,
                "nmax": int(nmin * math.exp(rng.uniform(math.log(2), math.log(24)))),
                "precision": "fp32"}
    kernel = rng.choice(["laplace", "laplace", "ralpha", "helmholtz"])
    split = "orig" if kernel == "laplace" and rng.random() < 0.2 else "dm"
    precision = rng.choice(["fp32", "fp32", "fp64"])
    top = {"exact": 60000, "solve": 300000}.get(kind, 700000 if precision == "fp32" else 250000)
    if kernel == "helmholtz":
        top //= 3
    n = int(math.exp(rng.uniform(math.log(500), math.log(top))))
    spacing = math.exp(rng.uniform(math.log(0.7), math.log(1.6)))  # mean point distance
    fx, fy = math.exp(rng.uniform(-0.7, 0.7)), math.exp(rng.uniform(-0.7, 0.7))
    side = spacing * n ** (1.0 / 3.0)
    box = [round(side * fx, 3), round(side * fy, 3), round(side / (fx * fy), 3)]
    order = rng.choice([4, 6, 6, 8, 8, 10])
    nderiv = rng.choice([None, None, None, 5, 10])
    rdir = round(spacing * rng.uniform(4.5, 9.0), 3)
    h = spacing * rng.uniform(0.75, 1.1)
    grid = [min(512, _fft_length(b, order, rdir, h)) for b in box]
    if rng.random() < 0.15:  # lengths with a factor 7, 11 or 13 are accepted too
        grid[rng.randrange(3)] = 4 * rng.choice([7, 11, 13]) * rng.choice([2, 3])
    # every axis keeps its points inside the charge octant
    grid = [g if g >= 4 * (order + 2) else 4 * (order + 2) for g in grid]
    return _case(kind, kernel, n, box, order, rdir, tuple(grid),
                 "fp64" if kind == "exact" else precision, split, nderiv,
                 alpha=rng.choice([-0.5, -0.5, -2.0, -3.0]), k0=round(rng.uniform(0.2, 0.9), 3))


# --- inputs ------------------------------------------------------------------

def _system(kernel, n, box, seed):
    """Points uniform in the box, charges uniform in [-1, 1] (real ones
    neutral)."""
    g = np.random.Generator(np.random.Philox(seed))
    coord = g.random((n, 3)) * np.asarray(box)
    if kernel == "helmholtz":
        return coord, g.uniform(-1, 1, n) + 1j * g.uniform(-1, 1, n)
    q = g.uniform(-1, 1, n)
    return coord, q - q.mean()


def _inputs(case, seed):
    return _system(case["kernel"], case["n"], (case["bx"], case["by"], case["bz"]), seed)


def _params(case):
    return api.make_params(case["kernel"], case["split"], case["rdir"], case["order"],
                           case["nderiv"], (case["n1"], case["n2"], case["n3"]),
                           alpha=case["alpha"] if case["kernel"] == "ralpha" else -1.0,
                           k0=case["k0"] if case["kernel"] == "helmholtz" else 0.0,
                           precision=case["precision"])


def _members(case):
    """(kernel, n, box) of a batch: log-uniform sizes and the serving mix of
    kernels (60 % 1/r, 25 % r^-0.5, 15 % Helmholtz) by a fixed rotation."""
    out = []
    for i in range(case["count"]):
        f = ((i + 0.5) * 0.6180339887498949) % 1.0
        n = int(case["nmin"] * (case["nmax"] / case["nmin"]) ** f)
        m = ((i + 0.5) * 0.7548776662466927) % 1.0
        kernel = "laplace" if m < 0.60 else ("ralpha" if m < 0.85 else "helmholtz")
        side = n ** (1.0 / 3.0)
        out.append((kernel, n, (side, side, side)))
    return out


def _batch_choice(kernel, n, box):
    return autotune.choose(kernel, n, tuple(box))


def _device(q):
    return torch.from_numpy(np.ascontiguousarray(q).view(np.float64)).cuda()


def prepare(case, seed):
    if case["kind"] == "batch":
        st = {"case": case, "batch": npme.api.Batch(), "solvers": [], "q": [], "V": [],
              "systems": []}
        for i, (kernel, n, box) in enumerate(_members(case)):
            coord, q = _system(kernel, n, box, seed * 1000 + i)
            ch = _batch_choice(kernel, n, box)
            p = api.make_params(kernel, "dm", ch["Rdir"], ch["order"], ch["nDeriv"], ch["grid"],
                                precision=case["precision"], **KERNEL[kernel])
            st["solvers"].append(npme.Solver(p).setup(coord))
            st["q"].append(_device(q))
            st["V"].append(torch.empty((n, 8 if kernel == "helmholtz" else 4),
                                       dtype=torch.float64, device="cuda"))
        return st
    coord, q = _inputs(case, seed)
    st = {"case": case, "solver": npme.Solver(_params(case)), "coord": coord, "q": q}
    if case["kind"] == "solve":
        # a program that moves points keeps its solver; its first geometry is another one
        other, _ = _inputs(case, seed + 7919)
        st["solver"].setup(other)
        return st
    st["solver"].setup(coord)
    if case["kind"] in ("step", "direct"):
        st["dq"] = _device(q)
        st["V"] = torch.empty((case["n"], 8 if case["kernel"] == "helmholtz" else 4),
                              dtype=torch.float64, device="cuda")
    return st


def run(st):
    kind = st["case"]["kind"]
    if kind in ("step", "direct"):
        s, stream = st["solver"], torch.cuda.current_stream().cuda_stream
        call = s.calcv_device if kind == "step" else s.direct_sum_device
        call(st["V"].data_ptr(), st["dq"].data_ptr(), stream)
        return st["V"]
    if kind == "batch":
        st["batch"].calcv(st["solvers"], [v.data_ptr() for v in st["V"]],
                          [q.data_ptr() for q in st["q"]], torch.cuda.current_stream().cuda_stream)
        return st["V"]
    if kind == "solve":
        V = st["solver"].setup(st["coord"]).calcv(st["q"])
    else:
        V = st["solver"].calcv_exact(st["q"])
    return V.view(np.float64)


# --- the work and the tolerance ----------------------------------------------

def _pairs(n, box, rdir):
    """Expected unordered pairs within rdir of n uniform points in a box."""
    a, b, c = box
    if rdir <= min(box):
        v = (a * b * c * 4.0 / 3.0 * math.pi * rdir ** 3
             - (a * b + b * c + c * a) * math.pi / 2.0 * rdir ** 4
             + (a + b + c) * 8.0 / 15.0 * rdir ** 5 - rdir ** 6 / 6.0)
        p = v / (a * b * c) ** 2
    else:
        g = np.random.Generator(np.random.Philox(7))
        d = (g.random((200000, 3)) - g.random((200000, 3))) * np.asarray(box)
        p = float((np.einsum("ij,ij->i", d, d) <= rdir * rdir).mean())
    return 0.5 * n * (n - 1.0) * p


def _work(kernel, n, box, order, nderiv, rdir, grid, precision, parts=("direct", "rec")):
    cx = 2 if kernel == "helmholtz" else 1
    flops = 0.0
    if "direct" in parts:  # per pair: distance 8, kernel and polynomials, both sums of both points
        flops += _pairs(n, box, rdir) * (29 + 4 * nderiv) * (3 if cx == 2 else 1)
    if "rec" in parts:
        N = float(grid[0]) * grid[1] * grid[2]
        # spread (2), interpolation with gradient (4 + 4), transforms of the octant's lines
        flops += n * order ** 3 * 4.0 * cx
        flops += 2.5 * cx * N * math.log2(N)
    return {"bytes": n * 8.0 * cx * 5, "flops": flops}


def work(case):
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for kernel, n, box in _members(case):
            ch = _batch_choice(kernel, n, box)
            w = _work(kernel, n, box, ch["order"], ch["nDeriv"], ch["Rdir"], ch["grid"],
                      case["precision"])
            total = {k: total[k] + w[k] for k in total}
        return total
    n, box = case["n"], (case["bx"], case["by"], case["bz"])
    cx = 2 if case["kernel"] == "helmholtz" else 1
    if case["kind"] == "exact":
        return {"bytes": n * (24.0 + 40.0 * cx), "flops": 0.5 * n * (n - 1.0) * 25 * cx}
    w = _work(case["kernel"], n, box, case["order"], case["nderiv"], case["rdir"],
              (case["n1"], case["n2"], case["n3"]), case["precision"],
              ("direct",) if case["kind"] == "direct" else ("direct", "rec"))
    if case["kind"] == "solve":
        w["bytes"] += 24.0 * n  # the coordinates
    return w


def tolerance(case):
    """About four times the distance from `exact` measured over listed and
    drawn cases: 1e-7 to 2e-6 in FP32 (r^alpha and high derivative orders the
    largest), up to 6e-15 in FP64, where r^alpha in flat boxes reached 6e-14
    against an independent program."""
    if case["precision"] == "fp64":
        return {"rel": 2e-13}
    return {"rel": 8e-6}


# --- the same numbers in 64 bits, by torch -------------------------------------

def _taylor(kernel, split, rdir, nderiv, alpha, k0):
    """Coefficients c_n of f_LR(r) = sum c_n (r^2 - rdir^2)^n, the derivative
    match at rdir: ((1/r) d/dr)^n f / (2^n n!)."""
    r2 = rdir * rdir
    f = []
    if kernel == "helmholtz":
        e = complex(math.cos(k0 * rdir), math.sin(k0 * rdir))
        f = [e / rdir, -e / rdir / r2 + 1j * k0 * e / r2]
        for n in range(2, nderiv + 1):
            f.append(-(2.0 * n - 1.0) / r2 * f[n - 1] - k0 * k0 / r2 * f[n - 2])
    else:
        a = -1.0 if kernel == "laplace" else alpha
        f = [rdir ** a]
        for n in range(1, nderiv + 1):
            f.append(f[n - 1] * (a - 2 * n + 2) / r2)
    return [v / (2.0 ** n * math.factorial(n)) for n, v in enumerate(f)]


def _horner(c, s):
    p = torch.full_like(s, c[-1]) if not isinstance(c[-1], complex) else \
        torch.full(s.shape, c[-1], dtype=torch.complex128, device=s.device)
    for v in reversed(c[:-1]):
        p = p * s + v
    return p


def _ewald_beta(rdir, tol=1e-6):
    c, x = math.log(math.sqrt(math.pi) * tol * rdir), 0.1
    for _ in range(1000):
        f = x * x + math.log(x) + c
        if abs(f) < 1e-13:
            break
        x -= f / (2 * x + 1 / x)
    return x / rdir


class _Kernel:
    """f and (1/r) df/dr of the full kernel and of its long-range part."""

    def __init__(self, kernel, split, rdir, nderiv, alpha, k0):
        self.kernel, self.split, self.rdir = kernel, split, rdir
        self.alpha = -1.0 if kernel == "laplace" else alpha
        self.k0 = k0
        if split == "orig":
            self.beta = _ewald_beta(rdir)
        else:
            self.c = _taylor(kernel, split, rdir, nderiv, alpha, k0)
            self.d = [2.0 * (n + 1) * v for n, v in enumerate(self.c[1:])]

    def full(self, r2):
        if self.kernel == "helmholtz":
            r = torch.sqrt(r2)
            e = torch.polar(1.0 / r, self.k0 * r)
            return e, e * (1j * self.k0 / r - 1.0 / r2)
        f = 1.0 / torch.sqrt(r2) if self.kernel == "laplace" else r2 ** (0.5 * self.alpha)
        return f, self.alpha * f / r2

    def short(self, r2):
        if self.split == "orig":
            r = torch.sqrt(r2)
            x = self.beta * r
            f = torch.erfc(x) / r
            return f, -(2.0 * self.beta / math.sqrt(math.pi) * torch.exp(-x * x) + f) / r2
        f, g = self.full(r2)
        s = r2 - self.rdir ** 2
        return f - _horner(self.c, s), g - _horner(self.d, s)

    def long(self, r2):
        if self.split == "orig":
            x = self.beta * torch.sqrt(r2)
            small = x < 1e-4
            v = torch.where(small, 2.0 / math.sqrt(math.pi) * (1.0 - x * x / 3.0),
                            torch.erf(x) / torch.where(small, torch.ones_like(x), x))
            return self.beta * v
        inside = r2 <= self.rdir ** 2
        outer, _ = self.full(torch.where(inside, torch.full_like(r2, self.rdir ** 2), r2))
        inner = _horner(self.c, torch.where(inside, r2, torch.zeros_like(r2)) - self.rdir ** 2)
        return torch.where(inside, inner, outer)

    def at_zero(self):
        if self.split == "orig":
            return 2.0 * self.beta / math.sqrt(math.pi)
        s = -self.rdir ** 2
        return sum(v * s ** n for n, v in enumerate(self.c))


def _pair_block(x, y, q, pair, rdir):
    """V, dV at the points x[..., a, 3] from the sources y[..., b, 3]."""
    d = [x[..., :, None, k] - y[..., None, :, k] for k in range(3)]
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    hit = r2 > 0
    if rdir is not None:
        hit &= r2 <= rdir * rdir
    f, g = pair(torch.where(hit, r2, torch.ones_like(r2)))
    w = torch.where(hit, q[..., None, :], torch.zeros((), dtype=q.dtype, device=q.device))
    g = g * w
    return torch.stack([(f * w).sum(-1)] + [(g * d[k]).sum(-1) for k in range(3)], -1)


def _pair_sum_all(coord, q, pair, rdir=None):
    n = coord.shape[0]
    step = max(1, int(2e7 // n))
    return torch.cat([_pair_block(coord[i:i + step], coord, q, pair, rdir)
                      for i in range(0, n, step)])


def _pair_sum_near(coord, q, pair, rdir):
    """Pairs within rdir by cells of edge >= rdir, padded to the fullest."""
    lo = coord.amin(0)
    ext = (coord.amax(0) - lo).tolist()
    nc = [max(1, int(e / rdir)) for e in ext]
    if max(nc) < 3 or coord.shape[0] < 6000:
        return _pair_sum_all(coord, q, pair, rdir)
    edge = torch.tensor([max(e, 1e-9) / m for e, m in zip(ext, nc)], device=coord.device,
                        dtype=torch.float64)
    dims = torch.tensor(nc, device=coord.device)
    ijk = torch.minimum(((coord - lo) / edge).long(), dims - 1)
    cell = (ijk[:, 0] * nc[1] + ijk[:, 1]) * nc[2] + ijk[:, 2]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=nc[0] * nc[1] * nc[2])
    width = int(count.max())
    start = torch.cumsum(count, 0) - count
    slot = start[cell[order]]
    rank = torch.arange(len(order), device=coord.device) - slot
    cells = count.numel()
    table = torch.full((cells + 1, width), -1, dtype=torch.long, device=coord.device)
    table[cell[order], rank] = order
    pos = torch.where((table >= 0)[..., None], coord[table.clamp(min=0)],
                      torch.full((), 1e9, dtype=torch.float64, device=coord.device))
    chg = torch.where(table >= 0, q[table.clamp(min=0)], torch.zeros((), dtype=q.dtype,
                                                                     device=q.device))
    V = torch.zeros((coord.shape[0], 4), dtype=q.dtype, device=q.device)
    ids = torch.arange(cells, device=coord.device)
    c3, c2, c1 = ids % nc[2], (ids // nc[2]) % nc[1], ids // (nc[1] * nc[2])
    step = max(1, int(2e7 // (width * width)))
    for i in range(0, cells, step):
        a = ids[i:i + step]
        tgt = pos[a]
        acc = torch.zeros((len(a), width, 4), dtype=q.dtype, device=q.device)
        for o in range(27):
            d1, d2, d3 = o // 9 - 1, (o // 3) % 3 - 1, o % 3 - 1
            m1, m2, m3 = c1[a] + d1, c2[a] + d2, c3[a] + d3
            ok = ((m1 >= 0) & (m1 < nc[0]) & (m2 >= 0) & (m2 < nc[1]) & (m3 >= 0) & (m3 < nc[2]))
            b = torch.where(ok, (m1 * nc[1] + m2) * nc[2] + m3, torch.full_like(m1, cells))
            # absent targets and sources sit on the same far point: distance 0, no pair
            acc += _pair_block(tgt, pos[b], chg[b], pair, rdir)
        t = table[a]
        V[t[t >= 0]] = acc[t >= 0]
    return V


def _bspline(order, u):
    """B_order(u + t) and its derivative at t = 0..order-1, each [order, n]."""
    c = torch.zeros((order,) + u.shape, dtype=u.dtype, device=u.device)
    c[0] = 1.0
    for j in range(1, order):
        if j == order - 1:
            prev = c.clone()
        new = torch.zeros_like(c)
        for k in range(j + 1):
            left = c[k] if k <= j - 1 else 0.0
            right = c[k - 1] if k >= 1 else 0.0
            new[k] = ((u + k) * left + (j + 1 - (u + k)) * right) / j
        c = new
    dw = torch.zeros_like(c)
    for t in range(order):
        dw[t] = (prev[t] if t <= order - 2 else 0.0) - (prev[t - 1] if t >= 1 else 0.0)
    return c, dw


def _ramp(x, a):
    z = 6.0 / a
    top = z / math.sqrt(1.0 + z * z)
    return 1.0 if x >= top else 0.0 if x <= -top else \
        0.5 * (1.0 + math.erf(a * x / math.sqrt(1.0 - x * x)))


def _window(x, X, Xmax, a):
    d = 0.5 * (Xmax - X)
    if x < -X:
        return _ramp((x + X + d) / d, a)
    return 1.0 if x <= X else _ramp((-x + X + d) / d, a)


def _axis_images(N, X, rdir, a=4.0):
    """Sample points of the half axis, their Fourier-extension images and the
    windows of both."""
    top, M = X + rdir, N // 2 + 1
    x1 = [i * 2 * top / N for i in range(M)]
    x2, t1, t2 = [], [], []
    for x in x1:
        if x > X:
            x2.append(x - 2 * top)
            t1.append(_window(x, X, 2 * top - X, a))
            t2.append(_window(x - 2 * top, X, 2 * top - X, a))
        else:
            x2.append(1.0)
            t1.append(1.0)
            t2.append(0.0)
    return [torch.tensor(v, dtype=torch.float64, device="cuda") for v in (x1, x2, t1, t2)]


def _reciprocal(coord, q, ker, order, rdir, grid):
    """The long-range part on the zero-padded grid: V and its gradient."""
    dev = coord.device
    lo, hi = coord.amin(0).tolist(), coord.amax(0).tolist()
    X, R, L = [], [], []
    for a in range(3):
        N = grid[a]
        a1, a2 = 1.0 - 2.0 * (order + 1) / N, 1.0 - 4.0 * (order + 1) / N
        x0 = hi[a] - lo[a]
        x = max(x0, x0 / a1 - rdir / 2.0 * a2 / a1)
        X.append(x)
        R.append(0.5 * (hi[a] + lo[a]) + 0.5 * (x0 - x))
        L.append(2 * (x + rdir))
    # kernel transform on the octant, even in every axis
    ax = [_axis_images(grid[a], X[a], rdir) for a in range(3)]
    M = [g // 2 + 1 for g in grid]
    cplx = q.is_complex()
    F = torch.zeros(M, dtype=q.dtype, device=dev)
    for s in range(8):
        p = [ax[a][(s >> a) & 1] for a in range(3)]
        w = [ax[a][2 + ((s >> a) & 1)] for a in range(3)]
        r2 = p[0][:, None, None] ** 2 + p[1][:, None] ** 2 + p[2] ** 2
        F += w[0][:, None, None] * w[1][:, None] * w[2] * ker.long(r2)
    for a in range(3):
        m = torch.arange(M[a], device=dev, dtype=torch.float64)
        C = torch.cos(2 * math.pi / grid[a] * (m[:, None] * m % grid[a]))
        C = C * torch.where((m == 0) | (m == M[a] - 1), 1.0, 2.0)
        b, _ = _bspline(order, torch.zeros(1, dtype=torch.float64, device=dev))
        ph = 2 * math.pi / grid[a] * m[:, None] * torch.arange(order, device=dev)
        lam = 1.0 / ((torch.cos(ph) * b[:, 0]).sum(1) ** 2 + (torch.sin(ph) * b[:, 0]).sum(1) ** 2)
        C = (C * lam[:, None]).to(q.dtype)
        F = torch.tensordot(C, F, ([1], [a])).movedim(0, a)
    # stencils
    o, wt, dwt = [], [], []
    for a in range(3):
        w = grid[a] / L[a] * (coord[:, a] - R[a])
        ms = torch.where(w < 0, torch.trunc(-w) + 1, -torch.trunc(w))
        b, db = _bspline(order, w + ms)
        o.append(ms.long() + grid[a] // 4)
        wt.append(b)
        dwt.append(db)
    H = [g // 2 for g in grid]
    Q = torch.zeros(H[0] * H[1] * H[2], dtype=q.dtype, device=dev)
    steps = [(i, j, k) for i in range(order) for j in range(order) for k in range(order)]
    for i, j, k in steps:
        at = ((o[0] + i) * H[1] + o[1] + j) * H[2] + o[2] + k
        Q.index_add_(0, at, q * (wt[0][i] * wt[1][j] * wt[2][k]))
    Q = Q.view(H)
    idx = [torch.arange(g, device=dev) for g in grid]
    fold = [torch.where(i <= g // 2, i, g - i) for i, g in zip(idx, grid)]
    if cplx:
        T = torch.fft.fftn(Q, s=grid)
        T *= F[fold[0]][:, fold[1]][:, :, fold[2]]
        T = torch.fft.ifftn(T)
    else:
        T = torch.fft.rfftn(Q, s=grid)
        T *= F[fold[0]][:, fold[1]]
        T = torch.fft.irfftn(T, s=grid)
    T = T[:H[0], :H[1], :H[2]].reshape(-1)
    V = torch.zeros((coord.shape[0], 4), dtype=q.dtype, device=dev)
    for i, j, k in steps:
        at = ((o[0] + i) * H[1] + o[1] + j) * H[2] + o[2] + k
        t = T[at]
        V[:, 0] += t * (wt[0][i] * wt[1][j] * wt[2][k])
        V[:, 1] += t * (dwt[0][i] * wt[1][j] * wt[2][k]) * (grid[0] / L[0])
        V[:, 2] += t * (wt[0][i] * dwt[1][j] * wt[2][k]) * (grid[1] / L[1])
        V[:, 3] += t * (wt[0][i] * wt[1][j] * dwt[2][k]) * (grid[2] / L[2])
    return V


def _solve(coord, q, kernel, split, order, nderiv, rdir, grid, alpha, k0, reciprocal=True):
    ker = _Kernel(kernel, split, rdir, nderiv, alpha, k0)
    coord, q = torch.from_numpy(coord).cuda(), torch.from_numpy(q).cuda()
    V = _pair_sum_near(coord, q, ker.short, rdir)
    if reciprocal:
        V += _reciprocal(coord, q, ker, order, rdir, list(grid))
        V[:, 0] -= ker.at_zero() * q
    return torch.view_as_real(V).reshape(len(q), 8) if V.is_complex() else V


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        for i, (kernel, n, box) in enumerate(_members(case)):
            coord, q = _system(kernel, n, box, seed * 1000 + i)
            ch = _batch_choice(kernel, n, box)
            out.append(_solve(coord, q, kernel, "dm", ch["order"], ch["nDeriv"], ch["Rdir"],
                              ch["grid"], KERNEL[kernel].get("alpha", -1.0),
                              KERNEL[kernel].get("k0", 0.0)))
        return out
    coord, q = _inputs(case, seed)
    kind = case["kind"]
    if kind == "exact":
        ker = _Kernel(case["kernel"], case["split"], case["rdir"], case["nderiv"], case["alpha"],
                      case["k0"])
        V = _pair_sum_all(torch.from_numpy(coord).cuda(), torch.from_numpy(q).cuda(), ker.full)
        V = (torch.view_as_real(V).reshape(len(q), 8) if V.is_complex() else V)
        return V.cpu().numpy()
    V = _solve(coord, q, case["kernel"], case["split"], case["order"], case["nderiv"],
               case["rdir"], (case["n1"], case["n2"], case["n3"]), case["alpha"], case["k0"],
               reciprocal=kind == "step" or kind == "solve")
    return V.cpu().numpy() if kind == "solve" else V
