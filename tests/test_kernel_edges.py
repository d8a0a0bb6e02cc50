"""Edges of the kernels' tilings and of the rules that choose between them:
transform lengths, B-spline orders, warps per target group, source zones,
runtime exponents, and what a non-finite charge reaches.

Tolerances (relative 2-norm): FP64 against the oracle 1e-12 (the same
algorithm; sums of up to 1e4 terms in another order), the two FP64 walks of
the same pairs 1e-13; FP32 against FP64 1e-5 for V and 3e-5 for the gradient
(the stated bound of the FP32 mode), the two FP32 walks 1e-6.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, rel
import npme_b200
from npme_b200 import api
from npme_b200.workloads import Workload
from oracle import orcbind as ob

pytestmark = pytest.mark.gpu

TOL = {"fp64": (1e-12, 1e-12), "fp32": (1e-5, 3e-5)}
WALKS = {"fp64": 1e-13, "fp32": 1e-6}


def check(V, Vo, prec, scale=1.0):
    assert rel(V[:, 0], Vo[:, 0]) < scale * TOL[prec][0]
    assert rel(V[:, 1:], Vo[:, 1:]) < scale * TOL[prec][1]


def system(n, func="laplace", split="dm", box=(10.0, 10.0, 10.0), grid=(48, 48, 48), order=6,
           Rdir=4.0, alpha=-0.5, k0=0.5, **kw):
    cplx = func == "helmholtz"
    return Workload("edge", n, box, func, split, order, grid, Rdir, alpha=alpha,
                    k0=k0 if cplx else 0.0, complex_charge=cplx, seed=7000 + n, **kw)


def direct(s, q):
    import torch
    cplx = np.iscomplexobj(q)
    dq = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    dV = torch.zeros((len(q), 8 if cplx else 4), dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    s.direct_sum_device(dV.data_ptr(), dq.data_ptr(), st.cuda_stream)
    st.synchronize()
    V = dV.cpu().numpy()
    return V.view(np.complex128) if cplx else V


def both_walks(w, prec, monkeypatch):
    """The direct sum with every pair once and from both sides."""
    c, q = w.generate()
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("NPME_PAIRS_ONCE", mode)
        with npme_b200.Solver(api.params_from_workload(w, precision=prec)) as s:
            out[mode] = direct(s.setup(c), q)
    return c, q, out["0"], out["1"]


# Lengths: the shortest, every radix (2, 3, 4, 5, 6, 8, 9, 10, 12, 16) and odd
# ones, long ones in each place (2,048 is the longest), and one with a prime
# factor above 5, which the library's own transforms leave to cuFFT.
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("func", ["laplace", "helmholtz"])
@pytest.mark.parametrize("grid,order", [
    ((20, 20, 20), 4), ((24, 36, 60), 4), ((100, 72, 40), 6), ((108, 80, 64), 6),
    ((64, 96, 144), 6), ((180, 48, 200), 6), ((64, 28, 96), 6), ((2048, 32, 36), 6),
    ((32, 2048, 60), 6), ((32, 40, 2048), 6), ((1920, 32, 32), 6), ((32, 36, 2000), 6),
    ((36, 32, 1620), 6)])
def test_transform_lengths(grid, order, func, prec):
    w = system(300, func, grid=grid, order=order)
    c, q = w.generate()
    with npme_b200.Solver(api.params_from_workload(w, precision=prec)) as s:
        V = s.setup(c).calcv(q)
    check(V, ob.calcv(ob.params_from_workload(w), c, q), prec)


# Orders up to 8 accumulate a brick in registers, larger ones in shared memory;
# one point, points that fill one brick (several batches a warp) with two far
# corners, and a uniform system.
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("func", ["laplace", "helmholtz"])
@pytest.mark.parametrize("order", [4, 6, 8, 10])
@pytest.mark.parametrize("shape", ["one", "brick", "uniform"])
def test_spread_orders(shape, order, func, prec):
    w = system({"one": 1, "brick": 2746, "uniform": 1500}[shape], func, order=order)
    c, q = w.generate()
    q = q + 1.5  # one sign: the smooth part is as large as the rest
    if shape == "brick":
        g = np.arange(14) * 0.06 + 5.0
        c[:2744] = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        c[2744:] = [[0.0, 0.0, 0.0], [10.0, 10.0, 10.0]]
    Vo = ob.calcv(ob.params_from_workload(w), c, q)
    with npme_b200.Solver(api.params_from_workload(w, precision=prec)) as s:
        V = s.setup(c).calcv(q)
    if shape == "one":  # a cancellation: against the scale of its terms
        assert np.abs(V - Vo).max() <= TOL[prec][0] * np.abs(q[0])
    else:
        check(V, Vo, prec)


def bspline(P, u):
    """B_P(u + t), t = 0 .. P-1, in 64 bits, [P][len(u)]."""
    x = u + np.arange(P)[:, None]
    b = ((x >= 0) & (x < 1)).astype(float)
    for n in range(2, P + 1):
        below = np.vstack([np.zeros_like(u), b[:-1]])  # B_{n-1}(x - 1)
        b = (x * b + (n - x) * below) / (n - 1)
    return b


# FP32 spreading weights: multiples of 2^-24 whose sum is the FP32 scale exactly; the
# tails (below 2^-7) within half a quantum and a quarter for the rounding of the
# recursion (0.15 in a restatement), so that they keep their digits.
def test_fp32_spreading_weights(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    lib = tmp_path / "libweights.so"
    subprocess.run([nvcc, "-std=c++17", "-O3", "-Xcompiler", "-fPIC", "-shared", "-gencode",
                    "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I" + os.path.join(ROOT, "npme_b200", "csrc"),
                    os.path.join(ROOT, "tests", "user_kernel", "spline_weights.cu"),
                    "-o", str(lib)], check=True)
    run = ctypes.CDLL(str(lib)).spline_weights
    u = np.linspace(0, 1, 20001).astype(np.float32)
    halvings = {0: 0, 1: 0, 2: 1, 3: 2, 4: 2, 5: 2, 11: 4, 13: 4, 14: 4, 15: 4}  # else 3
    for P in (4, 6, 8, 10, 12, 14, 16):
        w = np.empty((P, len(u)), np.float32)
        ptr = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_float)) for a in (u, w)]
        assert run(P, len(u), *ptr) == 0
        w = w.astype(float)
        scale = np.prod([j * 0.5 ** halvings.get(j, 3) for j in range(2, P)])
        assert (np.ldexp(w, 24) % 1 == 0).all()
        assert (w.sum(0) == np.float32(scale)).all()
        exact = scale * bspline(P, np.minimum(u.astype(float), 1 - 2.0 ** -53))
        tail = exact < 2.0 ** -7
        tail[P // 2] = False  # takes the rest
        assert (np.abs(w - exact)[tail] <= 1.25 * 2.0 ** -25).all()


# The FP32 grid of bricks that are taken in many windows (1e5 points of one sign in a
# few bricks), of sheets (one plane of each brick, shared out over the warps) and of
# bricks on both sides of a window: the smooth part against FP64.  Sums in 64-bit
# fixed point, rounded once, are off by up to 3e-7, 7e-7 and 6e-6 at orders 4, 6 and
# 8 (sheets and clusters have a rough grid, whose rounding the division by the
# splines' transform enlarges); FP32 registers without an end were by up to 5e-6,
# 1.3e-5 and 9e-5.
@pytest.mark.parametrize("func", ["laplace", "helmholtz"])
@pytest.mark.parametrize("order,tol", [(4, 1e-6), (6, 1e-6), (8, 1e-5)])
@pytest.mark.parametrize("shape", ["cluster", "sheet0", "sheet1", "sheet2", "window"])
def test_spread_dense_bricks(shape, order, tol, func):
    import torch
    n = 100000 if shape == "cluster" else 60000
    w = system(n, func, order=order, box=(60.0, 60.0, 60.0), grid=(96, 96, 96), Rdir=1.0)
    c, q = w.generate()
    q = np.abs(q.real) + 0.5 + (1j * np.abs(q.imag) if func == "helmholtz" else 0)
    if shape == "cluster":
        c = 31.0 + c / 12.0
    elif shape == "window":  # points within one grid cell each
        m = [1023, 1024, 1025, 2049]
        c, q = c[:sum(m)] / 120.0, q[:sum(m)]
        c += np.repeat([3.0, 20.0, 37.0, 50.0], m)[:, None]
    else:
        c[:, int(shape[5])] = 30.0 + 1e-3 * c[:, int(shape[5])]
    c[:2] = [[0.0] * 3, [60.0] * 3]
    smooth = {}
    for prec in ("fp64", "fp32"):
        with npme_b200.Solver(api.params_from_workload(w, precision=prec)) as s:
            smooth[prec] = s.setup(c).calcv(q) - direct(s, q)
    assert rel(smooth["fp32"], smooth["fp64"]) < tol


# Warps per group of 32 targets: 16 up to 148 groups, 8 up to 592, 4 up to
# 2,960, else one; sources by target halves from 18,944 points (FP64) and
# 94,720 (FP32 r^alpha and Helmholtz).
@pytest.mark.parametrize("func,split,prec,n", [
    (f, s, p, n)
    for f, s, p, sizes in [
        ("laplace", "dm", "fp32", (31, 3000, 15000, 60000, 100001)),
        ("laplace", "orig", "fp32", (31, 15000, 100001)),
        ("ralpha", "dm", "fp32", (31, 3000, 94719, 94720)),
        ("helmholtz", "dm", "fp32", (31, 3000, 15000, 94719, 94720)),
        ("laplace", "dm", "fp64", (31, 3000, 18943, 18944, 100001)),
        ("laplace", "orig", "fp64", (3000, 18944)),
        ("ralpha", "dm", "fp64", (3000, 18943, 18944)),
        ("helmholtz", "dm", "fp64", (31, 3000, 18943, 18944, 100001))]
    for n in sizes])
def test_group_splits_and_zones(func, split, prec, n, monkeypatch):
    side = max(n, 1000) ** (1 / 3)
    w = system(n, func, split, box=(side, 1.5 * side, side / 1.5), Rdir=3.5)
    _, _, two, one = both_walks(w, prec, monkeypatch)
    assert rel(one[:, 0], two[:, 0]) < WALKS[prec]
    assert rel(one[:, 1:], two[:, 1:]) < WALKS[prec]


# The bound of the segment lists (2^31 in all): a set-up just within it, 2.4 million
# points in a thin sheet with a cutoff of 38 column edges, and one beyond.
def test_segment_bound():
    import torch
    if torch.cuda.mem_get_info()[0] < 60e9:
        pytest.skip("needs 60 GB")
    n = 2400000
    c = np.random.default_rng(1).random((n, 3)) * [44.0, 44.0, 0.2]
    c[:2] = [[0.0, 0.0, 0.0], [44.0, 44.0, 0.2]]
    for Rdir, fits in ((19.05, True), (20.0, False)):
        # segments: (n/32 + columns + 1) x the fine columns within reach of a group, squared
        e = np.cbrt(32 * 44.0 * 44.0 * 0.25 * Rdir / n)
        nc = int(np.ceil(44.0 / e))
        bound = (n // 32 + nc * nc + 1) * (int((1 + 2 * Rdir * nc / 44.0) * 2) + 4) ** 2
        assert (bound < 2 ** 31) == fits
        with npme_b200.Solver(api.make_params("laplace", "dm", Rdir, 4, 3, (48, 48, 48))) as s:
            if fits:
                assert s.setup(c).info()["nGroups"] >= n // 32
            else:
                with pytest.raises(api.NPMEError, match="2\\^31"):
                    s.setup(c)


# Zones are built for the walks that use them alone: the others stage the same sources
# whatever the precision (candidates per point), where FP64 1/r leaves some out.
def test_zones_only_where_they_are_walked(monkeypatch):
    def candidates(func, split, prec, once):
        monkeypatch.setenv("NPME_PAIRS_ONCE", once)
        w = system(20000, func, split, box=(27.0, 27.0, 27.0), Rdir=3.5)
        with npme_b200.Solver(api.params_from_workload(w, precision=prec)) as s:
            return s.setup(w.generate()[0]).info()["pairsOnceCandidatesPerPoint"]
    plain = candidates("laplace", "dm", "fp32", "1")  # no zones at this size
    assert candidates("laplace", "dm", "fp64", "1") < 0.97 * plain
    assert candidates("laplace", "orig", "fp64", "1") == plain
    assert candidates("laplace", "dm", "fp64", "0") == plain


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("alpha,nd", [(1.0, 6), (3.0, 3), (0.5, 8), (-3.0, 6), (-2.5, 10),
                                      (-1.0, 3)])
def test_exponents(alpha, nd, prec, monkeypatch):
    w = system(2500, "ralpha", alpha=alpha, nDeriv=nd)
    c, q, two, one = both_walks(w, prec, monkeypatch)
    Vo = ob.direct(ob.params_from_workload(w), c, q)
    for V in (two, one):
        check(V, Vo, prec)


# Damped waves, and |k0| Rdir on both sides of 1e5, above which the FP64 pairs
# are evaluated from both sides with the library's sine and cosine.  At order 2
# the matched polynomial's terms reach (k0 Rdir)^2 times the sum, so the walks
# differ by their rounding (eps 1e10 at most), relative to the polynomial.
@pytest.mark.parametrize("k0,nd,tol", [(0.5, 6, 1e-13), (1.1 + 0.2j, 8, 1e-12),
                                       (3.0 - 0.4j, 4, 1e-12), (0.5, 3, 1e-13),
                                       (0.5, 5, 1e-13), (0.5, 15, 1e-11), (24999.0, 2, 1e-9),
                                       (25001.0, 2, 1e-9)])
def test_fp64_helmholtz_wave_numbers(k0, nd, tol, monkeypatch):
    w = system(1500, "helmholtz", k0=k0, nDeriv=nd)
    c, q, two, one = both_walks(w, "fp64", monkeypatch)
    assert rel(one, two) < tol
    with npme_b200.Solver(api.params_from_workload(w, precision="fp64")) as s:
        assert s.setup(c).info()["pairsOnce"] == (abs(k0) < 25000)
    if abs(k0) < 100:
        Vo = ob.direct(ob.params_from_workload(w), c, q)
        assert rel(one, Vo) < 10 * tol


# The two parts of FP64 Helmholtz carry the same matching polynomial, also where
# its coefficients cancel (1e3 times the sum at |k0| Rdir = 10): their rounding,
# eps times that (4e-14 at order 8, 1.6e-13 at 10), must not show in the total,
# whose own rounding is 5e-15 and 1e-14.
@pytest.mark.parametrize("k0,Rdir,nd,order,tol", [(0.5, 4.0, 6, 6, 1e-14),
                                                  (0.85, 12.0, 8, 8, 2.5e-14),
                                                  (0.85, 12.0, 10, 8, 6e-14)])
def test_fp64_helmholtz_parts_match(k0, Rdir, nd, order, tol):
    w = system(1500, "helmholtz", k0=k0, Rdir=Rdir, nDeriv=nd, order=order, grid=(64, 64, 64))
    c, q = w.generate()
    with npme_b200.Solver(api.params_from_workload(w, precision="fp64")) as s:
        V = s.setup(c).calcv(q)
    assert rel(V, ob.calcv(ob.params_from_workload(w), c, q)) < tol


# The same for 1/r and r^alpha, at cutoffs whose powers are not exact: were one part's
# coefficients rounded in another form, the total would be off by 3e-14 to 1e-13 at
# order 10, 2e-13 to 3e-13 at 12 and 3e-12 at 15.  The oracle's own rounding of its
# coefficients of r^2n is 4e-15, 2e-14 and 1e-13; three times that is allowed.
@pytest.mark.parametrize("once", ["1", "0"])
@pytest.mark.parametrize("nd,tol", [(10, 1.4e-14), (12, 6e-14), (15, 3e-13)])
@pytest.mark.parametrize("Rdir", [5.3, 7.123])
@pytest.mark.parametrize("func", ["laplace", "ralpha"])
def test_fp64_real_parts_match(func, Rdir, nd, tol, once, monkeypatch):
    monkeypatch.setenv("NPME_PAIRS_ONCE", once)
    w = system(3000, func, Rdir=Rdir, nDeriv=nd, order=8, grid=(64, 64, 64),
               box=(16.0, 16.0, 16.0))
    c, q = w.generate()
    with npme_b200.Solver(api.params_from_workload(w, precision="fp64")) as s:
        V = s.setup(c).calcv(q)
    assert rel(V, ob.calcv(ob.params_from_workload(w), c, q)) < tol


# Near pairs in FP64, 1e-5 apart, on coordinates of 35 bits: offsets from a group's
# centre are exact, so the gradient, which is the sum here, has the rounding of its
# formula (1e-15).  A coordinate scaled by 1/Rdir before the subtraction would leave
# 1e-16 / 1e-5.
@pytest.mark.parametrize("once", ["1", "0"])
@pytest.mark.parametrize("n", [600, 20000])
@pytest.mark.parametrize("func", ["laplace", "ralpha", "helmholtz"])
def test_fp64_near_pairs(func, n, once, monkeypatch):
    monkeypatch.setenv("NPME_PAIRS_ONCE", once)
    w = system(n, func, Rdir=2.3, box=(n ** (1 / 3),) * 3)
    c, q = w.generate()
    d = np.random.default_rng(5).standard_normal((n // 2, 3))
    c[1::2] = c[0::2] + 1e-5 * d / np.linalg.norm(d, axis=1)[:, None]
    c = np.ldexp(np.round(np.ldexp(c, 30)), -30)
    with npme_b200.Solver(api.params_from_workload(w, precision="fp64")) as s:
        V = direct(s.setup(c), q)
    assert rel(V, ob.direct(ob.params_from_workload(w), c, q)) < 1e-14


# The exact sum: partial groups, coincident points (whose gradients are not
# finite) and target subsets, which divide the sources among several CTAs.
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("func,alpha", [("laplace", -1.0), ("ralpha", 2.0), ("helmholtz", -1.0)])
@pytest.mark.parametrize("n", [1, 2, 33, 257, 5001])
def test_exact_sum_shares(n, func, alpha, prec):
    w = system(n, func, alpha=alpha)
    c, q = w.generate()
    q = q + 0.5
    same = [0, n // 2, n - 1] if n > 2 else []
    c[same] = c[:1]
    targets = np.unique(np.linspace(0, n - 1, 37).astype(np.uint32))
    with npme_b200.Solver(api.params_from_workload(w, precision=prec)) as s:
        s.setup(c)
        V, Vs = s.calcv_exact(q), s.calcv_exact_subset(targets, q)
        V1 = s.calcv_exact_subset(targets[-1:], q)
    Vo = ob.exact(ob.params_from_workload(w), c, q)
    single = np.setdiff1d(np.arange(n), same)
    scale = np.abs(Vo[single]).max() if n > 1 else 1.0
    for got, rows in ((V, np.arange(n)), (Vs, targets), (V1, targets[-1:])):
        ok = np.isin(rows, single)
        assert (np.abs(got[ok] - Vo[rows[ok]]) <= 1e-12 * scale).all()
        assert not np.isfinite(got[~ok, 1:]).any()


# A non-finite charge reaches the points within the cutoff and no others.
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("func,split,prec", [
    ("laplace", "dm", "fp32"), ("laplace", "orig", "fp32"), ("ralpha", "dm", "fp32"),
    ("helmholtz", "dm", "fp32"), ("laplace", "dm", "fp64"), ("ralpha", "dm", "fp64"),
    ("helmholtz", "dm", "fp64")])
@pytest.mark.parametrize("n", [3000, 20000])
def test_non_finite_charge_stays_local(n, func, split, prec, bad):
    side = n ** (1 / 3)
    w = system(n, func, split, box=(side, side, side), Rdir=3.5)
    c, q = w.generate()
    k = n // 3
    with npme_b200.Solver(api.params_from_workload(w, precision=prec)) as s:
        s.setup(c)
        q[k] = 0.0
        V0 = direct(s, q)
        q[k] = bad
        V = direct(s, q)
    r = np.linalg.norm(c - c[k], axis=1)
    far = r > w.Rdir * (1 + 1e-6)
    assert rel(V[far], V0[far]) < WALKS[prec]
    assert not np.isfinite(V[(r > 0) & (r < 0.9 * w.Rdir), 0]).any()


# Batches: the members' classes (function, order, exponent) with few and many
# groups, beside each other, against each member's own CalcV.
def test_batch_classes():
    import torch
    members = [system(40), system(1200, order=8, nDeriv=8), system(9000, box=(20.0, 20.0, 20.0)),
               system(40000, box=(33.0, 33.0, 33.0), grid=(64, 80, 96)),
               system(3000, split="orig"), system(2000, "ralpha"),
               system(2000, "ralpha", alpha=2.0),
               system(2500, "helmholtz"), system(12000, "helmholtz", box=(20.0, 20.0, 24.0)),
               system(1000, grid=(56, 48, 44))]
    solvers, qs, outs, alone = [], [], [], []
    for w in members:
        c, q = w.generate()
        s = npme_b200.Solver(api.params_from_workload(w, precision="fp32")).setup(c)
        alone.append(s.calcv(q))
        solvers.append(s)
        qs.append(torch.from_numpy(np.ascontiguousarray(q)).cuda())
        outs.append(torch.empty((w.n, 8 if np.iscomplexobj(q) else 4), dtype=torch.float64,
                                device="cuda"))
    torch.cuda.synchronize()
    b = api.Batch()
    b.calcv(solvers, [o.data_ptr() for o in outs], [q.data_ptr() for q in qs])
    b.sync()
    for o, V in zip(outs, alone):
        got = o.cpu().numpy()
        got = got.view(np.complex128) if np.iscomplexobj(V) else got
        assert rel(got[:, 0], V[:, 0]) < 1e-6 and rel(got[:, 1:], V[:, 1:]) < 1e-6
    b.close()
    for s in solvers:
        s.close()
