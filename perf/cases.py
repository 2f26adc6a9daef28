"""The work a user of the library has it do, as cases that can be timed and compared.

Two kinds of case, both through the Python binding of the C ABI (host arrays in, host arrays out):
  solve  one frequency (``Context.solve_frequency``) or a sweep (``Context.solve_batch``) of a deck of
         one or more bodies: Green functions, assembly, linear solve, force reductions, and the
         field-point potentials where the deck asks for them;
  green  ``Context.eval_green``, the Green function at point pairs a user hands over.
The bodies are those of ``meshgen`` (cylinders and boxes) at the sizes of the decks under tests/golden
and of the benchmark arrays; lengths, depths, frequencies and headings move a little with the seed.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hams-mrel_b200"))
import hams_b200  # noqa: E402
import meshgen  # noqa: E402

G0 = 9.81


def _solve(name, **kw):
    """A solve case with its defaults: one cylinder of 234 panels in 70 m, one frequency, fp64, LU."""
    case = dict(name=name, kind="solve", form="fp64", shape="cylinder", nx=1, ny=1, radius=5.0, draft=10.0, pitch=20.0,
                n_theta=18, n_z=9, n_r=4, depth=70.0, lids=False, blocks=False, nfreq=1, w0=0.9, w1=0.9, nbeta=1,
                field=0)
    case.update(kw)
    return case


def listed():
    return [
        # Green functions at a handful of pairs, near and far: a host loop that probes the kernel
        dict(name="green_64", kind="green", n=64, depth=50.0, rmin=1e-4, rmax=2.0, omega=1.1),
        # a table of Green functions over an odd number of pairs, as a host-side assembly asks for it
        dict(name="green_200k", kind="green", n=200003, depth=50.0, rmin=0.05, rmax=2.0, omega=1.1),
        # the smallest deck: one body of 234 panels in 70 m of water, one frequency
        _solve("one_body"),
        # three bodies of 234 panels, 12 frequencies, three headings: an ordinary interaction deck
        _solve("three_bodies_sweep", nx=3, pitch=30.0, nfreq=12, w0=0.3, w1=1.8, nbeta=3),
        # one body of 800 panels in infinite depth over a sweep
        _solve("deep_water_sweep", n_theta=40, n_z=15, n_r=5, depth=-1.0, nfreq=15, w0=0.1, w1=3.0),
        # a cylinder and a box with water-plane lids against irregular frequencies, mixed precision
        _solve("lids_mixed", form="mixed", shape="both", nx=2, radius=6.0, draft=7.0, pitch=50.0, n_theta=28, n_z=13,
               n_r=9, depth=60.0, lids=True, nfreq=4, w0=0.5, w1=1.7),
        # ten bodies of 234 panels in 14.5 m, twelve headings, pressures wanted at 100 points of the fluid
        _solve("field_points", nx=5, ny=2, radius=3.0, draft=5.0, pitch=15.0, depth=14.5, nfreq=2, w0=0.7, w1=1.3,
               nbeta=12, field=100),
        # four bodies of 600 panels with the iterative solver (ACA products, block preconditioner)
        _solve("array_gmres", form="gmres", nx=2, ny=2, radius=4.0, draft=8.0, pitch=30.0, n_theta=40, n_z=10, n_r=5,
               depth=40.0, w0=1.0, w1=1.0, nbeta=4),
        # the benchmark array (3 x 3 bodies of 600 panels), one frequency in plain FP64, every pair computed
        _solve("array_fp64", nx=3, ny=3, radius=4.0, draft=8.0, n_theta=40, n_z=10, n_r=5, depth=50.0, w0=1.2,
               w1=1.2, nbeta=4),
        # the same array, one frequency in mixed precision, identical body pairs computed once
        _solve("array_mixed", form="mixed", nx=3, ny=3, radius=4.0, draft=8.0, n_theta=40, n_z=10, n_r=5, depth=50.0,
               blocks=True, w0=1.5, w1=1.5, nbeta=4),
        # the benchmark's own form: the judged surrogate over a sweep of the array
        _solve("array_surrogate_sweep", form="surrogate", nx=3, ny=3, radius=4.0, draft=8.0, n_theta=40, n_z=10,
               n_r=5, depth=50.0, blocks=True, nfreq=10, w0=0.2, w1=2.2, nbeta=4),
        # the farm: 6 x 6 bodies of 560 panels (20,160), one frequency
        _solve("farm_mixed", form="mixed", nx=6, ny=6, radius=3.0, draft=6.0, pitch=12.0, n_theta=40, n_z=9, n_r=5,
               depth=40.0, blocks=True, w0=1.0, w1=1.0, nbeta=3),
    ]


def draw(rng):
    """Another case of the same ranges: a table of Green functions, or a deck of 1 to 9 bodies of about 80 to
    800 panels (at most 4,000 in all) in 0.9 m (model scale) to 200 m or infinite depth."""
    if rng.random() < 0.15:
        near = rng.random() < 0.3
        n = int(round(math.exp(rng.uniform(math.log(50), math.log(3000 if near else 200000)))))
        return dict(kind="green", n=n, depth=round(rng.uniform(12.0, 150.0), 2), rmin=1e-4 if near else 0.05,
                    rmax=round(rng.uniform(1.0, 3.0), 2), omega=round(rng.uniform(0.4, 2.0), 3))
    nx, ny = rng.choice([(1, 1), (1, 1), (2, 1), (2, 1), (3, 1), (2, 2), (5, 1), (3, 2), (3, 3)])
    nb = nx * ny
    per = min(800.0, 4000.0 / nb, math.exp(rng.uniform(math.log(80), math.log(800))))
    n_theta = 2 * max(4, int(round(math.sqrt(per / 2.5) * rng.uniform(0.8, 1.2))))
    rows = max(4, int(per / n_theta))
    n_r = max(2, int(rows * rng.uniform(0.25, 0.4)))
    scale = 0.05 if rng.random() < 0.15 else 1.0  # model scale: example decks at 0.9 m
    radius = rng.uniform(3.0, 8.0)
    draft = radius * rng.uniform(0.8, 2.0)
    depth = -1.0 if rng.random() < 0.25 else min(200.0, max(18.0, 1.35 * draft) * math.exp(rng.uniform(0.0, 2.4)))
    form = rng.choice(["fp64", "fp64", "fp64", "mixed", "mixed", "mixed", "surrogate", "gmres"])
    if form == "surrogate" and (depth < 0 or draft > 0.45 * depth):
        form = "mixed"  # the network serves finite depth and the upper half of the water
    lids = form in ("fp64", "mixed") and rng.random() < 0.25
    shape = rng.choice(["cylinder", "cylinder", "box"])
    w0 = rng.uniform(0.3, 1.4) / math.sqrt(scale)
    nfreq = 1 if form == "gmres" else rng.choice([1, 1, 2, 3, 5, 8])
    return dict(kind="solve", form=form, shape=shape, nx=nx, ny=ny, radius=round(radius * scale, 4),
                draft=round(draft * scale, 4), pitch=round(radius * rng.uniform(2.8, 6.0) * scale, 4),
                n_theta=n_theta, n_z=rows - n_r, n_r=n_r, depth=round(depth * scale, 4) if depth > 0 else -1.0,
                lids=lids, blocks=nb > 1 and not lids and rng.random() < 0.5, nfreq=nfreq, w0=round(w0, 4),
                w1=round(w0 * (rng.uniform(1.2, 1.9) if nfreq > 1 else 1.0), 4), nbeta=rng.choice([1, 1, 2, 4, 7]),
                field=rng.choice([0, 0, 0, 0, 37, 150]))


def _points(case, seed):
    """Point pairs (xq, yq, zq, xp, yp, zp) and near/far flags: horizontal distances spread over
    [rmin, rmax] depths (over their logarithm where that is more than a factor of a hundred), depths in
    the upper 40 % of the water."""
    r, n, h = np.random.RandomState(seed % (1 << 31)), case["n"], case["depth"]
    lo, hi = case["rmin"], case["rmax"]
    d = np.exp(r.uniform(math.log(lo), math.log(hi), n)) if hi > 100 * lo else r.uniform(lo, hi, n)
    th = r.uniform(0.0, 2.0 * math.pi, n)
    pts = np.zeros((n, 6), order="F")
    pts[:, 0], pts[:, 1] = r.uniform(-h, h, n), r.uniform(-h, h, n)
    pts[:, 3], pts[:, 4] = pts[:, 0] + d * h * np.cos(th), pts[:, 1] + d * h * np.sin(th)
    pts[:, 2], pts[:, 5] = r.uniform(-0.4 * h, -0.01 * h, n), r.uniform(-0.4 * h, -0.01 * h, n)
    return pts, (r.uniform(size=n) < 0.5).astype(np.int32), case["omega"] * r.uniform(0.97, 1.03)


def _deck(case, rng):
    """Bodies, lids and centres of a solve case; lengths move by up to 2 % with the seed."""
    j = lambda x: x * (1.0 + 0.02 * rng.uniform(-1.0, 1.0))
    radius, draft, pitch = j(case["radius"]), j(case["draft"]), j(case["pitch"])
    nt, nz, nr = case["n_theta"], case["n_z"], case["n_r"]
    bodies, lids, centres = [], [], []
    for iy in range(case["ny"]):
        for ix in range(case["nx"]):
            x, y = pitch * ix, pitch * iy
            if case["shape"] == "box" or (case["shape"] == "both" and (ix + iy) % 2):
                nl, nb = max(2, nt // 3), max(2, nt // 6)
                bodies.append(meshgen.box(2.0 * radius, radius, draft, nl, nb, nz, x, y))
                lids.append(meshgen.rect_lid(1.96 * radius, 0.98 * radius, max(1, nl // 2), max(1, nb // 2), x, y))
            else:
                bodies.append(meshgen.cylinder(radius, draft, nt, nz, nr, x, y))
                lids.append(meshgen.disc_lid(radius, nt, max(1, nr // 2), x, y))
            centres.append((x, y, 0.0))
    return bodies, lids, np.array(centres), radius, draft


class _State:
    """What a program keeps between calls: the context (freed with the state), waves, headings or points."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    rng = random.Random(seed)
    if case["kind"] == "green":
        pts, flag, omega = _points(case, seed)
        xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(4.0, 4.0, 8, 2, 2)])
        geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((1, 3)))
        ctx = hams_b200.Context(geom, case["depth"], rho=1025.0, g=G0)
        return _State(kind="green", ctx=ctx, wave=ctx.wave(omega), pts=pts, flag=flag)
    bodies, lids, centres, radius, draft = _deck(case, rng)
    xyz, ncn, ncon, cnt = meshgen.combine(bodies)
    geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, centres)
    if case["lids"]:
        lx, ln, lc, lcnt = meshgen.combine(lids)
        geom["ixyz_p"] = hams_b200.prepare_geometry(lx, ln, lc, lcnt, centres)["xyz_p"]
    form = case["form"]
    ctx = hams_b200.Context(geom, case["depth"], rho=1025.0, g=G0, irsp=1 if case["lids"] else 0,
                            precision=hams_b200.PREC_MIXED if form in ("mixed", "surrogate") else hams_b200.PREC_FP64,
                            solver=hams_b200.SOLVER_GMRES if form == "gmres" else hams_b200.SOLVER_LU,
                            body_blocks=1 if case["blocks"] else 0)
    if form == "surrogate":
        params = np.fromfile(os.path.join(os.path.dirname(hams_b200.__file__), "surrogate_w128x4.f32"), dtype=np.float32)
        ctx.set_surrogate(params, hams_b200.SURROGATE_FAR, hams_b200.SURROGATE_K_RANGE)
        ctx.set_surrogate_tolerance(hams_b200.SURROGATE_TOL)
    if case["field"]:
        # points of the fluid between and around the bodies, below every draft where the depth allows it
        m, low = case["field"], (0.97 * case["depth"] if case["depth"] > 0 else 3.0 * draft)
        span = np.abs(centres).max() + 3.0 * radius
        p = np.array([[rng.uniform(-3.0 * radius, span), rng.uniform(-3.0 * radius, span),
                       -rng.uniform(min(1.1 * draft, 0.9 * low), low)] for _ in range(m)])
        ctx.set_field_points(p)
    om = np.linspace(case["w0"], case["w1"], case["nfreq"]) * rng.uniform(0.98, 1.02)
    betas = [rng.uniform(0.0, 2.0 * math.pi) for _ in range(case["nbeta"])]
    return _State(kind="solve", ctx=ctx, waves=[ctx.wave(w) for w in om], betas=betas, field=case["field"])


def run(state):
    if state.kind == "green":
        return state.ctx.eval_green(state.wave, state.pts, state.flag)
    if len(state.waves) == 1:
        out = list(state.ctx.solve_frequency(state.waves[0], state.betas))
    else:
        out = list(state.ctx.solve_batch(state.waves, state.betas))
    if state.field:
        out += [state.ctx.field_potentials(len(state.betas), k) for k in range(len(state.waves))]
    return out


def _pair_flops(depth):
    """Operations of one pair's Green function and gradient: in finite depth about 30 modes (three terms of
    4 operations) and three epsilon tables of about 30 x 30 / 2 entries at 3 operations (the Bessel functions
    belong to a distance, not to a pair); in infinite depth the polynomials of the approximation."""
    return 400.0 if depth < 0 else 30 * 12 + 3 * 450 * 3


def work(case):
    """Inputs and outputs once, the pairs' Green functions (copied blocks of identical bodies not counted),
    the complex LU (8/3 n^3) and its solves; GMRES as 30 dense products per right-hand side instead."""
    if case["kind"] == "green":
        return dict(bytes=case["n"] * (6 * 8 + 4 + 64), flops=case["n"] * _pair_flops(case["depth"]))
    nb = case["nx"] * case["ny"]
    cyl = case["n_theta"] * (case["n_z"] + case["n_r"])
    nl, nw = max(2, case["n_theta"] // 3), max(2, case["n_theta"] // 6)
    box = 2 * case["n_z"] * (nl + nw) + nl * nw
    per = {"cylinder": cyl, "box": box, "both": (cyl + box) / 2}[case["shape"]]
    n, nrhs = per * nb, 6 * nb + case["nbeta"]
    lid = 0.2 * n if case["lids"] else 0
    blocks = (2 * case["nx"] - 1) * (2 * case["ny"] - 1) if case["blocks"] else nb * nb
    solve = 30 * 8.0 * n * n * nrhs if case["form"] == "gmres" else 8.0 / 3.0 * n ** 3 + 8.0 * n * n * nrhs
    flops = per * per * blocks * (1 + lid / n) * _pair_flops(case["depth"]) + solve + 8.0 * n * n * lid
    flops += 8.0 * 2 * case["field"] * n * nrhs
    byts = n * 200 + case["nfreq"] * (16.0 * 36 * nb * nb + 16.0 * 6 * nb * case["nbeta"] + 16.0 * case["field"] * nrhs)
    return dict(bytes=byts, flops=case["nfreq"] * flops)


def _roots(v, h, m):
    """k0 of k tanh(kh) = v and the first m roots of k tan(kh) = -v."""
    k = max(v, math.sqrt(v / h))
    for _ in range(100):
        t = math.tanh(k * h)
        k -= (k * t - v) / (t + k * h * (1.0 - t * t))
    n = np.arange(1, m + 1)
    a, b = (n - 0.5) * math.pi / h, n * math.pi / h
    for _ in range(200):
        c = 0.5 * (a + b)
        up = c * np.sin(c * h) * np.cos(n * math.pi) + v * np.cos(c * h) * np.cos(n * math.pi) > 0.0
        a, b = np.where(up, a, c), np.where(up, c, b)
    return k, 0.5 * (a + b)


def exact(case, seed):
    """The eigenfunction (John) series of the finite-depth Green function, summed in 64 bits, for tables of
    pairs at R/h >= 0.05, where 190 modes reach rounding.  Closer pairs and the solves have no such value:
    the Green functions they are built on are defined by truncated, extrapolated and fitted series
    (FinGreen3D, HavelockGF), whose own error is far above rounding."""
    if case["kind"] != "green" or case["rmin"] < 0.05:
        return None
    pts, flag, omega = _points(case, seed)
    h, v = case["depth"], omega * omega / G0
    k0, km = _roots(v, h, 190)
    dx, dy = pts[:, 0] - pts[:, 3], pts[:, 1] - pts[:, 4]
    zq, zp, r = pts[:, 2], pts[:, 5], np.hypot(dx, dy)
    tb = torch.special
    fn = lambda f, x: f(torch.from_numpy(np.ascontiguousarray(x))).numpy()
    p = math.pi / (h / 2.0 * (1.0 + math.sinh(2.0 * k0 * h) / (2.0 * k0 * h))) * np.cosh(k0 * (zp + h))
    hank0 = -fn(tb.bessel_y0, k0 * r) + 1j * fn(tb.bessel_j0, k0 * r)
    hank1 = -fn(tb.bessel_y1, k0 * r) + 1j * fn(tb.bessel_j1, k0 * r)
    g = p * np.cosh(k0 * (zq + h)) * hank0
    gr = -k0 * p * np.cosh(k0 * (zq + h)) * hank1
    gz = k0 * p * np.sinh(k0 * (zq + h)) * hank0
    for k in km:
        c = 4.0 / (h * (1.0 + math.sin(2.0 * k * h) / (2.0 * k * h))) * np.cos(k * (zp + h))
        b0, b1 = fn(tb.modified_bessel_k0, k * r), fn(tb.modified_bessel_k1, k * r)
        g += c * np.cos(k * (zq + h)) * b0
        gr -= c * k * np.cos(k * (zq + h)) * b1
        gz -= c * k * np.sin(k * (zq + h)) * b0
    gx, gy = gr * dx / r, gr * dy / r
    near, rr = flag == 1, np.sqrt(r * r + (zq - zp) ** 2)  # near pairs leave 1/r to the panel integrals
    for out, d in ((g, 1.0 / rr), (gx, -dx / rr ** 3), (gy, -dy / rr ** 3), (gz, -(zq - zp) / rr ** 3)):
        out[near] -= d[near]
    return np.asfortranarray(np.stack([g, gx, gy, gz], axis=1))
