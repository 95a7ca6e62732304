"""The work a user of momwire_b200 has it do, as measurable cases.

``listed()`` names the standing cases, ``draw(rng)`` makes one more of the
same ranges; ``prepare`` builds what a program holds before the call (the
solver objects, or host arrays for the block sampler), ``run`` makes one pass
through the public entry points, ``work`` counts what a pass cannot do
without and ``exact`` restates a pass in plain float64 torch / numpy.

Antenna programs keep one ``BSplineSolver`` per structure and step the
frequency (``compute_port_solution_swept``, ``compute_y_matrix_swept``), or
hand many structures to ``sweep.grouped_mixed_sweep``; H-matrix hosts call
the off-edge block assembler with host arrays.  Sizes are those of the
repository's configurations, tests and benchmark: a 21-segment dipole up to
the 16 x 16 array of 41-segment dipoles (10,496 unknowns, 256 ports).
"""

import functools
import math

import numpy as np
import torch

from momwire_b200 import BSplineSolver, accel, sweep

C_LIGHT = 299_792_458.0
EPS, MU = 8.8541878188e-12, 1.25663706127e-6  # the solver's own constants
C_SOLVER = 1.0 / math.sqrt(EPS * MU)
N_QP = 4  # the solver's default pair quadrature


def listed():
    return [
        # a single 21-segment dipole at one frequency: the smallest call, all latency
        dict(name="dipole_21", kind="array", nx=1, ny=1, nseg=21, degree=2, precision="fp64", nk=1),
        # a Yagi over perfect ground with the extended kernel, two frequencies: an ordinary small design
        dict(name="yagi_ek_pec", kind="yagi", elements=6, nseg=51, ek=True, pec=True, nk=2),
        # ground-plane vertical with sixteen copper radials, degree 1, reflection-coefficient ground (junction KCL)
        dict(name="radials_refl", kind="radials", radials=16, nseg=23, degree=1, loaded=True, nk=2),
        # inverted V over Sommerfeld ground, the upper end of the Sommerfeld workload's segment counts
        dict(name="vee_sommerfeld", kind="vee", nseg=200, precision="fp64", nk=1),
        # wire-grid plate with a monopole over Sommerfeld ground: hundreds of KCL rows beside the ports
        dict(name="plate_sommerfeld", kind="plate", cells=20, jports=3, precision="fp64"),
        # an 8 x 8 dipole array, every element a port: a mid-size dense solve in the default precision
        dict(name="array_8x8", kind="array", nx=8, ny=8, nseg=41, degree=2, precision="fp64", nk=1),
        # the 16 x 16 array in the default precision: the largest solve of the benchmark
        dict(name="array_16x16", kind="array", nx=16, ny=16, nseg=41, degree=2, precision="fp64", nk=1),
        # an odd-sided array in mixed precision
        dict(name="array_7x9_mixed", kind="array", nx=7, ny=9, nseg=45, degree=2, precision="mixed", nk=1),
        # the 16 x 16 array in mixed precision: the benchmark's headline step
        dict(name="array_16x16_mixed", kind="array", nx=16, ny=16, nseg=41, degree=2, precision="mixed", nk=1),
        # one Yagi's Y matrix over 64 frequencies in the default precision
        dict(name="yagi_sweep", kind="sweep", elements=6, nseg=51, precision="fp64", pec=False, nk=64),
        # many Yagis x 64 frequencies through the grouped sweep: the benchmark's sweep workload, a share of it
        dict(name="yagi_group_sweep", kind="group", structures=24, nk=64),
        # one admissible block of an H-matrix host, asked for whole
        dict(name="offedge_block", kind="block", n_i=1025, n_j=1311, degree=2),
    ]


def _odd(n):
    return int(n) | 1


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["array", "array", "array", "yagi", "radials", "vee", "plate", "sweep", "group", "block"])
    if kind == "array":
        # unknowns over the whole range, on their logarithm
        n = _log_int(rng, 21, 10496)
        nseg = rng.randint(11, 61)
        side = max(1, min(256, n // nseg))
        nx = max(1, min(16, int(round(math.sqrt(side) * rng.uniform(0.7, 1.4)))))
        ny = max(1, min(16, side // nx))
        nseg = max(8, min(nseg, 10496 // (nx * ny)))
        return dict(kind=kind, nx=nx, ny=ny, nseg=nseg, degree=rng.choice([1, 2, 2]),
                    precision=rng.choice(["fp64", "mixed"]), nk=1)
    if kind == "yagi":
        return dict(kind=kind, elements=rng.randint(3, 12), nseg=_odd(rng.randint(11, 100)),
                    ek=rng.choice([True, False]), pec=rng.choice([True, False]), nk=rng.randint(1, 3))
    if kind == "radials":
        return dict(kind=kind, radials=rng.randint(4, 32), nseg=rng.randint(6, 40), degree=rng.choice([1, 2]),
                    loaded=rng.choice([True, False]), nk=rng.randint(1, 3))
    if kind == "vee":
        return dict(kind=kind, nseg=2 * rng.randint(10, 100), precision=rng.choice(["fp64", "mixed"]), nk=1)
    if kind == "plate":
        return dict(kind=kind, cells=rng.randint(6, 22), jports=rng.randint(1, 5),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "sweep":
        return dict(kind=kind, elements=rng.randint(3, 10), nseg=_odd(rng.randint(11, 70)),
                    precision=rng.choice(["fp64", "mixed"]), pec=rng.choice([True, False]), nk=rng.randint(8, 64))
    if kind == "group":
        return dict(kind=kind, structures=rng.randint(6, 24), nk=rng.randint(16, 64))
    return dict(kind="block", n_i=_log_int(rng, 40, 1600), n_j=_log_int(rng, 40, 1600), degree=rng.choice([1, 2]))


# ------------------------------------------------------------- structures
def _array(case, rng):
    """nx x ny z-directed dipoles at half-wave pitch, centre-fed, lengths
    jittered by 1 %."""
    lam = C_LIGHT / 300e6
    wires = []
    for ix in range(case["nx"]):
        for iy in range(case["ny"]):
            L = 0.48 * lam * (1 + rng.uniform(-0.01, 0.01))
            x, y = ix * 0.5 * lam, iy * 0.5 * lam
            wires.append(np.array([[x, y, -L / 2], [x, y, L / 2]]))
    return dict(wires=wires, nsegs=case["nseg"], degree=case["degree"], wire_radius=0.5e-3, wavelength=lam,
                feeds=[(w, None, 1.0) for w in range(len(wires))])


def _yagi(rng, elements, npe, ek=False, pec=False):
    """Parallel z-directed elements along x, the second one fed; over perfect
    ground the lowest tip is 0.1 wavelength above it."""
    lam = C_LIGHT / 28e6
    x, wires = 0.0, []
    z0 = 0.4 * lam if pec else 0.0
    for e in range(elements):
        if e:
            x += rng.uniform(0.10, 0.30) * lam
        L = rng.uniform(0.40, 0.55) * lam
        wires.append(np.array([[x, 0.0, z0 - L / 2], [x, 0.0, z0 + L / 2]]))
    kw = dict(wires=wires, n_per_edge_per_wire=npe, degree=2, wavelength=lam, feeds=[(1, None, 1.0)],
              wire_radius=float(np.exp(rng.uniform(np.log(0.5e-3), np.log(10e-3)))), extended_kernel=ek)
    if pec:
        kw["ground_z"] = 0.0
    return kw


def _radials(case, rng):
    lam = C_LIGHT / 14.1e6
    base = np.array([0.0, 0.0, 0.06 * lam * (1 + rng.uniform(-0.05, 0.05))])
    n = case["radials"]
    wires = [np.array([base, base + [0.0, 0.0, 0.25 * lam * (1 + rng.uniform(-0.02, 0.02))]])]
    for i in range(n):
        a, L = 2.0 * np.pi * i / n, 0.25 * lam * (1 + rng.uniform(-0.02, 0.02))
        wires.append(np.array([base, base + L * np.array([np.cos(a), np.sin(a), -0.1])]))
    kw = dict(wires=wires, nsegs=case["nseg"], degree=case["degree"], wire_radius=1e-3, wavelength=lam,
              junctions=[[(w, "start") for w in range(n + 1)]], feeds=[(0, 0.5 * 0.25 * lam / case["nseg"], 1.0)],
              ground_z=0.0, ground_eps=(13.0, 0.005))
    if case["loaded"]:
        kw["wire_conductivity"] = 5.8e7
    return kw


def _vee(case, rng):
    lam = C_LIGHT / 14.1e6
    apex = np.radians(rng.uniform(100.0, 140.0))
    leg = 0.25 * lam
    dz, dy = leg * np.cos(apex / 2), leg * np.sin(apex / 2)
    top = np.array([0.0, 0.0, 0.15 * lam + dz])
    n = case["nseg"] // 2
    return dict(wires=[np.array([top - [0.0, dy, dz], top, top + [0.0, dy, -dz]])], n_per_edge_per_wire=[[n, n]],
                degree=2, wire_radius=1e-3, wavelength=lam, ground_z=0.0, ground_eps=(13.0, 0.005),
                ground_model="sommerfeld")


def _plate(case, rng):
    """Square wire grid, two segments per cell edge, over Sommerfeld ground
    with a monopole from its centre node and a few junction ports."""
    m, lam = case["cells"] + 1, C_LIGHT / 14.1e6
    size, z = 10.0 * (1 + rng.uniform(-0.02, 0.02)), 2.0
    step = size / case["cells"]
    xy = lambda i, j: (-size / 2 + i * step, -size / 2 + j * step, z)  # noqa: E731
    wires, nodes = [], {}
    for di, dj in ((1, 0), (0, 1)):
        for j in range(m - dj):
            for i in range(m - di):
                wires.append(np.array([xy(i, j), xy(i + di, j + dj)]))
                nodes.setdefault((i, j), []).append((len(wires) - 1, "start"))
                nodes.setdefault((i + di, j + dj), []).append((len(wires) - 1, "end"))
    c = (case["cells"] // 2, case["cells"] // 2)
    cx, cy, _ = xy(*c)
    wires.append(np.array([(cx, cy, z), (cx, cy, z + 10.0)]))
    nodes[c].append((len(wires) - 1, "start"))
    keys = sorted(nodes)
    cand = [i for i, k in enumerate(keys) if k != c]
    ports = sorted(int(x) for x in rng.choice(cand, size=case["jports"], replace=False))
    return dict(wires=wires, n_per_edge_per_wire=[2] * (len(wires) - 1) + [10], degree=2, wire_radius=1e-3,
                wavelength=lam, junctions=[nodes[k] for k in keys], junction_ports=ports,
                feeds=[(len(wires) - 1, 0.5, 1.0)], ground_z=0.0, ground_eps=(13.0, 5e-3),
                ground_model="sommerfeld")


def _group(case, rng):
    structs = []
    for _ in range(case["structures"]):
        n_el = int(rng.integers(3, 13))
        structs.append(_yagi(rng, n_el, [int(2 * rng.integers(5, 51) + 1) for _ in range(n_el)]))
    return structs


def _inputs(case, seed):
    """(constructor keywords -- a list of them for a group --, wavenumbers)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "array":
        kw, f = _array(case, rng), 300e6
    elif kind in ("yagi", "sweep"):
        kw = _yagi(rng, case["elements"], [case["nseg"]] * case["elements"], case.get("ek", False), case["pec"])
        f = 28e6
    elif kind == "radials":
        kw, f = _radials(case, rng), 14.1e6
    elif kind == "vee":
        kw, f = _vee(case, rng), 14.1e6
    elif kind == "plate":
        kw, f = _plate(case, rng), 14.1e6
    else:
        kw, f = _group(case, rng), 28e6
    nk = case.get("nk", 1)
    band = np.linspace(0.9, 1.1, nk) if nk > 1 else np.ones(1)
    return kw, 2 * np.pi * f * band / C_SOLVER


def _block_inputs(case, seed):
    """The block assembler's arguments for two groups of parallel wires a
    wavelength apart, as an H-matrix host holds them."""
    rng = np.random.default_rng(seed)
    lam = 1.0
    sides = []
    for n, x0 in ((case["n_i"], 0.0), (case["n_j"], 3.0 * lam)):
        wires, left, i = [], n, 0
        while left > 0:
            nb = min(left, 40)  # bases of one wire: its segments + degree - 2
            L = 0.48 * lam * (1 + rng.uniform(-0.01, 0.01))
            x, y = x0 + 0.5 * lam * (i % 4), 0.5 * lam * (i // 4)
            wires.append((np.array([x, y, -L / 2]), np.array([x, y, L / 2]), nb + 2 - case["degree"]))
            left -= nb
            i += 1
        b = _bases([(p, q, s, False, False) for p, q, s in wires], case["degree"])
        sides.append((b["supp"], b["polys"], b["seg_l"], b["seg_r"], b["tan"]))
    k = 2 * np.pi / lam * (1 + rng.uniform(-0.02, 0.02))
    t, w = np.polynomial.legendre.leggauss(N_QP)
    return (*sides[0], *sides[1], (0.5e-3) ** 2, k, k * C_SOLVER, EPS, MU, case["degree"], 0.5 * (t + 1), 0.5 * w)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "block":
        return kind, _block_inputs(case, seed), None
    kw, ks = _inputs(case, seed)
    if kind == "group":
        return kind, kw, ks
    return kind, BSplineSolver(**kw, precision=case.get("precision", "fp64")), ks


def run(state):
    kind, obj, ks = state
    if kind == "block":
        return accel.bspline_assemble_offedge_block(*obj)
    if kind == "group":
        return sweep.grouped_mixed_sweep(obj, ks)
    if kind == "sweep":
        return obj.compute_y_matrix_swept(ks)
    return [(s.y, s.coeffs) for s in obj.compute_port_solution_swept(ks)]


# ----------------------------------------------------------------- counts
def _sizes(case):
    """(segments, unknowns, ports, right-hand sides, image fills) of one solve."""
    kind = case["kind"]
    if kind == "array":
        w = case["nx"] * case["ny"]
        n_seg, n, p, m, img = w * case["nseg"], w * (case["nseg"] + case["degree"] - 2), w, w, 0
    elif kind in ("yagi", "sweep"):
        n_seg = case["elements"] * case["nseg"]
        n, p, m, img = n_seg, 1, 1, int(case["pec"])
    elif kind == "radials":
        w = case["radials"] + 1
        n_seg, n, p, m, img = w * case["nseg"], w * (case["nseg"] + case["degree"] - 1), 1, 2, 1
    elif kind == "vee":
        n_seg, n, p, m, img = case["nseg"], case["nseg"], 1, 1, 1
    else:
        e = 2 * case["cells"] * (case["cells"] + 1)
        n_seg, n, p = 2 * e + 10, 4 * e + 11, 1 + case["jports"]
        m, img = p + (case["cells"] + 1) ** 2 - case["jports"], 1
    return n_seg, n, p, m, img


def _solve_work(n_seg, n, p, m, img, degree, out_coeffs):
    """One frequency: tables in, Y (and coefficients) out; the n_qp^2 kernel
    samples and moments of every segment pair, the Galerkin contraction of
    every basis pair, the factorisation and the solves."""
    nm = degree + 1
    pair = N_QP * N_QP * 20.0 + nm * nm * N_QP * N_QP * 4.0
    gal = nm * nm * (2.0 * nm * nm + 2.0 * degree * degree) * 2.0
    flops = (1 + img) * (n_seg * n_seg * pair + n * n * gal) + 8.0 / 3.0 * n**3 + 8.0 * n * n * m
    bytes_ = 96.0 * n_seg + 8.0 * nm * nm * n + 16.0 * p * p + (16.0 * n * p if out_coeffs else 0.0)
    return np.array([bytes_, flops])


def work(case):
    kind, nk = case["kind"], case.get("nk", 1)
    if kind == "block":
        d1, n_i, n_j = case["degree"] + 1, case["n_i"], case["n_j"]
        # each segment pair's n_qp^2 samples once, then the contraction
        b, f = 16.0 * n_i * n_j + (n_i + n_j) * (72.0 + 8.0 * d1 * d1), n_i * n_j * (
            N_QP * N_QP * (20.0 + 4.0 * d1 * d1) + d1 * d1 * 4.0 * (d1 * d1 + case["degree"] ** 2))
    elif kind == "group":
        b = f = 0.0
        for s in _group(case, np.random.default_rng(0)):
            n = int(sum(s["n_per_edge_per_wire"]))
            b, f = np.array([b, f]) + nk * _solve_work(n, n, 1, 1, 0, 2, False)
    else:
        b, f = nk * _solve_work(*_sizes(case), case.get("degree", 2), kind != "sweep")
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------- the same results in 64 bits
@functools.lru_cache(maxsize=None)
def _unit_polys(n, d):
    """Monomial coefficients [segment, active basis, power] of the clamped
    degree-d B-splines on n unit segments."""
    knots = np.concatenate([np.zeros(d), np.arange(n + 1.0), np.full(d, float(n))])
    us = np.linspace(0.0, 1.0, d + 1)
    vander = np.vander(us, d + 1, increasing=True)
    out = np.zeros((n, d + 1, d + 1))
    for s in range(n):
        x, span = s + us, s + d
        N = np.zeros((d + 1, d + 1))
        N[:, 0] = 1.0
        for j in range(1, d + 1):  # Cox-de Boor on this span
            saved = np.zeros(d + 1)
            for r in range(j):
                lo, hi = knots[span + 1 - j + r], knots[span + r + 1]
                t = N[:, r] / (hi - lo)
                N[:, r] = saved + (hi - x) * t
                saved = (x - lo) * t
            N[:, j] = saved
        out[s] = np.linalg.solve(vander, N).T
    return out


def _bases(wires, d):
    """Tables of straight wires [(p, q, segments, start held, end held)]:
    segments, per-basis supports (-1: none) and polynomials in arc length,
    each wire's first segment and first basis, the held end bases."""
    seg_l, seg_r, tan, h, wire, supp, polys, first, held = [], [], [], [], [], [], [], [], []
    off = 0
    for w, (p, q, n, hs, he) in enumerate(wires):
        L = float(np.linalg.norm(q - p))
        t = np.arange(n + 1.0)[:, None] / n
        pts = (1 - t) * p + t * q
        seg_l.append(pts[:-1])
        seg_r.append(pts[1:])
        tan.append(np.tile((q - p) / L, (n, 1)))
        h.append(np.full(n, L / n))
        wire.append(np.full(n, w))
        c = _unit_polys(n, d) / (L / n) ** np.arange(d + 1)
        first.append((off, len(supp)))
        for j in range(0 if hs else 1, n + d if he else n + d - 1):
            sm, pm = np.full(d + 1, -1, dtype=np.int64), np.zeros((d + 1, d + 1))
            for a, s in enumerate(range(max(0, j - d), min(n, j + 1))):
                sm[a], pm[a] = off + s, c[s, j - s]
            if (hs and j == 0) or (he and j == n + d - 1):
                held.append((w, "start" if j == 0 else "end", len(supp)))
            supp.append(sm)
            polys.append(pm)
        off += n
    return dict(seg_l=np.vstack(seg_l), seg_r=np.vstack(seg_r), tan=np.vstack(tan), h=np.concatenate(h),
                wire=np.concatenate(wire), supp=np.array(supp), polys=np.array(polys), first=first, held=held)


def _ek(R, a, k):
    """NEC's coaxial factor of the extended kernel, and its value at k = 0."""
    t1, t2 = 0.25 * (a / R) ** 4, 0.5 * (a / R) ** 2
    c1 = 1.0 + 1j * k * R
    return 1.0 + t1 * (3.0 * c1 - (k * R) ** 2) - t2 * c1, 1.0 + 3.0 * t1 - t2


def _static_moments(h, n, a, d, ek):
    """[delta, p, P]: the integrals of u^p v^P K(u - v - delta h) over [0, h]^2
    for K = 1 / (4 pi R) (with the static extended-kernel factor), by panels
    graded towards the kernel's peak."""
    x20, w20 = np.polynomial.legendre.leggauss(20)
    edges = [0.0]
    while edges[-1] < 0.5 * h:
        edges.append(min(0.5 * h, max(0.5 * a, 2.0 * edges[-1])))
    e = np.array(edges)
    half = np.concatenate([e, (h - e)[::-1][1:]])
    e = np.concatenate([-half[::-1], half[1:]])
    t = (0.5 * (e[1:] + e[:-1])[:, None] + 0.5 * np.diff(e)[:, None] * x20).ravel()
    wt = (0.5 * np.diff(e)[:, None] * w20).ravel()
    W = np.zeros((d + 1, d + 1, t.size))  # integral of u^p (u - t)^P over the overlap
    at = np.abs(t)
    for p in range(d + 1):
        for P in range(d + 1):
            lo, hi = (p, P), (P, p)
            for (i, o), sel in ((lo, t >= 0), (hi, t < 0)):
                acc = sum(math.comb(i, r) * at ** (i - r) * (h - at) ** (o + r + 1) / (o + r + 1)
                          for r in range(i + 1))
                W[p, P] = np.where(sel, acc, W[p, P])
    delta = np.arange(-(n - 1), n)
    R = np.sqrt((t[None, :] - delta[:, None] * h) ** 2 + a * a)
    K = 1.0 / (4 * np.pi * R)
    if ek:
        K = K * _ek(R, a, 0.0)[1]
    return np.einsum("dt,pqt->dpq", K * wt, W)


def _smooth_moments(h, n, a, d, k, ek, t, w):
    """The same integrals of K_k - K_0 by the n_qp^2 rule."""
    delta = np.arange(-(n - 1), n)
    R = np.sqrt((h * (t[:, None] - t[None, :])[None] - delta[:, None, None] * h) ** 2 + a * a)
    num = -2.0 * np.sin(0.5 * k * R) ** 2 - 1j * np.sin(k * R)
    if ek:
        fac = _ek(R, a, k)[0]
        t1, t2 = 0.25 * (a / R) ** 4, 0.5 * (a / R) ** 2
        num = num * fac + (t1 * (3j * k * R - (k * R) ** 2) - t2 * 1j * k * R)
    G = num / (4 * np.pi * R)
    f = (w * h) * (t * h) ** np.arange(d + 1)[:, None]
    return np.einsum("pq,dqr,Pr->dpP", f, G, f)


def _fill(b, d, k, a, pec, ek, eps_t, static, dev):
    """The Galerkin impedance matrix of the tables ``b`` at wavenumber k."""
    f64, c128 = torch.float64, torch.complex128
    T = lambda x, dt=f64: torch.as_tensor(np.ascontiguousarray(x), dtype=dt, device=dev)  # noqa: E731
    tn, wn = np.polynomial.legendre.leggauss(N_QP)
    tn, wn = 0.5 * (tn + 1), 0.5 * wn
    n, N, d1 = b["supp"].shape[0], b["h"].size, d + 1
    om = k * C_SOLVER
    pts = T((1 - tn)[None, :, None] * b["seg_l"][:, None, :] + tn[None, :, None] * b["seg_r"][:, None, :])
    supp = np.maximum(b["supp"], 0)
    u = b["h"][supp][..., None] * tn  # (n, wing, q)
    pw = u[..., None] ** np.arange(d1)
    dp = np.arange(d1) * u[..., None] ** np.maximum(np.arange(d1) - 1, 0)
    wq = np.where(b["supp"] >= 0, b["h"][supp], 0.0)[..., None] * wn
    fA = T(np.einsum("naqp,nap->naq", pw, b["polys"]) * wq)
    fP = T(np.einsum("naqp,nap->naq", dp, b["polys"]) * wq)
    sup = T(supp, torch.int64)
    tan, wire = T(b["tan"]), T(b["wire"], torch.int64)
    mid = T(0.5 * (b["seg_l"] + b["seg_r"]))
    flip = T([1.0, 1.0, -1.0])
    Z = torch.zeros((n, n), dtype=c128, device=dev)
    order = [np.argsort(supp[:, w], kind="stable") for w in range(d1)]
    starts = [np.searchsorted(supp[o, w], np.arange(N + 1)) for w, o in enumerate(order)]
    step = max(1, int(1.6e7 // (N * N_QP * N_QP)))
    # direct pairs, then (over a ground) the mirrored sources
    for image in range(2 if pec or eps_t is not None else 1):
        src = pts * flip if image else pts
        stan, smid = (tan * flip, mid * flip) if image else (tan, mid)
        for i0 in range(0, N, step):
            i1 = min(N, i0 + step)
            diff = pts[i0:i1, :, None, None, :] - src[None, None]
            R = torch.sqrt((diff * diff).sum(-1) + a * a)  # (c, q, N, r)
            del diff
            G = torch.polar(1.0 / (4 * math.pi * R), -k * R)
            same = wire[i0:i1, None] == wire[None, :]
            if ek:  # every structure with the extended kernel has parallel wires: one axis per wire
                G = torch.where(same[:, None, :, None], G * _ek(R, a, k)[0], G)
            del R
            if not image:
                G = torch.where(same[:, None, :, None], torch.zeros((), dtype=c128, device=dev), G)
            td = tan[i0:i1] @ stan.T
            wA, wP = td.to(c128), torch.ones_like(td, dtype=c128)
            if image and eps_t is not None:  # Fresnel dyad, plane-wave charge weight at normal incidence
                dd = mid[i0:i1, None, :] - smid[None]
                hyp = torch.hypot(dd[..., 0], dd[..., 1])
                cth = dd[..., 2] / torch.sqrt((dd * dd).sum(-1))
                safe = hyp > 1e-30
                inv = 1.0 / torch.where(safe, hyp, torch.ones_like(hyp))
                px = torch.where(safe, -dd[..., 1] * inv, torch.ones_like(hyp))
                py = torch.where(safe, dd[..., 0] * inv, torch.zeros_like(hyp))
                P = ((tan[i0:i1, None, 0] * px + tan[i0:i1, None, 1] * py)
                     * (stan[None, :, 0] * px + stan[None, :, 1] * py))
                root = torch.sqrt(eps_t - (1.0 - cth * cth).to(c128))
                rv, rh = (eps_t * cth - root) / (eps_t * cth + root), (cth - root) / (cth + root)
                r0 = np.sqrt(eps_t)
                wA, wP = rv * (td - P) - rh * P, wP * complex((r0 - 1) / (r0 + 1))
            XA = torch.zeros((i1 - i0, N_QP, n), dtype=c128, device=dev)
            XP = torch.zeros_like(XA)
            for w in range(d1):
                g = G[:, :, sup[:, w], :]  # (c, q, n, r)
                XA += wA[:, sup[:, w]][:, None, :] * (g * fA[:, w]).sum(-1)
                XP += wP[:, sup[:, w]][:, None, :] * (g * fP[:, w]).sum(-1)
                del g
            XA, XP = 1j * om * MU * XA, XP / (1j * om * EPS)
            sign = -1.0 if image else 1.0
            for w in range(d1):
                m = order[w][starts[w][i0]:starts[w][i1]]
                if m.size:
                    mt = T(m, torch.int64)
                    s = sup[mt, w] - i0
                    Z[mt] += sign * ((fA[mt, w].to(c128)[:, None, :] @ XA[s])
                                     + (fP[mt, w].to(c128)[:, None, :] @ XP[s]))[:, 0, :]
    # pairs on one wire: static part exactly, the rest by the n_qp^2 rule
    ends = [f[1] for f in b["first"][1:]] + [n]
    for w, ((s0, m0), m1) in enumerate(zip(b["first"], ends)):
        ns = int((b["wire"] == w).sum())
        J = T(static[w] + _smooth_moments(b["h"][s0], ns, a, d, k, ek, tn, wn), c128)
        sp, pl = T(np.maximum(b["supp"][m0:m1] - s0, 0), torch.int64), T(b["polys"][m0:m1]).to(c128)
        dl = pl[..., 1:] * torch.arange(1, d1, device=dev)
        blk = torch.zeros((m1 - m0, m1 - m0), dtype=c128, device=dev)
        for i in range(d1):
            for j in range(d1):
                j4 = J[sp[None, :, j] - sp[:, None, i] + ns - 1]
                blk += 1j * om * MU * torch.einsum("mp,mnpq,nq->mn", pl[:, i], j4, pl[:, j])
                blk += torch.einsum("mp,mnpq,nq->mn", dl[:, i], j4[..., :d, :d], dl[:, j]) / (1j * om * EPS)
        Z[m0:m1, m0:m1] += blk
    return Z


def _internal_impedance(omega, a, sigma):
    """Series impedance per metre of a round conductor, I0 / I1 by Miller's
    backward recurrence."""
    kc = np.sqrt(1j * omega * MU * sigma)
    x, r = kc * a, 0.0
    for m in range(400, 0, -1):
        r = 1.0 / (2.0 * m / x + r)  # I_m / I_(m-1)
    return kc / (2.0 * np.pi * a * sigma) / r


def _add_loading(Z, b, omega, a, sigma, dev):
    zw = _internal_impedance(omega, a, sigma)
    d1 = b["polys"].shape[1]
    pq = np.arange(d1)[:, None] + np.arange(d1)[None, :] + 1.0
    by_seg = {}
    for m, row in enumerate(b["supp"]):
        for w, s in enumerate(row):
            if s >= 0:
                by_seg.setdefault(int(s), []).append((m, w))
    S = np.zeros(Z.shape)
    for s, wings in by_seg.items():
        H = b["h"][s] ** pq / pq
        for m, i in wings:
            for q, j in wings:
                S[m, q] += b["polys"][m, i] @ H @ b["polys"][q, j]
    return Z + zw * torch.as_tensor(S, device=dev).to(Z.dtype)


def _exact_solutions(kw, ks, dev):
    """[(y, coeffs)] of a straight-wire structure (free space, perfect or
    reflection-coefficient ground)."""
    wires, d, a = kw["wires"], kw["degree"], float(kw["wire_radius"])
    held = {e for j in kw.get("junctions", []) for e in j}
    npe = kw.get("n_per_edge_per_wire") or [kw["nsegs"]] * len(wires)
    b = _bases([(p[0], p[1], n, (w, "start") in held, (w, "end") in held)
                for w, (p, n) in enumerate(zip(wires, npe))], d)
    n, ek = b["supp"].shape[0], kw.get("extended_kernel", False)
    B = np.zeros((n, len(kw["feeds"])))
    for p, (w, arc, _v) in enumerate(kw["feeds"]):
        h = b["h"][b["first"][w][0]]
        s_f = 0.5 * h * npe[w] if arc is None else arc
        s = min(npe[w] - 1, int(math.floor(s_f / h + 1e-12)))
        at = b["supp"] == b["first"][w][0] + s
        B[:, p] = (at[..., None] * b["polys"] * (s_f - s * h) ** np.arange(d + 1)).sum((1, 2))
    A = np.zeros((len(kw.get("junctions", [])), n))
    for w, end, m in b["held"]:
        for r, j in enumerate(kw["junctions"]):
            if (w, end) in j:
                A[r, m] = 1.0 if end == "start" else -1.0
    static = [_static_moments(b["h"][b["first"][w][0]], npe[w], a, d, ek) for w in range(len(wires))]
    R = torch.as_tensor(np.hstack([B, A.T]), device=dev).to(torch.complex128)
    Bd, Ad, out = R[:, : B.shape[1]], R[:, B.shape[1]:].T, []
    for k in ks:
        eps_t = None
        if "ground_eps" in kw:
            eps_t = complex(kw["ground_eps"][0], -kw["ground_eps"][1] / (k * C_SOLVER * EPS))
        Z = _fill(b, d, float(k), a, "ground_z" in kw and eps_t is None, ek, eps_t, static, dev)
        if "wire_conductivity" in kw:
            Z = _add_loading(Z, b, k * C_SOLVER, a, kw["wire_conductivity"], dev)
        X = torch.linalg.solve(Z, R)
        W, Xc = X[:, : B.shape[1]], X[:, B.shape[1]:]
        if A.shape[0]:
            W = W - Xc @ torch.linalg.solve(Ad @ Xc, Ad @ W)
        out.append(((Bd.T @ W).cpu().numpy(), W.cpu().numpy()))
    return out


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind in ("vee", "plate"):
        return None  # Sommerfeld integrals: no plain restatement runs in seconds
    if kind == "block":
        sI, pI, lI, rI, tI, sJ, pJ, lJ, rJ, tJ, a2, k, om, eps, mu, d, t, w = _block_inputs(case, seed)
        T = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev)  # noqa: E731

        def side(s, p, left, right, tan):
            s0 = np.maximum(s, 0)
            L = np.linalg.norm(right - left, axis=1)[s0]
            x = (1 - t)[:, None] * left[s0][:, :, None, :] + t[:, None] * right[s0][:, :, None, :]
            u = L[..., None] * t
            e = np.arange(d + 1)
            wq = np.where(s >= 0, L, 0.0)[..., None] * w
            f = np.einsum("nwqp,nwp->nwq", u[..., None] ** e, p) * wq
            df = np.einsum("nwqp,nwp->nwq", e * u[..., None] ** np.maximum(e - 1, 0), p) * wq
            n = s.shape[0]
            tq = np.repeat(tan[s0][:, :, None, :], t.size, axis=2)
            return T(x.reshape(n, -1, 3)), T(f.reshape(n, -1)), T(df.reshape(n, -1)), T(tq.reshape(n, -1, 3))

        (xI, fI, gI, uI), (xJ, fJ, gJ, uJ) = side(sI, pI, lI, rI, tI), side(sJ, pJ, lJ, rJ, tJ)
        Z = torch.zeros((sI.shape[0], sJ.shape[0]), dtype=torch.complex128, device=dev)
        for q in range(xI.shape[1]):
            for r in range(xJ.shape[1]):
                R = torch.sqrt(((xI[:, None, q] - xJ[None, :, r]) ** 2).sum(-1) + a2)
                G = torch.polar(1.0 / (4 * math.pi * R), -k * R)
                Z += 1j * om * mu * (fI[:, q, None] * fJ[None, :, r]) * (uI[:, q] @ uJ[:, r].T) * G
                Z += (gI[:, q, None] * gJ[None, :, r]) * G / (1j * om * eps)
        return Z.cpu().numpy()
    kw, ks = _inputs(case, seed)
    if kind == "group":
        return {i: np.array([y for y, _c in _exact_solutions(s, ks, dev)]) for i, s in enumerate(kw)}
    sols = _exact_solutions(kw, ks, dev)
    return np.array([y for y, _c in sols]) if kind == "sweep" else sols
