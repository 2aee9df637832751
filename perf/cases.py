"""The work a user of this framework has it do, as cases that can be timed and checked.

Every case is posed as a user's program poses it: a plan (``lightsmith_b200.plan.make_plan``) of the problem, an engine
built from it once (``Engine.from_plan``, ``BlochBatch`` or ``AdjointRun``), and a pass that advances the run by the
chunks lightsmith's run loop takes (``Engine.make_runner``: dft_stride steps, a DFT sample, the status check), by a
batched launch, or by a whole forward and backward of the adjoint. Waveforms are ramped continuous waves, so that a
run can be advanced for as long as it is timed.

``prepare`` and ``exact`` share the problem's plain arrays (``_problem``); ``exact`` steps them in float64 with torch
alone (``_Reference``): Yee updates, CPML, TF/SF tables, point currents, mode sources, Bloch columns, dispersive nodes,
running DFTs, and torch autograd through the steps for the gradients.
"""

import math

import numpy as np
import torch

from lightsmith_b200.adjoint import AdjointRun
from lightsmith_b200.batch import BlochBatch
from lightsmith_b200.engine import Engine
from lightsmith_b200.plan import (ColumnSource, DFTMonitor, DipoleSource, DispersiveGroup, Medium, ModeSource, PMLSpec,
                                  Pole, TablePoints, TableSource, make_plan)

EV = 197.3269804  # hbar c in eV nm
# the sphere benchmark's metal (Drude and two Lorentz poles): eps_inf, (sigma, omega0, gamma) per pole
METAL = (5.9, (((9.0 / EV) ** 2, 0.0, 0.07 / EV), (1.3 * (2.6 / EV) ** 2, 2.6 / EV, 0.6 / EV),
               (1.5 * (3.7 / EV) ** 2, 3.7 / EV, 1.0 / EV)))


def listed():
    return [
        # a 2D device on a plane of three nodes (invariant z axis periodic), a mode launched at a port: the smallest
        # steps, where launches and latency count (the repository's 2D device fixtures: 123 x 139)
        {"name": "device2d", "kind": "device", "n0": 123, "n1": 139, "pml": 10, "stride": 20, "calls": 2, "nf": 5,
         "double": False},
        # lightsmith's default pose of a small particle: a quarter of the 49^3 grid of the repository's sphere solves
        # between two mirror planes, subpixel interface cells of the metal (mixed groups)
        {"name": "sphere49mirror", "kind": "scatter", "n0": 26, "n1": 26, "n2": 49, "mirror": True, "pml": 8,
         "stride": 10, "calls": 4, "nf": 9, "mixed": True, "double": False},
        # the same sphere solve without symmetry, staircase
        {"name": "sphere49", "kind": "scatter", "n0": 49, "n1": 49, "n2": 49, "mirror": False, "pml": 8, "stride": 10,
         "calls": 4, "nf": 9, "mixed": False, "double": False},
        # the full-size sphere solve (129^3, CPML 12, 81 wavelengths, one chunk of 100 steps)
        {"name": "sphere129", "kind": "scatter", "n0": 129, "n1": 129, "n2": 129, "mirror": False, "pml": 12,
         "stride": 100, "calls": 1, "nf": 81, "mixed": False, "double": False},
        # the precision a user asks for to check a result: float64, subpixel, a middling ragged grid
        {"name": "sphere97double", "kind": "scatter", "n0": 97, "n1": 89, "n2": 101, "mirror": False, "pml": 10,
         "stride": 20, "calls": 1, "nf": 21, "mixed": True, "double": True},
        # a particle cluster's grid (the layouts lightsmith sizes to a cluster are odd along every axis)
        {"name": "cluster", "kind": "scatter", "n0": 201, "n1": 215, "n2": 199, "mirror": False, "pml": 12,
         "stride": 16, "calls": 1, "nf": 24, "mixed": False, "double": False},
        # the plain solver's throughput case at three sizes: i.i.d. permittivity, CPML on every face, point currents,
        # a 16-frequency DFT plane
        {"name": "bulk100", "kind": "bulk", "n0": 100, "n1": 100, "n2": 100, "pml": 16, "stride": 31, "calls": 1,
         "nf": 16, "double": False},
        {"name": "bulk256", "kind": "bulk", "n0": 256, "n1": 256, "n2": 256, "pml": 16, "stride": 31, "calls": 1,
         "nf": 16, "double": False},
        {"name": "bulk640", "kind": "bulk", "n0": 640, "n1": 640, "n2": 640, "pml": 16, "stride": 31, "calls": 1,
         "nf": 16, "double": False},
        # oblique runs of periodic cells (30 to 60 cells a period, 200 along z), batched in one launch
        {"name": "sweep", "kind": "sweep", "runs": 14, "nz": 200, "pml": 12, "lo": 300, "hi": 600, "steps": 64,
         "batched": True},
        # the gradient of a slab device: forward from rest with checkpoints, then backward
        {"name": "gradient", "kind": "gradient", "n0": 200, "n1": 200, "n2": 120, "pml": 12, "box": 48, "steps": 400,
         "stride": 10, "checkpoint": 200, "metal": False},
        # the gradient around a metal particle (dispersive nodes, TF/SF plane wave, scattered flux), odd grid
        {"name": "gradmetal", "kind": "gradient", "n0": 113, "n1": 109, "n2": 117, "pml": 10, "box": 0, "steps": 192,
         "stride": 16, "checkpoint": 96, "metal": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "scatter", "scatter", "bulk", "bulk", "sweep", "gradient"])
    if kind == "device":
        return {"kind": kind, "n0": _log(rng, 60, 400), "n1": _log(rng, 60, 400), "pml": rng.randint(8, 14),
                "stride": rng.randint(5, 30), "calls": rng.randint(1, 3), "nf": rng.randint(1, 12),
                "double": rng.random() < 0.2}
    if kind == "scatter":
        m = _log(rng, 45, 200)
        n = [int(m * rng.uniform(0.85, 1.15)) | 1 for _ in range(3)]
        mirror = rng.random() < 0.3
        if mirror:
            n[0], n[1] = n[0] // 2 + 2, n[1] // 2 + 2
        return {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "mirror": mirror, "pml": 8 if m < 80 else 12,
                "stride": rng.randint(8, 40), "calls": rng.randint(1, 2), "nf": rng.randint(4, 60),
                "mixed": rng.random() < 0.5, "double": rng.random() < 0.2}
    if kind == "bulk":
        m = _log(rng, 64, 420)
        n = [max(48, int(m * rng.uniform(0.8, 1.2))) for _ in range(3)]
        if rng.random() < 0.7:  # rows of a multiple of four nodes, as a user of the throughput path chooses them
            n[2] = (n[2] + 3) // 4 * 4
        return {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "pml": rng.randint(8, 18), "stride": rng.randint(16, 32),
                "calls": 1, "nf": rng.randint(1, 24), "double": rng.random() < 0.2}
    if kind == "sweep":
        lo = rng.randint(300, 450)
        return {"kind": kind, "runs": rng.randint(1, 14), "nz": rng.randint(150, 210), "pml": rng.randint(8, 14), "lo": lo,
                "hi": lo + rng.randint(20, 150), "steps": rng.randint(24, 64), "batched": rng.random() < 0.6}
    if rng.random() < 0.5:
        return {"kind": kind, "n0": rng.randint(90, 200), "n1": rng.randint(70, 200), "n2": rng.randint(60, 120), "pml": 10,
                "box": rng.randint(16, 40), "steps": 20 * rng.randint(10, 18), "stride": 10, "checkpoint": 100,
                "metal": False}
    n = [rng.randint(70, 115) for _ in range(3)]
    return {"kind": kind, "n0": n[0], "n1": n[1], "n2": n[2], "pml": 8, "box": 0, "steps": 16 * rng.randint(6, 12),
            "stride": 16, "checkpoint": rng.choice([48, 96]), "metal": True}


# --- the problems as plain arrays -----------------------------------------------------------------------------------


def _flat(c, i, j, k, n):
    return ((np.asarray(c, np.int64) * n[0] + i) * n[1] + j) * n[2] + k


def _grid(*r):
    return [v.ravel() for v in np.meshgrid(*[np.arange(a, b) for a, b in r], indexing="ij")]


def _horizon(cells):
    """Steps the waveforms last: enough for any timing of a grid of that many cells."""
    return int(min(2_000_000, max(20_000, 4e11 / cells)))


def _ramped(omega, dt, n, phase=0.0):
    t = np.arange(n) * (omega * dt)
    return np.sin(t + phase) * np.minimum(1.0, t / (4 * math.pi)) ** 2


def _plane(axis, k, r, n, omega, energy):
    """The two tangential E components on node plane k normal to axis over node ranges r of the two other axes (in
    the order axis + 1, axis + 2), each with the H component it pairs with on planes k - 1 and k."""
    b, c = (axis + 1) % 3, (axis + 2) % 3
    B, C = _grid(*r)

    def at(comp, kk):
        x = [None] * 3
        x[axis], x[b], x[c] = np.full(B.size, kk), B, C
        return _flat(comp, *x, n)
    return {"omega": omega, "e": np.concatenate([at(b, k), at(c, k)]), "h1": np.concatenate([at(c, k - 1), at(b, k - 1)]),
            "h2": np.concatenate([at(c, k), at(b, k)]), "energy": energy, "of": None}


def _box_faces(lo, hi, n, omega, energy, mirror=(0, 0, 0)):
    """The faces of the node box [lo, hi] as one monitor (along a mirror axis only the high one), and the sign of
    each point in the outward flux."""
    got, sign = [], []
    for a in range(3):
        r = [(lo[(a + 1) % 3], hi[(a + 1) % 3] + 1), (lo[(a + 2) % 3], hi[(a + 2) % 3] + 1)]
        for side, k in ((-1.0, lo[a]), (1.0, hi[a])):
            if mirror[a] and side < 0:
                continue
            got.append(_plane(a, k, r, n, omega, energy))
            m = len(got[-1]["e"]) // 2
            sign.append(np.repeat([side, -side], m))
    cat = {k: np.concatenate([g[k] for g in got]) for k in ("e", "h1", "h2")}
    return {"omega": omega, "energy": energy, "of": None, **cat}, np.concatenate(sign)


def _base(n, dx, dt, pml, stride, double, **more):
    p = {"n": tuple(n), "dx": tuple(dx), "dt": dt, "pml": pml, "stride": stride, "double": double,
         "per": (False,) * 3, "bloch": (0.0,) * 3, "mirror": (0, 0, 0), "groups": [], "alpha": 0.0, "eps_ref": 1.0}
    p.update(more)
    return p


def _device(case, seed):
    """A 2D device of random strips between two waveguide ports: a mode of E_z launched on one port plane, recorded
    on both."""
    rng = np.random.default_rng(seed)
    n = (case["n0"], case["n1"], 3)
    dx, p = 25.0, case["pml"]
    dt = 0.99 * dx / math.sqrt(3)
    om = 2 * np.pi / np.linspace(1500.0, 1600.0, case["nf"])
    eps = np.full(n, 1.44 ** 2)
    w = max(4, n[1] // 8)
    mid = n[1] // 2 + int(rng.integers(-3, 4))
    eps[:, mid - w // 2:mid + w // 2] = 2.8 ** 2
    x0, x1 = n[0] // 3, 2 * n[0] // 3
    strips = rng.uniform(1.44 ** 2, 2.8 ** 2, (x1 - x0, n[1] - 2 * p - 4, 1))
    eps[x0:x1, p + 2:n[1] - p - 2] = strips
    js = np.arange(p + 2, n[1] - p - 2)
    xs = p + 5
    prof = np.exp(-((js - mid) / (0.7 * w)) ** 2)
    steps = _horizon(n[0] * n[1] * 3)
    wave = _ramped(float(om[0]), dt, steps, rng.uniform(0, 6.28))
    src = {"kind": "mode", "h": _flat(1, xs - 1, js, 1, n), "mH": (-0.4 * prof)[:, None], "tE": wave[:, None],
           "e": _flat(2, xs, js, 1, n), "mE": (0.3 * prof)[:, None], "tH": np.roll(wave, 1)[:, None]}
    r = [(p + 1, n[1] - p - 1), (1, 2)]
    mons = [_plane(0, p + 3, r, n, om, 1), _plane(0, n[0] - p - 4, r, n, om, 1)]
    return _base(n, (dx,) * 3, dt, ((p, p), (p, p), (0, 0)), case["stride"], case["double"], per=(False, False, True),
                 alpha=0.05 * float(om[0]), eps_ref=1.44 ** 2, inv_eps=1 / eps, sources=[src], monitors=mons)


def _scatter(case, seed):
    """A metal sphere in a medium under a table-fed TF/SF plane wave along z, with the scattered- and total-field flux
    boxes and the incident reference view of lightsmith's scattering driver; with mirror planes, its quarter around
    the planes at node 1 of x (E antisymmetric) and y (symmetric)."""
    rng = np.random.default_rng(seed)
    n = (case["n0"], case["n1"], case["n2"])
    mirror = (-1, 1, 0) if case.get("mirror") else (0, 0, 0)
    p, dx, nb = case["pml"], 4.0 if case["n2"] < 80 else 2.0, 1.33
    dt = 0.99 * dx / math.sqrt(3)
    wl = np.linspace(400.0, 800.0, case["nf"])
    om = 2 * np.pi / wl
    lo = [1 if mirror[a] else p for a in range(3)]  # the outer ends of the region without CPML
    hi = [n[a] - 1 - p for a in range(3)]
    gap = [max(3, (hi[a] - lo[a]) // (5 if not mirror[a] else 3)) for a in range(3)]
    tl = [1 if mirror[a] else lo[a] + gap[a] for a in range(3)]  # the total-field box, nodes [tl, th]
    th = [hi[a] - gap[a] for a in range(3)]
    half = [(th[a] - tl[a]) / (1 if mirror[a] else 2) for a in range(3)]
    rad = min(half) * rng.uniform(0.6, 0.7)
    ctr = [1.0 if mirror[a] else 0.5 * (tl[a] + th[a]) + rng.uniform(-0.5, 0.5) for a in range(3)]
    inv = np.full((3,) + n, 1 / nb ** 2)
    idx, mix, frac = [], [], []
    for c in range(3):
        box = [slice(max(0, int(ctr[a] - rad) - 2), min(n[a] - 1, int(ctr[a] + rad) + 3)) for a in range(3)]
        pos = np.meshgrid(*[np.arange(s.start, s.stop) + (0.5 if a == c else 0.0) - ctr[a] for a, s in enumerate(box)],
                          indexing="ij")
        d = np.sqrt(sum(v * v for v in pos)) - rad
        first = [(2 if mirror[a] < 0 and a != c else 1) if mirror[a] else 0 for a in range(3)]
        ok = np.ones(d.shape, bool)
        for a in range(3):
            sh = [1, 1, 1]
            sh[a] = -1
            ok &= (np.arange(box[a].start, box[a].stop) >= first[a]).reshape(sh)
        pure = (d < (-0.5 if case["mixed"] else 0.0)) & ok
        part = (np.abs(d) <= 0.5) & ok if case["mixed"] else np.zeros(d.shape, bool)
        flat = _flat(c, *[v + s.start for v, s in zip(np.indices(d.shape), box)], n)
        inv[c][tuple(box)][pure | part] = 1.0
        idx.append(flat[pure])
        mix.append(flat[part])
        frac.append(0.5 - d[part])
    groups = [{"idx": np.concatenate(idx), "frac": None, "w": None}]
    if case["mixed"]:
        f = np.clip(np.concatenate(frac), 0.02, 0.98)
        groups.append({"idx": np.concatenate(mix), "frac": np.stack([1 - f, f]), "w": rng.uniform(0, 1, len(f))})
    # the incident wave E_x (H_y = n E_x) g(t - nb z), one row of a table in steps of m dt, read with each plane's delay
    m = 4
    steps = _horizon(n[0] * n[1] * n[2])
    rows = steps // m + 400
    table = _ramped(2 * np.pi / rng.uniform(450, 700), m * dt, rows)
    cmax = rows - 6

    def times(z, half_step):  # whole and fractional fine time at step 0 of the wave at height z (cells)
        t = 8.0 * m + (n[2] + 8 - z) * nb * dx / dt + (0.5 if half_step else 0.0)
        i0 = np.floor(t).astype(np.int64)
        return i0, t - i0
    c_e, c_h = dt / dx / nb ** 2, dt / dx

    def face(comp, r, z, coef, half_step):
        i, j, k = _grid(*r)
        i0, u0 = times(np.broadcast_to(np.asarray(z(k), float), k.shape), half_step)
        return _flat(comp, i, j, k, n), i0, u0, np.full(k.shape, coef)
    xs = (max(tl[0], 1), th[0])  # E_x over [tl, th) along x, nodes [tl, th] along y (odd components from node 2)
    ys = (max(tl[1], 1), th[1] + 1)
    # H_y next to the x faces reads E_x nowhere (E_x is normal there); E_z at the x faces reads H_y; E_x at the z faces
    # reads H_y; H_y below/above the z faces and H_z beside the y faces read E_x
    E = [face(0, (xs, ys, (tl[2], tl[2] + 1)), lambda k: k - 0.5, c_e * nb, True),
         face(0, (xs, ys, (th[2], th[2] + 1)), lambda k: k + 0.5, -c_e * nb, True)]
    H = [face(1, (xs, ys, (tl[2] - 1, tl[2])), lambda k: k + 1.0, c_h, False),
         face(1, (xs, ys, (th[2], th[2] + 1)), lambda k: k + 0.0, -c_h, False),
         face(2, (xs, (th[1], th[1] + 1), (tl[2], th[2] + 1)), lambda k: k + 0.0, c_h, False)]
    E.append(face(2, ((th[0], th[0] + 1), ys, (tl[2], th[2])), lambda k: k + 0.5, c_e * nb, True))
    if not mirror[0]:
        E.append(face(2, ((tl[0], tl[0] + 1), ys, (tl[2], th[2])), lambda k: k + 0.5, -c_e * nb, True))
    if not mirror[1]:
        H.append(face(2, (xs, (tl[1] - 1, tl[1]), (tl[2], th[2] + 1)), lambda k: k + 0.0, -c_h, False))
    E, H = ([np.concatenate([f[q] for f in g]) for q in range(4)] for g in (E, H))
    vi, vu = times(np.full(3, 0.5 * (tl[2] + th[2])), False)
    src = {"kind": "table", "table": table, "m": m, "cmax": cmax, "E": E, "H": H,
           "inc": np.stack([table, 0 * table, 0 * table]), "view": (vi, vu)}
    sca, sign = _box_faces([1 if mirror[a] else tl[a] - 2 for a in range(3)], [th[a] + 2 for a in range(3)], n, om, 1,
                           mirror)
    tot, _ = _box_faces([1 if mirror[a] else tl[a] + 1 for a in range(3)], [th[a] - 1 for a in range(3)], n, om, 2,
                        mirror)
    view = {"omega": om, "e": np.arange(3), "h1": None, "h2": None, "energy": 0, "of": "view"}
    cells = tuple((0 if mirror[a] else p, p) for a in range(3))
    return _base(n, (dx,) * 3, dt, cells, case["stride"], case["double"], mirror=mirror, alpha=0.05 * float(om.min()),
                 eps_ref=nb ** 2, inv_eps=inv, groups=groups, sources=[src], monitors=[sca, tot, view], sign=sign,
                 inside=([0.5 * (tl[a] + th[a]) for a in range(3)], min(half)))


def _bulk(case, seed):
    """The throughput case: i.i.d. permittivity in [1, 12.25], a cloud of point currents between the CPML slabs, the
    running DFT on the centre z plane."""
    rng = np.random.default_rng(seed)
    n = (case["n0"], case["n1"], case["n2"])
    dx, p = 20.0, case["pml"]
    dt = 0.99 * dx / math.sqrt(3)
    om = 2 * np.pi / np.linspace(1000.0, 2000.0, case["nf"])
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    inv = 1 / (1 + 11.25 * torch.rand(n, generator=g, device="cuda", dtype=torch.float32))
    m = max(64, n[0] * n[1] * n[2] // 65536)
    at = [rng.integers(p + 2, n[a] - p - 2, m) for a in range(3)]
    idx = np.unique(_flat(rng.integers(0, 3, m), *at, n))
    wave = _ramped(float(om.max()), dt, _horizon(n[0] * n[1] * n[2]), rng.uniform(0, 6.28))
    src = {"kind": "dipole", "e": idx, "coef": rng.normal(size=len(idx)), "wave": wave}
    mon = _plane(2, n[2] // 2, [(1, n[0] - 1), (1, n[1] - 1)], n, om, 1)
    return _base(n, (dx,) * 3, dt, ((p, p),) * 3, case["stride"], case["double"], alpha=0.05 * 2 * math.pi / 2000.0,
                 inv_eps=inv, sources=[src], monitors=[mon])


def _cell(case, period, rng):
    """One oblique run of a pillar on a substrate: a square periodic cell under a Bloch phase, a TF/SF plane fed by a
    3 x 3 x nz column with the same phases, planes above and below, the column's probe."""
    nc = int(math.ceil(period / 10.0))
    d, dz, nz, p = period / nc, 10.0, case["nz"], case["pml"]
    n = (nc + 2, nc + 2, nz)
    dt = 0.99 / math.sqrt(2 / d ** 2 + 1 / dz ** 2)
    ks, kr, kt = p + 10, p + 4, nz - p - 4
    xc = (((np.arange(n[0]) - 1) % nc) + 0.5) * d - 0.5 * period
    pillar = xc[:, None] ** 2 + xc[None, :] ** 2 <= (0.3 * period) ** 2
    eps = np.ones(n)
    z1 = min(ks + 68, kt - 8)
    eps[:, :, z1:] = 1.45 ** 2
    eps[:, :, ks + 8:z1][pillar] = 2.4 ** 2
    om = 2 * np.pi / rng.uniform(450, 750)
    th, ph = math.radians(rng.uniform(1, 60)), math.radians(rng.uniform(0, 90))
    kx, ky = om * math.sin(th) * math.cos(ph), om * math.sin(th) * math.sin(ph)
    ax = rng.uniform(0, 6.28)
    i, j = np.meshgrid(np.arange(nc), np.arange(nc), indexing="ij")
    shared = {"per": (True, True, False), "bloch": (kx, ky, 0.0), "alpha": 0.01}
    col = _base((3, 3, nz), (d, d, dz), dt, ((0, 0), (0, 0), (p, p)), 1, False, inv_eps=np.ones((3, 3, nz)), sources=[],
                monitors=[], **shared)
    src = {"kind": "column", "col": col, "k_src": ks, "k_launch": ks - 1, "phase": np.exp(1j * (kx * i + ky * j) * d),
           "amp": (complex(math.cos(ax), 0.2), complex(math.sin(ax), -0.1)),
           "wave": _ramped(om, dt, _horizon(n[0] * n[1] * nz)), "cE": dt / dz, "cH": dt / dz}
    omega = np.array([om])
    r = [(1, n[0] - 1), (1, n[1] - 1)]
    probe = {**_plane(2, ks + 3, [(1, 2), (1, 2)], (3, 3, nz), omega, 0), "of": "column"}
    stride = max(1, int(2 * np.pi / (2.6 * 2 * np.pi / 450) / dt))
    return _base(n, (d, d, dz), dt, ((0, 0), (0, 0), (p, p)), stride, False, inv_eps=1 / eps, sources=[src],
                 monitors=[_plane(2, kr, r, n, omega, 1), _plane(2, kt, r, n, omega, 1), probe], **shared)


def _slab(case, seed):
    """A slab waveguide along x with a random design region: a sheet of E_y before it, E_y on a plane after it."""
    rng = np.random.default_rng(seed)
    n = (case["n0"], case["n1"], case["n2"])
    dx, p = 20.0, case["pml"]
    dt = 0.99 * dx / math.sqrt(3)
    zc, h = n[2] // 2, 5
    eps = np.full(n, 1.44 ** 2)
    eps[:, :, zc - h:zc + h + 1] = 3.48 ** 2
    x0 = (n[0] - case["box"]) // 2
    box = ((x0, x0 + case["box"]), (p + 6, n[1] - p - 6), (zc - h, zc + h + 1))
    sl = tuple(slice(a, b) for a, b in box)
    eps[sl] = 1.44 ** 2 + rng.uniform(0, 1, eps[sl].shape[:2])[:, :, None] * (3.48 ** 2 - 1.44 ** 2)
    om = 2 * np.pi / 1550.0

    def sheet(x):
        _, j, k = _grid((x, x + 1), (p + 3, n[1] - p - 3), (zc - 2 * h, zc + 2 * h + 1))
        return _flat(1, x, j, k, n), np.cos(0.2 * (k - zc))
    e, amp = sheet(x0 - 4)
    at, w = sheet(x0 + case["box"] + 4)
    src = {"kind": "dipole", "e": e, "coef": 0.3 * amp, "wave": _ramped(om, dt, case["steps"] + 8, rng.uniform(0, 6.28))}
    mon = {"omega": np.array([om]), "e": at, "h1": None, "h2": None, "energy": 0, "of": None}
    return _base(n, (dx,) * 3, dt, ((p, p),) * 3, case["stride"], False, alpha=0.05 * om, eps_ref=1.44 ** 2,
                 inv_eps=1 / eps, sources=[src], monitors=[mon], box=box, w=w)


def _shell(case, seed):
    """The scattering case with a design box around the particle and the scattered flux, summed over the
    wavelengths, as the objective."""
    p = _scatter({**case, "mirror": False, "mixed": False, "nf": 8, "double": False}, seed)
    mid, half = p["inside"]
    p["box"] = tuple((int(mid[a] - 0.7 * half) - 2, int(mid[a] + 0.7 * half) + 4) for a in range(3))
    return p


def _problem(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        sizes = np.random.default_rng(case["runs"] + 1000 * case["lo"] + case["hi"])  # the periods: the case's, not the seed's
        rng = np.random.default_rng(seed)
        return [_cell(case, sizes.uniform(case["lo"], case["hi"]), rng) for _ in range(case["runs"])]
    if kind == "gradient":
        return _shell(case, seed) if case["metal"] else _slab(case, seed)
    return {"device": _device, "scatter": _scatter, "bulk": _bulk}[kind](case, seed)


def _objective(p, acc_e, acc_h):
    """The real scalar a gradient case differentiates, of the first monitor's accumulators."""
    if "w" in p:
        a = (torch.as_tensor(p["w"], dtype=torch.complex128, device=acc_e.device) * acc_e[0]).sum()
        return (a * a.conj()).real
    s = torch.as_tensor(p["sign"], dtype=torch.float64, device=acc_e.device)
    return 0.5 * ((acc_e * acc_h.conj()).real * s).sum()


# --- through the framework ------------------------------------------------------------------------------------------


def _plan(p):
    """The framework's plan of a problem."""
    src, views = [], {}
    metal = Medium(METAL[0], tuple(Pole(*q) for q in METAL[1]))
    for s in p["sources"]:
        if s["kind"] == "table":
            def points(q):
                return TablePoints(q[0], np.zeros(len(q[0]), np.int64), q[1], q[2], q[3])
            rows = len(s["table"])
            view = views["view"] = object()
            src.append(TableSource(s["table"], s["inc"].reshape(-1), s["m"], s["cmax"], points(s["E"]), points(s["H"]),
                                   (rows * np.arange(3), *s["view"]), view))
        elif s["kind"] == "dipole":
            src.append(DipoleSource(s["e"], s["coef"], s["wave"]))
        elif s["kind"] == "mode":
            src.append(ModeSource(s["h"], s["mH"], s["tE"], s["e"], s["mE"], s["tH"]))
        else:
            src.append(ColumnSource(_plan(s["col"]), s["k_src"], s["k_launch"], s["phase"], s["amp"], s["wave"],
                                    s["cE"], s["cH"]))
            views["column"] = src[-1]
    groups = [DispersiveGroup(g["idx"], [metal] if g["w"] is None else [Medium(1.33 ** 2), metal],
                              np.ones((1, len(g["idx"]))) if g["w"] is None else g["frac"], g["w"]) for g in p["groups"]]
    mons = [DFTMonitor(m["omega"], m["e"], m["h1"], m["h2"], energy=m["energy"],
                       source=None if m["of"] is None else views[m["of"]]) for m in p["monitors"]]
    inv = p["inv_eps"]
    on_gpu = isinstance(inv, torch.Tensor)
    plan = make_plan(shape=p["n"], dx=p["dx"], dt=p["dt"], single=not p["double"],
                     inv_eps=np.broadcast_to(1.0, p["n"]) if on_gpu else inv, groups=groups,
                     pml=PMLSpec(cells=p["pml"], alpha_max=p["alpha"], eps_ref=p["eps_ref"]), sources=src,
                     monitors=mons, dft_stride=p["stride"], periodic=p["per"], bloch=p["bloch"], mirror=p["mirror"])
    if on_gpu:
        plan["inv_eps"] = inv
    return plan


def prepare(case, seed):
    p = _problem(case, seed)
    if case["kind"] == "sweep":
        engines = [Engine.from_plan(_plan(q)) for q in p]
        if case["batched"]:
            return {"engines": engines, "batch": BlochBatch(engines, min(len(q["sources"][0]["wave"]) for q in p) - 1),
                    "steps": case["steps"]}
        return {"engines": engines, "runners": [e.make_runner(True)[0] for e in engines]}
    if case["kind"] == "gradient":
        run_ = AdjointRun(_plan(p), p["box"], checkpoint=case["checkpoint"], objective=lambda e, h: _objective(p, e, h))
        return {"adjoint": run_, "steps": case["steps"]}
    eng = Engine.from_plan(_plan(p))
    return {"engine": eng, "runner": eng.make_runner(True)[0], "calls": case["calls"]}


def _accs(eng):
    return [[m["acc_e"]] + ([] if m["acc_h"] is None else [m["acc_h"]]) for m in eng.monitors]


def run(state):
    if "adjoint" in state:
        a = state["adjoint"]
        J, (acc_e, acc_h) = a.forward(state["steps"])
        return {"J": J, "acc": [acc_e] if acc_h is None else [acc_e, acc_h], "grad": a.backward()}
    if "engines" in state:
        if "batch" in state:
            state["batch"].run(state["steps"])
        else:
            for r in state["runners"]:
                r()
        return [[e.E, e.H, *_accs(e)[0]] for e in state["engines"]]
    for _ in range(state["calls"]):
        state["runner"]()
    eng = state["engine"]
    return {"E": eng.E, "H": eng.H, "acc": _accs(eng), "energy": eng.energy}


# --- the same in float64, with torch alone --------------------------------------------------------------------------


class _Reference:
    def __init__(self, p):
        self.p, self.n, self.t = p, p["n"], 0
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.cx = any(p["bloch"])
        self.ft = torch.complex128 if self.cx else torch.float64
        self.E, self.H = (torch.zeros((3,) + self.n, dtype=self.ft, device=self.dev) for _ in range(2))
        inv = self.d(p["inv_eps"])
        self.coef = [p["dt"] * inv] * 3 if inv.dim() == 3 else [p["dt"] * inv[c] for c in range(3)]
        del inv
        self.region = {k: [[self._range(k, c, a) for a in range(3)] for c in range(3)] for k in "EH"}
        self.slabs, self.psi = self._cpml()
        self.sources = [{**s, "ref": _Reference(s["col"])} if s["kind"] == "column" else dict(s) for s in p["sources"]]
        for s in self.sources:
            for k in ("e", "h", "coef", "wave", "mH", "tE", "mE", "tH", "table", "phase"):
                if k in s:
                    s[k] = self.d(s[k], keep=True)
            if s["kind"] == "table":
                s["E"], s["H"] = ([self.d(v, keep=True) for v in s[k]] for k in "EH")
                s["now"] = torch.zeros(3, dtype=torch.float64, device=self.dev)
        self.groups = [self._group(g) for g in p["groups"]]
        self.acc = [[torch.zeros((len(m["omega"]), len(m["e"])), dtype=torch.complex128, device=self.dev)
                     for _ in range(1 if m["h1"] is None else 2)] for m in p["monitors"]]
        self.energy = torch.zeros(2, dtype=torch.float64, device=self.dev)

    def d(self, v, keep=False):
        v = torch.as_tensor(v, device=self.dev)
        return v if keep and not v.is_floating_point() else v.to(torch.float64)

    def _range(self, kind, c, a):
        n, per, m = self.n[a], self.p["per"][a], self.p["mirror"][a]
        if kind == "E":
            return ((2 if m < 0 and a != c else 1) if m else (1 if per or a != c else 0)), n - 1
        top = n if a == c and not per else n - 1
        return ((2 if m < 0 and a == c else 1) if m else (1 if per else 0)), top

    def _cpml(self):
        slabs, psi = [], []
        for a, (lo, hi) in enumerate(self.p["pml"]):
            if not (lo or hi):
                continue
            n, h, dt = self.n[a], self.p["dx"][a], self.p["dt"]
            smax = 0.8 * 4 / (math.sqrt(self.p["eps_ref"]) * h)
            for kind in "HE":
                u = torch.arange(n, dtype=torch.float64, device=self.dev) + (0.5 if kind == "H" else 0.0)
                rho = torch.zeros_like(u)
                if lo:
                    rho = torch.maximum(rho, ((lo - u) / lo).clamp(0, 1))
                if hi:
                    rho = torch.maximum(rho, ((u - (n - 1 - hi)) / hi).clamp(0, 1))
                sig, al = smax * rho ** 3, self.p["alpha"] * (1 - rho) * (rho > 0)
                b = torch.exp(-(sig + al) * dt)
                c = torch.where(sig > 0, sig * (b - 1) / (sig + al).clamp(min=1e-300), torch.zeros_like(sig))
                for comp in range(3):
                    if comp == a:
                        continue
                    start, stop = self.region[kind][comp][a]
                    for x0, x1 in ([(start, min(stop, lo + 1))] if lo else []) + (
                            [(max(start, n - 2 - hi), stop)] if hi else []):
                        r = list(self.region[kind][comp])
                        r[a] = (x0, x1)
                        shape = [1, 1, 1]
                        shape[a] = x1 - x0
                        slabs.append((kind, comp, a, tuple(slice(*q) for q in r), b[x0:x1].view(shape),
                                      c[x0:x1].view(shape)))
                        psi.append(torch.zeros([q[1] - q[0] for q in r], dtype=self.ft, device=self.dev))
        return slabs, psi

    def _group(self, g):
        idx = self.d(g["idx"], keep=True)
        z = torch.zeros(len(idx), dtype=self.ft, device=self.dev)
        dt, poles = self.p["dt"], []
        for s, w0, ga in METAL[1]:
            den = 1 + ga * dt / 2
            poles.append(((2 - w0 ** 2 * dt ** 2) / den, -(1 - ga * dt / 2) / den, s * dt ** 2 / den))
        out = {"idx": idx, "poles": poles, "w": None, "state": [z] * (4 + 4 * len(poles))}
        if g["w"] is not None:
            out["w"], out["f"] = self.d(g["w"]), self.d(g["frac"])
        return out

    def _diff(self, F, comp, axis, r, forward):
        s = list(r)
        k = 1 if forward else -1
        s[axis] = slice(r[axis].start + k, r[axis].stop + k)
        v = F[comp][tuple(s)] - F[comp][r] if forward else F[comp][r] - F[comp][tuple(s)]
        return v * (1 / self.p["dx"][axis])

    def _half(self, kind):
        tgt, src, fwd = (self.H, self.E, True) if kind == "H" else (self.E, self.H, False)
        for c in range(3):
            r = tuple(slice(*q) for q in self.region[kind][c])
            curl = self._diff(src, (c + 2) % 3, (c + 1) % 3, r, fwd) - self._diff(src, (c + 1) % 3, (c + 2) % 3, r, fwd)
            tgt[c][r] += curl * (-self.p["dt"]) if kind == "H" else curl * self.coef[c][r]
        for q, (k, c, a, r, b, cc) in enumerate(self.slabs):
            if k != kind:
                continue
            first = a == (c + 1) % 3
            der = self._diff(src, (c + 2) % 3 if first else (c + 1) % 3, a, r, fwd)
            sgn = (1.0 if first else -1.0) * (-1.0 if kind == "H" else 1.0)
            scale = sgn * cc * self.p["dt"] if kind == "H" else sgn * cc * self.coef[c][r].detach()
            self.psi[q] = b * self.psi[q] + scale * der
            tgt[c][r] += self.psi[q]

    def _ghosts(self, F, low):
        for a in range(3):
            if self.p["per"][a]:
                n = self.n[a]
                dst, src = (0, n - 2) if low else (n - 1, 1)
                kl = self.p["bloch"][a] * (n - 2) * self.p["dx"][a] * (-1 if low else 1)
                v = F.select(a + 1, src).clone()
                F.select(a + 1, dst).copy_(v * complex(math.cos(kl), math.sin(kl)) if self.cx else v)

    def _read(self, s, i0, u0):
        """The table's waveform at fine times n + i0 + u0, quintic Lagrange interpolation on six samples."""
        q = self.t + i0
        c = torch.clamp(q // s["m"], max=s["cmax"])
        u = (q % s["m"] + u0) / s["m"]
        out = torch.zeros_like(u)
        for j in range(6):
            w = torch.ones_like(u)
            for k in range(6):
                if k != j:
                    w = w * (u - (k - 2)) / (j - k)
            out = out + w * s["table"][c + j]
        return out

    def _correct(self, kind):
        F = self.H if kind == "H" else self.E
        flat = F.view(-1)
        for s in self.sources:
            if s["kind"] == "table":
                idx, i0, u0, coef = s[kind]
                flat.index_add_(0, idx, coef * self._read(s, i0, u0))
            elif s["kind"] == "dipole" and kind == "E":
                flat.index_add_(0, s["e"], -s["coef"] * s["wave"][self.t])
            elif s["kind"] == "mode":
                i, m, t = (s["h"], s["mH"], s["tE"]) if kind == "H" else (s["e"], s["mE"], s["tH"])
                flat.index_add_(0, i, m @ t[self.t])
            elif s["kind"] == "column":
                ref, k = s["ref"], s["k_src"]
                src, at, z, cf = (ref.E, k, k - 1, s["cH"]) if kind == "H" else (ref.H, k - 1, k, -s["cE"])
                ph = s["phase"].to(self.ft)
                F[0, 1:-1, 1:-1, z] -= cf * ph * src[1, 1, 1, at]
                F[1, 1:-1, 1:-1, z] += cf * ph * src[0, 1, 1, at]

    def _poles(self, g, at, drive):
        tot = 0
        for k, (c1, c2, c3) in enumerate(g["poles"]):
            p0, p1 = g["state"][at + 2 * k], g["state"][at + 2 * k + 1]
            new = c1 * p0 + c2 * p1 + c3 * drive
            g["state"][at + 2 * k], g["state"][at + 2 * k + 1] = new, p0
            tot = tot + new
        return tot

    def _disperse(self, g):
        """state: D, the E before, the harmonic and the arithmetic path's E, then the poles of either path."""
        st, flat, np_ = g["state"], self.E.view(-1), len(g["poles"])
        D = st[0] + (flat[g["idx"]] - st[1])
        if g["w"] is None:
            e = (D - self._poles(g, 4, st[1])) / METAL[0]
        else:
            eh = (D - self._poles(g, 4, st[2])) / METAL[0]
            ea = (D - g["f"][1] * self._poles(g, 4 + 2 * np_, st[3])) / (g["f"][0] * 1.33 ** 2 + g["f"][1] * METAL[0])
            e = g["w"] * (g["f"][0] / 1.33 ** 2 * D + g["f"][1] * eh) + (1 - g["w"]) * ea
            st[2], st[3] = eh, ea
        flat.index_copy_(0, g["idx"], e)
        st[0], st[1] = D, e

    def half_h(self):
        self._ghosts(self.E, False)
        self._half("H")

    def half_e(self):
        self._ghosts(self.H, True)
        for a in range(3):
            if self.p["mirror"][a] > 0:
                for c in ((a + 1) % 3, (a + 2) % 3):
                    self.H[c].select(a, 0).copy_(-self.H[c].select(a, 1))
        self._half("E")

    def step(self):
        self.half_h()
        self._correct("H")
        cols = [s for s in self.sources if s["kind"] == "column"]
        for s in cols:
            s["ref"].half_h()
        self.half_e()
        self._correct("E")
        for g in self.groups:
            self._disperse(g)
        for s in cols:
            s["ref"].half_e()
            for c in range(2):
                s["ref"].E[c, 1, 1, s["k_launch"]] += s["amp"][c] * s["wave"][self.t]
        for s in self.sources:
            if s["kind"] == "table":
                s["now"][0] = self._read(s, *(self.d(v[:1], keep=True) for v in s["view"]))[0]
        self.t += 1

    def sample(self):
        en = [None, None]
        for m, acc in zip(self.p["monitors"], self.acc):
            E, H = self.E.view(-1), self.H.view(-1)
            for s in self.sources:
                if m["of"] == "view" and s["kind"] == "table":
                    E = s["now"]
                if m["of"] == "column" and s["kind"] == "column":
                    E, H = s["ref"].E.view(-1), s["ref"].H.view(-1)
            om = self.d(m["omega"])
            te = self.t * self.p["dt"]
            e = E[self.d(m["e"], keep=True)].to(torch.complex128)
            acc[0] = acc[0] + torch.exp(1j * om * te)[:, None] * e
            if m["h1"] is not None:
                h = 0.5 * (H[self.d(m["h1"], keep=True)] + H[self.d(m["h2"], keep=True)]).to(torch.complex128)
                acc[1] = acc[1] + torch.exp(1j * om * (te - 0.5 * self.p["dt"]))[:, None] * h
                if m["energy"]:
                    v = (e.abs() ** 2).sum() + (h.abs() ** 2).sum()
                    en[m["energy"] - 1] = v if en[m["energy"] - 1] is None else en[m["energy"] - 1] + v
        for k, v in enumerate(en):
            if v is not None:
                self.energy[k] = v.detach()

    def advance(self, steps):
        for _ in range(steps):
            self.step()
            if self.t % self.p["stride"] == 0:
                self.sample()

    # the state the adjoint's segments start from
    def state(self):
        return [self.E, self.H, *self.psi, *[v for g in self.groups for v in g["state"]]]

    def set_state(self, v, t):
        self.E, self.H, rest, self.t = v[0], v[1], list(v[2:]), t
        self.psi = rest[:len(self.psi)]
        rest = rest[len(self.psi):]
        for g in self.groups:
            g["state"] = rest[:len(g["state"])]
            rest = rest[len(g["state"]):]


def _gradient(p, steps):
    """(J, accumulators of the first monitor, dJ/d(1/eps) over the box) by torch autograd, a segment at a time."""
    r = _Reference(p)
    seg = p["stride"] * max(1, 16 // p["stride"])
    kept = []
    with torch.no_grad():
        for t in range(0, steps, seg):
            kept.append((t, [v.clone() for v in r.state()]))
            r.advance(min(seg, steps - t))
    acc = [a.clone().requires_grad_(True) for a in r.acc[0]]
    J = _objective(p, acc[0], acc[1] if len(acc) > 1 else None)
    g_acc = torch.autograd.grad(J, acc)
    sl = tuple(slice(a, b) for a, b in p["box"])
    coef = r.coef
    total, bar = 0, None
    for t, s0 in reversed(kept):
        leaf = [v.detach().requires_grad_(True) for v in s0]
        boxes = [c[sl].detach().clone().requires_grad_(True) for c in coef]
        r.coef = [c.detach().clone() for c in coef]
        for c, b in zip(r.coef, boxes):
            c[sl] = b
        r.set_state([v.clone() for v in leaf], t)
        r.acc = [[torch.zeros_like(x) for x in a] for a in r.acc]
        r.advance(min(seg, steps - t))
        out, weight = list(r.acc[0]), [g for g in g_acc]
        if bar is not None:
            pairs = [(o, b) for o, b in zip(r.state(), bar) if b is not None and o.requires_grad]
            out, weight = out + [o for o, _ in pairs], weight + [b for _, b in pairs]
        use = [(o, w) for o, w in zip(out, weight) if o.requires_grad]
        if not use:
            continue
        got = torch.autograd.grad([o for o, _ in use], boxes + leaf, [w for _, w in use], allow_unused=True)
        total = total + sum(g for g in got[:3] if g is not None)
        bar = got[3:]
        r.acc = [[x.detach() for x in a] for a in r.acc]
    return float(J), [a.detach() for a in acc], total * p["dt"]


def exact(case, seed):
    p = _problem(case, seed)
    if case["kind"] == "gradient":
        J, acc, grad = _gradient(p, case["steps"])
        return {"J": J, "acc": acc, "grad": grad}
    with torch.no_grad():
        if case["kind"] == "sweep":
            out = []
            for q in p:
                r = _Reference(q)
                r.advance(case["steps"] if case["batched"] else q["stride"])
                out.append([r.E, r.H, *r.acc[0]])
            return out
        r = _Reference(p)
        r.advance(case["calls"] * case["stride"])
    return {"E": r.E, "H": r.H, "acc": r.acc, "energy": r.energy}


# --- what a pass cannot do without, and how exact it is -------------------------------------------------------------


def work(case):
    """State, coefficients and accumulators moved once a pass, and the steps' arithmetic: 30 operations a cell for the
    two curls and their updates (36 where spacings differ), 24 for each axis whose CPML holds the cell; four times
    that for complex values, and twice for the reverse steps and the recomputed forward ones of a gradient."""
    kind = case["kind"]
    if kind == "sweep":
        mean = ((case["lo"] + case["hi"]) / 20 + 2) ** 2 * case["nz"] * case["runs"]
        slab = mean * (2 * case["pml"] + 2) / case["nz"]
        steps = case["steps"] if case["batched"] else 8
        return {"bytes": mean * 100 + slab * 64, "flops": steps * 2 * (36 * mean + 24 * slab)}
    n = [case["n0"], case["n1"], case.get("n2", 3)]
    cells = n[0] * n[1] * n[2]
    pairs = 0
    for a in range(3):
        sides = 0 if kind == "device" and a == 2 else (1 if case.get("mirror") and a < 2 else 2)
        pairs += sides * (case["pml"] + 1) * cells // n[a]
    size = 8 if case.get("double") else 4
    steps = case["steps"] if kind == "gradient" else case["calls"] * case["stride"]
    coef = 3 if kind == "scatter" or case.get("metal") else 1
    flops = steps * (30 * cells + 24 * pairs)
    state = size * ((12 + coef) * cells + 8 * pairs)
    return {"bytes": state * (3 if kind == "gradient" else 1), "flops": flops * (3 if kind == "gradient" else 1)}


def tolerance(case):
    """About four times the distance from ``exact`` that was measured: 3e-16 at most in float64; in float32 up to 3e-7
    for fields, 9e-7 for accumulators and 1.3e-6 for gradients."""
    if case.get("double"):
        return {"rel": 2e-15, "max": 1e-12}
    return {"rel": 6e-6, "max": 3e-4}
