"""The framework's workloads as callable cases.

A case is a dict of plain values.  ``prepare`` makes what a program holds
before a tracking call (particles, a compiled lattice or a job), ``run`` is
one pass through the public entry points, ``work`` what the pass cannot do
without and ``exact`` the same result from plain float64 torch code.

Kinds:

* ``ring``    -- until-turn tracking of a long synthetic ring (drifts,
                 quadrupole-led multipoles of order 1-10, shifts, rotations,
                 cavities, elliptic apertures) on device-resident particles;
                 ``cells`` = 4000 is the 20,000-element ring.  A polar
                 amplitude grid is a dynamic-aperture study (it loses
                 particles), a Gaussian beam an ordinary one.
* ``fodo``    -- the same call on the short FODO ring, many turns.
* ``line``    -- ``track_line`` through a section of the ring.
* ``job``     -- ``TrackJob`` on host buffers: push, track, collect; with
                 ``output`` "monitor" (turn-by-turn) or "elements"
                 (element-by-element) the stored records are collected too.
* ``beams``   -- FODO ring with 4D / 6D beam-beam and space-charge kicks.
* ``tricub``  -- FODO ring with field-map kicks on one shared grid.
* ``adjoint`` -- differentiable tracking: forward, loss, backward.
* ``batch``   -- several ring variants in one persistent launch.

``mode`` is the arithmetic policy: "exact" (the default of every entry
point) or "fast".
"""

import math
from functools import lru_cache

import numpy as np
import torch

from sixtracklib_gb300.autodiff import DifferentiableLattice, coordinates
from sixtracklib_gb300.batch import BatchTracker
from sixtracklib_gb300.beam_elements import Elements, bb6d_data
from sixtracklib_gb300.device import DeviceTracker
from sixtracklib_gb300.particles import ParticlesSet
from sixtracklib_gb300.trackjob import TrackJob

P0C, MASS0 = 7e12, 938272088.16
EPS0, CLIGHT = 8.854187817620e-12, 299792458.0
QE_BB, QE_SC, QE_PART = 1.60217662e-19, 1.602176634e-19, 1.602176634e-19
KINDS = ("ring", "fodo", "line", "job", "beams", "tricub", "adjoint", "batch")
GRID = (100, 100, 50, 0.25e-3, 0.25e-3, 0.02)  # nodes and steps of the field map


def listed():
    return [
        # the smallest call: a job on host buffers, one turn of a short ring
        dict(name="job_1k_fodo_1turn", kind="job", n=1000, turns=1, mode="exact", output="none"),
        # turn-by-turn monitor data of a beam with an odd particle count
        dict(name="job_5k_monitor", kind="job", n=5003, turns=16, mode="exact", output="monitor"),
        # element-by-element output, the debugging and optics use
        dict(name="job_777_elements", kind="job", n=777, turns=1, mode="exact", output="elements"),
        # ordinary beam, many turns of a short ring, default arithmetic
        dict(name="fodo_10k_exact", kind="fodo", n=10000, turns=100, mode="exact", beam="gauss"),
        # the headline: a dynamic-aperture scan of the 20,000-element ring
        dict(name="ring_1m_polar_fast", kind="ring", n=1000000, cells=4000, turns=1, mode="fast", beam="polar"),
        # the same ring, ordinary beam, default arithmetic
        dict(name="ring_131k_exact", kind="ring", n=131072, cells=4000, turns=1, mode="exact", beam="gauss"),
        # a section of the ring, ragged particle count
        dict(name="line_20k_exact", kind="line", n=20011, cells=800, begin=501, end=3333, mode="exact", beam="gauss"),
        # colliding beams with space charge: round and elliptic strong beams
        dict(name="beams_round_65k_fast", kind="beams", n=65536, turns=2, mode="fast", elliptic=False),
        dict(name="beams_elliptic_33k_fast", kind="beams", n=33333, turns=1, mode="fast", elliptic=True),
        # electron-cloud style field-map kicks
        dict(name="tricub_65k_fast", kind="tricub", n=65536, turns=2, mode="fast"),
        # gradients of a loss on the final coordinates
        dict(name="adjoint_16k_20turns", kind="adjoint", n=16384, turns=20, mode="fast"),
        # a scan over lattice variants of different size and beam
        dict(name="batch_9_fast", kind="batch", n=40000, variants=9, cells=400, turns=2, mode="fast"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(KINDS)
    mode = rng.choice(("exact", "fast"))
    beam = rng.choice(("gauss", "polar"))
    if kind == "ring":
        cells = _log(rng, 60, 4000)
        return dict(kind=kind, n=_log(rng, 500, 400000), cells=cells, turns=max(1, 4000 // cells // 4), mode=mode, beam=beam)
    if kind == "fodo":
        return dict(kind=kind, n=_log(rng, 100, 200000), turns=_log(rng, 1, 100), mode=mode, beam=beam)
    if kind == "line":
        cells = _log(rng, 60, 2000)
        b = rng.randrange(0, 2 * cells)
        return dict(kind=kind, n=_log(rng, 500, 200000), cells=cells, begin=b, end=rng.randrange(b + 1, 4 * cells), mode=mode, beam="gauss")
    if kind == "job":
        out = rng.choice(("none", "monitor", "elements"))
        top = {"none": 100000, "monitor": 6000, "elements": 1000}[out]
        return dict(kind=kind, n=_log(rng, 64, top), turns=1 if out == "elements" else rng.randint(1, 16), mode=mode, output=out)
    if kind == "beams":
        return dict(kind=kind, n=_log(rng, 1000, 100000), turns=1, mode=mode, elliptic=rng.random() < 0.5)
    if kind == "tricub":
        return dict(kind=kind, n=_log(rng, 1000, 200000), turns=rng.randint(1, 4), mode=mode)
    if kind == "adjoint":
        return dict(kind=kind, n=_log(rng, 500, 20000), turns=rng.randint(2, 20), mode=mode)
    return dict(kind=kind, n=_log(rng, 2000, 50000), variants=rng.randint(3, 9), cells=_log(rng, 60, 400), turns=rng.randint(1, 4), mode=mode)


# ------------------------------------------------- lattices as plain tuples
def _fodo():
    e = []
    for _ in range(64):
        e += [("d", 2.0), ("m", (0.0, 0.05)), ("d", 2.0), ("m", (0.0, -0.05))]
    return e + [("c", 6e6, 400e6, 180.0), ("b", -0.02, 0.02, -0.02, 0.02)]


@lru_cache(maxsize=64)
def _ring(cells, seed=20240601):
    """FODO cells with a slow ramp of quadrupole strengths, multipole errors,
    and the extras in the proportions of the 20,000-element ring."""
    rng = np.random.default_rng(seed)
    k = np.sort(rng.uniform(0.01, 0.05, cells))
    k = np.concatenate([k[0::2], k[1::2][::-1]])
    length = rng.uniform(0.5, 5.0, cells)
    orders = rng.integers(1, 11, size=2 * cells)
    split = set(int(i) for i in rng.choice(2 * cells, size=cells // 4, replace=False))
    extra = {}
    for kind, num in (("x", cells // 4), ("r", cells // 4), ("e", cells // 4)):
        for s in rng.choice(2 * cells, size=num):
            extra.setdefault(int(s), []).append(kind)
    n_cav = max(1, cells // 250)
    cav = set(int(i) for i in np.linspace(0, 2 * cells, n_cav, endpoint=False))
    e = []
    for j in range(2 * cells):
        half = float(length[j // 2])
        e += [("d", 0.5 * half)] * 2 if j in split else [("d", half)]
        knl = [0.0, float(k[j // 2] if j % 2 == 0 else -k[j // 2])]
        knl += [float(rng.normal(0.0, 1e-4 * 10.0 ** -n)) for n in range(2, int(orders[j]) + 1)]
        e.append(("m", tuple(knl)))
        if j in cav:
            e.append(("c", 6e6 / n_cav, 400e6, 180.0))
        for kind in extra.get(j, ()):
            if kind == "x":
                e.append(("x", float(rng.normal(0, 1e-5)), float(rng.normal(0, 1e-5))))
            elif kind == "r":
                a = float(rng.normal(0.0, 1e-4))
                e.append(("r", math.cos(a), math.sin(a)))
            else:
                e.append(("e", 0.015, 0.01))
    return tuple(e)


@lru_cache(maxsize=4)
def _beams(elliptic):
    """FODO ring, 4 6D beam-beam (21 slices), 4 4D beam-beam, 200 space-charge kicks."""
    rng = np.random.default_rng(7)
    s, ns = 16.7e-6, 21
    sy = 1.3 * s if elliptic else s
    z = tuple(float(np.sqrt(2) * 0.0755 * v) for v in torch.special.erfinv(
        torch.linspace(-1, 1, 2 * ns + 1, dtype=torch.float64)[1::2]).numpy())
    e = _fodo()
    for _ in range(4):
        e += [("6", float(rng.uniform(1e-4, 2e-4)), float(rng.uniform(0, 0.5)), float(rng.normal(0, 1e-6)),
               float(rng.normal(0, 1e-6)), 1.15e11 / ns, z, s, sy), ("d", 1.0)]
    for _ in range(4):
        e += [("4", 1.15e11, s, sy, 1.0, float(rng.normal(0, 1e-6)), float(rng.normal(0, 1e-6))), ("d", 1.0)]
    return tuple(e + [("s", 1e11, 0.1, 1e-3, 1.2e-3 if elliptic else 1e-3, 0.1)] * 200)


@lru_cache(maxsize=1)
def _field_map():
    """Node table of a Gaussian potential bump and its scaled derivatives."""
    nx, ny, nz, dx, dy, dz = GRID
    ax = []
    for n, d, s in ((nx, dx, 3e-3), (ny, dy, 2.5e-3), (nz, dz, 0.2)):
        u = d * (np.arange(n) - 0.5 * (n - 1))
        g = np.exp(-0.5 * (u / s) ** 2)
        ax.append((g, -u / (s * s) * g * d))
    t = np.empty((nz, ny, nx, 8))
    for k, (a, b, c) in enumerate(((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1))):
        t[..., k] = 2e-11 * ax[2][c][:, None, None] * ax[1][b][None, :, None] * ax[0][a][None, None, :]
    return t


def _tricub():
    e = []
    for i, o in enumerate(_fodo()):
        e.append(o)
        if i % 4 == 3:
            e.append(("t", 0.5))
    return e


def _learnable():
    rng = np.random.default_rng(4)
    e, quads, sexts = [], [], []
    for c in range(64):
        sext = c % 4 == 0
        e.append(("d", 2.0))
        quads.append(len(e))
        if sext:
            sexts.append(len(e))
        e.append(("m", (0.0, 0.05, float(rng.normal(0, 0.1))) if sext else (0.0, 0.05)))
        e += [("d", 2.0), ("m", (0.0, -0.05))]
    e += [("c", 6e6, 400e6, 180.0), ("b", -0.02, 0.02, -0.02, 0.02)]
    return e, [(q, "knl", 1) for q in quads] + [(s, "knl", 2) for s in sexts]


def _plain_elements(case):
    kind = case["kind"]
    if kind in ("ring", "line"):
        return _ring(case["cells"])
    return {"fodo": _fodo, "job": _fodo, "tricub": _tricub}[kind]() if kind != "beams" else _beams(case["elliptic"])


def _elements(plain):
    e = Elements()
    maps = sum(o[0] == "t" for o in plain)
    for o in plain:
        k = o[0]
        if k == "d":
            e.Drift(length=o[1])
        elif k == "m":
            e.Multipole(knl=list(o[1]))
        elif k == "c":
            e.Cavity(voltage=o[1], frequency=o[2], lag=o[3])
        elif k == "x":
            e.XYShift(dx=o[1], dy=o[2])
        elif k == "r":
            e.SRotation(cos_z=o[1], sin_z=o[2])
        elif k == "e":
            e.LimitEllipse(a=o[1], b=o[2])
        elif k == "b":
            e.LimitRect(min_x=o[1], max_x=o[2], min_y=o[3], max_y=o[4])
        elif k == "6":
            e.BeamBeam6D(data=bb6d_data(
                q_part=QE_PART, phi=o[1], alpha=o[2], delta_x=o[3], delta_y=o[4], n_part_per_slice=np.full(len(o[6]), o[5]),
                z_slices=np.array(o[6]), sigmas=(o[7] ** 2, 0.0, 0.0, 0.0, 1e-12, 0.0, 0.0, o[8] ** 2, 0.0, 1e-12)))
        elif k == "4":
            e.BeamBeam4D(charge=o[1], sigma_x=o[2], sigma_y=o[3], beta_r=o[4], min_sigma_diff=1e-10, x_bb=o[5], y_bb=o[6],
                         d_px=0.0, d_py=0.0, enabled=1.0)
        elif k == "s":
            e.SCQGaussProfile(number_of_particles=o[1], bunchlength_rms=o[2], sigma_x=o[3], sigma_y=o[4], length=o[5],
                              x_co=0.0, y_co=0.0, min_sigma_diff=1e-10, q_param=1.0, enabled=1)
        elif k == "t":
            e.TriCub(data=len(plain), length=o[1])
    if maps:
        nx, ny, nz, dx, dy, dz = GRID
        e.TriCubData(nx=nx, ny=ny, nz=nz, x0=-0.5 * (nx - 1) * dx, y0=-0.5 * (ny - 1) * dy, z0=-0.5 * (nz - 1) * dz,
                     dx=dx, dy=dy, dz=dz, table_addr=_field_map().reshape(-1))
    return e


_IMAGES = {}


def _image(key, plain):
    """A lattice's buffer; a program builds it once and keeps it."""
    if key not in _IMAGES:
        while len(_IMAGES) >= 64:
            _IMAGES.pop(next(iter(_IMAGES)))
        _IMAGES[key] = _elements(plain).cbuffer.to_image()
    return _IMAGES[key]


# ------------------------------------------------------------------- beams
def _beam(n, seed, beam="gauss"):
    """A 21 x n column block: 7 TeV protons, a Gaussian beam (1 mm, 10 urad,
    5 cm, 1e-4) or a polar amplitude grid up to 20 mm."""
    rng = np.random.default_rng(seed)
    f = np.zeros((21, n))
    e0 = math.sqrt(P0C * P0C + MASS0 * MASS0)
    f[0], f[1], f[2], f[3], f[4], f[15], f[16] = 1.0, MASS0, P0C / e0, e0 / MASS0, P0C, 1.0, 1.0
    if beam == "polar":
        r, th = np.meshgrid(np.linspace(0.0, 0.02, -(-n // 11)), np.linspace(0.0, 0.5 * np.pi, 11), indexing="ij")
        f[6], f[7] = (r * np.cos(th)).reshape(-1)[:n], (r * np.sin(th)).reshape(-1)[:n]
        delta = rng.uniform(-3e-4, 3e-4, n)
    else:
        f[6], f[7] = rng.normal(0, 1e-3, n), rng.normal(0, 1e-3, n)
        f[8], f[9] = rng.normal(0, 1e-5, n), rng.normal(0, 1e-5, n)
        f[10], delta = rng.normal(0, 0.05, n), rng.normal(0, 1e-4, n)
    b0 = f[2]
    ptau_b0 = np.sqrt((delta * b0) ** 2 + 2.0 * delta * b0 * b0 + 1.0) - 1.0
    f[11], f[12], f[13], f[14] = ptau_b0 / (b0 * b0), delta, 1.0 / (1.0 + delta), (1.0 + delta) / (1.0 + ptau_b0)
    k = f.view(np.int64)
    k[17], k[18], k[19], k[20] = np.arange(n), 0, 0, 1
    return f


def _columns(n, seed, beam):
    return torch.from_numpy(_beam(n, seed, beam).view(np.int64)).cuda()


def _variants(case):
    """(cells, particles) of the variants of a batch, spread around the case's."""
    rng = np.random.default_rng(case["variants"] * 1000 + case["cells"])
    return [(int(max(16, case["cells"] * rng.uniform(0.2, 1.0))), int(max(100, case["n"] * rng.uniform(0.05, 1.0))))
            for _ in range(case["variants"])]


# --------------------------------------------------------------- the calls
def prepare(case, seed):
    kind, cfg = case["kind"], "mode=" + case.get("mode", "exact")
    key = tuple(sorted((k, v) for k, v in case.items() if k in ("kind", "cells", "elliptic")))
    if kind == "job":
        lat = _elements(_fodo())
        if case["output"] == "monitor":
            lat.BeamMonitor(num_stores=case["turns"], start=0, skip=1, is_rolling=False, is_turn_ordered=True)
        ps = ParticlesSet()
        p = ps.Particles(num_particles=case["n"])
        block = _beam(case["n"], seed).view(np.uint64)
        p.set_block(block)
        job = TrackJob(lat, ps, until_turn_elem_by_elem=1 if case["output"] == "elements" else 0, config_str=cfg)
        return dict(case=case, job=job, p=p, block=block, keep=(lat, ps))
    if kind == "adjoint":
        plain, params = _learnable()
        lat = DifferentiableLattice(_elements(plain), params, cfg)
        cols = _columns(case["n"], seed, "gauss")
        return dict(case=case, lat=lat, cols=cols, coords=coordinates(cols).clone().requires_grad_(True),
                    values=torch.tensor(lat.initial_values, dtype=torch.float64, device="cuda", requires_grad=True))
    if kind == "batch":
        sizes = _variants(case)
        trk = [DeviceTracker(_image(("v", c, i), _ring(c, 100 + i)), cfg) for i, (c, _) in enumerate(sizes)]
        cols = [_columns(n, seed * 100 + i, "gauss") for i, (_, n) in enumerate(sizes)]
        work = [c.clone() for c in cols]
        bt = BatchTracker(trk)
        bt.set_particles(work)
        return dict(case=case, bt=bt, cols=cols, work=work)
    if kind == "tricub":
        cfg += " track_tricub=enabled"
    cols = _columns(case["n"], seed, case.get("beam", "gauss"))
    return dict(case=case, trk=DeviceTracker(_image(key, _plain_elements(case)), cfg), cols=cols, work=cols.clone())


#: Rows of a column block that share a scale.
_ROWS = {"reference_s": (0, 6), "x_y": (6, 8), "px_py": (8, 10), "zeta": (10, 11), "energy": (11, 13), "ratios": (13, 17)}


def _out(cols, prefix=""):
    """A column block by groups of columns: float64 rows and whole numbers."""
    real = cols[:17].view(np.float64 if isinstance(cols, np.ndarray) else torch.float64)
    whole = cols[17:].view(np.int64) if isinstance(cols, np.ndarray) else cols[17:]
    return {**{prefix + k: real[a:b] for k, (a, b) in _ROWS.items()}, prefix + "whole": whole}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "job":
        job, p = state["job"], state["p"]
        p.set_block(state["block"])
        job.push_particles()
        if case["output"] == "elements":
            job.track_elem_by_elem(case["turns"])
        else:
            job.track_until(case["turns"])
        job.collect_particles()
        out = _out(p.block)
        if case["output"] != "none":
            job.collect_output()
            out.update(_out(job.output_particles(0).block, "stored_"))
        return out
    if kind == "adjoint":
        coords, values = state["coords"], state["values"]
        coords.grad = values.grad = None
        fin, alive = state["lat"].track(coords, values, state["cols"], case["turns"], checkpoint_every=10)
        loss = (fin[0] ** 2 + fin[2] ** 2).sum()
        loss.backward()
        return {"final": fin.detach(), "state": alive, "g_coords": coords.grad, "g_values": values.grad}
    if kind == "batch":
        for w, c in zip(state["work"], state["cols"]):
            w.copy_(c)
        if state["bt"].track_until(0, case["turns"]) != 0:
            raise RuntimeError("batch tracking failed")
        return [_out(w) for w in state["work"]]
    work, trk = state["work"], state["trk"]
    work.copy_(state["cols"])
    if kind == "line":
        st = trk.track_line(work, case["begin"], case["end"], False)
    else:
        st = trk.track_until(work, case["turns"])
    if st != 0:
        raise RuntimeError("tracking failed")
    return _out(work)


# ------------------------------------------------------------ what it takes
_FLOPS = {"d": 17, "c": 45, "x": 2, "r": 12, "e": 5, "b": 0, "t": 381}


def _flops(plain):
    """Operations of one particle through the elements, from the formulas."""
    total = 0.0
    for o in plain:
        if o[0] == "m":
            total += 8 * (len(o[1]) - 1) + 4
        elif o[0] == "6":
            total += 228 + len(o[6]) * (119 + 41 + (73 if o[7] == o[8] else 88 + 2 * 250))
        elif o[0] in "4s":
            same = o[2] == o[3] if o[0] == "4" else o[3] == o[4]
            total += 26 + (21 if same else 38 + 2 * 250)
        else:
            total += _FLOPS[o[0]]
    return total


def work(case):
    kind, n, turns = case["kind"], case["n"], case.get("turns", 1)
    column = 8.0 * n
    if kind == "batch":
        sizes = _variants(case)
        return {"bytes": sum(8.0 * m * (21 + 13) for _, m in sizes),
                "flops": sum(turns * m * _flops(_ring(c, 100 + i)) for i, (c, m) in enumerate(sizes))}
    if kind == "adjoint":
        return {"bytes": column * (21 + 13 + 12), "flops": 3.0 * turns * n * _flops(_learnable()[0])}
    plain = _plain_elements(case)
    if kind == "line":
        plain = plain[case["begin"]:case["end"]]
    size = column * (21 + 13)
    if kind == "job":
        size += column * 21 * {"none": 0, "monitor": turns, "elements": len(plain)}[case["output"]]
    return {"bytes": size, "flops": turns * n * _flops(plain)}


# ------------------------------------------- the same in plain float64 torch
def _w(z):
    """Faddeeva function for Im z >= 0 (J. A. C. Weideman, SIAM J. Numer.
    Anal. 31 (1994) 1497), 40 terms."""
    n = 40
    m = 2 * n
    k = np.arange(-m + 1, m)
    lim = math.sqrt(n / math.sqrt(2.0))
    t = lim * np.tan(0.5 * k * np.pi / m)
    f = np.concatenate([[0.0], np.exp(-t * t) * (lim * lim + t * t)])
    a = np.real(np.fft.fft(np.fft.fftshift(f)))[1:n + 1] / (2 * m)
    zz = (lim + 1j * z) / (lim - 1j * z)
    p = torch.zeros_like(z)
    for c in a[::-1]:
        p = p * zz + c
    return 2.0 * p / (lim - 1j * z) ** 2 + (1.0 / math.sqrt(math.pi)) / (lim - 1j * z)


def _field(x, y, sxx, syy, round_):
    """Transverse field of a Gaussian beam and its G terms."""
    k = 1.0 / (2.0 * math.pi * EPS0)
    if round_:
        r2 = x * x + y * y
        u = r2 / (2.0 * sxx)
        e = torch.exp(-u)
        t = -torch.expm1(-u) * k / r2
        ex, ey = t * x, t * y
        gx = 0.5 / r2 * (y * ey - x * ex + k / sxx * x * x * e)
        gy = 0.5 / r2 * (x * ex - y * ey + k / sxx * y * y * e)
        return ex, ey, gx, gy
    # taller than wide: the long axis is y
    sx, sy = sxx ** 0.5, syy ** 0.5
    s = (2.0 * (syy - sxx)) ** 0.5
    ax, ay = x.abs(), y.abs()
    e = torch.exp(-0.5 * (x * x / sxx + y * y / syy))
    w1 = _w(torch.complex(ay / s, ax / s))
    w2 = _w(torch.complex(sx / sy * ay / s, sy / sx * ax / s))
    fact = 1.0 / (2.0 * EPS0 * math.sqrt(math.pi) * s)
    ey = torch.sign(y) * fact * (w1.imag - e * w2.imag)
    ex = torch.sign(x) * fact * (w1.real - e * w2.real)
    xe = x * ex + y * ey
    i2 = 1.0 / (2.0 * (sxx - syy))
    return ex, ey, -i2 * (xe + k * (sy / sx * e - 1.0)), i2 * (xe + k * (sx / sy * e - 1.0))


def _new_delta(v, d):
    b0 = v["b0"]
    q = torch.sqrt((d * b0) ** 2 + 2.0 * d * b0 * b0 + 1.0)
    v["d"], v["psigma"] = d, (q - 1.0) / (b0 * b0)
    v["rpp"], v["rvv"] = 1.0 / (1.0 + d), (1.0 + d) / q


def _energy(v, de):
    """A change of the energy by de / energy0, zeta scaled with the velocity."""
    b0 = v["b0"]
    q = torch.sqrt((v["d"] * b0) ** 2 + 2.0 * v["d"] * b0 * b0 + 1.0)
    pt = (de + q - 1.0) / b0
    old = v["rvv"]
    r = pt * pt + 2.0 * pt / b0
    v["d"], v["psigma"] = r / (torch.sqrt(1.0 + r) + 1.0), pt / b0
    v["rpp"], v["rvv"] = 1.0 / (1.0 + v["d"]), (1.0 + v["d"]) / (1.0 + pt * b0)
    v["zeta"] = v["zeta"] * (v["rvv"] / old)


def _boost(v, o):
    sp, cp, tp, sa, ca = math.sin(o[1]), math.cos(o[1]), math.tan(o[1]), math.sin(o[2]), math.cos(o[2])
    x, y, s = v["x"] - o[3], v["y"] - o[4], v["zeta"]
    px, py, d = v["px"], v["py"], v["d"]
    h = d + 1.0 - torch.sqrt((1.0 + d) ** 2 - px * px - py * py)
    px, py, d = px / cp - h * ca * tp / cp, py / cp - h * sa * tp / cp, d - px * ca * tp - py * sa * tp + h * tp * tp
    pz = torch.sqrt((1.0 + d) ** 2 - px * px - py * py)
    hx, hy, hs = px / pz, py / pz, 1.0 - (d + 1.0) / pz
    proj = ca * sp * x + sa * sp * y
    return x + hx * proj + ca * tp * s, px, y + hy * proj + sa * tp * s, py, hs * proj + s / cp, d


def _beam_beam_6d(v, o, q0, p0):
    """Hirata's synchro-beam map of an uncoupled strong beam."""
    sp, cp, tp, sa, ca = math.sin(o[1]), math.cos(o[1]), math.tan(o[1]), math.sin(o[2]), math.cos(o[2])
    x, px, y, py, s, d = _boost(v, o)
    for z in o[6]:
        big = 0.5 * (s - z / cp)
        s22 = 1e-12 / (cp * cp)
        sxx, syy, ds = o[7] ** 2 + s22 * big * big, o[8] ** 2 + s22 * big * big, 2.0 * s22 * big
        xb, yb = x + px * big - ca * tp * z, y + py * big - sa * tp * z
        ex, ey, gx, gy = _field(xb, yb, sxx, syy, o[7] == o[8])
        ksl = o[5] * QE_PART * q0 / (p0 * CLIGHT)
        fx, fy, fz = ksl * ex, ksl * ey, 0.5 * ksl * ds * (gx + gy)
        d = d + fz + 0.5 * (fx * (px + 0.5 * fx) + fy * (py + 0.5 * fy))
        x, px, y, py = x - big * fx, px + fx, y - big * fy, py + fy
    pz = torch.sqrt((1.0 + d) ** 2 - px * px - py * py)
    hx, hy, hs = px / pz, py / pz, 1.0 - (d + 1.0) / pz
    # [x y s] = (1 + h (ca sp, sa sp, 0)) u + (ca tp, sa tp, 1 / cp) w solved for u = (x0, y0), w
    one = torch.ones_like(x)
    m = torch.stack([torch.stack([1.0 + hx * ca * sp, hx * sa * sp, ca * tp * one], -1),
                     torch.stack([hy * ca * sp, 1.0 + hy * sa * sp, sa * tp * one], -1),
                     torch.stack([hs * ca * sp, hs * sa * sp, one / cp], -1)], -2)
    u = torch.linalg.solve(m, torch.stack([x, y, s], -1).unsqueeze(-1)).squeeze(-1)
    h = (d + 1.0 - pz) * cp * cp
    px, py = px * cp + h * ca * tp, py * cp + h * sa * tp
    d = d + px * ca * tp + py * sa * tp - h * tp * tp
    v["x"], v["y"], v["zeta"], v["px"], v["py"] = u[:, 0] + o[3], u[:, 1] + o[4], u[:, 2], px, py
    _new_delta(v, d)


def _hermite(u):
    """Cubic Hermite basis (f0, f1, d0, d1) at u and its derivative."""
    b = torch.stack([1.0 - 3.0 * u ** 2 + 2.0 * u ** 3, 3.0 * u ** 2 - 2.0 * u ** 3, u - 2.0 * u ** 2 + u ** 3, u ** 3 - u ** 2])
    return b, torch.stack([6.0 * u * (u - 1.0), 6.0 * u * (1.0 - u), 1.0 - 4.0 * u + 3.0 * u ** 2, 3.0 * u ** 2 - 2.0 * u])


def _map_kick(v, length, table):
    nx, ny, nz, dx, dy, dz = GRID
    at, basis, slope = [], [], []
    for u, n, d in ((v["x"], nx, dx), (v["y"], ny, dy), (v["zeta"] / (v["b0"] * v["rvv"]), nz, dz)):
        f = (u + 0.5 * (n - 1) * d) / d
        i = torch.floor(f).clamp(0, n - 2)
        at.append(i.long())
        b, s = _hermite(f - i)
        basis.append(b)
        slope.append(s)
    kick = [0.0, 0.0, 0.0]
    order = ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1))
    for c in range(8):
        i, j, k = c & 1, (c >> 1) & 1, c >> 2
        node = table[at[2] + k, at[1] + j, at[0] + i]
        for m, (a, b, e) in enumerate(order):
            bx, by, bz = basis[0][2 * a + i], basis[1][2 * b + j], basis[2][2 * e + k]
            kick[0] = kick[0] + node[:, m] * slope[0][2 * a + i] * by * bz
            kick[1] = kick[1] + node[:, m] * bx * slope[1][2 * b + j] * bz
            kick[2] = kick[2] + node[:, m] * bx * by * slope[2][2 * e + k]
    v["px"] = v["px"] - kick[0] * (length / dx)
    v["py"] = v["py"] - kick[1] * (length / dy)
    _energy(v, -kick[2] * (length / dz) * P0C / math.sqrt(P0C * P0C + MASS0 * MASS0))


def _apply(v, o, table=None, knl=None):
    k = o[0]
    if k == "d":
        xp, yp = v["px"] * v["rpp"], v["py"] * v["rpp"]
        v["x"], v["y"] = v["x"] + xp * o[1], v["y"] + yp * o[1]
        v["zeta"] = v["zeta"] + o[1] * (v["rvv"] - (1.0 + 0.5 * (xp * xp + yp * yp)))
        return (v["x"].abs() < 1.0) & (v["y"].abs() < 1.0)
    if k == "m":
        b = o[1] if knl is None else knl
        n = len(b) - 1
        re, im = b[n] / math.factorial(n), 0.0
        for j in range(n - 1, -1, -1):
            re, im = b[j] / math.factorial(j) + re * v["x"] - im * v["y"], re * v["y"] + im * v["x"]
        v["px"], v["py"] = v["px"] - re, v["py"] + im
    elif k == "c":
        tau = v["zeta"] / (v["b0"] * v["rvv"])
        e0 = math.sqrt(P0C * P0C + MASS0 * MASS0)
        _energy(v, o[1] / e0 * torch.sin(math.pi / 180.0 * o[3] - 2.0 * math.pi / CLIGHT * o[2] * tau))
    elif k == "x":
        v["x"], v["y"] = v["x"] - o[1], v["y"] - o[2]
    elif k == "r":
        c, s = o[1], o[2]
        v["x"], v["y"] = c * v["x"] + s * v["y"], c * v["y"] - s * v["x"]
        v["px"], v["py"] = c * v["px"] + s * v["py"], c * v["py"] - s * v["px"]
    elif k == "e":
        return (v["x"] / o[1]) ** 2 + (v["y"] / o[2]) ** 2 <= 1.0
    elif k == "b":
        return (v["x"] >= o[1]) & (v["x"] <= o[2]) & (v["y"] >= o[3]) & (v["y"] <= o[4])
    elif k == "6":
        _beam_beam_6d(v, o, QE_BB, P0C / CLIGHT * QE_BB)
    elif k == "4":
        beta = v["b0"] / v["rvv"]
        f = o[1] * QE_PART * QE_BB * (1.0 + beta * o[4]) / (P0C * QE_BB * (beta + o[4]))
        ex, ey, _, _ = _field(v["x"] - o[5], v["y"] - o[6], torch.full_like(beta, o[2] ** 2), torch.full_like(beta, o[3] ** 2), o[2] == o[3])
        v["px"], v["py"] = v["px"] + f * ex, v["py"] + f * ey
    elif k == "s":
        beta, z = v["b0"] * v["rvv"], v["zeta"] / v["rvv"]
        f = o[5] * o[1] * QE_SC ** 2 * (1.0 - v["b0"] * beta) / (P0C * QE_SC * beta)
        f = f * torch.exp(-z * z / (2.0 * o[2] ** 2)) / (math.sqrt(2.0 * math.pi) * o[2])
        ex, ey, _, _ = _field(v["x"], v["y"], torch.full_like(beta, o[3] ** 2), torch.full_like(beta, o[4] ** 2), o[3] == o[4])
        v["px"], v["py"] = v["px"] + f * ex, v["py"] + f * ey
    elif k == "t":
        _map_kick(v, o[1], table)
    return None


_NAMES = {5: "s", 6: "x", 7: "y", 8: "px", 9: "py", 10: "zeta", 11: "psigma", 12: "d", 13: "rpp", 14: "rvv"}


def _start(f):
    v = {name: f[row] for row, name in _NAMES.items()}
    v["b0"] = f[2]
    return v


def _track(f, plain, turns, line=False, record=None):
    """The 17 real columns after tracking; particles outside an aperture stop
    there.  ``record`` is called with the columns before every element."""
    f = torch.as_tensor(f[:17]).cuda()
    fin, live = f.clone(), torch.arange(f.shape[1], device="cuda")
    table = torch.as_tensor(_field_map()).cuda() if any(o[0] == "t" for o in plain) else None
    v = _start(f)

    def store(to, sel):
        for row, name in _NAMES.items():
            to[row, live[sel]] = v[name][sel]

    for _ in range(turns):
        for i, o in enumerate(plain):
            if record is not None:
                now = f.clone()
                store(now, torch.ones_like(live, dtype=torch.bool))
                record(i, now)
            ok = _apply(v, o, table)
            if o[0] == "d":
                v["s"] = v["s"] + o[1]
            if ok is not None and not bool(ok.all()):
                store(fin, ~ok)
                v = {name: t[ok] for name, t in v.items()}
                live = live[ok]
                f = f[:, ok]
        if not line:
            if record is not None:
                now = f.clone()
                store(now, torch.ones_like(live, dtype=torch.bool))
                record(len(plain), now)
            v["s"] = torch.zeros_like(v["s"])
    store(fin, torch.ones_like(live, dtype=torch.bool))
    return fin


def _real(fin, prefix=""):
    return {**{prefix + k: None if fin is None else fin[a:b] for k, (a, b) in _ROWS.items()}, prefix + "whole": None}


def exact(case, seed):
    kind, n, turns = case["kind"], case["n"], case.get("turns", 1)
    if kind == "batch":
        return [_real(_track(_beam(m, seed * 100 + i), _ring(c, 100 + i), turns)) for i, (c, m) in enumerate(_variants(case))]
    f = _beam(n, seed, case.get("beam", "gauss"))
    if kind == "adjoint":
        plain, params = _learnable()
        c = torch.as_tensor(np.ascontiguousarray(f[[6, 8, 7, 9, 10, 12]])).cuda().requires_grad_(True)
        val = torch.tensor([plain[e][1][k] for e, _, k in params], dtype=torch.float64, device="cuda", requires_grad=True)
        at = {(e, k): j for j, (e, _, k) in enumerate(params)}
        v = dict(x=c[0], px=c[1], y=c[2], py=c[3], zeta=c[4], b0=torch.as_tensor(f[2]).cuda())
        _new_delta(v, c[5])
        for _ in range(turns):
            for i, o in enumerate(plain):
                knl = [val[at[i, k]] if (i, k) in at else b for k, b in enumerate(o[1])] if o[0] == "m" else None
                ok = _apply(v, o, knl=knl)
                if ok is not None and not bool(ok.all()):
                    return None  # a lost particle's gradient starts where it stopped
        fin = torch.stack([v[k] for k in ("x", "px", "y", "py", "zeta", "d")])
        (fin[0] ** 2 + fin[2] ** 2).sum().backward()
        return {"final": fin.detach(), "state": None, "g_coords": c.grad, "g_values": val.grad}
    plain = list(_plain_elements(case))
    if kind == "line":
        return _real(_track(f, plain[case["begin"]:case["end"]], 1, line=True))
    kept, want = [], case.get("output", "none")

    def record(i, now):
        if want == "elements" and i < len(plain) or want == "monitor" and i == len(plain):
            kept.append(now)

    out = _real(_track(f, plain, turns, record=record if want != "none" else None))
    if want != "none":
        out.update(_real(torch.cat(kept, 1) if all(k.shape[1] == n for k in kept) else None, "stored_"))
    return out
