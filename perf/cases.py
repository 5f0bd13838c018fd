"""Performance cases: what a user of the dose engine has it do.

Every case is a plain dict.  ``prepare`` makes what a program has in hand
before the call (phantom, beams, engine), ``run`` is one pass through the
package's public entry points, ``exact`` the same outputs in float64 by plain
torch and numpy, ``work`` the bytes and operations the path cannot do without.

Kinds of case:

* ``call``         ``Conehead().calculate`` from host arrays to a host dose;
* ``beam``         one beam on a resident phantom, ``DoseEngine.run``;
* ``intermediates`` the same, every per-voxel intermediate returned as well;
* ``batch``        several beams of one phantom, ``DoseEngine.run_batch``;
* ``graph``        a captured batch over several phantom sizes, replayed;
* ``plan``         the MLC beams of one RT plan, blocks uploaded and run;
* ``gradient``     dose and gradient of beamlet weights (autograd);
* ``radiological`` the density-scaled cone distance extension.
"""
import math
import os
import random
from types import SimpleNamespace

import numpy as np
import torch

SETTINGS = {
    "sPri": 0.90924, "sAnn": 2.887e-3, "zAnn": 4.0, "rInner": 0.2, "rOuter": 1.4,
    "zExp": 12.5, "sExp": 8.289e-3, "kExp": 0.4816, "softRatio": 0.0025,
    "softLimit": 20, "hornRatio": 0.0065, "fluenceResampling": 3,
    "energy_weights": {"0.5": 0.08196, "1.0": 0.12385, "1.5": 0.10605, "2.0": 0.08307,
                       "2.5": 0.05881, "3.0": 0.03911, "3.5": 0.02131, "4.0": 0.02426,
                       "4.5": 0.0, "5.0": 0.00881, "5.5": 0.0, "6.0": 0.00498},
}
GRAPH_SIZES = (64, 96, 128, 160)


def _case(kind, n, spacing, field, beams=1, jitter=0.0, collimator=True, hetero=True, samples=3):
    """field: side of the jaw opening in cm (jitter: the range added to it)."""
    sp = spacing if isinstance(spacing, tuple) else (spacing,) * 3
    return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "sx": sp[0], "sy": sp[1], "sz": sp[2],
            "beams": beams, "field": field, "jitter": jitter, "collimator": collimator, "hetero": hetero,
            "samples": samples}


def listed():
    cube = lambda n: (n, n, n)  # noqa: E731
    named = {
        # the smallest whole call: 40^3 water, 0.5 cm, 10 x 10, host to host (latency, launches)
        "call_water_40": _case("call", cube(40), 0.5, 10.0, collimator=False, hetero=False),
        # the reference's example: SimplePhantom, 201^3 at 2 mm, 10 x 10, host to host
        "call_water_201": _case("call", cube(201), 0.2, 10.0, collimator=False, hetero=False),
        # one beam while a user looks at it: a small resident grid
        "beam_slab_64": _case("beam", cube(64), 0.25, 6.0),
        # the same on the headline grid, 5 x 5 cm
        "beam_slab_128": _case("beam", cube(128), 0.25, 5.0, collimator=False),
        # one large field on a ragged, anisotropic grid, as CT volumes are cropped
        "beam_ragged_150": _case("beam", (150, 130, 83), (0.25, 0.25, 0.3), 14.0),
        # the headline workload: 32 beams of 5 x 5 cm on one 128^3 phantom per call
        "batch_slab_128x32": _case("batch", cube(128), 0.25, 5.0, beams=32, collimator=False),
        # a request of the dose server on its largest phantom; an odd count
        "batch_slab_192x7": _case("batch", cube(192), 0.25, 5.0, beams=7, jitter=5.0),
        # beams of several phantoms captured once and replayed, jaws 2-20 cm
        "graph_mixed_64": _case("graph", cube(160), 0.25, 2.0, beams=64, jitter=18.0),
        # a treatment plan: MLC beams on a ragged CT-like grid
        "plan_mlc_9": _case("plan", (140, 101, 112), 0.3, 16.0, beams=9),
        # commissioning: every per-voxel quantity of one beam
        "intermediates_96": _case("intermediates", cube(96), 0.25, 10.0),
        # an optimiser's step: dose and gradient of 40 x 40 beamlets of 0.5 cm
        "gradient_128": _case("gradient", cube(128), 0.25, 20.0),
        # the density-scaled cone distance (an option, far dearer than the stock cone)
        "radiological_48": _case("radiological", cube(48), 0.4, 5.0),
    }
    return [dict(c, name=k) for k, c in named.items()]


def draw(rng):
    """One more case: sizes spread over their logarithm, odd and unequal ones among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "beam", "beam", "beam", "batch", "batch", "batch", "graph", "plan", "plan",
                       "intermediates", "gradient", "gradient", "radiological"])
    lo, hi = {"call": (24, 201), "beam": (24, 208), "batch": (32, 192), "graph": (48, 160), "plan": (48, 150),
              "intermediates": (32, 120), "gradient": (32, 150), "radiological": (24, 52)}[kind]
    n = size(lo, hi)
    if kind == "graph" or rng.random() < 0.35:
        dims = (n, n, n)
    elif rng.random() < 0.4:
        dims = (n, n, size(lo, hi))                     # square in x and y: the densities are read swapped
    else:
        dims = (n, size(lo, hi), size(lo, hi))
    base = rng.choice([0.2, 0.25, 0.3, 0.4])
    spacing = (base, base, rng.choice([base, base, 0.25, 0.3])) if kind != "gradient" else (base,) * 3
    extent = min(d * s for d, s in zip(dims, spacing))
    field = round(min(rng.uniform(2.0, 20.0), max(2.0, 0.9 * extent)), 2)
    if kind == "radiological":
        field = min(field, 6.0)
    vox = dims[0] * dims[1] * dims[2]
    most = max(1, min(32, int(32 * 128 ** 3 / vox)))
    beams = {"batch": min(most, size(2, 32)), "graph": min(most, size(4, 32)),
             "plan": min(most, size(2, 12))}.get(kind, 1)
    samples = rng.choice([3, 3, 3, 3, 2, 4, 5]) if kind in ("beam", "batch", "call") else 3
    hetero = kind != "call" or rng.random() < 0.5
    return _case(kind, dims, spacing, field, beams=beams, jitter=round(rng.uniform(0, 4), 2) if beams > 1 else 0.0,
                 collimator=rng.random() < 0.7, hetero=hetero, samples=samples)


# --------------------------------------------------------------- inputs --
def _settings(case):
    s = dict(SETTINGS, fluenceResampling=case["samples"])
    if case["kind"] == "radiological":
        s["coneDistance"] = "radiological"
    return s


def _dims(case):
    return [case["nx"], case["ny"], case["nz"]], [case["sx"], case["sy"], case["sz"]]


def _origin(case, n, sp):
    """Centred on the isocentre; water calls have their surface on it (the reference's phantoms)."""
    o = [-(k - 1) * s / 2 for k, s in zip(n, sp)]
    if not case["hetero"]:
        o[1] = sp[1] / 2
    return np.array(o, dtype=np.float32)


def _densities(case, n, sp, seed):
    """Water, or a lung and a bone slab in water with 20 random cuboids."""
    rho = np.ones(n, dtype=np.float32)
    rng = np.random.default_rng(seed)
    if not case["hetero"]:
        # water with the few per mille of a scanner's noise, so that no two inputs are the same
        return rho + rng.uniform(-0.004, 0.004, size=n).astype(np.float32)
    depth = (np.arange(n[1]) + 0.5) * sp[1]
    rho[:, (depth >= 5.0) & (depth < 12.0), :] = 0.25
    rho[:, (depth >= 14.0) & (depth < 16.0), :] = 1.85
    for _ in range(20):
        ext = [int(rng.integers(max(1, k // 32), max(2, k // 6))) for k in n]
        lo = [int(rng.integers(0, k - e)) for k, e in zip(n, ext)]
        rho[lo[0]:lo[0] + ext[0], lo[1]:lo[1] + ext[1], lo[2]:lo[2] + ext[2]] = rng.uniform(0.2, 2.0)
    return rho


def _volumes(case, seed):
    """(size, spacing, origin, densities) of every phantom of the case."""
    n, sp = _dims(case)
    if case["kind"] == "graph":
        sizes = [max(16, int(round(k * case["nx"] / 160))) for k in GRAPH_SIZES]
        dims = [[k, k, k] for k in sizes]
    else:
        dims = [n]
    return [(d, sp, _origin(case, d, sp), _densities(case, d, sp, 1000 * seed + i)) for i, d in enumerate(dims)]


def _beams(case, seed):
    """Per beam: phantom index, gantry, collimator and jaw opening (x1, x2, z1, z2) in cm."""
    rng = random.Random(7919 * seed + 17)
    out = []
    for i in range(case["beams"]):
        gantry = 0.0 if not case["hetero"] else rng.uniform(0.0, 359.9)
        coll = rng.uniform(0.0, 90.0) if case["collimator"] else 0.0
        fx, fz = (case["field"] + case["jitter"] * rng.random() for _ in range(2))
        out.append((i % len(GRAPH_SIZES) if case["kind"] == "graph" else 0, gantry, coll,
                    (-fx / 2, fx / 2, -fz / 2, fz / 2)))
    return out


def _leaves(case, seed, i):
    """60 leaf pairs of an MLC (mm): boundaries, ends (bank A then B), jaws X and Y."""
    rng = random.Random(104729 * seed + i)
    bounds = [-200.0 + 10 * k for k in range(11)] + [-100.0 + 5 * k for k in range(1, 41)] + \
             [100.0 + 10 * k for k in range(1, 11)]
    half = 5 * case["field"]
    a, b = [], []
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        mid = min(1.0, abs(lo + hi) / 2 / half)
        w = half * math.sqrt(max(0.0, 1 - mid * mid))
        a.append(round(-w * rng.uniform(0.6, 1.0), 1))
        b.append(round(w * rng.uniform(0.6, 1.0), 1) if w > 0 else a[-1])
    return bounds, a + b, [-half, half], [-half, half]


def _plan(case, seed):
    """An RT plan as a DICOM reader hands it over: one static beam per entry."""
    def beam(i):
        bounds, ends, jx, jy = _leaves(case, seed, i)
        devices = [SimpleNamespace(RTBeamLimitingDeviceType="MLCX", LeafPositionBoundaries=bounds)]
        positions = [SimpleNamespace(RTBeamLimitingDeviceType=k, LeafJawPositions=v)
                     for k, v in (("ASYMX", jx), ("ASYMY", jy), ("MLCX", ends))]
        return SimpleNamespace(BeamType="STATIC", BeamLimitingDeviceSequence=devices,
                               ControlPointSequence=[SimpleNamespace(BeamLimitingDevicePositionSequence=positions)])
    return SimpleNamespace(BeamSequence=[beam(i) for i in range(case["beams"])])


def _weights(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((40, 40), generator=g, device="cuda", dtype=torch.float32) + 0.05


def _target(case, seed):
    """The dose an optimiser wants: a smooth bump around the isocentre, [x][y][z]."""
    n, sp = _dims(case)
    ax = [(torch.arange(k, device="cuda", dtype=torch.float32) - (k - 1) / 2) * s for k, s in zip(n, sp)]
    r2 = ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2
    return (1.5 + 0.1 * (seed % 5)) * torch.exp(-r2 / 18.0)


def _beamlet_cells(case):
    return max(1, int(round(case["field"] * 100 / 40)))


_ENGINE = {}


def _engine(case, n, sp):
    """The engine a program keeps for its grids (one at a time here)."""
    from conehead_gb300.engine import DoseEngine
    key = (case["kind"], tuple(n), tuple(sp))
    if key not in _ENGINE:
        _ENGINE.clear()
        eng = DoseEngine(0)
        eng.set_kernel(SETTINGS["energy_weights"])
        eng.prepare(n, sp)
        _ENGINE[key] = eng
    return _ENGINE[key]


def prepare(case, seed):
    from conehead_gb300 import Block, Conehead, GridPhantom, Source
    kind, settings = case["kind"], _settings(case)
    phantoms = [GridPhantom(rho, origin, sp) for _, sp, origin, rho in _volumes(case, seed)]
    beams = []
    for vol, gantry, coll, rect in _beams(case, seed):
        src, blk = Source(), Block()
        src.gantry, src.collimator = gantry, coll
        blk.set_rect(*rect)
        beams.append((vol, src, blk))
    state = {"kind": kind, "settings": settings}
    if kind == "call":
        return dict(state, calc=Conehead(), source=beams[0][1], block=beams[0][2], phantom=phantoms[0])
    n, sp = _dims(case)
    eng = _engine(case, n, sp)
    state["eng"] = eng
    if kind == "gradient":
        from conehead_gb300.adjoint import BeamletDose, BeamletGrid
        op = BeamletDose(eng, phantoms[0], beams[0][1], BeamletGrid(40, 40, _beamlet_cells(case)), settings)
        return dict(state, op=op, weights=_weights(case, seed).requires_grad_(True), target=_target(case, seed))
    rhos = [eng.upload_densities(p.densities) for p in phantoms]
    if kind == "plan":
        plan = _plan(case, seed)
        pairs = [(b[1], Block.from_plan(plan, beam=i)) for i, b in enumerate(beams)]
        return dict(state, phantom=phantoms[0], rho=rhos[0], pairs=pairs)
    jobs = [eng.job(phantoms[v], rhos[v], src, eng.block_for(blk), settings) for v, src, blk in beams]
    if kind == "graph":
        state["graph"] = eng.capture(jobs)
    return dict(state, jobs=jobs)


def run(state):
    kind = state["kind"]
    if kind == "call":
        return state["calc"].calculate(state["source"], state["block"], state["phantom"], state["settings"])
    if kind in ("beam", "radiological"):
        return state["eng"].run(state["jobs"][0])
    if kind == "intermediates":
        dose, inter = state["eng"].run(state["jobs"][0], intermediates=True)
        return dict(inter, dose=dose)
    if kind == "batch":
        return state["eng"].run_batch(state["jobs"])
    if kind == "graph":
        return state["graph"].launch()
    if kind == "plan":
        eng = state["eng"]
        jobs = [eng.job(state["phantom"], state["rho"], src, eng.block_for(blk), state["settings"])
                for src, blk in state["pairs"]]
        return eng.run_batch(jobs)
    from conehead_gb300.adjoint import beamlet_dose
    w = state["weights"]
    w.grad = None
    dose = beamlet_dose(w, state["op"])
    ((dose - state["target"]) ** 2).sum().backward()
    return {"dose": dose.detach(), "grad": w.grad}


# ----------------------------------------------------------------- work --
def _fft_flops(n):
    """Forward and inverse real transforms of the padded grid, zero lines left out, and the product."""
    P = [2 * k - 1 for k in n]
    lines = (n[0] * n[1], n[0] * P[2] / 2, P[1] * P[2] / 2)
    per = (2.5 * P[2] * math.log2(P[2]), 5 * P[1] * math.log2(P[1]), 5 * P[0] * math.log2(P[0]))
    return sum(2 * a * b for a, b in zip(lines, per)) + 3 * P[0] * P[1] * P[2]


def _reached(case, n, sp):
    """Voxels a beam reaches, and the voxels a ray crosses on its way out."""
    area = (case["field"] + case["jitter"] / 2) ** 2
    depth = max(k * s for k, s in zip(n, sp))
    vox = min(float(n[0] * n[1] * n[2]), area * depth / (sp[0] * sp[1] * sp[2]))
    if case["kind"] == "intermediates":
        vox = float(n[0] * n[1] * n[2])
    return vox, 0.75 * sum(n) / 3 * 1.5


def work(case):
    n, sp = _dims(case)
    if case["kind"] == "graph":
        dims = [[max(16, int(round(k * case["nx"] / 160)))] * 3 for k in GRAPH_SIZES]
        per = [dims[i % len(dims)] for i in range(case["beams"])]
    else:
        dims, per = [n], [n] * case["beams"]
    vol = lambda d: float(d[0] * d[1] * d[2])  # noqa: E731
    read, write, flops = sum(4 * vol(d) for d in dims), 0.0, 0.0
    for d in per:
        vox, steps = _reached(case, d, sp)
        write += 4 * vol(d)
        flops += vox * (3 * steps + 10 * case["samples"] ** 3 + 12 * 12)
        if case["kind"] == "radiological":
            flops += vox * 576 * steps * 6
        else:
            flops += _fft_flops(d)
    if case["kind"] == "intermediates":
        write += 32 * vol(n)
    if case["kind"] == "gradient":
        read += 8 * vol(n)                   # the target and dL/d(dose)
        write += 4 * vol(n)
        flops += _fft_flops(n) + 4 * vol(n)
    return {"bytes": read + write, "flops": flops}


# ---------------------------------------------------------------- exact --
# mass attenuation of water (cm^2/g, NIST) at the spectrum's bins, as float32
_MU = (0.09687, 0.07072, 0.05754, 0.04942, 0.044555, 0.03969, 0.03686, 0.03403, 0.03217, 0.03031, 0.029005, 0.0277)
_F64 = dict(device="cuda", dtype=torch.float64)


def _kernel_table():
    """K [48][5996] (cumulative, 0.05 .. 60 cm) and the cone angles of the settings' spectrum."""
    here = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    pack = np.load(os.path.join(here, "conehead_gb300", "data", "edknrc_6mv.npz"))
    diff, raw = 0.0, None
    for label, w in SETTINGS["energy_weights"].items():
        raw = pack["E1.5" if label == "1.0" else "E" + label].astype(np.float32)
        d = raw[:, 2].reshape(48, 24)
        diff = diff + d / d.sum() * w
    diff = diff / diff.sum()
    r = np.linspace(0.05, 60.0, 5996)
    radii = np.unique(raw[:, 1])
    K = np.stack([np.interp(r, radii, row) for row in np.asarray(diff, dtype=np.float64).cumsum(axis=1)])
    return K, np.unique(raw[:, 0])


def _walks(n, sp):
    """The 576 cone walks from a voxel centre: offsets [m][576][3], exit t (float32 DDA), alive."""
    f = np.float32
    K, phis = _kernel_table()
    th = np.repeat(np.linspace(0, 330, 12, dtype=f).astype(np.float64), 48) * np.pi / 180.0
    ph = np.tile(phis.astype(f).astype(np.float64), 12) * np.pi / 180.0
    d = np.stack([f(np.cos(th) * np.sin(ph)), f(np.cos(ph)), f(np.sin(th) * np.sin(ph))], axis=1).astype(f)
    d = d / np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])[:, None]
    s = np.array(sp, dtype=f)
    a = np.abs(d)
    with np.errstate(divide="ignore"):
        t = np.where(a == 0, f(1e9), (s * f(0.5)) / a).astype(f)
        dt = np.where(a == 0, f(1e9), s / a).astype(f)
    step = np.where(d < 0, -1, 1)
    o = np.zeros((576, 3), dtype=np.int64)
    rows = np.arange(576)
    offs, ts, alive = [], [], []
    ok = np.ones(576, bool)
    while True:
        ok = ok & (np.abs(o) <= np.array(n) - 1).all(axis=1)
        if not ok.any():
            return K, np.array(offs), np.array(ts), np.array(alive)
        a01 = t[:, 0] < t[:, 1]
        ax = np.where(a01 & (t[:, 0] < t[:, 2]), 0, np.where(~a01 & (t[:, 1] < t[:, 2]), 1, 2))
        offs.append(o.copy())
        ts.append(t[rows, ax].copy())
        alive.append(ok.copy())
        t[rows, ax] = t[rows, ax] + dt[rows, ax]
        o[rows, ax] += step[rows, ax]


def _index(t):
    return np.minimum(np.abs(np.floor(t.astype(np.float64) * 100.0 - 5.0)), 5995).astype(np.int64)


def _spectrum(n, sp):
    """FFT of the cone stencil on the grid padded to twice its size."""
    K, offs, ts, alive = _walks(n, sp)
    row = np.tile(np.arange(48), 12)
    P = [2 * k for k in n]
    S = np.zeros(P)
    prev = np.zeros(576)
    for o, t, ok in zip(offs, ts, alive):
        k = K[row, _index(t)]
        np.add.at(S, tuple(o[ok].T), (k - prev)[ok])
        prev = k
    return torch.fft.rfftn(torch.from_numpy(S).to("cuda"))


def _convolve(T, Sf, transpose=False):
    n = T.shape
    P = [2 * k for k in n]
    F = torch.fft.rfftn(T, s=P)
    D = torch.fft.irfftn(F * (Sf.conj() if transpose else Sf), s=P)
    return D[:n[0], :n[1], :n[2]].contiguous()


def _geometry(gantry, coll):
    """Source position, beam axis and world-to-beam matrix (float64)."""
    rad, g, c = (((90 - gantry) % 360) * np.pi / 180, gantry * np.pi / 180, -coll * np.pi / 180)
    pos = np.array([100.0 * np.cos(rad), -100.0 * np.sin(rad), 0.0])
    rc = np.array([[np.cos(c), 0, np.sin(c)], [0, 1, 0], [-np.sin(c), 0, np.cos(c)]])
    rg = np.array([[np.cos(g), -np.sin(g), 0], [np.sin(g), np.cos(g), 0], [0, 0, 1]])
    vx, vy, vz = rg @ (rc @ np.array([1.0, 0, 0])), rg @ np.array([0, 1.0, 0]), rg @ (rc @ np.array([0, 0, 1.0]))
    return pos, vy, np.linalg.inv(np.array([vx, vy, vz]).transpose())


def _project(geo, p):
    """(ray to the source, xb, zb) of float32 points p[3]: float64 steps stored as float32."""
    src, vy, m = geo
    srcf = src.astype(np.float32).astype(np.float64)
    rd = [(src[k] - p[k].double()).float() for k in range(3)]
    r = [x.double() for x in rd]
    si = -float(vy @ srcf) / (vy[0] * r[0] + vy[1] * r[1] + vy[2] * r[2])
    pp = [(srcf[k] + si * r[k]).float().double() for k in range(3)]
    xb, zb = ((m[i][0] * pp[0] + m[i][1] * pp[1] + m[i][2] * pp[2]).float() for i in (0, 2))
    return rd, xb, zb


def _map_cells(xb, zb):
    """Block map row and column of a projected point, and whether it is on the map."""
    c0, c1 = (torch.floor(v * 100.0).clamp(-1e6, 1e6).long() + 2000 for v in (xb, zb))
    on = (c0 >= 0) & (c0 <= 3999) & (c1 >= 0) & (c1 <= 3999)
    return (c0 - 1) % 4000, (c1 - 1) % 4000, on


def _block_map(case, seed, i, rect):
    """The beam's 4000 x 4000 transmission map (float32)."""
    m = np.zeros((4000, 4000), dtype=np.float32)
    if case["kind"] != "plan":
        lo = [max(0, int(2000 + v * 100)) for v in rect]
        m[lo[0]:lo[1], lo[2]:lo[3]] = 1.0
        return m
    bounds, ends, jx, jy = _leaves(case, seed, i)
    b = np.floor(np.array(bounds, dtype=np.float32) * 10).astype(int) + 2000
    e = np.floor(np.array(ends) * 10).astype(int) + 2000
    ramp = np.linspace(1.0, 0.0, 15)
    m[:] = 1.0
    for k in range(len(b) - 1):
        w = b[k + 1] - b[k]
        prof = np.ones(w, dtype=np.float32)
        for row, v in ((0, 0.20), (1, 0.50), (2, 0.75), (w - 1, 0.20), (w - 2, 0.50), (w - 3, 0.75)):
            prof[row] = v
        ends_a, ends_b = e[k], e[k + len(b) - 1]
        leaf = np.ones((w, ends_a)) * prof[:, None]
        leaf[:, -15:] *= ramp
        m[b[k]:b[k + 1], :ends_a] = np.float32(1) - leaf.astype(np.float32)
        leaf = np.ones((w, 3999 - ends_b)) * prof[:, None]
        leaf[:, -15:] *= ramp
        m[b[k]:b[k + 1], ends_b:3999] = np.float32(1) - leaf.astype(np.float32)[::-1, ::-1]
    jx, jy = (np.floor(np.array(v) * 10).astype(int) + 2000 for v in (jx, jy))
    open_ = np.zeros_like(m)
    open_[jy[0]:jy[1], jx[0]:jx[1]] = 1.0
    return m * open_


def _sample_cells(geo, pos, sp, S, part):
    """Map cells of sub-sample `part` of every voxel centre pos[3] (float32)."""
    i = (part // (S * S), part // S % S, part % S)
    p = []
    for k in range(3):
        s = float(np.float32(sp[k]))
        off = float(np.float32(sp[k]) / np.float32(S))
        p.append((((pos[k].double() - s * 0.5) + off * 0.5) + off * i[k]).float())
    _, xb, zb = _project(geo, p)
    return _map_cells(xb, zb)


def _depth(geo, rd, vox, rho, n, sp):
    """Radiological depth from the centres of voxels vox[3] to the grid's edge."""
    r = torch.stack([x.double() for x in rd])
    d = r / r.square().sum(0).sqrt()
    s = torch.tensor([float(np.float32(k)) for k in sp], **_F64)[:, None]
    t = torch.where(d == 0, 1e9, s / 2 / d.abs())
    dt = torch.where(d == 0, 1e9, s / d.abs())
    step = torch.where(d < 0, -1, 1)
    at = torch.stack(vox).clone()
    top = torch.tensor(n, device="cuda")[:, None]
    flat = rho.reshape(-1)
    deff, last = torch.zeros(at.shape[1], **_F64), torch.zeros(at.shape[1], **_F64)
    inside = torch.ones(at.shape[1], dtype=torch.bool, device="cuda")
    k = 0
    while True:
        a01 = t[0] < t[1]
        ax = torch.where(a01 & (t[0] < t[2]), 0, torch.where(~a01 & (t[1] < t[2]), 1, 2))[None]
        tm = t.gather(0, ax)[0]
        here = flat[((at[0] * n[1] + at[1]) * n[2] + at[2]) * inside]
        deff = torch.where(inside, deff + here * (tm - last), deff)
        last = torch.where(inside, tm, last)
        t.scatter_add_(0, ax, dt.gather(0, ax))
        at.scatter_add_(0, ax, step.gather(0, ax))
        inside = inside & ((at >= 0) & (at < top)).all(0)
        k += 1
        if k % 16 == 0 and not bool(inside.any()):
            return deff


def _terma(case, geo, vol, look, S, every):
    """Per-voxel quantities on the grid; look(rows, cols, on) gives a sample's transmission."""
    n, sp, origin, rho = vol
    rho = torch.from_numpy(rho).to("cuda").double()
    if n[0] == n[1]:
        rho = rho.transpose(0, 1).contiguous()            # the reference's resampling swaps x and y
    ax = [(float(origin[k]) + float(np.float32(sp[k])) * torch.arange(n[k], **_F64)).float() for k in range(3)]
    N = n[0] * n[1] * n[2]
    blocked = torch.zeros(N, **_F64)
    for lo in range(0, N, 1 << 22):
        v = torch.arange(lo, min(N, lo + (1 << 22)), device="cuda")
        pos = [ax[0][v // (n[1] * n[2])], ax[1][v // n[2] % n[1]], ax[2][v % n[2]]]
        for part in range(S ** 3):
            blocked[v] += look(*_sample_cells(geo, pos, sp, S, part)) / S ** 3
    v = torch.arange(N, device="cuda") if every else torch.nonzero(blocked).reshape(-1)
    vox = [v // (n[1] * n[2]), v // n[2] % n[1], v % n[2]]
    rd, xb, zb = _project(geo, [ax[k][vox[k]] for k in range(3)])
    c = SETTINGS
    oad = (xb * xb + zb * zb).sqrt()
    mag = torch.stack([x.double() for x in rd]).square().sum(0).sqrt()
    ring = oad * c["zAnn"] / 100.0
    ann = torch.where((ring >= c["rInner"]) & (ring <= c["rOuter"]),
                      c["sAnn"] * (100.0 - c["zAnn"]) ** 2 / (mag - c["zAnn"]) ** 2, 0.0)
    o = oad.double()
    rexp = o.clamp(min=2.0) * c["zExp"] / 100.0
    ext = c["sExp"] / rexp * torch.exp(-c["kExp"] * rexp) * (100.0 - c["zExp"]) ** 2 / (mag - c["zExp"]) ** 2
    fl = (c["sPri"] * (100.0 / mag) ** 2 + ann + ext) * blocked[v]
    fs = torch.where(oad < c["softLimit"], 1.0 / (1.0 - c["softRatio"] * o), 1.0)
    fh = 1.0 + o * c["hornRatio"]
    deff = _depth(geo, rd, vox, rho, n, sp)
    T = torch.zeros_like(fl)
    for (label, w), mu in zip(c["energy_weights"].items(), _MU):
        mu = float(np.float32(mu))
        T += float(np.float32(w)) * fl * torch.exp(-mu * fs * deff) * float(label) * mu * fh
    T = T * blocked[v]

    def full(x):
        g = torch.zeros(N, **_F64)
        g[v] = x.double()
        return g.reshape(n)

    return {"blocked": blocked.reshape(n), "d_eff": full(deff), "oad": full(oad), "fluence": full(fl),
            "f_soften": full(fs), "f_horn": full(fh), "terma": full(T)}


def _radiological_dose(T, vol):
    """The cone walks with the kernel read at the density-scaled distance."""
    n, sp, _, rho = vol
    if n[0] == n[1]:
        rho = rho.transpose(1, 0, 2)
    rho = torch.from_numpy(np.ascontiguousarray(rho)).to("cuda").reshape(-1)
    K, offs, ts, alive = _walks(n, sp)
    K = torch.from_numpy(K).to("cuda").reshape(-1)
    src = torch.nonzero(T.reshape(-1)).reshape(-1)
    x, y, z = src // (n[1] * n[2]), src // n[2] % n[1], src % n[2]
    amount = T.reshape(-1)[src]
    dose = torch.zeros(T.numel(), **_F64)
    offs, ts, alive = (torch.from_numpy(a).to("cuda") for a in (offs, ts, alive))
    for d0 in range(0, 576, 72):
        row = ((torch.arange(d0, d0 + 72, device="cuda") % 48) * 5996)[:, None]
        rad = torch.zeros((72, len(src)), device="cuda")
        ok = torch.ones_like(rad, dtype=torch.bool)
        prev, last = torch.zeros((72, len(src)), **_F64), torch.zeros((72, 1), device="cuda")
        for m in range(len(ts)):
            o = offs[m, d0:d0 + 72, :, None]
            tx, ty, tz = x + o[:, 0], y + o[:, 1], z + o[:, 2]
            ok = ok & alive[m, d0:d0 + 72, None] & (tx >= 0) & (tx < n[0]) & (ty >= 0) & (ty < n[1]) & \
                (tz >= 0) & (tz < n[2])
            at = ((tx * n[1] + ty) * n[2] + tz) * ok
            t = ts[m, d0:d0 + 72, None]
            rad = rad + rho[at] * (t - last)
            last = t
            k = K[row + (rad.double() * 100.0 - 5.0).floor().abs().clamp(max=5995).long()]
            dose.index_add_(0, at.reshape(-1), (amount * (k - prev) * ok).reshape(-1))
            prev = k
    return dose.reshape(n)


def exact(case, seed):
    vols, kind = _volumes(case, seed), case["kind"]
    spectra, out = {}, []
    for i, (v, gantry, coll, rect) in enumerate(_beams(case, seed)):
        n, sp = vols[v][0], vols[v][1]
        geo = _geometry(gantry, coll)
        if kind == "gradient":
            return _exact_gradient(case, seed, geo, vols[v])
        m = torch.from_numpy(_block_map(case, seed, i, rect)).to("cuda").double()
        q = _terma(case, geo, vols[v], lambda r, c, on: m[r, c] * on, case["samples"], kind == "intermediates")
        if kind == "radiological":
            return _radiological_dose(q["terma"], vols[v])
        if v not in spectra:
            spectra[v] = _spectrum(n, sp)
        dose = _convolve(q["terma"], spectra[v])
        if kind == "intermediates":
            return dict(q, dose=dose)
        out.append(dose)
    if kind == "call":
        return out[0].cpu().numpy()
    return out[0] if kind == "beam" else out


def _exact_gradient(case, seed, geo, vol):
    n, sp, origin, _ = vol
    cell = _beamlet_cells(case)
    r0 = 2000 - 20 * cell
    w = _weights(case, seed).double().reshape(-1)

    def beamlet(r, c, on):
        i, j = torch.div(r - r0, cell, rounding_mode="floor"), torch.div(c - r0, cell, rounding_mode="floor")
        on = on & (i >= 0) & (i < 40) & (j >= 0) & (j < 40)
        return torch.where(on, i * 40 + j, 1600)

    wide = torch.cat([w, torch.zeros(1, **_F64)])
    q = _terma(case, geo, vol, lambda r, c, on: wide[beamlet(r, c, on)], 3, False)
    Sf = _spectrum(n, sp)
    dose = _convolve(q["terma"], Sf)
    back = _convolve(2.0 * (dose - _target(case, seed).double()), Sf, transpose=True)
    v = torch.nonzero(q["terma"].reshape(-1)).reshape(-1)
    T, b = q["terma"].reshape(-1)[v], q["blocked"].reshape(-1)[v]
    per = back.reshape(-1)[v] * 2.0 * T / b / 27.0
    at = [v // (n[1] * n[2]), v // n[2] % n[1], v % n[2]]
    pos = [(float(origin[k]) + float(np.float32(sp[k])) * at[k].double()).float() for k in range(3)]
    grad = torch.zeros(1601, **_F64)
    for part in range(27):
        grad.index_add_(0, beamlet(*_sample_cells(geo, pos, sp, 3, part)), per)
    return {"dose": dose, "grad": grad[:1600].reshape(40, 40)}
