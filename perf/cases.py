"""The dose engine's work, as its users have it done: dose runs of beams, dose
influence columns of beamlets, and a server that shares one GPU between
requests, each through the public Python entry points of `ompmc_b200.engine`.

A pass is one call that a planning program makes (one dose run, one matrix of
columns, one load of requests).  What such a program keeps between calls --
physics tables, phantom, engine, server -- is made in `prepare`.

Physics data are not part of this repository, so this file writes files of
the formats the engine reads (PEGS4 media, XCOM cross sections, form factors,
multiple-scattering surface, spin table) from textbook formulas: collision
losses by Berger and Seltzer, Moller, Bhabha and Heitler cross sections,
complete-screening bremsstrahlung and smooth fits of the photon cross
sections.  They are within some ten per cent of the tabulated ones, so
histories take the steps, events and branches they take with the real data.

Every result is a Monte Carlo estimate: its value depends on the random
streams and on the rounding of each trajectory, and no formula gives it, so
`exact` has nothing to say.  The same seed gives the same histories, hence
the same result up to the order of the FP64 sums.
"""
from __future__ import annotations

import functools
import math
import tempfile
from pathlib import Path

import numpy as np

from ompmc_b200 import assets
from ompmc_b200.engine import EVENT_FP32, EVENT_FP64, PLAIN_FP64, Engine, Server, Tables, bixel_grid, load_spectrum

RM = 0.5109989461           # electron rest energy, MeV
R02 = 0.079407877           # classical electron radius squared, barn
NA = 0.60221408             # Avogadro's number x 1e-24
FSC = 1.0 / 137.035999

# ------------------------------------------------------------ physics data
#: Media by mass: density, mean excitation energy (eV), (Z, A, mass fraction).
_H, _C, _N, _O = (1, 1.008), (6, 12.011), (7, 14.007), (8, 15.999)
MEDIA = {
    "H2O521ICRU": (1.0, 75.0, [(*_H, 0.1119), (*_O, 0.8881)]),
    "LUNG521ICRU": (0.26, 75.3, [(*_H, 0.103), (*_C, 0.105), (*_N, 0.031), (*_O, 0.761)]),
    "ICRUTISSUE521ICRU": (1.0, 74.9, [(*_H, 0.101), (*_C, 0.111), (*_N, 0.026), (*_O, 0.762)]),
    "ICRPBONE521ICRU": (1.85, 106.4, [(*_H, 0.047), (*_C, 0.144), (*_N, 0.042), (*_O, 0.446), (15, 30.974, 0.105),
                                     (20, 40.078, 0.216)]),
    "AIR521ICRU": (1.2048e-3, 85.7, [(*_C, 0.0001), (*_N, 0.7553), (*_O, 0.2318), (18, 39.948, 0.0128)]),
}
AE, AP, UE, UP = 0.521, 0.01, 50.511, 50.0
MEKE = 176


def _collision(t, te, mean_i, positron):
    """Restricted collision loss bracket L of dE/dx = 2 pi r0^2 n m / beta^2 L
    (Berger and Seltzer); t in units of m, te the Moller threshold."""
    beta2 = t * (t + 2) / (t + 1) ** 2
    base = np.log(2 * (t + 2) / mean_i ** 2)
    if positron:
        d = np.minimum(te, t)
        y = 1 / (t + 2)
        f = np.log(t * d) - beta2 / t * (t + 2 * d - 1.5 * d ** 2 * y - (d - d ** 3 / 3) * y ** 2
                                         - (d ** 2 / 2 - t * d ** 3 / 3 + d ** 4 / 4) * y ** 3)
    else:
        d = np.minimum(te, t / 2)
        f = -1 - beta2 + np.log((t - d) * d) + t / (t - d) + (d ** 2 / 2 + (2 * t + 1) * np.log(1 - d / t)) / (t + 1) ** 2
    x = np.log10(np.sqrt(t * (t + 2)))
    delta = np.where(x > 0.24, 4.606 * x - 3.5 + 0.0912 * np.maximum(2.8 - x, 0) ** 3.48, 0.0)
    return base + f - np.maximum(delta, 0)


def _electron_tables(medium):
    """PEGS4 arrays of one medium per cm: energy grid and the 7 functions of
    ln E (sigma, loss and branching ratios of e- and e+), with scalars."""
    rho, mean_i, parts = medium
    ne = rho * NA * sum(w * z / a for z, a, w in parts)            # electrons per barn cm
    rlc = 1 / (rho * sum(w * z * (z + 1) * math.log(287 / math.sqrt(z)) / (716.4 * a) for z, a, w in parts))
    te = AE - RM
    e = np.exp(np.linspace(math.log(te), math.log(UE - RM), MEKE))
    t, c = e / RM, te / RM
    beta2 = t * (t + 2) / (t + 1) ** 2
    k = 2 * math.pi * R02 * ne * RM
    loss = [k / beta2 * _collision(t, c, mean_i * 1e-6 / RM, p) for p in (False, True)]
    loss = [s + 4 / 3 * AP / rlc * (e + RM) / (e + 1.5 * RM) for s in loss]
    y = np.minimum(AP / e, 1.0)                                   # complete screening, softened at low energy
    brem = (4 / 3 * (-np.log(y) - 1 + y) + (1 - y ** 2) / 2) / rlc * e / (e + 0.4)
    g = t + 1
    c1, c2 = (t / g) ** 2, (2 * g - 1) / g ** 2
    e0 = np.minimum(te / e, 0.5)
    moller = k / (beta2 * e) * (c1 * (0.5 - e0) + 1 / e0 - 1 / (1 - e0) - c2 * np.log((1 - e0) / e0))
    moller = np.where(e > 2 * te, np.maximum(moller, 0), 0.0)
    yy = 1 / (t + 2)
    yp = 1 - 2 * yy
    b4, b2, b1 = yp ** 3, yp * (3 + yy ** 2), 2 - yy ** 2
    b3 = b4 + yp ** 2
    u = np.linspace(0, 1, 401)[:, None]
    eps = np.exp(np.log(np.minimum(te / e, 1.0)) * (1 - u))         # log grid from the threshold to 1
    f = (1 / (eps * beta2) - b1 + eps * (b2 - eps * (b3 - eps * b4)))
    bhabha = np.maximum(k / e * np.sum((f[1:] + f[:-1]) / 2 * np.diff(np.log(eps), axis=0), axis=0), 0)
    q = np.sqrt(g ** 2 - 1)
    annih = ne * math.pi * R02 / (g + 1) * ((g ** 2 + 4 * g + 1) / (g ** 2 - 1) * np.log(g + q) - (g + 3) / q)
    sige, sigp = brem + moller, brem + bhabha + annih
    sige = np.maximum(sige, 1e-12)
    zs = sum(w / a * z * (z + 1) for z, a, w in parts)
    ze = sum(w / a * z * (z + 1) * math.log(z ** (-2 / 3)) for z, a, w in parts)
    zx = sum(w / a * z * (z + 1) * math.log(1 + 3.34 * (FSC * z) ** 2) for z, a, w in parts)
    blcc = 6680.0 * rho * zs * math.exp((ze - zx) / zs)
    xcc = 22.696 * math.pi / 180 * math.sqrt(zs * rho)
    zt = sum(w / a * z * (z + 1) for z, a, w in parts)
    zg = -sum(w / a * z * (z + 1) * math.log(z) / 3 for z, a, w in parts) / zt
    delcm = 136 * RM * math.exp(zg)
    fs = [sige * rlc, sigp * rlc, loss[0] * rlc, loss[1] * rlc, brem / sige, brem / sigp, (brem + bhabha) / sigp,
          np.full(MEKE, 0.01)]
    return e, fs, rlc, blcc * rlc, xcc * math.sqrt(rlc), delcm


def _write_pegs(path):
    """The media above in the PEGS4 text format (one block a medium)."""
    out = []
    for name, medium in MEDIA.items():
        rho, _, parts = medium
        e, fs, rlc, blcc, xcc, delcm = _electron_tables(medium)
        eke1 = (MEKE - 1) / math.log(e[-1] / e[0])
        eke0 = 1 - eke1 * math.log(e[0])
        out.append(f" MEDIUM={name:24s}STERNCID={name:24s}")
        out.append(f" MIXT,RHO= {rho:.6E},NE={len(parts):2d}, IUNRST=0, EPSTFL=0, IAPRIM=1")
        unit = min(w / a for _, a, w in parts)
        for z, a, w in parts:
            out.append(f" ASYM=X ,Z={z:3d}.,A={a:9.4f},PZ= {w / a / unit:.6E},RHOZ= {w / unit:.6E}")
        out.append(f"  {rlc:.7E}  {AE:.7E}  {AP:.7E}  {UE:.7E}  {UP:.7E}")
        out.append(f"    0    0    0  {MEKE:3d}    0    0    0")
        out += ["  0.0 0.0 0.0 0.0 0.0 0.0"] * 7
        head = [0.952, delcm, 0, 0, 0, 0, 0, 0, 0, 0, blcc, xcc, eke0, eke1]
        out.append(" ".join(f"{v:.9E}" for v in head))
        le = np.log(e)
        rows = np.zeros((MEKE, 16))
        for c, v in enumerate(fs):
            a1 = np.append(np.diff(v) / np.diff(le), 0.0)
            a1[-1] = a1[-2]
            rows[:, 2 * c], rows[:, 2 * c + 1] = v - a1 * le, a1
        out += [" ".join(f"{v:.9E}" for v in r) for r in rows]
    path.write_text("\n".join(out) + "\n")


def _write_element_data(root):
    """XCOM-like cross sections per element (ln MeV, ln barn) and form factors."""
    e = np.exp(np.linspace(math.log(0.001), math.log(100.0), 80))
    k = e / RM
    shape = np.interp(np.log(k), np.log([2.0, 4.0, 11.7, 40.0, 200.0]), [0.45, 0.9, 3.05, 6.5, 9.0])
    files = {"photo": [], "rayleigh": [], "pair": [], "triplet": []}
    for z in range(1, 51):
        photo = 148 * (z / 8) ** 4.4 * (0.01 / e) ** 3.15 * (1 + (e / 0.4) ** 2)
        rayl = 6 * (z / 8) ** 2.4 * np.where(e > 0.01, (0.01 / e) ** 1.7, (0.01 / e) ** 0.4)
        files["photo"].append((e, photo))
        files["rayleigh"].append((e, rayl))
        for name, thr, f in (("pair", 2 * RM, z * z), ("triplet", 4 * RM, z)):
            m = e > 1.05 * thr
            files[name].append((e[m], FSC * R02 * f * shape[m] * (1 - thr / e[m]) ** 3))
    for name, rows in files.items():
        text = []
        for x, s in rows:
            text.append(str(len(x)))
            text += [f"{a:.8E} {b:.8E}" for a, b in zip(np.log(x), np.log(s))]
        (root / f"xcom_{name}.data").write_text("\n".join(text) + "\n")
    x = np.concatenate([[0.0], np.exp(np.linspace(math.log(0.005), math.log(6000.0), 99))])
    text = [" ".join(f"{v:.6E}" for v in x)]
    for z in range(1, 51):
        ff = z / (1 + (x / (0.25 * z ** (1 / 3))) ** 2) ** 1.6
        text.append(" ".join(f"{v:.6E}" for v in ff))
    (root / "pgs4form.dat").write_text("\n".join(text) + "\n")


def _write_ms_surface(path):
    """Multiple-scattering surface: 64 x 8 rows of nodes, densities and aliases."""
    u = np.linspace(0, 1, 32)
    text = []
    for i in range(64):
        for j in range(8):
            f = 1 + 0.25 * np.cos(math.pi * u * (1 + 0.1 * j)) * (1 + i / 128)
            w = 0.7 + 0.3 * np.cos(1.7 * np.arange(31) + 0.3 * i + j) ** 2
            a = np.arange(31) // 2 + 1
            text += [" ".join(f"{v:.7f}" for v in r) for r in (u, f, w)] + [" ".join(str(v) for v in a)]
    path.write_text("\n".join(text) + "\n")


@functools.lru_cache(maxsize=None)
def _data():
    """The folder with the files above, written once in a process."""
    keep = tempfile.TemporaryDirectory(prefix="omc_cases_")
    root = Path(keep.name)
    _write_pegs(root / "media.pegs4dat")
    _write_element_data(root)
    _write_ms_surface(root / "msnew.data")
    assets.write_spin_standin(root / "spinms.data", zmax=20)
    for s in assets.SPECTRA:
        assets.write_spectrum(root / f"{s}.spectrum", s)
    return keep, root


@functools.lru_cache(maxsize=None)
def _tables(media):
    root = _data()[1]
    return Tables(root / "media.pegs4dat", root / "pgs4form.dat", root, media)


# ---------------------------------------------------------------- phantoms
@functools.lru_cache(maxsize=4)
def _phantom(kind, n, fine):
    """One patient's (or one test's) phantom: water or slab cube of n^3
    voxels, or the CT-like body on n x n x 3n/4 voxels; `fine` names the voxel
    size in millimetres."""
    if kind == "water":
        return assets.water_cube(n, fine / 10)
    if kind == "slab":
        return assets.slab_phantom(n, fine / 10)
    size = n * fine / 10 / 38.4
    return assets.ct_phantom(n, n, (n * 3) // 4, fine / 10, seed=1234, scale=(size, size, size))


# ------------------------------------------------------------------- cases
def listed():
    beam = dict(kind="beam", form="fp32", source="6mv", charge=0, nsplit=1, batches=10, field=5.0)
    return [
        # a spot check while a plan is edited: the smallest run that the batch statistics still make sense of
        dict(beam, name="beam_water30_1e4", phantom="water", n=30, mm=10.0, histories=10_000),
        # the slab phantom of the tests and of the benchmark's second workload, at a draft's and a result's histories
        dict(beam, name="beam_slab64_1e6", phantom="slab", n=64, mm=2.5, histories=1_000_000),
        dict(beam, name="beam_slab64_1e7", phantom="slab", n=64, mm=2.5, histories=10_000_000),
        # a patient-sized CT grid under a 10 x 10 cm field, with an odd history count
        dict(beam, name="beam_ct128_5e6", phantom="ct", n=128, mm=3.0, histories=5_000_003, field=10.0),
        # a fine CT grid (6 M voxels) and the high-energy spectrum: tallies and results larger than L2
        dict(beam, name="beam_ct200_18mv", phantom="ct", n=200, mm=2.0, source="18mv", histories=1_000_000,
             field=10.0),
        # an electron field (charge -1), one energy
        dict(beam, name="beam_electron_6mev", phantom="water", n=47, mm=5.0, source="mono", energy=6.0, charge=-1,
             histories=200_000, field=4.0),
        # photon splitting, the variance reduction that the input file's nsplit asks for
        dict(beam, name="beam_slab64_nsplit20", phantom="slab", n=64, mm=2.5, nsplit=20, histories=100_000),
        # FP64 transport: the accuracy study's form
        dict(beam, name="beam_ct64_fp64", phantom="ct", n=64, mm=6.0, form="fp64", histories=300_000),
        # the form with fixed scratch that a plan optimiser calls in its loop
        dict(beam, name="noalloc_water30", phantom="water", n=30, mm=10.0, form="noalloc", histories=20_000),
        # dose influence columns of a small field, as matRad asks for them
        dict(kind="dij", name="dij_ct64_36", phantom="ct", n=64, mm=6.0, source="6mv", beams=1, side=6,
             histories=10_000, batches=10),
        # the benchmark's serving load in small: seven beams' bixels, histories spread over a decade
        dict(kind="serve", name="serve_ct128_63", phantom="ct", n=128, mm=3.0, source="6mv", beams=7, side=3,
             histories=60_000, batches=10),
        # one request at a time on the same server, the sequential loop of a user without batching
        dict(kind="serve", name="serve_ct128_single", phantom="ct", n=128, mm=3.0, source="6mv", beams=1, side=1,
             histories=60_000, batches=10),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """A case of the same ranges: any phantom, grid, source, form and count."""
    kind = rng.choice(["beam"] * 6 + ["noalloc", "dij", "serve", "serve"])
    phantom = rng.choice(["water", "slab", "ct"])
    n = int(_log(rng, 20, 144 if phantom == "ct" else 72))
    extent = {"water": 300.0, "slab": 160.0, "ct": 384.0}[phantom]
    # odd sizes: the pitch is whatever fits the extent, to a tenth of a millimetre
    grid = dict(phantom=phantom, n=n, mm=round(extent / n, 1))
    source = rng.choice(["6mv", "6mv", "18mv"])
    if kind in ("beam", "noalloc"):
        c = dict(kind="beam", form="fp32", source=source, charge=0, nsplit=1, batches=rng.choice([10, 10, 10, 5, 20]),
                 field=round(rng.uniform(1.0, 12.0), 1), **grid)
        if kind == "noalloc":
            c.update(phantom="water", n=rng.randrange(20, 41), form="noalloc", histories=int(_log(rng, 1e4, 2.5e4)))
            c["mm"] = round(300.0 / c["n"], 1)
            return c
        what = rng.choice(["photon", "photon", "photon", "electron", "split", "fp64"])
        if what == "electron":
            c.update(source="mono", energy=round(rng.uniform(1.0, 12.0), 2), charge=rng.choice([-1, -1, 1]),
                     histories=int(_log(rng, 1e4, 1e6)))
        elif what == "split":
            c.update(nsplit=rng.choice([5, 10, 20]), histories=int(_log(rng, 1e4, 2e5)))
        elif what == "fp64":
            c.update(form="fp64", histories=int(_log(rng, 1e4, 6e5)))
        else:
            c.update(histories=int(_log(rng, 1e4, 5e6)))
        return c
    c = dict(source=source, batches=10, phantom="ct", n=int(_log(rng, 32, 128)))
    c["mm"] = round(384.0 / c["n"], 1)
    if kind == "dij":
        return dict(c, kind="dij", beams=rng.randrange(1, 4), side=rng.randrange(2, 7), histories=int(_log(rng, 5e3, 4e4)))
    return dict(c, kind="serve", beams=rng.randrange(1, 8), side=rng.randrange(1, 4), histories=int(_log(rng, 2e4, 6e4)))


# ------------------------------------------------------------------ passes
def _source(case):
    if case["source"] == "mono":
        return dict(mono_energy=case["energy"], charge=case["charge"])
    return dict(spectrum=load_spectrum(_data()[1] / f"{case['source']}.spectrum"))


class _Matrix:
    """The plan's sparse dose matrix: columns one after the other in arrays of
    a fixed capacity, row -1 and value 0 where there is no entry."""

    def __init__(self, columns, nvox):
        capacity = columns * min(nvox, 200_000)
        self.nnz = np.zeros(columns, dtype=np.int64)
        self.rows = np.full(capacity, -1, dtype=np.int32)
        self.vals, self.var = np.zeros(capacity), np.zeros(capacity)

    def take(self, nnz, rows, vals, var):
        before, total = int(self.nnz.sum()), int(np.sum(nnz))
        self.nnz[:] = nnz
        for to, parts, none in ((self.rows, rows, -1), (self.vals, vals, 0.0), (self.var, var, 0.0)):
            np.concatenate(parts, out=to[:total])
            to[total:before] = none
        return dict(nnz=self.nnz, rows=self.rows, vals=self.vals, var=self.var)


def prepare(case, seed):
    """Tables, phantom, engine (and server) that the user's program keeps, and
    the beam that this plan asks for: its place, and its histories' seed."""
    rng = np.random.default_rng(seed)
    ph = _phantom(case["phantom"], case["n"], case["mm"])
    tables = _tables(tuple(ph.media))
    if case["kind"] == "beam":
        engine = Engine(tables, ph, nsplit=case["nsplit"])
        dx, dy = rng.uniform(-1.0, 1.0, 2)
        h = case["field"] / 2
        call = dict(ncase=case["histories"], nbatch=case["batches"], seed=1 + seed,
                    collimator=(dx - h, dx + h, dy - h, dy + h), **_source(case))
        return dict(case=case, engine=engine, call=call)
    engine = Engine(tables, ph)
    gantry = (np.array([0.0, 51.0, 103.0, 154.0, 206.0, 257.0, 309.0])[:case["beams"]] + rng.uniform(0, 20)).tolist()
    bl = bixel_grid(ph, gantry, bixel=0.5, field=(0.5 * case["side"], 0.5 * case["side"]))
    bl.update(_source(case))
    state = dict(case=case, engine=engine, beamlets=bl, seed=1 + seed, matrix=_Matrix(len(bl["corner"]), ph.nvox))
    if case["kind"] == "serve":
        nb = len(bl["corner"])
        state["server"] = Server(engine, max_requests=min(64, nb), seed=1 + seed)
        state["set"] = state["server"].beamlet_set(bl)
        # a decade of histories over the requests, around the case's count
        state["jobs"] = [(int(b), int(case["histories"] * 10 ** (f - 0.5)) if nb > 1 else case["histories"])
                         for b, f in zip(rng.permutation(nb), rng.uniform(0, 1, nb))]
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "beam":
        if case["form"] == "noalloc":
            dose, unc, stats = state["engine"].run_beam_noalloc(**state["call"])
        else:
            mode = {"fp32": EVENT_FP32, "fp64": EVENT_FP64, "plain": PLAIN_FP64}[case["form"]]
            dose, unc, stats = state["engine"].run_beam(mode=mode, **state["call"])
        return dict(dose=dose, unc=unc, edep=stats["edep"], esrc=stats["esrc"], histories=int(stats["histories"]))
    if case["kind"] == "dij":
        colptr, rows, vals, var, _ = state["engine"].run_beamlets(state["beamlets"], case["histories"], case["batches"],
                                                                  1e-4, seed=state["seed"])
        return state["matrix"].take(np.diff(colptr), [rows], [vals], [var])
    server = state["server"]
    ids = [server.submit_beamlet(state["set"], b, n, case["batches"], 1e-4, seed=state["seed"] * 4096 + b + 1)
           for b, n in state["jobs"]]
    while server.step(8) > 0:
        pass
    columns = [server.result_sparse(i) for i in ids]
    server.completed()
    for i in ids:
        server.release(i)
    return state["matrix"].take([len(c[0]) for c in columns], *([c[k] for c in columns] for k in range(3)))


def exact(case, seed):
    """A Monte Carlo estimate has no value that a formula gives."""
    return None


def work(case):
    """The phantom read and the result written once, and the arithmetic of the
    histories: some 50 transport steps each (photon splitting: times the
    splitting factor's share of charged particles) of about 400 operations."""
    n = case["n"]
    nvox = n * n * ((n * 3) // 4 if case["phantom"] == "ct" else n)
    if case["kind"] == "beam":
        histories, out = case["histories"], 16 * nvox
        steps = 50.0 if case["charge"] == 0 else 150.0
        steps *= case["nsplit"] / 2 if case["nsplit"] > 1 else 1
    else:
        columns = case["beams"] * case["side"] ** 2
        histories, out = columns * case["histories"], columns * 20 * nvox // 20
        steps = 50.0
    return dict(bytes=5.0 * nvox + out, flops=histories * steps * 400.0)
