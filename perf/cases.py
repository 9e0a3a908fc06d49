"""Measured workloads of the dose engine: what its users have it compute.

Every case is one whole call of the Python API: a dose job (``Engine.run``),
a dose-influence matrix (``Engine.run_dij``), history-by-history scoring or a
round trip of the dose server.  Phantoms and spectra come from
``ompmc_gb300.workloads``; the physics tables are built by the library from
files in the reference's formats (pegs4, form factors, XCOM, msnew, spinms).
Those files are generated here from textbook formulas, so that the cases run
where no copy of the real data is at hand; they give water, lung, bone and
air their usual mean free paths, stopping powers and scattering strengths.

The engine is a Monte Carlo program whose particles are processed in an
order that differs from run to run, so two runs of the same seeds agree
within their statistical noise.  Phantoms, fields and history counts are
chosen so that this noise is about one per cent of the dose (2-norm), which
is also what a planning dose is computed to.  There is no closed-form value
of a dose, hence no ``exact``.
"""

from __future__ import annotations

import math
import os
import tempfile

import numpy as np

from ompmc_gb300 import api, spinms
from ompmc_gb300 import workloads as W

RM = 0.5109989461  # electron rest energy, MeV
TE, AP, UE, UP = 0.700 - RM, 0.010, 50.511, 50.0
RE2N = 0.0794079 * 0.60221408  # classical electron radius squared (barn) times Avogadro (1e24)

# Name -> (density, {Z: (A, atoms per formula)}, mean excitation energy / eV, radiation length g/cm2)
MEDIA = {
    W.WATER: (1.0, {1: (1.008, 2.0), 8: (15.999, 1.0)}, 75.0, 36.08),
    W.LUNG: (0.26, {1: (1.008, 10.2), 6: (12.011, 0.86), 7: (14.007, 0.22), 8: (15.999, 4.68)}, 75.3, 36.5),
    W.BONE: (1.85, {1: (1.008, 4.7), 6: (12.011, 1.2), 7: (14.007, 0.3), 8: (15.999, 2.79), 15: (30.974, 0.226),
                    20: (40.078, 0.525)}, 106.4, 27.8),
    W.AIR: (0.0012048, {7: (14.007, 1.56), 8: (15.999, 0.42), 18: (39.948, 0.01)}, 85.7, 36.62),
}
SLAB4 = ((0.0, 5.0, W.WATER, 1.0), (5.0, 15.0, W.LUNG, 0.26), (15.0, 18.0, W.BONE, 1.85), (18.0, 30.0, W.WATER, 1.0))


# ---- physics files -----------------------------------------------------------
def _fmt(values):
    return " ".join("%.10g" % v for v in values)


def _electron_tables(rho, elements, i_ev, x0):
    """Per-energy cross sections and restricted stopping powers (per cm):
    Moller and Bhabha above TE, Born-approximation bremsstrahlung above AP,
    Heitler annihilation, Bethe-Bloch below TE."""
    mass = sum(a * p for a, p in elements.values())
    ne = RE2N * rho * sum(z * p for z, (a, p) in elements.items()) / mass  # r_e^2 * electrons per cm3, 1/cm
    n = 150
    t = np.exp(np.linspace(math.log(0.9995 * TE), math.log(UE - RM), n))  # a track's last energies lie inside
    tau = t / RM
    b2 = tau * (tau + 2) / (tau + 1) ** 2
    c = 2 * math.pi * ne / b2
    eps = np.minimum(TE / t, 0.5)
    moller = c / tau * ((tau / (tau + 1)) ** 2 * (0.5 - eps) + 1 / eps - 1 / (1 - eps)
                        - (2 * tau + 1) / (tau + 1) ** 2 * np.log((1 - eps) / eps))
    moller = np.where(t > 2 * TE, np.maximum(moller, 0.0), 0.0)
    eb = np.minimum(TE / t, 1.0)
    bhabha = np.where(t > TE, c / tau * np.maximum(1 / eb - 1 + b2 * (0.5 - 2) * np.log(1 / eb) * 0.5, 0.0), 0.0)
    g = tau + 1
    annih = math.pi * ne / (g + 1) * ((g * g + 4 * g + 1) / (g * g - 1) * np.log(g + np.sqrt(g * g - 1))
                                      - (g + 3) / np.sqrt(g * g - 1))
    y = np.minimum(AP / t, 1.0)
    soft = t / (t + 1.0)  # the Born logarithm falls off below a few MeV
    brems = soft * rho / x0 * (4 / 3 * np.log(1 / y) - 4 / 3 * (1 - y) + 0.5 * (1 - y * y))
    x = np.log10(np.sqrt(tau * (tau + 2)))
    delta = np.where(x < 0.24, 0.0, 4.6052 * x - 3.502 + 0.0912 * np.maximum(2.8 - x, 0.0) ** 3.477)
    d = np.minimum(TE / RM, tau / 2)
    f = -1 - b2 + np.log((tau - d) * d) + tau / (tau - d) + (d * d / 2 + (2 * tau + 1) * np.log(1 - d / tau)) / g ** 2
    dedx = RM * c * (np.log(2 * (tau + 2) / (i_ev * 1e-6 / RM) ** 2) + f - np.maximum(delta, 0.0))
    dedx += soft * rho / x0 * 4 / 3 * AP
    esig, psig = moller + brems, bhabha + annih + brems
    cols = (esig * x0 / rho, psig * x0 / rho, dedx * x0 / rho, dedx * x0 / rho, brems / esig, brems / psig,
            (brems + bhabha) / psig, np.ones(n))
    return t, cols


def _write_pegs(path):
    out = []
    for name, (rho, el, i_ev, x0) in MEDIA.items():
        mass = sum(a * p for a, p in el.values())
        zs = sum(p * z * (z + 1) for z, (a, p) in el.items())
        ze = sum(p * z * (z + 1) * math.log(z ** (-2 / 3)) for z, (a, p) in el.items())
        zx = sum(p * z * (z + 1) * math.log(1 + 3.34 * (z / 137.036) ** 2) for z, (a, p) in el.items())
        rlc = x0 / rho
        # Moliere's scattering parameters per cm; the file holds them per radiation length.
        blcc = 6702.33 * rho * zs / mass * math.exp((ze - zx) / zs)
        xcc = 0.1569 * rho * zs / mass
        t, cols = _electron_tables(rho, el, i_ev, x0)
        n = len(t)
        eke1 = (n - 1) / math.log(t[-1] / t[0])
        eke0 = 1 - eke1 * math.log(t[0])
        lt = np.log(t)
        out.append(" MEDIUM=%-24s,STERNCID=%s" % (name, name))
        out.append(" COMP,RHO=%.6g,NE=%d" % (rho, len(el)))
        for z, (a, p) in el.items():
            out.append(" ASYM=%d,Z=%d.,A=%.4f,PZ=%.5g,RHOZ=%.5g" % (z, z, a, p, a * p))
        out.append(_fmt((rlc, TE + RM, AP, UE, UP)))
        out.append("0 0 0 %d 0 0 0" % n)
        out.extend(["0 0 0 0 0 0"] * 6)
        zg = -sum(p * z * (z + 1) * math.log(z) for z, (a, p) in el.items()) / (3 * zs)
        out.append("0 0 0 0 0")
        out.append(_fmt((0.952, 136 * RM * math.exp(zg), 0, 0, 0, 0, 0, 0, 0, 0, blcc * rlc, math.sqrt(xcc * rlc),
                         eke0, eke1)))
        pairs = []
        for v in cols:
            slope = np.empty(n)
            slope[:-1] = (v[1:] - v[:-1]) * eke1
            slope[-1] = slope[-2]
            pairs += [v - slope * lt, slope]
        out.extend(_fmt(row) for row in np.stack(pairs, 1))
    with open(path, "w") as f:
        f.write("\n".join(out) + "\n")


def _write_xsec(path, energies, sigma):
    with open(path, "w") as f:
        for z in range(1, 51):
            f.write("%d\n%s\n" % (len(energies), _fmt(np.stack((np.log(energies), np.log(sigma(z))), 1).ravel())))


def write_physics(root):
    """Write the physics files under `root` (pegs4/ and data/); returns the
    .inp keys that name them."""
    pegs, data = os.path.join(root, "pegs4"), os.path.join(root, "data")
    os.makedirs(pegs, exist_ok=True)
    os.makedirs(data, exist_ok=True)
    _write_pegs(os.path.join(pegs, "700icru.pegs4dat"))
    # Photon cross sections in barn per atom: power laws pinned to oxygen at 10 keV; pair and triplet with
    # their thresholds.
    e = np.exp(np.linspace(math.log(1e-3), math.log(60.0), 80))
    _write_xsec(os.path.join(data, "xcom_photo.data"), e,
                lambda z: 148 * (z / 8) ** 4.2 * (e / 0.01) ** -3.3 * (1 + (e / 0.6) ** 2) ** 1.05)
    _write_xsec(os.path.join(data, "xcom_rayleigh.data"), e,
                lambda z: 6.7 * (z / 8) ** 2.4 * 2.0 / (1.0 + (e / 0.01) ** 1.85))
    for name, eth, weight in (("pair", 2 * RM, lambda z: z * z), ("triplet", 4 * RM, lambda z: 0.8 * z)):
        ep = np.exp(np.linspace(math.log(1.02 * eth), math.log(60.0), 60))
        sig = 5.795e-4 * (1 - eth / ep) ** 3 * np.clip(2.7 + 1.18 * np.log(ep / 2), 1.5, 6.5)
        _write_xsec(os.path.join(data, "xcom_%s.data" % name), ep, lambda z: weight(z) * sig)
    x = np.concatenate(([0.0], np.exp(np.linspace(math.log(5e-3), math.log(1e6), 99))))
    with open(os.path.join(pegs, "pgs4form.dat"), "w") as f:
        f.write(_fmt(x) + "\n")
        for z in range(1, 51):
            # (falls as x^-0.8: the cumulative distribution stays strictly increasing in single precision)
            f.write(_fmt(z * (1 + (x / (0.45 * z ** (1 / 3))) ** 2) ** -0.4) + "\n")
    # Multiple-scattering surface: the variable u is uniform (screened Rutherford scattering), no aliases.
    row = "\n".join((_fmt(np.arange(32) / 31.0), _fmt(np.ones(32)), _fmt(np.ones(31)), _fmt(np.arange(1, 32))))
    with open(os.path.join(data, "msnew.data"), "w") as f:
        f.write("\n".join([row] * (64 * 8)) + "\n")
    spinms.write_spin_neutral(os.path.join(data, "spinms.data"))
    for name, spec in (("6mv", W.spectrum_6mv()), ("250kvp", W.spectrum_250kvp())):
        W.write_spectrum(os.path.join(data, name + ".spectrum"), name, *spec)
    return {"pegs": os.path.join(pegs, "700icru.pegs4dat"), "pgs4form": os.path.join(pegs, "pgs4form.dat"),
            "data_folder": data + os.sep}


_files = {}


def _physics():
    if not _files:
        _files.update(write_physics(tempfile.mkdtemp(prefix="omc_physics_")))
    return _files


# ---- cases ---------------------------------------------------------------------
def _case(name=None, call="run", phantom="slab", nx=20, ny=20, nz=20, vox=1.5, source="6mv", charge=0, field=10.0,
          histories=1_000_000, nbatch=10, nsplit=1, fp32=True, inflight=0, beamlets=0, jobs=0):
    c = dict(call=call, phantom=phantom, nx=nx, ny=ny, nz=nz, vox=vox, source=source, charge=charge, field=field,
             histories=histories, nbatch=nbatch, nsplit=nsplit, fp32=fp32, inflight=inflight, beamlets=beamlets,
             jobs=jobs)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest call: a 5 MeV electron pencil beam on a little water box, launch and drain latency.
        _case("electron_pencil", phantom="water", nx=12, ny=12, nz=12, vox=0.5, source="mono5", charge=-1, field=0.0,
              histories=100_000),
        # The plain small job: 1.25 MeV parallel photons on water in the reference's arithmetic.
        _case("water_fp64", phantom="water", nx=12, ny=12, nz=12, vox=2.5, source="mono1.25", histories=4_000_000,
              fp32=False),
        # The 6 MV slab on a coarse grid, a planning-size job.
        _case("slab_6mv", nx=30, ny=30, nz=30, vox=1.0, histories=40_000_000),
        # The 6 MV slab on its 2 mm grid: a small (radiosurgery) field, scored to about one per cent.
        _case("slab_2mm", nx=150, ny=150, nz=150, vox=0.2, field=1.5, histories=80_000_000),
        # The same slab in the reference's arithmetic.
        _case("slab_fp64", field=5.0, histories=8_000_000, fp32=False),
        # 250 kVp: photo-electric absorption, Rayleigh scattering and photons below the electron cut-off.
        _case("kvp_250", source="250kvp", field=5.0, histories=6_000_000),
        # A positron field (Bhabha, annihilation), the other charge of the electron tables.
        _case("positron_field", phantom="water", nx=15, ny=13, nz=11, vox=0.5, source="mono5", charge=1, field=2.0,
              histories=1_000_000),
        # Photon splitting, the variance reduction users turn on, with its queues bounded by `inflight`.
        _case("slab_split16", field=5.0, histories=1_000_000, nsplit=16, inflight=2_000_000),
        # History-by-history uncertainties beside the batch sums.
        _case("slab_history", call="history", field=4.0, histories=6_000_000),
        # A new patient: phantom upload and dose of a blob phantom with odd sizes, four media.
        _case("ct_new_phantom", call="upload", phantom="ct", nx=61, ny=67, nz=33, vox=0.8, field=5.0,
              histories=60_000_000),
        # matRad's dose-influence matrix: beamlets of three gantry angles in one launch.
        _case("dij_ct", call="dij", phantom="ct", nx=33, ny=35, nz=31, vox=1.0, histories=32_400_000, beamlets=36),
        # The dose server: jobs of three phantoms and two spectra submitted together.
        _case("server_mix", call="server", nx=20, ny=20, nz=20, vox=1.5, field=5.0, histories=32_000_000, jobs=4),
    ]


def _needed(vox, field):
    """Histories for a noise of about two per cent between two runs: it falls
    with the square root of the histories per beam area and of the voxel
    volume."""
    return 1.3e6 * max(field, vox) ** 2 / vox ** 3


def draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "history", "upload", "dij", "server"))
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    if kind == "run" and rng.random() < 0.35:  # charged particles
        n = [rng.randint(9, 40) for _ in range(3)]
        fp32 = rng.random() < 0.75
        field = rng.choice((0.0, 2.0 if fp32 else 1.0))
        hist = log(1.2e6 if field else 2e5, 3e6) / (1 if fp32 else 3)
        return _case(phantom="water", nx=n[0], ny=n[1], nz=n[2], vox=round(log(0.3, 0.7), 3), source="mono5",
                     charge=rng.choice((-1, 1)), field=field, histories=int(hist), nbatch=rng.choice((5, 10)),
                     fp32=fp32)
    vox = log(0.8, 2.0)
    # The box stays near 30 cm, the axes differ.
    n = [max(6, int(round(30.0 / vox * rng.uniform(0.85, 1.15)))) for _ in range(3)]
    box = dict(nx=n[0], ny=n[1], nz=n[2], vox=round(vox, 3))
    if kind == "dij":
        beamlets = 3 * rng.choice((4, 9, 12))
        return _case(call="dij", phantom="ct", field=3.0, beamlets=beamlets, **box,
                     histories=beamlets * int(min(1e6, 9e5 * max(1.0, vox ** 2) / vox ** 3)))
    phantom = "ct" if kind == "upload" else rng.choice(("water", "slab", "slab", "ct"))
    source = "6mv" if kind == "history" else rng.choice(("6mv", "6mv", "mono1.25", "250kvp"))
    # A field as wide as the option's speed allows at the wanted noise.
    most, fp32, nsplit, inflight, scale = 6e7, True, 1, 0, 1.0
    jobs = rng.choice((2, 3, 5)) if kind == "server" else 0
    if kind == "run":
        option = rng.random()
        if option < 0.25:
            most, fp32 = 1e7, False
        elif option < 0.45:
            nsplit, inflight, scale = rng.choice((4, 8, 16)), 2_000_000, 0.5
            most = 6e7 / nsplit
    elif kind == "history":
        most, scale = 1.2e7, 1.2
    scale *= max(1, jobs)
    widest = math.sqrt(most / scale / _needed(vox, 1.0) * max(1.0, vox ** 2))
    field = round(min(8.0, widest, max(vox, rng.uniform(2.0, 8.0))), 2)
    return _case(call=kind, phantom=phantom, source=source, field=field, nsplit=nsplit, fp32=fp32, inflight=inflight,
                 jobs=jobs, histories=int(scale * _needed(vox, field) * rng.uniform(1.0, 1.3)), **box)


def _phantom(c, seed, kind=None):
    kind = kind or c["phantom"]
    nxyz = (c["nx"], c["ny"], c["nz"])
    if kind == "water":
        return W.homogeneous(vox=c["vox"], nxyz=nxyz)
    if kind == "slab":
        layers = SLAB4[:-1] + ((18.0, 1e3, W.WATER, 1.0),)
        return W.slab(vox=c["vox"], nxyz=nxyz, layers=layers)
    return W.ct_like(*nxyz, vox=c["vox"], seed=seed)


def _job_text(c, seed, histories, source=None):
    """The .inp text of the job, with the seed's RANMAR seed pair and a field
    moved by up to half a millimetre."""
    rng = np.random.default_rng(seed)
    P = _physics()
    source = source or c["source"]
    h, (dx, dy) = 0.5 * c["field"], rng.uniform(-0.05, 0.05, 2)
    kw = dict(mono_energy=float(source[4:])) if source.startswith("mono") else dict(
        spectrum_file=os.path.join(P["data_folder"], source + ".spectrum"))
    ssd = 1e8 if source == "mono1.25" else 100.0
    return W.Job("(in memory)", P["pegs"], P["pgs4form"], P["data_folder"], P["data_folder"], ncase=histories,
                 nbatch=c["nbatch"], seeds=(int(rng.integers(1, 31328)), int(rng.integers(1, 30081))),
                 charge=c["charge"], collimator=(dx - h, dx + h, dy - h, dy + h), ssd=ssd, nsplit=c["nsplit"],
                 **kw).text()


def _problem(c, seed, histories, kind=None, source=None):
    ph = _phantom(c, seed, kind)
    phantom = api.Phantom.from_arrays(ph.media, ph.xb, ph.yb, ph.zb, ph.med, ph.rho)
    return api.Problem(api.Input(text=_job_text(c, seed, histories, source)), phantom=phantom)


def prepare(case, seed):
    c = dict(case)
    prec = api.FP32 if c["fp32"] else api.FP64
    s = {"case": c, "precision": prec}
    if c["call"] == "server":
        kinds = ("water", "slab", "ct")
        s["problems"] = [_problem(c, seed + 7919 * j, c["histories"] // c["jobs"], kinds[j % 3],
                                  ("6mv", "mono1.25")[j % 2]) for j in range(c["jobs"])]
        seeds = s["problems"][0].seeds
        s["server"] = api.Server(list(MEDIA), _job_text(c, seed, 1000), precision=prec, seeds=seeds)
        return s
    s["problem"] = p = _problem(c, seed, c["histories"])
    s["engine"] = e = api.Engine(0).load(p)
    if c["call"] == "dij":
        per = c["beamlets"] // 3
        side = int(math.ceil(math.sqrt(per)))
        zc = 0.5 * (p.phantom.s.nz * c["vox"])
        bl = W.beamlets(gantry_deg=(0.0, 51.43, 308.57), iso=(0.0, 0.0, zc), bixel=1.0, field=float(side))
        keep = np.concatenate([np.flatnonzero(bl.ibeam == b)[:per] for b in range(3)])
        e.set_beamlets(W.Beamlets(bl.ibeam[keep], bl.source, bl.corner[keep], bl.side1[keep], bl.side2[keep]))
        s["per_beamlet"] = c["histories"] // c["beamlets"]
    return s


def run(state):
    c = state["case"]
    if c["call"] == "server":
        srv = state["server"]
        ids = [srv.submit_problem(p) for p in state["problems"]]
        done = [srv.wait(i) for i in ids]
        return {"edep": [d[0] for d in done], "edep2": [d[1] for d in done]}
    eng, prob = state["engine"], state["problem"]
    if c["call"] == "dij":
        col, row, val, _ = eng.run_dij(rel_threshold=1e-4, nperbatch=state["per_beamlet"], nbatch=1,
                                       precision=state["precision"], fp32_values=True)
        # The matrix a planner multiplies with, dense: its sparsity pattern follows the noise.
        dij = np.zeros((c["beamlets"], prob.nreg - 1), np.float32)
        for b in range(c["beamlets"]):
            dij[b, row[col[b]:col[b + 1]]] = val[col[b]:col[b + 1]]
        return {"dij": dij}
    if c["call"] == "upload":
        eng.set_geometry(prob)
    a, a2, _ = eng.run(precision=state["precision"], inflight=c["inflight"],
                       history_stats=1 if c["call"] == "history" else 0)
    out = {"edep": a, "edep2": a2}
    if c["call"] == "history":
        out["sum"], out["sum2"], n, _ = eng.history_sums()
        out["histories"] = n
    return out


def work(case):
    """Bytes: the phantom's voxel records (medium and density) once and the
    results once.  Operations: per history, 12 per voxel crossing (about 7
    per cm of the phantom's depth in photons, one chord in electrons), 150 per
    photon interaction and 350 per electron step; the counts are those of a
    6 MV history in water (3 interactions, 45 steps in millimetre voxels,
    25 in centimetre voxels), scaled by the photon energy."""
    c = case
    nvox = c["nx"] * c["ny"] * c["nz"]
    per_voxel = 8 + 8 * 2
    if c["call"] == "history":
        per_voxel += 16
    if c["call"] == "dij":
        per_voxel = 8 + 4 * c["beamlets"]
    if c["call"] == "server":
        per_voxel *= c["jobs"]
    depth = c["nz"] * c["vox"]
    cross = 1.3 * depth / c["vox"]
    steps = 25 + 4 / c["vox"]
    if c["charge"]:
        steps, cross, inter = 3 * steps, 0.0, 1
    else:
        inter = {"6mv": 3, "mono1.25": 3, "250kvp": 6}[c["source"]]
        steps *= {"6mv": 1.0, "mono1.25": 0.45, "250kvp": 0.0}[c["source"]]
    flops = 12 * cross + 150 * inter + 350 * steps
    return {"bytes": float(nvox * per_voxel), "flops": float(c["histories"] * c["nsplit"] * flops)}


def exact(case, seed):
    return None
