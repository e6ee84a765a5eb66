"""Workloads that the performance of this library is measured on.

Every case is one call that a program makes through the Python binding: a
transport run into device tallies, the same into host buffers with a new
activity map, a list-mode (PSF) run, a dose run, the gradient of the
log-likelihood, several phantoms in one batch, and a batch captured in a CUDA
graph.  The phantoms and scanners are those of mcpet.inputs (water cube,
head, body; 15 to 256 rings) at the sizes that the tests and the benchmark
use and at ragged ones between them, from 2e4 to 1e9 decays, with the lanes
of the reference program (replayable, the default) and balanced ones.

The material tables are written here, once per process, from textbook
models (Klein-Nishina, power laws fitted to the published attenuation of
water and air, hydrogen-like form factors and Compton profiles) in the
format and on the energy grid of the tables that users have: 50 eV steps from
5 keV, water with 3 Compton shells and air with 9.
"""
from __future__ import annotations

import atexit
import math
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcgpu-pet_b200"))

import mcpet  # noqa: E402
from mcpet import grad as mcpet_grad  # noqa: E402
from mcpet import inputs  # noqa: E402

# --------------------------------------------------------------- materials

# electrons, ionisation energy (eV), Compton profile at p = 0 (atomic units)
SHELLS = {
    "water": [(6.0, 12.6, 0.55), (2.0, 28.5, 0.66), (2.0, 538.0, 0.115)],
    "air": [(3.12, 13.0, 0.52), (1.56, 24.5, 0.74), (1.56, 401.6, 0.132), (0.84, 13.6, 0.50), (0.42, 28.5, 0.66),
            (0.42, 538.0, 0.115), (0.05, 15.9, 0.45), (0.02, 285.0, 0.16), (0.01, 3203.0, 0.05)],
}
# nominal density (g/cm3), electrons per gram / 1e23
BULK = {"water": (1.0, 3.343), "air": (0.00120479, 3.006)}
INV_FINE_STRUCTURE = 137.035999


def _compton_per_electron(e):
    """Klein-Nishina total cross section (cm2)."""
    k = e / 510998.95
    l2 = np.log1p(2 * k)
    return 2 * math.pi * 7.9407877e-26 * ((1 + k) / k ** 2 * (2 * (1 + k) / (1 + 2 * k) - l2 / k) + l2 / (2 * k)
                                          - (1 + 3 * k) / (1 + 2 * k) ** 2)


def _write_material(path, name, e_max):
    rho, n_e = BULK[name]
    e = np.arange(5.0e3, e_max, 50.0)
    x = e / 1.0e5
    mu_c = n_e * 1e23 * _compton_per_electron(e)
    mu_p = 2.76e-3 * x ** -3.1 * (1.0 if name == "water" else 0.93)
    mu_r = 5.0e-3 / (x * x + 0.006)
    # squared form factor (1 + x2/b2)^-4 of x2 = (sin(theta/2)/lambda)^2 in 1/A^2, and its cumulative
    b2 = 0.55 ** 2
    xs = np.concatenate([[0.0], np.geomspace(1.0e-4, 1.1 * (e_max * 8.0655e-5) ** 2, 127)])
    cum = lambda t: 1.0 - (1.0 + t / b2) ** -3  # noqa: E731
    c = cum(xs) / cum(xs[-1])
    pdf = 3.0 / b2 * (1.0 + xs / b2) ** -4 / cum(xs[-1])
    slope = np.diff(c) / np.diff(xs)
    b = np.append(1.0 - slope ** 2 / (pdf[:-1] * pdf[1:]), 0.0)
    a = np.append(slope / pdf[:-1] - b[:-1] - 1.0, 0.0)
    lo = np.clip(np.searchsorted(c, np.arange(128) / 127.0, side="right"), 1, 127)
    hi = np.clip(np.searchsorted(c, np.arange(1, 129) / 127.0, side="left") + 1, lo + 1, 128)
    pmax = cum((e * 8.065535669e-5) ** 2) / cum(xs[-1])
    with open(path, "w") as f:
        f.write("#[MATERIAL DEFINITION]\n#[NOMINAL DENSITY (g/cm^3)]\n# %.8f\n#[NUMBER OF DATA VALUES]\n# %d\n"
                "#[MEAN FREE PATHS (cm)]\n#[Energy (eV) | Rayleigh | Compton | Photoelectric | TOTAL | "
                "Rayleigh: max cumul prob F^2]\n" % (rho, len(e)))
        np.savetxt(f, np.stack([e, 1 / (mu_r * rho), 1 / (mu_c * rho), 1 / (mu_p * rho),
                                1 / ((mu_r + mu_c + mu_p) * rho), pmax], 1), fmt="  %.10E")
        f.write("#[RAYLEIGH INTERACTIONS (RITA sampling of atomic form factor)]\n#[DATA VALUES TO SAMPLE SQUARED "
                "MOLECULAR FORM FACTOR (F^2)]\n# 128\n#[SAMPLING DATA: X, P, A, B, ITL, ITU]\n")
        for i in range(128):
            f.write("  %.10E  %.10E  %.10E  %.10E  %d  %d\n" % (xs[i], c[i], a[i], b[i], lo[i], hi[i]))
        f.write("#[COMPTON INTERACTIONS (relativistic impulse model with approximated one-electron analytical "
                "profiles)]\n#[NUMBER OF SHELLS]\n# %d\n#[SHELL INFORMATION: FCO, UICO, FJ0, KZCO, KSCO]\n"
                % len(SHELLS[name]))
        for n, u, j0 in SHELLS[name]:
            f.write("  %.8E  %.8E  %.8E  8  30\n" % (n, u, j0 * INV_FINE_STRUCTURE))


_work = None


def _workdir():
    global _work
    if _work is None:
        _work = tempfile.mkdtemp(prefix="mcpet_cases_")
        atexit.register(shutil.rmtree, _work, True)
    return _work


def _materials(extended):
    """Material files of the ten tissue slots: air, then water."""
    top = 1.25e6 if extended else 5.15e5
    paths = []
    for name in ("air", "water"):
        p = os.path.join(_workdir(), "%s_%d" % (name, extended))
        if not os.path.exists(p):
            _write_material(p, name, top)
        paths.append(p)
    return [paths[0]] + [paths[1]] * 9


# ------------------------------------------------------------------- cases

SMALL = dict(phantom="cube", nx=9, ny=9, nz=9, voxel_cm=1.0, rings=15, radial=147, angles=168, mrd=14, span=1)
HEAD = dict(phantom="head", nx=128, ny=128, nz=64, voxel_cm=0.2, rings=64, radial=256, angles=256, mrd=63, span=1)
HEAD32 = dict(HEAD, rings=32, radial=128, mrd=31)
BATCH = dict(phantom="head", nx=112, ny=112, nz=112, voxel_cm=0.3, rings=32, radial=128, angles=128, mrd=31, span=1)
BODY = dict(phantom="body", nx=128, ny=128, nz=200, voxel_cm=0.4, rings=256, radial=192, angles=384, mrd=38, span=11)


def listed():
    return [
        # the smallest call: a check run of the sample geometry, as one makes after installing, default options
        dict(SMALL, name="cube_2e4", call="device", lanes="reference", decays=2.0e4),
        # the sample simulation at its stated size, replayable lanes: three hot voxels among 729
        dict(SMALL, name="cube_1e7", call="device", lanes="reference", decays=1.0e7),
        # list-mode output: PSF and sinogram of the sample geometry, records put in time order
        dict(SMALL, name="cube_psf_1e6", call="psf", lanes="reference", decays=1.0e6),
        # a short frame of a small ragged head
        dict(phantom="head", nx=61, ny=47, nz=37, voxel_cm=0.41, rings=32, radial=101, angles=128, mrd=31, span=1,
             name="head_frame_1e6", call="device", lanes="balanced", decays=1.0e6),
        # the head phantom in replayable lanes on the 32-ring scanner
        dict(HEAD32, name="head32_reference_1e8", call="device", lanes="reference", decays=1.0e8),
        # the head workload at full size: 1e9 decays into 5.3e8-bin sinograms
        dict(HEAD, name="head_1e9", call="device", lanes="balanced", decays=1.0e9),
        # one iteration of a reconstruction: new activity from the host, tallies back to pinned host buffers
        dict(HEAD32, name="head32_host_1e7", call="host", lanes="balanced", decays=1.0e7, angles=128),
        # forward and backward: log-likelihood with its gradient in activity and density
        dict(HEAD, name="head_gradient_5e7", call="grad", lanes="balanced", decays=5.0e7),
        # material and voxel dose beside the sinogram, a decaying source
        dict(HEAD32, name="head32_dose_2e7", call="dose", lanes="balanced", decays=2.0e7),
        # six phantoms of uneven size in one batch, every second one with a 1157 keV prompt gamma
        dict(BATCH, name="batch_6x3e6", call="batch", lanes="balanced", decays=3.0e6, scenes=6),
        # small phantoms regenerated by replays of a captured graph
        dict(BATCH, nx=45, ny=45, nz=45, voxel_cm=0.35, radial=64, angles=64, name="graph_8x2e5", call="graph",
             lanes="balanced", decays=2.0e5, scenes=8),
        # two bed positions of a body on the long-axial scanner, one phantom in one batch
        dict(BODY, name="beds_2x5e7", call="beds", lanes="balanced", decays=5.0e7, scenes=2),
    ]


def draw(rng):
    """Another case of the same kinds: sizes over their whole range, odd ones
    among them; at most a fifth of the largest listed case's decays."""
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    call = rng.choice(["device", "device", "device", "host", "psf", "dose", "grad", "batch", "graph", "beds"])
    c = dict(call=call, lanes=rng.choice(["balanced", "balanced", "reference"]), span=1)
    n = int(log(30, 150))
    if call == "psf" or (call == "device" and rng.random() < 0.3):
        c.update(SMALL, decays=float(int(log(2e4, 5e6))))
    elif call == "beds":
        c.update(BODY, nx=rng.randint(60, 128), ny=rng.randint(60, 128), nz=rng.randint(90, 200), scenes=rng.randint(1, 3),
                 radial=rng.randint(60, 192), decays=float(int(log(2e6, 5e7))))
    else:
        rings = rng.choice([16, 23, 32, 48, 64])
        angles = rng.choice([64, 96, 128, 256])
        c.update(phantom="head", nx=n, ny=max(24, int(n * rng.uniform(0.7, 1.1))),
                 nz=max(20, int(n * rng.uniform(0.4, 1.1))), voxel_cm=round(min(rng.uniform(0.2, 0.4), 28.0 / n), 3),
                 rings=rings, radial=rng.randint(50, angles), angles=angles, mrd=rng.randint(rings // 2, rings - 1),
                 decays=float(int(log(1e5, 2e8 if call == "device" else 3e7))))
    if call in ("batch", "graph"):
        c.update(scenes=rng.randint(2, 8), decays=float(int(log(5e4, 3e6))))
    return c


def _phantom(c, k, rng_seed):
    """(material, density, activity, voxel size) of the case's k-th phantom."""
    shape = (c["nz"], c["ny"], c["nx"])
    if c["phantom"] == "cube":
        mat, rho, act, vs = inputs.water_cube_phantom(c["decays"])
        r = np.random.default_rng(rng_seed)
        act = act * r.uniform(0.8, 1.2, act.shape)
        return mat, rho, (act * (c["decays"] / act.sum())).astype(np.float32), vs
    if c["phantom"] == "body":
        return inputs.body_phantom(shape, c["voxel_cm"], seed=rng_seed, total_bq=c["decays"])[:4]
    if c["call"] in ("batch", "graph") and k:   # uneven sizes: from a quarter of the case's to all of it
        f = (1.0, 0.55, 0.8, 0.35, 0.7, 0.25, 0.9, 0.45)[k % 8]
        shape = tuple(max(16, int(s * f)) for s in shape)
    return inputs.head_phantom(shape, c["voxel_cm"], seed=rng_seed, total_bq=c["decays"])[:4]


def _scene(c, k, seed, phantom, **more):
    mat, rho, act, vs = phantom
    prompt = c["call"] == "batch" and k % 2 == 1
    kw = dict(seed=1 + (seed * 7919 + k * 104729) % 2147480000, n_rows=c["rings"], n_crystals=2 * c["angles"],
              n_angles=c["angles"], n_radial=c["radial"], n_z_slices=2 * c["rings"] - 1, max_ring_difference=c["mrd"],
              span=c["span"])
    if c["phantom"] == "cube":
        kw.update(detector_radius=-40.0, detector_height=20.0, fov_z=20.0)
    else:
        kw.update(detector_radius=-39.0 if c["phantom"] == "body" else -41.0, detector_height=0.4 * c["rings"],
                  fov_z=0.4 * c["rings"])
    if prompt:
        kw.update(prompt_gamma_energy=1157020.0, prompt_gamma_yield=1.0)
    kw.update(more)
    spec = inputs.spec_for(_materials(c["call"] == "batch"), "unused.vox", **kw)
    sc = mcpet.Scene.from_arrays(inputs.config_from_spec(spec, _workdir()), mat, rho, act, vs)
    sc.to_device()
    return sc


KEYS = ("trues", "scatter", "image_trues", "image_scatter", "spectrum")


def prepare(case, seed):
    c, call = dict(case), case["call"]
    lanes = mcpet.LANES_REFERENCE if c["lanes"] == "reference" else mcpet.LANES_BALANCED
    s = {"call": call, "opts": mcpet.RunOptions(lane_mode=lanes)}
    base = seed % 1000003
    if call in ("batch", "graph", "beds"):
        if call == "beds":
            ph = _phantom(c, 0, base)
            size = [n * c["voxel_cm"] for n in (c["nx"], c["ny"], c["nz"])]
            centers = inputs.bed_centers(size, c["scenes"], 20.0)
            s["scenes"] = [_scene(c, k, seed, ph, detector_center=centers[k], detector_radius=39.0)
                           for k in range(c["scenes"])]
        else:
            s["scenes"] = [_scene(c, k, seed, _phantom(c, k, base + k)) for k in range(c["scenes"])]
        s["tallies"] = [mcpet.device_tallies_for(x) for x in s["scenes"]]
        if call == "graph":
            s["graph"] = mcpet.BatchGraph(s["scenes"], s["tallies"], s["opts"])
        return s
    more = {}
    if call == "psf":
        more = dict(tally_psf_sinogram=0, psf_size=2 * int(0.25 * c["decays"] + 1000))
    if call == "dose":
        more = dict(material_dose=True, voxel_dose=True, mean_life_s=9.5e3,
                    dose_roi=(1, c["nx"], 1, c["ny"], 1, c["nz"]))
    ph = _phantom(c, 0, base)
    sc = s["scene"] = _scene(c, 0, seed, ph, **more)
    if call == "host":
        s["activity"] = ph[2]
        cfg, info = sc.config, sc.info
        sizes = (cfg.n_bins, cfg.n_bins, info.n_voxels, info.n_voxels, cfg.n_energy_bins)
        s["host"] = {k: torch.empty(int(n), dtype=torch.int32, pin_memory=True) for k, n in zip(KEYS, sizes)}
        return s
    t = s["tallies"] = mcpet.device_tallies_for(sc, psf_capacity=more.get("psf_size", 0))
    if call == "psf":
        t["psf"].zero_()
    if call == "dose":
        t["material_dose"] = torch.zeros(mcpet.MAX_MATERIALS * 2, dtype=torch.int64, device="cuda")
        t["voxel_dose"] = torch.zeros(int(sc.info.n_dose_voxels) * 2, dtype=torch.int64, device="cuda")
    if call == "grad":
        # a measurement: about one detected pair per 17 decays, spread like a smooth object over the sinogram
        nb = int(sc.config.n_bins)
        g = torch.Generator(device="cuda").manual_seed(seed)
        mean = c["decays"] / 17.0 / nb
        s["measured"] = torch.poisson(torch.full((nb,), mean, device="cuda"), generator=g)
        s["background"] = torch.full((nb,), 0.05 * mean, device="cuda")
    return s


def _tallies(t):
    return {k: t[k] for k in KEYS + ("material_dose", "voxel_dose") if k in t}


def run(s):
    call, opts = s["call"], s["opts"]
    if call == "host":
        s["scene"].set_activity(s["activity"])
        r = s["scene"].run_into(s["host"], opts)
        return [s["host"][k] for k in KEYS] + [r["coincidences"], r["total_histories"]]
    if call == "grad":
        r = mcpet_grad.grad(s["scene"], s["measured"], s["background"], opts, tallies=s["tallies"])
        return [r.grad_activity, r.grad_density_scale, r.loglik, _tallies(s["tallies"])]
    if call in ("batch", "beds"):
        mcpet.Scene.run_batch_device(s["scenes"], s["tallies"], opts)
        return [_tallies(t) for t in s["tallies"]]
    if call == "graph":
        s["graph"].launch()
        return [_tallies(t) for t in s["tallies"]]
    s["scene"].run_device(s["tallies"], opts)
    out = _tallies(s["tallies"])
    if call == "psf":
        # records by time of emission (words 0, 1), pairs of one time by voxel (word 3); unused ones are zero and first
        w = s["tallies"]["psf"].view(torch.int32).view(-1, 22)
        by_voxel = torch.argsort(w[:, 3], stable=True)
        time = (w[:, 1].long() << 32) | (w[:, 0].long() & 0xFFFFFFFF)
        out["psf"] = w[by_voxel][torch.argsort(time[by_voxel], stable=True)]
    return out


def work(case):
    c = case
    n_scenes = c.get("scenes", 1)
    # sinogram planes: 2 rings - 1 - 2 |d| of each ring difference d, about 1/span of them with a span
    planes = sum(2 * c["rings"] - 1 - 2 * abs(d) for d in range(-c["mrd"], c["mrd"] + 1)) // c["span"]
    bins = planes * c["radial"] * c["angles"]
    voxels = c["nx"] * c["ny"] * c["nz"]
    out = n_scenes * 4 * (2 * bins + 2 * voxels + 700)
    if c["call"] == "grad":
        out += 8 * bins + 8 * voxels         # measured and background read, both gradients written
    if c["call"] == "dose":
        out += 16 * voxels
    if c["call"] == "psf":
        out += 88 * int(0.04 * c["decays"])
    # 32-bit operations of a decay: pair emission, decay time and detector about 460, 50 for each Woodcock step, 360
    # for each Compton scattering (5.1 and 2.4 of them in the head, 1.9 and 0.7 in the 9 cm cube)
    ops = {"cube": 810, "head": 1570, "body": 1570}[c["phantom"]]
    return {"bytes": out + n_scenes * 6 * voxels, "flops": n_scenes * c["decays"] * ops}


def tolerance(case):
    """Counts and doses are whole numbers that follow from the seed alone:
    any schedule of the lanes gives the same ones.  (Other rounding does not:
    a build without multiply-add contraction moves up to three quarters of
    the voxel counts of the 1e9-decay head, as every later history of a lane
    changes with the first that draws another number.)  The gradients are
    32-bit sums in no fixed order."""
    return {"rel": 1e-5, "differ": 0.0} if case["call"] == "grad" else "exact"


def exact(case, seed):
    """None: a history has no value in 64 bits to be compared with, it parts
    from this one at the first decision that rounds the other way.  The
    statistical comparison is in the test suite."""
    return None
