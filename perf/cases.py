"""The engine's measured cases: dose runs through the public Python API over the
range of calls its users make, from a few hundred histories of a real-time loop
to the statistics of a finished plan.

A case is a dict of plain values:

  path        run       DoseEngine.reset, run, dose: one phantom, tallies of this call only
              noalloc   DoseEngine.run_noalloc into the caller's device array
              phantoms  DoseEngine.reset, run_phantoms, tallies: several phantoms at once
              adjoint   autograd.voxel_dose forward and backward
  phantom     water, slab (water/lung/bone/water), perturbed (water, densities
              1 +- 10%), ragged (water and bone, uneven planes), batched
              (workloads.batch_problem)
  edge, dx    voxels along an edge and their size in cm (uneven planes: the mean)
  beam        pencil, field (a 10 x 10 cm rectangle or what fits), spectrum
              (the field with a 0.1-6 MeV spectrum), phsp (a phase space of
              photons, electrons and positrons)
  charge, energy, ecut   source particle, its kinetic energy (MeV), electron cut-off (MeV, total)
  histories, batches     per call
  precision, bca, howfarless   engine options (egsgpu_config)
  phantoms    number of phantoms (path phantoms)

The state of another seed has other random numbers, and for the perturbed,
ragged and batched phantoms other densities or planes too.
"""
import numpy as np
import torch

import egsnrc_gb300 as eg
from egsnrc_gb300 import workloads as W
from egsnrc_gb300.autograd import voxel_dose

BASE = dict(path="run", phantom="water", edge=30, dx=1.0, beam="field", charge=0, energy=6.0, ecut=0.521,
            histories=100000, batches=10, precision=32, bca=0, howfarless=0, phantoms=1)


def listed():
    def case(name, **kw):
        return dict(BASE, name=name, **kw)
    return [
        # a real-time loop: a few hundred histories into a device array that the caller owns
        case("noalloc_slab64_512", path="noalloc", phantom="slab", edge=64, dx=0.25, beam="spectrum", ecut=0.7,
             histories=512, batches=1),
        # a quick look at a pencil beam, the configuration of water30 with 1/1000 of its histories
        case("water30_1e4", beam="pencil", energy=2.0, ecut=0.7, histories=10000),
        # water30 at a tenth of its histories: one depth dose
        case("water30_1e6", beam="pencil", energy=2.0, ecut=0.7, histories=1000000),
        # slab64 for a planning-grade estimate
        case("slab64_2e6", phantom="slab", edge=64, dx=0.25, beam="spectrum", ecut=0.7, histories=2000000),
        # slab64 at its full statistics, as the benchmark's default runs it (one batch)
        case("slab64_1e8", phantom="slab", edge=64, dx=0.25, beam="spectrum", ecut=0.7, histories=100000000, batches=1),
        # water128e: 20 MeV electrons in fine voxels, 10 batches
        case("water128e_2e5", edge=128, dx=0.2, charge=-1, energy=20.0, histories=200000),
        # perturbed64: heterogeneous densities under a 6 MeV photon field; a ragged history count
        case("perturbed64_777777", phantom="perturbed", edge=64, dx=0.3, histories=777777),
        # a linac phase space (photons, electrons, positrons) into uneven planes and two media,
        # with PRESTA-I boundary crossing as DOSXYZnrc users run it
        case("phsp_ragged_presta1_3e5", phantom="ragged", edge=41, dx=0.5, beam="phsp", energy=15.0, ecut=0.7,
             histories=300000, bca=1),
        # the HOWFARLESS option on a homogeneous water phantom
        case("howfarless128e_1e6", edge=128, dx=0.2, charge=-1, energy=20.0, histories=1000000, howfarless=1),
        # several independent small plans in one call
        case("phantoms12_3e5", path="phantoms", phantom="batched", edge=48, dx=0.2, ecut=0.7, histories=300000,
             phantoms=12),
        # the FP64 engine: precision reference runs
        case("slab64_fp64_2e5", phantom="slab", edge=64, dx=0.25, beam="spectrum", ecut=0.7, histories=200000,
             precision=64),
        # gradient of a dose objective with respect to the densities (forward, then the seed-replay adjoint)
        case("adjoint_perturbed32_1e5", path="adjoint", phantom="perturbed", edge=32, dx=0.6, histories=100000),
    ]


def steps_per_history(c):
    """Photon voxel crossings and charged-particle steps of one history, roughly."""
    size = c["edge"] * c["dx"]
    if c["phantom"] == "batched":
        size, e, half = 9.6, 9.5, True
    else:
        e, half = (1.7 if c["beam"] == "spectrum" else c["energy"]), False
    electrons = min(e, 2.0 * size) * (25.0 + (0 if c["howfarless"] else 8.0 / c["dx"]))
    photons = 2.5 * size / (size if c["howfarless"] else c["dx"])
    if c["charge"] != 0:
        return 0.3 * photons, electrons
    absorbed = min(1.0, 0.025 * size)
    return photons * (0.75 if half else 1.0), electrons * absorbed * (5.0 if half else 1.0)


def cost(c):
    """Relative cost of a pass, in FP32 photon crossings: the steps of all
    histories, and for each batch the longest track, whose steps follow one
    another."""
    p, e = steps_per_history(c)
    track = c["energy"] * (25.0 + 8.0 / c["dx"])
    n = c["histories"] * (p + 20.0 * e) + c["batches"] * track * 5e6
    return n * (10.0 if c["precision"] == 64 else 1.0) * (4.0 if c["path"] == "adjoint" else 1.0)


def draw(rng):
    def logint(a, b):
        return int(round(float(np.exp(rng.uniform(np.log(a), np.log(b))))))
    top = cost(listed()[4])
    while True:
        c = dict(BASE)
        c["path"] = rng.choice(["run"] * 8 + ["noalloc", "phantoms", "adjoint"])
        c["batches"] = rng.choice([1, 5, 10, 20])
        c["histories"] = logint(2000, 50000000)
        if c["path"] == "noalloc":
            c.update(histories=rng.randint(100, 2048), batches=1)
        elif c["path"] == "adjoint":
            c.update(histories=logint(20000, 200000), batches=10)
        if c["path"] == "phantoms":
            c.update(phantom="batched", ecut=0.7, edge=rng.randint(24, 64), dx=0.2, phantoms=rng.randint(4, 24),
                     histories=logint(100000, 1000000), batches=rng.choice([1, 5, 10]))
            return c
        c["phantom"] = "perturbed" if c["path"] == "adjoint" else rng.choice(["water", "slab", "perturbed", "ragged"])
        c["edge"] = rng.randint(15, 40) if c["path"] == "adjoint" else logint(12, 140)
        c["dx"] = round(rng.uniform(14.0, 30.0) / c["edge"], 3)
        c["beam"] = rng.choice(["pencil", "field", "spectrum", "phsp"] if c["path"] == "run" else ["field", "spectrum"])
        c["energy"] = round(rng.uniform(1.0, 18.0), 2)
        if c["beam"] in ("pencil", "field"):
            c["charge"] = rng.choice([0, 0, -1]) if c["path"] == "adjoint" else rng.choice([0, 0, 0, -1, -1, 1])
        elif c["beam"] == "spectrum":
            c["energy"] = 6.0
        c["ecut"] = rng.choice([0.521, 0.7])
        if c["path"] == "run":
            o = rng.random()
            if o < 0.12:
                c.update(precision=64, batches=rng.choice([1, 5]))
            elif o < 0.24:
                c["bca"] = 1
            elif o < 0.36 and c["phantom"] == "water":
                c["howfarless"] = 1
        if cost(c) < 0.5 * top:
            return c


def spectrum_source(half):
    return eg.ParallelBeam(charge=0, spectrum=W.bremsstrahlung_spectrum(), position=(0.0, 0.0, -1.0),
                           rectangle=(-half, half, -half, half))


def phase_space(c, rng, half):
    """Particles as a linac head's exit plane has them: mostly photons with a
    falling spectrum, a few electrons and positrons, slightly divergent."""
    n = 20000
    p = np.zeros((n, 7), dtype=np.float32)
    kind = rng.random(n)
    p[:, 0] = np.where(kind < 0.97, 0, np.where(kind < 0.992, -1, 1))
    p[:, 1] = np.clip(c["energy"] * rng.beta(1.0, 4.0, n), 0.05, c["energy"])
    p[:, 2:4] = rng.uniform(-half, half, (n, 2))
    p[:, 4:6] = p[:, 2:4] / 100.0 + rng.normal(0.0, 0.005, (n, 2))
    p[:, 6] = 1.0
    return eg.PhaseSpaceSource(p, position=(0.0, 0.0, -0.5))


def geometry(c, rng):
    n, dx = c["edge"], c["dx"]
    if c["phantom"] == "water":
        return [W.WATER], W.centred_geometry(n, dx)
    if c["phantom"] == "perturbed":
        return [W.WATER], W.centred_geometry(n, dx, 0, 1.0 + 0.1 * rng.uniform(-1.0, 1.0, n ** 3))
    size = n * dx
    if c["phantom"] == "slab":
        z = (np.arange(n) + 0.5) / n * 16.0
        medz = np.where(z < 3, 0, np.where(z < 9, 1, np.where(z < 11, 2, 0))).astype(np.int32)
        return [W.WATER, W.LUNG, W.BONE], W.centred_geometry(n, dx, np.broadcast_to(medz[:, None, None], (n, n, n)).ravel())
    # ragged: uneven planes (widths within a factor of about three), bone blocks in water
    def planes(lo):
        w = rng.uniform(0.5, 1.5, n)
        return lo + np.concatenate([[0.0], np.cumsum(w / w.sum() * size)])
    med = (rng.random((n, n, n)) < 0.2).astype(np.int32)
    return [W.WATER, W.BONE], eg.XYZGeometry(planes(-size / 2), planes(-size / 2), planes(0.0), med.ravel())


def source(c, rng):
    half = min(5.0, 0.4 * c["edge"] * c["dx"])
    if c["beam"] == "spectrum":
        return spectrum_source(half)
    if c["beam"] == "phsp":
        return phase_space(c, rng, half)
    rect = None if c["beam"] == "pencil" else (-half, half, -half, half)
    return eg.ParallelBeam(charge=c["charge"], energy=c["energy"], position=(0.0, 0.0, -1.0), rectangle=rect)


def prepare(case, seed):
    c = dict(BASE, **case)
    rng = np.random.default_rng(seed)
    st = dict(c=c, seed=1 + int(seed) % 2000000000)
    if c["path"] == "phantoms":
        eng = eg.DoseEngine(W.BATCH_MEDIA, ecut=c["ecut"], pcut=0.01)
        ks = 7 * (int(seed) % 100000) + np.arange(c["phantoms"])
        lo = max(16, c["edge"] // 2)      # edges from half of `edge` up to it, the same for every seed
        edges = [lo + (5 * j) % (c["edge"] - lo + 1) for j in range(c["phantoms"])]
        probs = [W.batch_problem(int(k), edge=(m, m), dx=c["dx"], hist=(1.0, 30.0)) for k, m in zip(ks, edges)]
        w = np.array([p["histories"] for p in probs], dtype=np.float64)
        for p, h in zip(probs, np.maximum(c["batches"], np.rint(w / w.sum() * c["histories"]))):
            p["histories"] = int(h)
        eng.set_phantoms(probs)
        st.update(eng=eng, probs=probs)
        return st
    media, geom = geometry(c, rng)
    src = source(c, rng)
    eng = eg.DoseEngine(media, ecut=c["ecut"], pcut=0.01, precision=c["precision"], bca_algorithm=c["bca"],
                        howfarless=c["howfarless"])
    eng.set_geometry(geom)
    eng.set_source(src)
    st.update(eng=eng, geom=geom, src=src)
    if c["path"] == "noalloc":
        st["dose"] = torch.zeros(geom.nvox, dtype=torch.float64, device="cuda")
    elif c["path"] == "adjoint":
        st["rhor"] = torch.tensor(geom.rhor, dtype=torch.float64, device="cuda")
    return st


def run(st):
    c, eng = st["c"], st["eng"]
    if c["path"] == "noalloc":
        eng.run_noalloc(st["dose"].data_ptr(), c["histories"], seed=st["seed"])
        return st["dose"]
    if c["path"] == "phantoms":
        eng.reset()
        eng.run_phantoms(nbatch=c["batches"])
        s, s2, _ = eng.tallies()
        return [s, s2]
    if c["path"] == "adjoint":
        rhor = st["rhor"].detach().requires_grad_()
        dose = voxel_dose(rhor, eng, st["geom"], c["histories"], seed=st["seed"], nbatch=c["batches"])
        scale = 1.0 / dose.detach().amax()
        (dose * scale).square().sum().backward()
        return [dose.detach(), rhor.grad]
    eng.reset()
    eng.run(c["histories"], nbatch=c["batches"], seed=st["seed"])
    dose, sigma = eng.dose()
    return [dose, sigma]


def work(case):
    """Each voxel's medium and density read once and its two results written
    once (the no-allocation entry point writes one); about 30 operations for
    a photon crossing and 300 for a charged-particle step, whose numbers the
    physics fixes."""
    c = dict(BASE, **case)
    vox = c["edge"] ** 3 * (0.5 * c["phantoms"] if c["path"] == "phantoms" else 1)
    p, e = steps_per_history(c)
    n = c["histories"] * (3 if c["path"] == "adjoint" else 1)
    return {"bytes": vox * (5 + (8 if c["path"] == "noalloc" else 16)), "flops": n * (30.0 * p + 300.0 * e)}


def exact(case, seed):
    """None: a Monte Carlo result is its own random walk; there is no closed form of it."""
    return None
