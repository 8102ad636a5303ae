"""What the framework's speed is measured on: photon simulations as its users run them.

Every case goes through a public entry point -- ``run``, ``run_batch``, ``diff.ReplayGradient``,
``diff.FluenceGradient`` -- with the host arrays that a program has in hand, and counts from that call to its
host outputs.  Workloads are the built-in benchmarks (60^3 cube, cube with a sphere, planar source), the layered
head, per-voxel absorption maps, replays, modulated sources and batches, from a first look of ten thousand
photons to 1e8.  The optical properties and the random seed differ from input to input, as in a fit or a sweep.

Detected photons are recorded in the order in which they arrive at a shared counter, which is not the same twice;
``run`` puts them into the order of their contents, so that two calls can be compared.
"""
import math

import numpy as np

import mcxcl_gb300
from mcxcl_gb300 import diff

C0 = 299.792458  # mm per ns


# ------------------------------------------------------------------------------------------------ the cases

def case(name, kind, volume, photons, **kw):
    """kind: which entry point; volume: what is simulated; the rest in plain values."""
    edge = kw.pop("edge", 60)
    c = dict(name=name, kind=kind, volume=volume, photons=int(photons), nx=edge, ny=edge, nz=edge, gates=1, reflect=1,
             detectors=0, source="pencil", output="flux", roulette=0.0, unit=1.0, omega=0.0, sims=1)
    c.update(kw)
    return c


def listed():
    return [
        # a first look while a setup is written: the smallest call, all latency and launches
        case("cube_1e4", "run", "cube", 1e4, reflect=0),
        # the built-in cube benchmark as shipped: four detectors, no reflection, 1e6 photons
        case("cube_1e6", "run", "cube", 1e6, reflect=0, detectors=4),
        # the same cube for a noise-free field: 1e8 photons, the largest call
        case("cube_1e8", "run", "cube", 1e8, reflect=0),
        # the cube with a scattering sphere: Fresnel, 50 time gates, detectors with partial paths and seeds
        case("sphere_1e6", "run", "sphere", 1e6, gates=50, detectors=4),
        case("sphere_2e7", "run", "sphere", 2e7, gates=50, detectors=4),
        # a layered head: 7.1 M voxels, five tissues, 10 gates, 16 detectors, roulette
        case("head_1e7", "run", "head", 1e7, nx=181, ny=217, nz=181, gates=10, reflect=0, detectors=16,
             roulette=1e-4),
        # wide-field illumination from above the tissue: photons enter through void, ragged volume, deposited energy
        case("planar_3e6", "run", "layers", 3e6, nx=75, ny=61, nz=43, source="planar", output="energy"),
        # a 100 MHz modulated source: complex field
        case("modulated_1e6", "run", "sphere", 1e6, omega=2 * math.pi * 1e8),
        # the sensitivity of each detector: a forward run's detected photons replayed
        case("replay_2e6", "replay", "sphere", 2e6, gates=10, detectors=4, output="jacobian"),
        # a fit of a per-voxel absorption map: detector readings and their gradient
        case("readings_1e6", "readings", "map", 1e6, edge=100, detectors=16),
        # a loss of the fluence field, its gradient per voxel in absorption and scattering
        case("fluence_1e6", "fluence", "sphere", 1e6, gates=5),
        # a training set's simulations in one call: cubes of many sizes, one after another
        case("batch_24", "batch", "cubes", 3e5, sims=24, edge=96),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run"] * 6 + ["replay", "readings", "fluence", "batch"])
    c = case("", kind, "cube", log(1e4, 1e7))
    del c["name"]
    c.update(nx=log(24, 128), ny=log(24, 128), nz=log(24, 128), unit=rng.choice([1.0, 1.0, 0.5]))
    if kind == "run":
        c.update(volume=rng.choice(["cube", "sphere", "layers", "map"]), gates=rng.choice([1, 1, 5, 10, 37, 50]),
                 reflect=rng.choice([0, 1, 1]), detectors=rng.choice([0, 1, 4, 16]),
                 source=rng.choice(["pencil", "pencil", "planar", "disk", "gaussian", "isotropic"]),
                 output=rng.choice(["flux", "flux", "fluence", "energy"]), roulette=rng.choice([0.0, 0.0, 1e-4, 1e-3]))
        if c["detectors"] == 16:
            c.update(photons=min(c["photons"], 4000000))  # all detected photons fit the record buffer
        if c["volume"] == "sphere" and rng.random() < 0.25:
            c.update(omega=2 * math.pi * 1e6 * rng.uniform(50, 500), photons=log(1e4, 3e6), detectors=0, output="flux",
                     roulette=0.0)
    elif kind == "replay":
        c.update(volume="sphere", photons=log(1e5, 1e7), gates=rng.choice([1, 10, 20]), detectors=rng.choice([1, 4]),
                 output=rng.choice(["jacobian", "jacobian", "wltof", "nscat"]))
    elif kind == "readings":
        c.update(volume="map", photons=log(1e5, 3e6), detectors=rng.choice([4, 16]))
    elif kind == "fluence":
        c.update(volume=rng.choice(["sphere", "map"]), photons=log(1e4, 3e6), gates=rng.choice([1, 5]))
    else:
        c.update(volume="cubes", photons=log(3e4, 3e5), sims=rng.randint(3, 40))
    return c


# ----------------------------------------------------------------------------------------------- the inputs

def grid(c):
    return np.ogrid[0:c["nx"], 0:c["ny"], 0:c["nz"]]


def ball(c, centre, radius):
    x, y, z = grid(c)
    return (x + 0.5 - centre[0]) ** 2 + (y + 0.5 - centre[1]) ** 2 + (z + 0.5 - centre[2]) ** 2 < radius * radius


def head(c):
    """Five nested ellipsoids, label k + 1 inside the k-th."""
    x, y, z = grid(c)
    shape = (c["nx"], c["ny"], c["nz"])
    vol = np.zeros(shape, np.uint8)
    mid = [np.float32((s - 1) / 2) for s in shape]
    for label, (a, b, h) in enumerate(((88, 106, 88), (84, 102, 84), (79, 97, 79), (77, 95, 77), (60, 75, 60)), 1):
        f = np.float32
        vol[((x - mid[0]) / f(a)) ** 2 + ((y - mid[1]) / f(b)) ** 2 + ((z - mid[2]) / f(h)) ** 2 <= 1] = label
    return vol


def smooth(shape, corr, rng):
    """A Gaussian random field of unit variance."""
    white = rng.standard_normal(shape).astype(np.float32)
    k2 = sum(np.meshgrid(*[np.fft.fftfreq(n) ** 2 for n in shape[:2]], np.fft.rfftfreq(shape[2]) ** 2, indexing="ij"))
    z = np.fft.irfftn(np.fft.rfftn(white) * np.exp(-2 * np.pi ** 2 * corr ** 2 * k2), s=shape)
    return (z - z.mean()) / z.std()


#: mua and mus (1/mm), g and n of each medium; row 0 is what is outside
MEDIA = {
    "cube": [[0, 0, 1, 1], [0.005, 1.0, 0.01, 1.37]],
    "sphere": [[0, 0, 1, 1], [0.005, 1.0, 0.01, 1.37], [0.002, 5.0, 0.9, 1.0]],
    "layers": [[0, 0, 1, 1], [0.02, 9.0, 0.89, 1.37], [0.004, 0.1, 0.89, 1.37], [0.05, 10.0, 0.9, 1.37]],
    "head": [[0, 0, 1, 1], [0.019, 7.8, 0.89, 1.37], [0.019, 7.8, 0.89, 1.37], [0.004, 0.009, 0.89, 1.37],
             [0.02, 9.0, 0.89, 1.37], [0.08, 40.9, 0.84, 1.37]],
    "map": [[0, 0, 1, 1], [0.01, 1.0, 0.9, 1.37]],
}


def medium(volume, rng):
    """The media with absorption and scattering a few per cent from their nominal values."""
    prop = np.array(MEDIA[volume], np.float64)
    prop[1:, :2] *= rng.uniform(0.95, 1.05, prop[1:, :2].shape)
    return prop.tolist()


def setup(c, rng):
    """The dictionary of one simulation."""
    nx, ny, nz, volume = c["nx"], c["ny"], c["nz"], c["volume"]
    cx, cy, top = nx // 2, ny // 2, 0
    cfg = dict(nphoton=c["photons"], prop=medium(volume, rng), tstart=0, tend=5e-9, tstep=5e-9 / c["gates"],
               seed=int(rng.integers(1, 2 ** 31 - 1)), isreflect=c["reflect"], outputtype=c["output"], issrcfrom0=1,
               unitinmm=c["unit"], srcdir=[0, 0, 1], issavedet=0)
    if volume == "cube":
        vol = np.ones((nx, ny, nz), np.uint8)
    elif volume == "sphere":
        vol = np.where(ball(c, (nx / 2 + rng.uniform(-1, 1), ny / 2 + rng.uniform(-1, 1), nz / 2), min(nx, ny, nz) / 4),
                       2, 1).astype(np.uint8)
    elif volume == "layers":
        vol = np.broadcast_to(np.searchsorted([0.15, 0.3], (np.arange(nz) + 0.5) / nz)[None, None] + 1,
                              (nx, ny, nz)).astype(np.uint8)
    elif volume == "head":
        vol = head(c)
        top = int(np.argmax(vol[cx, cy] > 0))
    else:
        vol = np.maximum(0.01 * (1 + 0.2 * smooth((nx, ny, nz), 5.0, rng)), 1e-4).astype(np.float32)[None]
    cfg["vol"] = vol
    cfg["srcpos"] = [cx, cy, top]
    if c["source"] == "planar":
        cfg.update(srctype="planar", srcpos=[nx / 6, ny / 6, -10], srcparam1=[nx / 1.5, 0, 0, 0],
                   srcparam2=[0, ny / 1.5, 0, 0])
    elif c["source"] in ("disk", "gaussian"):
        cfg.update(srctype=c["source"], srcparam1=[min(nx, ny) / 8, 0, 0, 0])
    elif c["source"] == "isotropic":
        cfg.update(srctype="isotropic", srcpos=[cx + 0.5, cy + 0.5, nz / 3])
    if c["detectors"]:
        ring, size = (30, 2) if volume == "head" else (min(10, nx // 3, ny // 3), 1)
        dets = []
        for k in range(c["detectors"]):
            ang = 2 * math.pi * k / c["detectors"]
            x, y = int(round(cx + ring * math.cos(ang))), int(round(cy + ring * math.sin(ang)))
            dets.append([x, y, int(np.argmax(vol[x, y] > 0)) if volume == "head" else 0, size])
        cfg.update(detpos=dets, issavedet=1, savedetflag="dsp" if volume != "map" else "dxv", issaveseed=1)
    if c["roulette"]:
        cfg["minenergy"] = c["roulette"]
    if c["omega"]:
        cfg["omega"] = c["omega"]
    return cfg


def cubes(c, rng):
    """The simulations of a batch: independent cubes of many sizes, media and photon counts, half of them with a ball."""
    got = []
    for n in np.random.default_rng([c["sims"], c["nx"]]).integers(32, max(33, c["nx"]) + 1, c["sims"]).tolist():
        d = dict(nx=n, ny=n, nz=n)

        def one():
            return [float(np.exp(rng.uniform(np.log(1e-3), np.log(1e-1)))), float(rng.uniform(0.5, 2)),
                    float(rng.uniform(0.6, 0.95)), float(rng.uniform(1.33, 1.45))]

        vol, prop = np.ones((n, n, n), np.uint8), [[0, 0, 1, 1], one()]
        if rng.random() < 0.5:
            r = rng.uniform(0.1, 0.3) * n
            vol[ball(d, rng.uniform(r, n - r, 3), r)] = 2
            prop.append(one())
        got.append(dict(nphoton=int(np.exp(rng.uniform(np.log(c["photons"] / 10), np.log(c["photons"])))), vol=vol,
                        prop=prop, tstart=0, tend=5e-9, tstep=5e-9, srcpos=[n / 2, n / 2, 0], srcdir=[0, 0, 1],
                        issrcfrom0=1, isreflect=1, issavedet=0, seed=int(rng.integers(1, 2 ** 31 - 1))))
    return got


def in_order(seeds):
    """Where each detected photon belongs by its launch state."""
    s = np.ascontiguousarray(seeds.T).view(np.uint64)
    return np.argsort(s[:, 0], kind="stable")


def table(records, rows):
    """Records by column in a table of a fixed number of rows: how many photons are detected is a matter of chance."""
    t = np.zeros((rows, records.shape[0]), records.dtype)
    n = min(rows, records.shape[1])
    t[:n] = records.T[:n]
    return t


def prepare(c, seed):
    rng = np.random.default_rng([20240607, int(seed)])
    if c["kind"] == "batch":
        return dict(kind="batch", cfgs=cubes(c, rng))
    cfg = setup(c, rng)
    if c["kind"] == "run":
        return dict(kind="run", cfg=cfg, rows=c["photons"] // 800 * c["detectors"],
                    width=7 if c["volume"] == "map" else 1 + 2 * (len(cfg["prop"]) - 1))
    if c["kind"] == "replay":
        # the forward run whose detected photons are asked about
        first = mcxcl_gb300.run(dict(cfg, outputtype="flux"))
        seeds, detp = first.get("seeds", np.zeros((16, 0), np.uint8)), first.get("detp", np.zeros((1, 0), np.float32))
        order = in_order(seeds)
        cfg.pop("nphoton")
        cfg.update(seed=np.asfortranarray(seeds[:, order]), detphotons=np.asfortranarray(detp[:, order]), replaydet=-1,
                   issaveseed=0, issavedet=1)
        return dict(kind="run", cfg=cfg, rows=0)
    if c["kind"] == "readings":
        mua = cfg.pop("vol")[0]
        for k in ("issavedet", "savedetflag", "issaveseed", "outputtype"):
            cfg.pop(k, None)
        return dict(kind="readings", sim=diff.ReplayGradient(cfg), mua=mua, pull=rng.standard_normal(c["detectors"]))
    shape = (c["nx"], c["ny"], c["nz"], c["gates"])
    return dict(kind="fluence", sim=diff.FluenceGradient(cfg), pull=rng.standard_normal(shape))


def run(state):
    kind = state["kind"]
    if kind == "batch":
        got = mcxcl_gb300.run_batch(state["cfgs"])
        return [r["flux"] for r in got] + [np.array([[r["stat"]["energytot"], r["stat"]["energyabs"]] for r in got])]
    if kind == "readings":
        values = state["sim"].forward(state["mua"])
        return [values, state["sim"].backward(state["pull"])]
    if kind == "fluence":
        field = state["sim"].forward()
        return [field, *state["sim"].backward(state["pull"])]
    r = mcxcl_gb300.run(state["cfg"])
    out = [r["flux"], r["stat"]["energytot"], r["stat"]["energyabs"], int(r["stat"]["detected"])]
    if state["rows"]:
        seeds = r.get("seeds", np.zeros((16, 0), np.uint8))
        detp = r.get("detp", np.zeros((state["width"], 0), np.float32))
        order = in_order(seeds)[:state["rows"]]
        out += [table(seeds[:, order], state["rows"]), table(detp[:, order], state["rows"])]
    return out


# ------------------------------------------------------------------------------------------------- the work

#: steps to a voxel face or a scattering site, and scatterings, of a mean photon
#: (cube, sphere, head: counted by the verification kernel; the others estimated), taken for all sizes
PATH = {"cube": (196, 78), "sphere": (344, 156), "layers": (330, 250), "head": (527, 443), "map": (300, 120),
        "cubes": (250, 100)}


def work(c):
    """Each input read and each output written once; 48 operations a step to the next face or scattering site, 65 a
    scattering, 20 a launch (the least arithmetic of the method; its random numbers, tests and table reads not counted)."""
    steps, scatterings = PATH[c["volume"]]
    voxels = c["nx"] * c["ny"] * c["nz"]
    photons, label = c["photons"], 4 if c["volume"] == "map" else 1
    fields = c["gates"] * (2 if c["omega"] else 1)
    if c["kind"] == "batch":
        photons, voxels = c["photons"] * 0.39 * c["sims"], voxels * 0.4 * c["sims"]
    if c["kind"] == "replay":
        photons, fields = photons * 0.005 * c["detectors"] / 4, c["gates"] * c["detectors"]
    if c["kind"] == "readings":
        fields = 1
    if c["kind"] == "fluence":
        photons *= 3  # forward, the loss of each photon, the gradient
    return {"bytes": float(voxels * (label + 4 * fields)), "flops": float(photons * (48 * steps + 65 * scatterings + 20))}


def exact(c, seed):
    """A photon's path follows from each comparison of a rounded number with a random one: in 64 bits other photons
    are detected and other voxels crossed, and the result is another sample of the same mean, not this one's value."""
    return None
