"""The kernel of the usual configurations (byte labels or float absorption) against the general one.

Both run the same photons with the same arithmetic, so every output is compared to the last bit where it is
summed exactly (energies, records, launch states) and to the rounding of the float remainders in the field:
a deposit's remainder is at most half a unit, the fields are rounded to float, and the float sums of the
remainders differ in order alone, far below one part in 1e6 of the field's norm.  A configuration whose
scattering limit ``gscatter`` is at most 2^24 takes the general kernel; no photon here scatters as often.
"""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _void_inside():
    """A closed cavity of label 0, an odd shape, three labels."""
    vol = np.ones((37, 29, 41), np.uint8)
    vol[10:20, 8:21, 12:30] = 2
    vol[13:17, 12:18, 18:24] = 0
    vol[:, :, 38:] = 3
    return vol


_ODD = dict(vol=_void_inside(), srcpos=[18, 14, 0], detpos=[[18, 6, 0, 2], [30, 14, 0, 3]],
            prop=[[0, 0, 1, 1], [0.01, 1, 0.5, 1.37], [0.02, 5, 0.9, 1.45], [0.3, 12, 0.0, 1.37]])
_MAP = (0.005 + 0.02 * np.random.RandomState(3).rand(37, 29, 41)).astype(np.float32)
_MAP[13:17, 12:18, 18:24] = 0
_MAP[30:, :, 20:] = 1e-8
_MUA = dict(vol=_MAP[None], srcpos=[18, 14, 0], detpos=[[18, 6, 0, 2], [30, 14, 0, 3]], prop=[[0, 0, 1, 1], [0.01, 1, 0.77, 1.37]])
CASES = {
    "default": {}, "plain": dict(issavedet=0, issaveseed=0), "paths": dict(savedetflag="dp"), "scatterings": dict(savedetflag="ds"),
    "both": dict(savedetflag="dsp"), "momentum": dict(savedetflag="dspm"), "id": dict(savedetflag="d"),
    "noreflect": dict(isreflect=0), "energy": dict(outputtype="energy"), "fluence": dict(outputtype="fluence"),
    "cyclic": dict(bc="ccrrcc", isreflect=0), "mirror": dict(bc="mmammm"), "reflecting": dict(bc="rrrrrr", isreflect=0),
    "facedet": dict(bc="aaaaaa001000", isreflect=0), "roulette": dict(minenergy=0.01), "unit": dict(unitinmm=0.5),
    "odd": _ODD, "odd noreflect": dict(_ODD, isreflect=0, savedetflag="dp"), "odd gates": dict(_ODD, tstart=1e-10, tend=1.7e-9, tstep=1e-10),
    "matched": dict(_ODD, prop=[[0, 0, 1, 1], [0.01, 1, 0.5, 1], [0.02, 5, 0.9, 1], [0.3, 12, 0.0, 1]]),
    "no absorption": dict(prop=[[0, 0, 1, 1], [0, 1, 0.5, 1.37], [1e-8, 5, 0.9, 1.45]]),
    "saved reflectance": dict(vol=cases._voidtop(), issaveref=1, srcpos=[20, 20, 0]),
    "one voxel": cases.VARIANTS["onevoxel"], "few photons": dict(nphoton=100), "specular": cases.VARIANTS["outside_src_specular"],
    "wide label": dict(vol=np.full((40, 40, 40), 127, np.uint8), prop=[[0, 0, 1, 1]] + [[0.01, 1, 0.5, 1.37]] * 127, savedetflag="d"),
    "angles": cases.VARIANTS["angleinvcdf"], "pattern": cases.VARIANTS["pattern"], "isotropic": cases.VARIANTS["isotropic"],
    "many gates": dict(tstep=2e-11), "one void step": dict(maxvoidstep=1), "two void steps": dict(maxvoidstep=2),
    # the most media whose records fit the general kernel's shared memory, and some fewer
    "72 media": dict(vol=np.arange(1, 41, dtype=np.uint8)[:, None, None] + np.zeros((1, 40, 40), np.uint8), savedetflag="dspm",
                     prop=[[0, 0, 1, 1]] + [[0.01, 1, 0.5, 1.37]] * 71),
    "60 media": dict(vol=np.arange(1, 41, dtype=np.uint8)[:, None, None] + np.zeros((1, 40, 40), np.uint8), savedetflag="dspm",
                     prop=[[0, 0, 1, 1]] + [[0.01, 1, 0.5, 1.37]] * 59), "backward": dict(prop=[[0, 0, 1, 1], [0.01, 2, -0.4, 1.37], [0.02, 5, 0.87, 1.45]]),
    # float absorption: voxels without any, and every record kind
    "mua": dict(_MUA, savedetflag="dxv"), "mua energy": dict(_MUA, outputtype="energy"), "mua plain": dict(_MUA, issavedet=0, issaveseed=0),
    "mua matched": dict(_MUA, isreflect=0, savedetflag="dspm", minenergy=0.01), "mua gates": dict(_MUA, tstart=1e-10, tend=1.7e-9, tstep=1e-10),
    "mua mirror": dict(_MUA, bc="mmammm"), "mua cyclic": dict(_MUA, bc="ccrrcc", isreflect=0),
    # modulated sources
    "rf": dict(omega=2 * np.pi * 1e8), "rf roulette": dict(omega=2 * np.pi * 3e8, minenergy=0.01, outputtype="fluence"),
    "rf odd": dict(_ODD, omega=2 * np.pi * 1e8, isreflect=0, issavedet=0, issaveseed=0),
    "rf no absorption": dict(omega=2 * np.pi * 1e8, prop=[[0, 0, 1, 1], [0, 1, 0.5, 1.37], [1e-8, 5, 0.9, 1.45]]), "no photon detected": dict(detpos=[[20, 20, 39, 1]], nphoton=50),
}


def _run(cfg, general):
    import mcxcl_gb300
    r = mcxcl_gb300.run(dict(cfg, **({"gscatter": 1 << 24} if general else {})))
    out = {"flux": np.asarray(r["flux"], np.complex128 if np.iscomplexobj(r["flux"]) else np.float64)}
    for k in ("energytot", "energyabs", "detected", "failedlaunch"):
        out[k] = r["stat"][k]
    if "dref" in r:
        out["dref"] = np.asarray(r["dref"], np.float64)
    rows = [np.ascontiguousarray(r[k].T).view(np.uint32) for k in ("seeds", "detp") if k in r]
    t = np.concatenate(rows, axis=1) if rows else np.zeros((0, 1), np.uint32)
    out["records"] = t[np.lexsort(t.T[::-1])]
    return out


@pytest.mark.parametrize("name", list(CASES))
def test_same_photons_as_the_general_kernel(name):
    cfg = cases.small_two_media(**dict(dict(nphoton=200000), **CASES[name]))
    a, b = _run(cfg, False), _run(cfg, True)
    assert sorted(a) == sorted(b)
    for k in ("energytot", "energyabs", "detected", "failedlaunch"):
        assert a[k] == b[k], (k, a[k], b[k])
    assert np.array_equal(a["records"], b["records"])
    for k in ("flux", "dref"):
        if k in a:
            assert np.linalg.norm(a[k] - b[k]) <= 1e-6 * np.linalg.norm(b[k]), k
            assert np.array_equal(a[k] != 0, b[k] != 0), k


@pytest.mark.parametrize("base", ["default", "odd", "mua", "roulette"])
@pytest.mark.parametrize("output", ["jacobian", "wltof", "nscat", "wm", "wptof", "flux", "energy"])
@pytest.mark.parametrize("det", [-1, 0, 2])
def test_replays_as_the_general_kernel(base, output, det):
    """A replay's deposits: weight x path or x scatterings, per detector and gate."""
    import mcxcl_gb300
    cfg = cases.small_two_media(**dict(dict(nphoton=50000, savedetflag="dsp", tstep=5e-10), **CASES[base]))
    if base == "mua":
        cfg["savedetweight"] = 1
    first = mcxcl_gb300.run(cfg)
    rep = dict(cfg, seed=first["seeds"], outputtype=output, replaydet=det, savedetflag="dsp")
    if base == "mua":
        rep.update(replayweight=first["detweight"][0], replaytof=first["detweight"][1].clip(0, 4.99e-9),
                   replaydetid=first["detp"][0].astype(np.int32))
    else:
        rep["detphotons"] = first["detp"]
    a, b = _run(rep, False), _run(rep, True)
    assert a["energytot"] == b["energytot"] and a["energyabs"] == b["energyabs"] and a["detected"] == b["detected"]
    assert np.linalg.norm(b["flux"]) > 0 and np.linalg.norm(a["flux"] - b["flux"]) <= 1e-6 * np.linalg.norm(b["flux"])


@pytest.mark.parametrize("name", ["default", "odd", "mua", "no absorption", "mua gates"])
def test_fluence_gradient_as_the_general_kernel(name):
    """The loss gradient's float sums add the same terms in another order: up to 1e5 terms of one sign in an
    element, each sum off by at most a few hundred roundings of 6e-8."""
    from mcxcl_gb300 import diff
    cfg = cases.small_two_media(**dict(dict(nphoton=50000), **CASES[name]))
    for k in ("issaveseed", "savedetflag"):
        cfg.pop(k, None)
    cfg["issavedet"] = 0
    got = []
    for extra in ({}, {"gscatter": 1 << 24}):
        g = diff.FluenceGradient(dict(cfg, **extra))
        f = g.forward()
        d = np.random.RandomState(1).standard_normal(f.shape)
        got.append((f, *g.backward(d)))
        g.close()
    for x, y in zip(*got):
        assert np.linalg.norm(y) > 0 and np.linalg.norm(x - y) <= 2e-5 * np.linalg.norm(y)


def _batch():
    """150 simulations (two waves) of different volumes, media, gates and outputs, in 1 to 3 photons a thread."""
    sims = []
    for k in range(150):
        name = ["default", "noreflect", "energy", "fluence", "cyclic", "mirror", "roulette", "unit", "matched", "no absorption", "odd gates",
                "isotropic", "few photons", "backward"][k % 14]
        cfg = cases.small_two_media(**dict(dict(nphoton=1500), **CASES[name]))
        for key in ("detpos", "savedetflag", "issaveseed"):
            cfg.pop(key, None)
        sims.append(dict(cfg, seed=k + 1, issavedet=0))
    return sims


@pytest.mark.parametrize("per_thread", [0, 3])
def test_batch_as_the_general_kernel(per_thread):
    import mcxcl_gb300
    sims = _batch()
    a = mcxcl_gb300.run_batch(sims, photons_per_thread=per_thread)
    b = mcxcl_gb300.run_batch([dict(c, gscatter=1 << 24) for c in sims], photons_per_thread=per_thread)
    for x, y in zip(a, b):
        assert x["stat"]["energytot"] == y["stat"]["energytot"] and x["stat"]["energyabs"] == y["stat"]["energyabs"]
        f, g = np.asarray(x["flux"], np.float64), np.asarray(y["flux"], np.float64)
        assert np.linalg.norm(g) > 0 and np.linalg.norm(f - g) <= 1e-6 * np.linalg.norm(g)


@pytest.mark.parametrize("extra", [{}, cases.VARIANTS["multisrc_id"], _ODD])
def test_complex_pairs_hold_the_planes(extra):
    """run()'s complex field, exported as pairs, against the two planes the C interface exports by default."""
    import ctypes

    import mcxcl_gb300
    from mcxcl_gb300 import _lib, pmcxcl
    cfg = cases.small_two_media(**dict(dict(nphoton=20000, omega=2 * np.pi * 1e8), **extra))
    flux = mcxcl_gb300.run(cfg)["flux"]
    L, C = _lib.load(), _lib.Config()
    try:
        pmcxcl.parse_config(cfg, C)
        L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
        L.mcx_run_simulation(ctypes.byref(C), None, None)
        pmcxcl._check(C)
        planes = np.ctypeslib.as_array(C.exportfield, shape=(2 * flux.size,)).copy()
    finally:
        L.mcx_clearcfg(ctypes.byref(C))
    assert flux.dtype == np.complex64 and flux.flags["F_CONTIGUOUS"] and np.abs(planes[flux.size:]).max() > 0
    want = (planes[:flux.size] + 1j * planes[flux.size:]).reshape(flux.shape, order="F")
    # two runs of the same photons: the order of the remainders' float sums
    assert np.abs(flux - want).max() <= 1e-6 * np.abs(want).max()
