"""The kernel of byte-label volumes against the general common-configuration one.

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
    "many gates": dict(tstep=2e-11), "no photon detected": dict(detpos=[[20, 20, 39, 1]], nphoton=50),
}


def _run(cfg, general):
    import mcxcl_gb300
    r = mcxcl_gb300.run(dict(cfg, **({"gscatter": 1 << 24} if general else {})))
    out = {"flux": np.asarray(r["flux"], np.float64)}
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
