"""Which kernel a call runs, in which shape, and what that must not change."""
import ctypes

import numpy as np
import pytest

import cases
from test_gpu_label import CASES

pytestmark = pytest.mark.gpu


def _session():
    """The device session that run(), run_batch() and the gradients share."""
    from mcxcl_gb300 import _lib, pmcxcl
    L, C = _lib.load(), _lib.Config()
    try:
        pmcxcl.parse_config(cases.small_two_media(nphoton=1000), C)
        L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
        s = L.mcx_prepare_simulation(ctypes.byref(C))
        pmcxcl._check(C)
    finally:
        L.mcx_clearcfg(ctypes.byref(C))
    return L, s


def _usual(L, s):
    return _kernel(L, s)[0]


def _kernel(L, s):
    usual, lanes = ctypes.c_int(-1), ctypes.c_int(-1)
    assert L.mcxg_get_kernel(s, ctypes.byref(usual), ctypes.byref(lanes)) == 0
    return usual.value, lanes.value


@pytest.mark.parametrize("name", list(CASES))
def test_which_kernel_ran(name):
    """The comparisons of the two kernels compare two kernels: 72 media with every record alone do not fit."""
    import mcxcl_gb300
    L, s = _session()
    cfg = cases.small_two_media(**dict(dict(nphoton=1000), **CASES[name]))
    mcxcl_gb300.run(cfg)
    assert _usual(L, s) == (name != "72 media")
    mcxcl_gb300.run(dict(cfg, gscatter=1 << 24))
    assert _usual(L, s) == 0


def test_batch_kernel():
    import mcxcl_gb300
    L, s = _session()
    sims = [dict(cases.small_two_media(nphoton=1000), issavedet=0, issaveseed=0, seed=k + 1) for k in range(3)]
    for c in sims:
        c.pop("detpos")
    mcxcl_gb300.run_batch(sims)
    assert _usual(L, s) == 1
    mcxcl_gb300.run_batch(sims[:2] + [dict(sims[2], gscatter=1 << 24)])
    assert _usual(L, s) == 0


def test_both_gradient_passes_on_one_kernel():
    """The second pass's float sums depend on what ran before it, so both passes are of the general kernel."""
    from mcxcl_gb300 import diff
    cfg = cases.small_two_media(nphoton=20000, issavedet=0, issaveseed=0)
    cfg.pop("detpos")
    g = diff.FluenceGradient(cfg)
    try:
        f = g.forward()
        assert _usual(g.L, g.s) == 1
        c = np.ascontiguousarray(np.ones(f.size, np.float32))
        assert g.L.mcxg_set_adjoint(g.s, c.ctypes.data, c.size) == 0
        for flag in (256, 512):
            assert g.L.mcxg_simulate(g.s, flag, ctypes.byref(ctypes.c_float())) == 0
            assert _usual(g.L, g.s) == 0
    finally:
        g.close()


def _launch(L, s):
    grid, block = ctypes.c_int(), ctypes.c_int()
    assert L.mcxg_get_launch(s, ctypes.byref(grid), ctypes.byref(block), None) == 0
    return grid.value, block.value


def _plain(**kw):
    cfg = cases.small_two_media(**dict(dict(issavedet=0, issaveseed=0), **kw))
    cfg.pop("detpos")
    return cfg


def test_a_tuned_shape_ends_with_its_run():
    """The shape that a small tuned run chose is not the next batch's or gradient's."""
    import mcxcl_gb300
    from mcxcl_gb300 import diff
    L, s = _session()
    sims = [_plain(nphoton=20000, seed=k + 1) for k in range(4)]
    mcxcl_gb300.run_batch(sims)
    batch = _launch(L, s), _usual(L, s)
    assert batch[1] == 1
    cfg, shapes = _plain(nphoton=2000000), []
    for before in ({}, dict(nphoton=50000, autotune=1), dict(nphoton=50000, autotune=1, gscatter=1 << 24), dict(nphoton=300, debuglevel="M")):
        mcxcl_gb300.run(_plain(**before))
        g = diff.FluenceGradient(cfg)
        try:
            f = g.forward()
            shapes.append((_launch(L, s), _usual(L, s)))
            g.backward(np.ones(f.shape))
        finally:
            g.close()
        mcxcl_gb300.run(_plain(**before))
        mcxcl_gb300.run_batch(sims)
        assert (_launch(L, s), _usual(L, s)) == batch
    assert shapes == [shapes[0]] * 4 and shapes[0][1] == 1


def test_tuned_runs_of_few_photons_spread_their_lanes():
    import mcxcl_gb300
    L, s = _session()
    mcxcl_gb300.run(_plain(nphoton=10000))
    assert _kernel(L, s)[0] == 1 and _kernel(L, s)[1] < 32
    mcxcl_gb300.run(_plain(nphoton=10000, autotune=1))
    grid, block = _launch(L, s)
    sms = mcxcl_gb300.gpuinfo()[0]["sm"]
    warps = grid // sms * block // 32
    assert _kernel(L, s)[1] == min(32, -(-(10000 // sms) // warps)) < 32


def test_the_kernels_are_tuned_apart():
    """A general run's tuned shape is not taken for the same problem on the usual configurations' kernel."""
    import mcxcl_gb300
    L, s = _session()
    sms = mcxcl_gb300.gpuinfo()[0]["sm"]
    cfg = _plain(nphoton=20000 * sms, autotune=1)
    mcxcl_gb300.run(dict(cfg, gscatter=1 << 24))
    assert _usual(L, s) == 0
    mcxcl_gb300.run(cfg)
    assert _usual(L, s) == 1 and _launch(L, s) == (3 * sms, 256)


@pytest.mark.parametrize("general", [0, 1 << 24])
@pytest.mark.parametrize("photons", [200, 20000, 200000])
def test_every_shape_runs_every_photon(general, photons):
    """Shapes of few warps and lanes, the caller's own included: the same energies as the automatic one."""
    from mcxcl_gb300 import _lib, pmcxcl
    L, C, got = _lib.load(), _lib.Config(), []
    try:
        pmcxcl.parse_config(dict(_plain(nphoton=photons), **({"gscatter": general} if general else {})), C)
        L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
        s = L.mcx_prepare_simulation(ctypes.byref(C))
        pmcxcl._check(C)
        for shape in ((0, 0), (256, 1), (256, 3), (256, 4), (128, 2), (32, 1), (64, 16)):
            for flags in (2, 16):                                        # plain and aggregated deposits
                assert L.mcxg_set_launch(s, *shape) == 0
                assert L.mcxg_simulate(s, flags, ctypes.byref(ctypes.c_float())) == 0
                esc, tot = ctypes.c_double(), ctypes.c_double()
                assert L.mcxg_get_energy(s, ctypes.byref(esc), ctypes.byref(tot)) == 0
                field = np.zeros(40 ** 3 * 20)
                assert L.mcxg_get_field_f64(s, field.ctypes.data) == 0
                got.append((_usual(L, s), tot.value, esc.value, field.sum()))
        assert L.mcxg_set_launch(s, 0, 0) == 0
    finally:
        L.mcx_clearcfg(ctypes.byref(C))
    assert len({g[0] for g in got}) == (1 if general else 2)
    for g in got:
        # the instantiations of the general kernel contract differently: a path may part from another's
        assert g[1] == photons and abs(g[2] - got[0][2]) <= 2e-3 * photons ** 0.5 * 10 and abs(g[3] / got[0][3] - 1) <= 0.02


_TWICE = '''
import ctypes, sys
sys.path[:0] = [%r, %r]
import numpy as np, cases
from mcxcl_gb300 import _lib, pmcxcl
L, C = _lib.load(), _lib.Config()
cfg = cases.small_two_media(nphoton=2000, savedetflag="dsp", prop=[[0, 0, 1, 1]] + [[0.01, 1, 0.5, 1.37]] * %d, **%r)
pmcxcl.parse_config(cfg, C)
L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
s = L.mcx_prepare_simulation(ctypes.byref(C))
pmcxcl._check(C)
for _ in range(2):
    assert L.mcxg_set_launch(s, 256, 4) == 0 and L.mcxg_simulate(s, 2, ctypes.byref(ctypes.c_float())) == 0
    g = ctypes.c_int()
    L.mcxg_get_launch(s, ctypes.byref(g), None, None)
    print(g.value)
'''


@pytest.mark.parametrize("media,extra,blocks", [(30, {}, 3), (60, {}, 1), (30, dict(gscatter=1 << 24), 3)])
def test_no_more_blocks_than_fit(media, extra, blocks):
    """Records of many media leave room for fewer blocks a SM (their shared memory: 2 x 1 KB a medium and block of 228 KB),
    in a process's first launch of a kernel as in its second."""
    import os
    import subprocess
    import sys

    import mcxcl_gb300
    here = os.path.dirname(os.path.abspath(__file__))
    p = subprocess.run([sys.executable, "-c", _TWICE % (os.path.dirname(here), here, media, extra)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    sms = mcxcl_gb300.gpuinfo()[0]["sm"]
    assert [int(x) // sms for x in p.stdout.split()] == [blocks, blocks]


def test_where_few_photons_end():
    """Other media formats and shared patterns, which gain less from few warps, take their full shape earlier."""
    import mcxcl_gb300
    L, s = _session()
    sms = mcxcl_gb300.gpuinfo()[0]["sm"]
    for variant, line, full in (("asf2h", 300, 3), ("svmc", 300, 3), ("pattern_share", 700, 4), ("gscatter", 1000, 4), ("angleinvcdf", 1000, 2)):
        cfg = cases.small_two_media(**dict(cases.VARIANTS[variant], issaveseed=0))
        for photons, blocks in ((line * sms, 1), ((line + 1) * sms, full)):
            mcxcl_gb300.run(dict(cfg, nphoton=photons))
            assert _launch(L, s) == (blocks * sms, 256)
            assert _kernel(L, s)[1] == (min(32, -(-line // 8)) if blocks == 1 else 32)


@pytest.mark.parametrize("general", [{}, dict(gscatter=1 << 24)])
def test_batch_labels_past_the_last_medium(general):
    """A caller of the C interface may hand in a volume that validation has not seen: labels past a simulation's media
    are its last medium, not another simulation's or an empty row."""
    from mcxcl_gb300 import _lib, pmcxcl
    L, got = _lib.load(), []
    one, two = [[0, 0, 1, 1], [0.01, 1, 0.5, 1.37]], [[0, 0, 1, 1], [0.01, 1, 0.5, 1.37], [0.02, 5, 0.9, 1.45]]
    for past in (False, True):
        Cs = [_lib.Config() for _ in range(4)]
        try:
            for k, C in enumerate(Cs):
                pmcxcl.parse_config(_plain(nphoton=3000, seed=k + 1, prop=two if k % 2 else one,
                                           vol=np.full((20, 20, 20), 1 + k % 2, np.uint8), srcpos=[10, 10, 0], **general), C)
                L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
                pmcxcl._check(C)
                if past:
                    np.ctypeslib.as_array(C.vol, shape=(8000,))[:] = (2, 3, 3, 120)[k]
            L.mcx_run_batch((ctypes.POINTER(_lib.Config) * 4)(*[ctypes.pointer(C) for C in Cs]), 4, ctypes.c_uint(0), ctypes.c_uint(0))
            pmcxcl._check(Cs[0])
            got.append([(C.energytot, C.energyesc) + tuple(np.ctypeslib.as_array(C.exportfield, shape=(8000 * 20,)).tolist()) for C in Cs])
        finally:
            for C in Cs:
                L.mcx_clearcfg(ctypes.byref(C))
    for a, b in zip(*got):
        assert a[:2] == b[:2] and 0 < a[1] < a[0] == 3000
        assert np.abs(np.array(a[2:]) - np.array(b[2:])).max() <= 1e-6 * max(a[2:])


def test_energies_of_more_simulations_than_a_grid_is_high():
    """65,540 simulations of two photons: the batch runs and its energies are summed (its fields are read in a grid whose
    second dimension ends at 65,535, so the call that wants them too refuses)."""
    from mcxcl_gb300 import _lib, pmcxcl
    L, s = _session()
    cfg = dict(nphoton=2, vol=np.ones((2, 2, 2), np.uint8), prop=[[0, 0, 1, 1], [0.01, 1, 0.5, 1.37]], srcpos=[1, 1, 0], srcdir=[0, 0, 1],
               issrcfrom0=1, tstart=0, tend=5e-9, tstep=5e-9, isreflect=0, issavedet=0, seed=3)
    n = 65540
    Cs = [_lib.Config() for _ in range(n)]
    try:
        for C in Cs:
            pmcxcl.parse_config(cfg, C)
            L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
        L.mcx_run_batch((ctypes.POINTER(_lib.Config) * n)(*[ctypes.pointer(C) for C in Cs]), n, ctypes.c_uint(0), ctypes.c_uint(0))
        assert L.mcxg_batch_simulate(ctypes.c_void_p(s), ctypes.c_uint(0), ctypes.byref(ctypes.c_float())) == 0
        e = np.zeros((n, 2))
        assert L.mcxg_batch_get_energy(ctypes.c_void_p(s), ctypes.c_void_p(e.ctypes.data)) == 0
    finally:
        for C in Cs:
            L.mcx_clearcfg(ctypes.byref(C))
    assert (e[:, 1] == 2).all() and (e == e[0]).all() and 0 < e[0, 0] <= 2


def test_the_precision_check_runs_the_kernel_it_vouches_for():
    import mcxcl_gb300
    from mcxcl_gb300 import _lib, pmcxcl
    L, C = _lib.load(), _lib.Config()
    for cfg, usual in ((_plain(nphoton=20000), 1), (cases.small_two_media(nphoton=20000), 1), (_plain(nphoton=20000, isreflect=0), 1),
                       (_plain(nphoton=20000, gscatter=1 << 24), 0)):
        try:
            pmcxcl.parse_config(cfg, C)
            L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
            s = L.mcx_prepare_simulation(ctypes.byref(C))
            pmcxcl._check(C)
            fields = []
            for flags in (2, 2 | 128):
                assert L.mcxg_simulate(s, flags, ctypes.byref(ctypes.c_float())) == 0
                assert _usual(L, s) == usual
                fields.append(np.zeros(40 ** 3 * 20))
                assert L.mcxg_get_field_f64(s, fields[-1].ctypes.data) == 0
            f64, plain, spill = np.zeros(fields[0].size), np.zeros(fields[0].size, np.float32), np.zeros(fields[0].size, np.float32)
            assert L.mcxg_get_verify(s, f64.ctypes.data, plain.ctypes.data, spill.ctypes.data) == 0
        finally:
            L.mcx_clearcfg(ctypes.byref(C))
        # the same photons as without the check, to the field's rounded remainders; the general kernel's instantiations
        # contract differently.  Plain sums of 2e4 terms of one sign are off by at most 2e4 half ulps, 1.2e-3 (the spill
        # field loses what two additions at once both carry over: it is what the others are measured against, not checked)
        norm = np.linalg.norm(f64)
        assert norm > 0 and np.linalg.norm(fields[1] - f64) <= 1e-6 * norm
        assert not usual or np.linalg.norm(fields[0] - f64) <= 1e-6 * norm
        assert np.linalg.norm(plain - f64) <= 1.2e-3 * norm and spill.any()
    sims = [_plain(nphoton=3000, seed=k + 1) for k in range(3)]
    for extra, usual in (({}, 1), (dict(gscatter=1 << 24), 0)):
        got = mcxcl_gb300.run_batch([dict(c, **extra) for c in sims], verify=True)
        assert _usual(L, s) == usual and max(o["stat"]["relerr_max"] for o in got) < 1e-6


@pytest.mark.parametrize("depth", [0.5, -9, -1000])
def test_weights_above_one_stay_within_the_fields_range(depth):
    """A fourierx source's weight grows with its modulation parameter: 501 at -1000.  What the field holds is what the
    photons left, to the roundings of weights (some 20 steps of 6e-8)."""
    import mcxcl_gb300
    cfg = dict(nphoton=1000000, vol=np.ones((6, 6, 6), np.uint8), prop=[[0, 0, 1, 1], [1.0, 1, 0.5, 1]], srcpos=[2, 2, 0],
               srctype="fourierx", srcdir=[0, 0, 1], srcparam1=[1, 0, 0, 1], srcparam2=[0, 0, 0, depth], issrcfrom0=1, seed=5,
               tstart=0, tend=5e-9, tstep=5e-9, isreflect=0, issavedet=0, outputtype="energy", isnormalized=0)
    r = mcxcl_gb300.run(cfg)
    tot, esc = r["stat"]["energytot"], r["stat"]["energyesc"]
    assert abs(tot / (1e6 * (2 - depth) / 2) - 1) < 1e-4
    assert abs(np.asarray(r["flux"], np.float64).sum() / (tot - esc) - 1) < 1e-5


def test_a_medium_that_adds_weight():
    """mua < 0 between mirrors: 1e6 photons grow to e^5.5 times their weight, which the energies and the field tell
    alike, but for the visit that the time window's end cuts short (at most 3.5 voxels of 1,094: 1.7 %)."""
    import mcxcl_gb300
    cfg = dict(nphoton=1000000, vol=np.ones((2, 2, 2), np.uint8), prop=[[0, 0, 1, 1], [-0.005, 1, 0.5, 1.37]], srcpos=[1, 1, 0.5],
               srcdir=[0, 0, 1], issrcfrom0=1, seed=5, tstart=0, tend=5e-9, tstep=5e-9, isreflect=0, bc="mmmmmm", issavedet=0,
               outputtype="energy", isnormalized=0)
    r = mcxcl_gb300.run(cfg)
    tot, esc = r["stat"]["energytot"], r["stat"]["energyesc"]
    assert tot == 1e6 and abs(esc / (1e6 * np.exp(0.005 * 299.792458 * 5 / 1.37)) - 1) < 0.02
    assert abs(np.asarray(r["flux"], np.float64).sum() / (tot - esc) - 1) < 0.018
