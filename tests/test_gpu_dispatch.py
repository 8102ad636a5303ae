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
    usual = ctypes.c_int(-1)
    assert L.mcxg_get_kernel(s, ctypes.byref(usual)) == 0
    return usual.value


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


@pytest.mark.parametrize("scale", [np.inf, np.nan, -np.inf, -2.0, 0.0, 3.0])
@pytest.mark.parametrize("omega", [0, 2 * np.pi * 1e8])
def test_untouched_elements_take_the_scale(scale, omega):
    """An element that no photon touched is 0 x scale: NaN under an infinite factor, as in a run that launched nothing."""
    from mcxcl_gb300 import _lib, pmcxcl
    L, C = _lib.load(), _lib.Config()
    try:
        pmcxcl.parse_config(cases.small_two_media(nphoton=300, omega=omega), C)
        L.mcx_validatecfg(ctypes.byref(C), None, None, 0)
        s = L.mcx_prepare_simulation(ctypes.byref(C))
        pmcxcl._check(C)
        assert L.mcxg_simulate(s, 2, ctypes.byref(ctypes.c_float())) == 0
        n = 40 ** 3 * 20
        raw, got = np.zeros((2, n), np.float32), np.zeros((2, n), np.float32)
        comps = 2 if omega else 1
        assert L.mcxg_get_field(s, raw.ctypes.data, 1.0) == 0 and L.mcxg_get_field(s, got.ctypes.data, scale) == 0
        with np.errstate(invalid="ignore"):
            want = (raw.astype(np.float64) * scale).astype(np.float32)
        assert (raw[:comps] == 0).mean() > 0.5 and (raw[:comps] != 0).any()
        # raw is rounded to float before the product here, and after it there
        assert np.allclose(got[:comps], want[:comps], rtol=2.5e-7, atol=0, equal_nan=True)
        if omega:
            pairs = np.zeros((n, 2), np.float32)
            assert L.mcxg_get_field_pairs(s, pairs.ctypes.data, scale) == 0
            assert np.array_equal(pairs.T, got, equal_nan=True)
        else:
            blocks, scales = np.zeros(n, np.float32), np.array([scale, 1.0] * 10)
            assert L.mcxg_get_field_blocks(ctypes.c_void_p(s), ctypes.c_void_p(blocks.ctypes.data),
                                           ctypes.c_void_p(scales.ctypes.data), ctypes.c_uint32(20)) == 0
            both = blocks.reshape(10, 2, -1)
            assert np.array_equal(both[:, 0], got[0].reshape(10, 2, -1)[:, 0], equal_nan=True)
            assert np.array_equal(both[:, 1], raw[0].reshape(10, 2, -1)[:, 1])
    finally:
        L.mcx_clearcfg(ctypes.byref(C))


def test_a_run_that_launches_nothing():
    import mcxcl_gb300
    cfg = cases.small_two_media(nphoton=300, maxvoidstep=1, issavedet=0, issaveseed=0)
    cfg.pop("detpos")
    r = mcxcl_gb300.run(cfg)
    assert r["stat"]["energytot"] == 0 and np.isnan(r["flux"]).all()
    many = mcxcl_gb300.run_batch([cfg, dict(cfg, maxvoidstep=1000)])
    assert np.isnan(many[0]["flux"]).all() and np.isfinite(many[1]["flux"]).all() and many[1]["flux"].max() > 0
