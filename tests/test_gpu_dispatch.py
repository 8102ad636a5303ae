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
