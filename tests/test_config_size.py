"""Config keeps the size and the last field that C programs were built with."""
import ctypes


def test_nothing_read_past_errormsg():
    """2,272 bytes on a 64-bit machine, the last four of them padding, which a copy of the structure need not keep."""
    from mcxcl_gb300 import build
    build.build()
    from mcxcl_gb300 import _lib
    L = _lib.load()
    last = max(_lib.Config._fields_, key=lambda f: getattr(_lib.Config, f[0]).offset)[0]
    assert last == "errormsg" and L.mcx_config_sizeof() == ctypes.sizeof(_lib.Config) == 2272
    assert L.mcx_config_offsetof(b"errormsg") == 2272 - 4 - 256
    assert L.mcx_config_offsetof(b"complexpairs") == ctypes.c_size_t(-1).value
