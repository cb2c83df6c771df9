"""Kernel attributes (the shared memory a launch may ask for) are set once on every device
that a process uses, not once per process: on a second device the FP64 entry points'
kernels could not be launched (CPU; the devices are numbers)."""
import ctypes as ct

from elphbolt_gb300 import _lib, build


def test_once_on_each_device():
    build.build()
    L = _lib.load()
    dev = [0, 0, 1, 0, 1, 7, 7, 64]
    ran = (ct.c_int * len(dev))()
    assert L.ephg_debug_once_per_device(len(dev), (ct.c_int * len(dev))(*dev), ran) == _lib.EPHG_OK
    assert list(ran) == [1, 0, 1, 0, 0, 1, 0, 1]
