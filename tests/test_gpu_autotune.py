"""What the batch autotuner measures (csrc/batch.cu, batch_step_time)."""
import ctypes
import time

import pytest

from conftest import ehd

pytestmark = pytest.mark.gpu


def params(nx, ny, nz):
    dz = 1.0 / (nz - 1)
    return ehd.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000)


def test_columns_are_timed():
    """Columns step on their own streams.  The time of a step of a batch of them is
    the one a clock on the host sees over many steps: 3,000 of them take some
    milliseconds, against which a launch is nothing."""
    steps = 3000
    with ehd.Batch([params(1, 1, 65), params(1, 1, 33)], "fp64") as b:
        for sim in b:
            sim.initialize()
        b.step(10)
        for sim in b:
            sim.synchronize()
        wall = []
        for _ in range(3):
            t = time.perf_counter()
            b.step(steps)
            for sim in b:
                sim.synchronize()
            wall.append(time.perf_counter() - t)
        step_time = getattr(ehd.lib(), "_ZN3ehd15batch_step_timeEP9ehd_batchiPf")
        step_time.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_float)]
        ms = ctypes.c_float()
        assert step_time(b.h, steps, ctypes.byref(ms)) == 0
        assert 0.5 < 1e-3 * ms.value * steps / min(wall) < 1.5, (ms.value * steps, wall)
