"""What the batch autotuner measures (csrc/batch.cu, batch_step_time) and what it tries."""
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


# (grid, storage, grouped launches, fields that reach no launch while lbm_kernel and
# poisson_path stay 0): a column; folded axes, on pairs, on the per-node kernel (odd
# NX) and, FP64, on rows; the split-y solve; run-time passes (BF16 storage), where all
# but lbm_kernel count
IDLE = [((1, 1, 33), "fp32", False, ("node_block_x", "fft_rows", "fft_cols", "poisson_path", "z_solve")),
        ((24, 22, 9), "fp32", False, ("node_block_x", "fft_rows", "fft_cols", "poisson_path")),
        ((23, 22, 9), "fp32", False, ("lbm_kernel", "fft_rows", "fft_cols", "poisson_path")),
        ((44, 22, 9), "fp64", False, ("node_block_x", "fft_rows", "fft_cols", "poisson_path")),
        ((64, 64, 33), "fp32", False, ("node_block_x", "fft_rows", "fft_cols", "z_solve")),
        ((64, 64, 33), "fp16", True, ("lbm_kernel", "fft_rows", "fft_cols", "z_solve")),
        ((24, 22, 9), "bf16", False, ("lbm_kernel", "poisson_path"))]


@pytest.mark.parametrize("shape,prec,grouped,idle", IDLE)
def test_fields_without_effect_are_not_tried(shape, prec, grouped, idle):
    """Trials of fields that change no launch time the same launches again, and noise
    chooses among them: three short autotunes leave such fields as they were, as long
    as the kernel and the path that make them idle are kept."""
    with ehd.Batch([params(*shape)] * 2, prec) as b:
        b.set_mode(0 if grouped else 1)
        start = b[0].get_tuning()
        for _ in range(3):
            b.autotune(trial_steps=1)
            t = b[0].get_tuning()
            if t["lbm_kernel"] == 0 and t["poisson_path"] == 0:
                for k in idle:
                    assert t[k] == start[k], (k, t, start)
            if "lbm_kernel" in idle:
                assert t["lbm_kernel"] == 0
