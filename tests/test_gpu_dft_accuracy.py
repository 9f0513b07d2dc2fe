"""The folded transforms (csrc/dft.cu) are no further from a 64-bit solve than the
run-time radix passes whose place they take, in FP32: BF16 storage computes in FP32
too and keeps the passes, so a Poisson solve of the same charge in such a context is
the comparison.  Charges as a convecting state has them, with 30 % noise; the
fluctuation of phi and the horizontal field, whose error is the transforms' alone, in
the root mean square over four charges.  Two computations of the same sums in another
order, so the folded one's error is asked to be below 1.1 times the other's.
"""
import numpy as np
import pytest

from conftest import ehd

pytestmark = pytest.mark.gpu

# smooth widths of 24 to 360 points, an odd one, a prime, and one axis of each with 64
SHAPES = [(24, 20, 33), (100, 80, 40), (160, 160, 33), (200, 210, 30), (303, 302, 25),
          (360, 90, 20), (64, 251, 20), (192, 64, 17)]


def charge(shape, seed):
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    x = 2 * np.pi * np.arange(nx) / nx
    y = 2 * np.pi * np.arange(ny)[:, None] / ny
    z = np.linspace(0.0, 1.0, nz)[:, None, None]
    roll = np.cos(x + rng.uniform(0, 6)) + 0.7 * np.cos(y + rng.uniform(0, 6))
    q = 10.0 / np.sqrt(1.0 + 6.0 * z) * (1.0 + 0.15 * np.sin(np.pi * z) * roll)
    q = q * (1.0 + 0.3 * rng.standard_normal((nz, ny, nx)))
    return q.astype(np.float32).astype(np.float64)


def fluctuation(a):
    return a - a.mean(axis=(1, 2), keepdims=True)


@pytest.mark.parametrize("shape", SHAPES)
def test_folded_sums_are_as_accurate_as_the_passes(shape):
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = ehd.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000)
    err = {"fp32": [], "bf16": []}
    for seed in range(4):
        out = {}
        for prec in ("fp64", "fp32", "bf16"):
            with ehd.Simulation(p, prec) as sim:
                sim.initialize()
                f = sim.get_fields()
                f["q"] = charge(shape, seed)
                sim.set_fields(f)
                sim.poisson()
                o = sim.get_fields(("phi", "ex", "ey"))
            out[prec] = (fluctuation(o["phi"]), o["ex"], o["ey"])
        for prec, e in err.items():
            e.append([np.linalg.norm(a - b) / np.linalg.norm(b)
                      for a, b in zip(out[prec], out["fp64"])])
    rms = {prec: np.sqrt((np.array(e) ** 2).mean(axis=0)) for prec, e in err.items()}
    assert (rms["fp32"] < 1.1 * rms["bf16"]).all(), rms
