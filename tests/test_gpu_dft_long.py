"""The folded transforms (csrc/dft.cu) at the longest widths that the rule gives them:
1021 (a prime) and 1022 (2 x 7 x 73), several tiles of outputs and the longest sums, and
primes and twice primes in between, on either axis and in both precisions; against
the oracle.  Each case asserts that its long axis is folded, so that a change of the
rule cannot empty it.  (1023 and 1024, the last widths the kernels could take, go to
run-time radix passes.)

Tolerances are those of the other Poisson tests (1e-10 FP64, 2e-6 FP32 of the largest
value): a folded sum of 511 terms has a rounding error of about 0.2 sqrt(511) units,
2.7e-7 in FP32, relative to its rms.
"""
import ctypes

import numpy as np
import pytest

from conftest import O, ehd, relerr

pytestmark = pytest.mark.gpu


def folded(n, y, rsize):
    f = getattr(ehd.lib(), "_ZN3ehd10dft_usableEibm")
    f.restype, f.argtypes = ctypes.c_bool, [ctypes.c_int, ctypes.c_bool, ctypes.c_size_t]
    return f(n, y, rsize)


@pytest.mark.parametrize("shape", [(1021, 3, 4), (3, 1021, 5), (1022, 2, 4), (2, 1022, 4),
                                   (251, 4, 5), (4, 251, 5), (386, 3, 6), (3, 386, 6), (509, 2, 5)])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 2e-6)])
def test_long_folded_axes_match_oracle(shape, prec, tol):
    import make_golden as M
    nx, ny, nz = shape
    rsize = 8 if prec == "fp64" else 4
    assert folded(max(nx, ny), ny > nx, rsize)
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000)
    f = M.random_fields(p, 8)
    o = O.Oracle(p)
    o.set_fields(f)
    o.poisson()
    o.efield()
    b = o.get_fields()
    o.close()
    with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), prec) as sim:
        sim.set_fields(f)
        sim.poisson()
        a = sim.get_fields()
    e = max(np.abs(b[k]).max() for k in ("ex", "ey", "ez"))
    assert relerr(a["phi"], b["phi"]) < tol, relerr(a["phi"], b["phi"])
    for k in ("ex", "ey", "ez"):
        assert np.abs(a[k] - b[k]).max() < tol * e, (k, np.abs(a[k] - b[k]).max() / e)
