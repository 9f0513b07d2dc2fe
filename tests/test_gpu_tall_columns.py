"""Grids too tall for the two-sided z solve, whose columns stay in shared memory:
the first depths beyond it (NZ = 882 in FP64, 1762 in FP32 are its last), where the
run-time sine transform takes over, and the first beyond that one (1464 and 2561),
left to the FP64 sweep through global memory; against the oracle, and each route by
its difference from the sweep's bits.

The tolerances are those of the other Poisson tests (1e-10 FP64, 2e-6 FP32 of the
largest value).
"""
import numpy as np
import pytest

from conftest import O, ehd, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,prec,tol,sweep", [
    (882, "fp64", 1e-10, False), (883, "fp64", 1e-10, False), (1464, "fp64", 1e-10, True),
    (1762, "fp32", 2e-6, False), (1763, "fp32", 2e-6, False), (1763, "mixed", 2e-6, False),
    (2561, "fp32", 2e-6, True)])
def test_tall_columns_leave_the_sweep_as_the_last_resort(nz, prec, tol, sweep):
    import make_golden as M
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(6, 3, nz, 6 * dz, 3 * dz, T=200, M=10, C=10, Fe=4000)
    f = M.random_fields(p, 19)
    o = O.Oracle(p)
    o.set_fields(f)
    o.poisson()
    o.efield()
    b = o.get_fields()
    o.close()
    out = []
    for z_solve in (0, 1):
        with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), prec) as sim:
            sim.set_tuning(z_solve=z_solve)
            sim.set_fields(f)
            sim.poisson()
            out.append(sim.get_fields())
    e = max(np.abs(b[k]).max() for k in ("ex", "ey", "ez"))
    for a in out:
        assert relerr(a["phi"], b["phi"]) < tol, relerr(a["phi"], b["phi"])
        for k in ("ex", "ey", "ez"):
            assert np.abs(a[k] - b[k]).max() < tol * e, (k, np.abs(a[k] - b[k]).max() / e)
    assert np.array_equal(out[0]["phi"], out[1]["phi"]) == sweep


@pytest.mark.parametrize("nz", [512, 513, 514, 641, 642, 643, 770])
def test_mean_mode_of_tall_columns(nz):
    """The two sides of the depth (512) from which the mean mode is summed by runs
    of planes, and runs that end before, at and after the last plane (640 interior
    planes are 128 runs of 5)."""
    import make_golden as M
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(3, 2, nz, 3 * dz, 2 * dz, T=200, M=10, C=10, Fe=4000)
    f = M.random_fields(p, 23)
    o = O.Oracle(p)
    o.set_fields(f)
    o.poisson()
    o.efield()
    b = o.get_fields()
    o.close()
    with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), "fp64") as sim:
        sim.set_fields(f)
        sim.poisson()
        a = sim.get_fields()
    assert relerr(a["phi"], b["phi"]) < 1e-10, relerr(a["phi"], b["phi"])
    assert relerr(a["ez"], b["ez"]) < 1e-10, relerr(a["ez"], b["ez"])
    # the planes' means alone
    ma, mb = a["phi"].mean(axis=(1, 2)), b["phi"].mean(axis=(1, 2))
    assert relerr(ma, mb) < 1e-10, relerr(ma, mb)
