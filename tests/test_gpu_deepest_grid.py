"""The deepest grid that the step's launches have room for (65,535 planes): FP32 and
mixed storage take it on the per-node kernel, the node-pair launch having one plane
of blocks too few, and the plane below it on pairs.
"""
import numpy as np
import pytest

from conftest import ehd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [65534, 65535])
@pytest.mark.parametrize("prec", ["fp32", "mixed"])
def test_deepest_grids_step(nz, prec):
    dz = 1.0 / (nz - 1)
    p = ehd.params_from_groups(2, 1, nz, 2 * dz, dz, T=200, M=10, C=10, Fe=4000)
    out = []
    for kern in (0, 1):
        with ehd.Simulation(p, prec) as sim:
            sim.set_tuning(lbm_kernel=kern)
            sim.initialize()
            sim.step(1)
            sim.step(1)
            out.append(sim.get_fields(("rho", "q")))
    for k in ("rho", "q"):
        assert np.isfinite(out[0][k]).all()
        assert np.array_equal(out[0][k], out[1][k]), k
