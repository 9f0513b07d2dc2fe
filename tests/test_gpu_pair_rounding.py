"""The node-pair step (csrc/lbm_pair.cu) beside the per-node step from one state.

After ehd_set_fields the first step runs on the per-node kernel in either run, so
the second starts from the same bits.  Up to the plane sums the two kernels do
the same FP32 operations on it in the same order (the pull with its shift of
references in one rounding, the sums over the directions), so rho and q, which
are read back from those sums, are the same bits: any tolerance is zero.
"""
import numpy as np
import pytest

from conftest import O, ehd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 1, 4), (6, 3, 5), (66, 7, 5), (64, 64, 33), (130, 9, 7)])
@pytest.mark.parametrize("prec", ["fp32", "fp16", "mixed"])
def test_density_and_charge_are_the_node_kernels_bits(shape, prec):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000,
                             exf=50.0, uw=0.01)
    f = M.random_fields(p, 17)
    out = []
    for kern in (0, 1):
        with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), prec) as sim:
            sim.set_tuning(lbm_kernel=kern)
            sim.set_fields(f)
            sim.step(1)
            sim.step(1)
            out.append(sim.get_fields())
    for k in ("rho", "q"):
        assert np.array_equal(out[0][k], out[1][k]), (k, np.abs(out[0][k] - out[1][k]).max())
