"""The column kernel (csrc/column.cu) with FP32 arithmetic beside the per-node kernel: one
step from one state.  rho, q, u and w of a step are sums over the pulled populations
(and E of the state before), which both kernels form from the same values with the same
FP32 operations in the same order, so they are the same bits: any tolerance is zero.
"""
import numpy as np
import pytest

from conftest import ehd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [4, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp16", "bf16"])
@pytest.mark.parametrize("lam", [(1.0 / 12.0, 1e-6), (0.25, 0.25)])
def test_moments_of_a_column_step_are_the_node_kernels_bits(nz, prec, lam):
    dz = 1.0 / (nz - 1)
    p = ehd.params_from_groups(1, 1, nz, dz, dz, T=250, M=9, C=8, Fe=4000, lambda_f=lam[0],
                               lambda_g=lam[1], exf=20.0)
    out = []
    for kern in (0, 1):
        with ehd.Simulation(p, prec) as sim:
            sim.initialize()
            sim.set_tuning(lbm_kernel=1)
            sim.step(100)
            sim.set_tuning(lbm_kernel=kern)
            sim.step(1)
            out.append(sim.get_fields())
    for k in ("rho", "q", "u", "w"):
        assert np.array_equal(out[0][k], out[1][k]), (k, np.abs(out[0][k] - out[1][k]).max())
