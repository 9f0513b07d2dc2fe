"""The two-nodes-per-thread step (csrc/lbm_pair.cu: FP32, FP16 and mixed storage,
even nx) at the edges of its runs of node pairs: one pair a row, rows and planes
that end inside a warp and inside a block, the smallest stack, and the general
sizes; against the oracle beside the per-node kernel.

Both kernels do the same FP32 arithmetic and round the same populations to their
storage once a step, in a different order of operations, so their distances from
the FP64 oracle have the same size: the pair kernel's is asked to be below twice
the per-node kernel's (the spread between two realisations of the same rounding)
plus 1e-6.
"""
import numpy as np
import pytest

from conftest import O, ehd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 1, 4), (2, 5, 5), (6, 3, 4), (34, 3, 6), (64, 4, 5), (66, 7, 5),
                                   (128, 2, 6), (130, 9, 7), (256, 4, 5), (302, 5, 6)])
@pytest.mark.parametrize("prec", ["fp16", "mixed", "fp32"])
def test_pair_kernel_is_as_near_the_oracle_as_the_node_kernel(shape, prec):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000,
                             exf=50.0, uw=0.01)
    f = M.random_fields(p, 31)
    o = O.Oracle(p)
    o.set_fields(f)
    o.step(8)
    b = o.get_fields()
    o.close()
    err = {}
    for kern in (0, 1):
        with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), prec) as sim:
            sim.set_tuning(lbm_kernel=kern)
            sim.set_fields(f)
            sim.step(5)
            sim.step(3)
            a = sim.get_fields()
            assert not sim.diagnostics()["nonfinite"]
        err[kern] = {k: np.linalg.norm(a[k] - b[k]) / max(np.linalg.norm(b[k]), 1e-30)
                     for k in O.FIELDS if np.abs(b[k]).max() > 1e-9}
    for k, e in err[1].items():
        assert err[0][k] < 2.0 * e + 1e-6, (k, err[0][k], e)
