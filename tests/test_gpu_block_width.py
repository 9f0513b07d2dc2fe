"""The per-node step at every block width, and at the width a context takes by
itself, where rows end inside a warp and inside a block: against the oracle.

FP64: the widths differ in the order of the plane sums alone, so each is held
to the 1e-10 of the step's own parity (8 steps of sums of at most 2 000 terms
at 1.1e-16 each, times the 1e2 by which the charge relations amplify a sum).
"""
import numpy as np
import pytest

from conftest import O, ehd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(15, 6, 5), (17, 5, 5), (70, 6, 5), (122, 5, 5), (126, 4, 5), (302, 5, 5)])
def test_block_widths_match_the_oracle(shape):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000,
                             exf=50.0, uw=0.01)
    f = M.random_fields(p, 17)
    o = O.Oracle(p)
    o.set_fields(f)
    o.step(8)
    b = o.get_fields()
    o.close()
    for bx in (0, 16, 32, 64, 128):
        with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), "fp64") as sim:
            sim.set_tuning(lbm_kernel=1, **({"node_block_x": bx} if bx else {}))
            sim.set_fields(f)
            sim.step(8)
            a = sim.get_fields()
        for k in O.FIELDS:
            top = np.abs(b[k]).max()
            if top > 1e-9:
                assert np.abs(a[k] - b[k]).max() < 1e-10 * top, (bx, k)
