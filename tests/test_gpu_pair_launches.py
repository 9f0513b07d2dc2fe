"""The node-pair step's two launch shapes in FP16 and mixed storage (csrc/lbm_pair.cu):
plane 0 with the pairs up to 5,000 blocks of pairs, in a launch of its own above.
128 x 100 x 101 has 5,000, 128 x 100 x 102 5,050; 302 x 266 x 38 ends inside a block.

rho and q of the second step, which both kernels take from the same state, are the
per-node kernel's bits.  Over more steps the two round the same populations in a
different order of the plane sums, so the pair kernel's distance from an FP64 run is
asked to be below twice the per-node kernel's, plus 1e-6 (as for the small grids).
"""
import numpy as np
import pytest

from conftest import O, ehd

pytestmark = pytest.mark.gpu

SHAPES = [(128, 100, 101), (128, 100, 102), (302, 266, 38)]


def case(shape):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000)
    return ehd.Params.from_dict(p.as_dict()), M.random_fields(p, 37)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec", ["fp16", "mixed"])
def test_both_launch_shapes_match_the_node_kernel(shape, prec):
    p, f = case(shape)
    with ehd.Simulation(p, "fp64") as sim:
        sim.set_fields(f)
        sim.step(7)
        ref = sim.get_fields()
    second, err = [], []
    for kern in (0, 1):
        with ehd.Simulation(p, prec) as sim:
            sim.set_tuning(lbm_kernel=kern)
            sim.set_fields(f)
            sim.step(1)
            sim.step(1)
            second.append(sim.get_fields(("rho", "q")))
            sim.step(5)  # four steps without the macroscopic fields, one with
            a = sim.get_fields()
            assert not sim.diagnostics()["nonfinite"]
        err.append({k: np.linalg.norm(a[k] - ref[k]) / max(np.linalg.norm(ref[k]), 1e-30)
                    for k in O.FIELDS if np.abs(ref[k]).max() > 1e-9})
    for k in ("rho", "q"):
        assert np.array_equal(second[0][k], second[1][k]), k
    for k, e in err[1].items():
        assert err[0][k] < 2.0 * e + 1e-6, (k, err[0][k], e)
