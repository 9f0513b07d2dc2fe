"""Long ehd_step calls: from 40 steps on, runs of eight steps are one CUDA graph
(csrc/api.cu, kManySteps), the remainder and the last step, which writes the
macroscopic fields, graphs of one.  The launches are the same ones in the same order,
so fields, time and step count are those of direct launches, bit for bit, from either
buffer parity, at the shortest such call, with every kind of remainder, and after a
change of launch shapes between two calls.
"""
import numpy as np
import pytest

from conftest import O, ehd

pytestmark = pytest.mark.gpu


def case(shape, seed):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000)
    return ehd.Params.from_dict(p.as_dict()), M.random_fields(p, seed)


# rows, pairs, the per-node kernel (odd nx); compile-time, folded and split-y transforms
@pytest.mark.parametrize("shape,prec", [((32, 12, 9), "fp64"), ((64, 64, 33), "fp32"),
                                        ((30, 22, 11), "fp16"), ((25, 16, 9), "bf16"),
                                        ((40, 10, 13), "mixed")])
@pytest.mark.parametrize("calls", [(40,), (1, 40), (2, 41, 48), (1, 57, 39)])
def test_runs_of_eight_steps_are_the_direct_launches(shape, prec, calls):
    p, f = case(shape, 13)
    out = []
    for graphs in (True, False):
        with ehd.Simulation(p, prec, graphs=graphs) as sim:
            sim.set_fields(f)
            for n in calls:
                sim.step(n)
            out.append((sim.get_fields(), sim.diagnostics()))
    for k in O.FIELDS:
        assert np.array_equal(out[0][0][k], out[1][0][k]), k
    assert out[0][1] == out[1][1]
    assert out[0][1]["step"] == sum(calls)


def test_new_launch_shapes_between_two_long_calls():
    p, f = case((30, 22, 11), 14)
    out = []
    for graphs in (True, False):
        with ehd.Simulation(p, "fp32", graphs=graphs) as sim:
            sim.set_fields(f)
            sim.step(45)
            sim.set_tuning(lbm_kernel=1, node_block_x=32, z_solve=1)
            sim.step(45)
            out.append(sim.get_fields())
    for k in O.FIELDS:
        assert np.array_equal(out[0][k], out[1][k]), k
