"""The column kernel (a 1 x 1 x NZ grid's steps in one launch, csrc/column.cu)
against the oracle and against the per-node kernel, at the sizes where its
block changes: the smallest grid, one warp and one more node, the last sizes
of either block, and the first grid beyond it (which stays per node).

Tolerances: the kernels do the same operations in another order, so FP64 runs
of some tens of steps agree to a few hundred units of round-off of the field's
largest value (1e-11), FP32 ones to 1e-5 as the row kernel's do, and 16-bit
storage to the rounding of its populations (2^-11 and 2^-8 of a deviation a
step, bounded here by 1e-2 and 5e-2 of the field).
"""
import numpy as np
import pytest

from conftest import O, ehd, relerr

pytestmark = pytest.mark.gpu


def column(nz, seed):
    import make_golden as M
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(1, 1, nz, dz, dz, T=300, M=10, C=10, Fe=4000, lambda_f=1.0 / 12.0,
                             lambda_g=1e-6, exf=20.0, uw=0.01)
    f = M.random_fields(p, seed)
    return p, f


def check(a, b, tol):
    vel = max(np.abs(b[k]).max() for k in ("u", "v", "w"))
    for k in O.FIELDS:
        if k in ("ex", "ey"):
            continue  # zero on a column
        s = vel if k in ("u", "v", "w") else np.abs(b[k]).max()
        assert np.abs(a[k] - b[k]).max() < tol * s, (k, np.abs(a[k] - b[k]).max() / s)


@pytest.mark.parametrize("nz", [4, 5, 31, 32, 33, 64, 65, 128, 129, 256, 257])
def test_column_steps_match_oracle(nz):
    p, f = column(nz, nz)
    o = O.Oracle(p)
    o.set_fields(f)
    with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), "fp64") as sim:
        sim.set_fields(f)
        sim.step(2)
        sim.step(1)
        sim.step(20)
        o.step(23)
        check(sim.get_fields(), o.get_fields(), 1e-11)
        d = sim.diagnostics()
    assert d["step"] == 23 and not d["nonfinite"]


@pytest.mark.parametrize("nz", [5, 33, 129])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-11), ("fp32", 1e-5), ("mixed", 1e-2),
                                      ("fp16", 1e-2), ("bf16", 5e-2)])
def test_column_kernel_continues_per_node_steps(nz, prec, tol, tmp_path):
    """Runs that change kernel on the way, one of them through a checkpoint,
    against one on the per-node kernel throughout."""
    p, f = column(nz, 3)
    q = ehd.Params.from_dict(p.as_dict())
    with ehd.Simulation(q, prec, row_kernel=False) as a, ehd.Simulation(q, prec) as b:
        a.set_fields(f)
        a.step(21)
        b.set_fields(f)
        b.step(8)
        b.set_tuning(lbm_kernel=1)
        b.step(3)
        b.set_tuning(lbm_kernel=0)
        b.step(5)
        b.checkpoint(tmp_path / "c")
        b.step(2)
        b.restore(tmp_path / "c")
        b.step(5)
        check(b.get_fields(), a.get_fields(), tol)


def test_batch_of_columns_is_bitwise_lone_columns():
    cases = [column(nz, nz) for nz in (9, 33, 40)]
    ps = [ehd.Params.from_dict(p.as_dict()) for p, _ in cases]
    with ehd.Batch(ps, "fp64") as b:
        for sim, (_, f) in zip(b, cases):
            sim.set_fields(f)
        b.step(1)
        b.step(17)
        got = [sim.get_fields() for sim in b]
    for p, (_, f), g in zip(ps, cases, got):
        with ehd.Simulation(p, "fp64") as sim:
            sim.set_fields(f)
            sim.step(18)
            one = sim.get_fields()
        for k in O.FIELDS:
            assert np.array_equal(one[k], g[k]), k
