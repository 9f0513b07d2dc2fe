"""Who runs the bulk-copy row kernel: lone FP64 contexts, and FP32 and mixed storage in
grouped batch steps (mode 0).  (Lone FP32 and mixed contexts of even nx step node
pairs.)  Graph against direct launches, contexts of different widths side by side, and
the grouped kernels on rows of whole warps and on rows that end inside one, of the
smallest and the largest width.
"""
import numpy as np
import pytest

from conftest import O, ehd, relerr

pytestmark = pytest.mark.gpu


def case(shape, seed, T=200.0):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=T, M=10, C=10, Fe=4000)
    return p, M.random_fields(p, seed)


def to_ehd(p):
    return ehd.Params.from_dict(p.as_dict())


@pytest.mark.parametrize("shape", [(128, 32, 17), (80, 12, 9)])
def test_fp64_rows_graphs_and_direct_launches_agree_bitwise(shape):
    p, f = case(shape, 9)
    out = []
    for graphs in (True, False):
        with ehd.Simulation(to_ehd(p), "fp64", graphs=graphs) as sim:
            sim.set_fields(f)
            sim.step(9)
            sim.step(4)
            out.append(sim.get_fields())
    for k in O.FIELDS:
        assert np.array_equal(out[0][k], out[1][k]), k


def test_fp64_rows_of_different_widths_share_the_kernel():
    """The larger first: the kernel's shared-memory attribute is per function."""
    cases = [case(s, 7) for s in ((128, 16, 9), (64, 16, 9), (96, 10, 6))]
    sims = []
    try:
        for p, f in cases:
            sim = ehd.Simulation(to_ehd(p), "fp64")
            sims.append(sim)
            sim.set_fields(f)
        for _ in range(3):
            for sim in sims:
                sim.step(1)
        for (p, f), sim in zip(cases, sims):
            o = O.Oracle(p)
            o.set_fields(f)
            o.step(3)
            a, b = sim.get_fields(), o.get_fields()
            o.close()
            for k in ("q", "phi", "rho"):
                assert relerr(a[k], b[k]) < 1e-10, (k, relerr(a[k], b[k]))
    finally:
        for sim in sims:
            sim.close()


@pytest.mark.parametrize("shape", [(32, 12, 9), (40, 10, 7), (64, 20, 11), (104, 6, 5), (256, 4, 5)])
@pytest.mark.parametrize("prec", ["fp32", "mixed"])
def test_grouped_rows_are_as_near_the_oracle_as_the_node_kernel(shape, prec):
    """Three instances of one grid in one group.  The same FP32 arithmetic and storage
    rounding as a lone context on the per-node kernel, in another order, so the
    distance from the FP64 oracle is asked to be below twice that context's plus 1e-6."""
    cases = [case(shape, 40 + i, T) for i, T in enumerate((150.0, 200.0, 300.0))]
    with ehd.Batch([to_ehd(p) for p, _ in cases], prec) as b:
        b.set_mode(0)
        for sim, (_, f) in zip(b, cases):
            sim.set_fields(f)
        b.step(5)
        b.step(3)
        group = [sim.get_fields() for sim in b]
    for (p, f), g in zip(cases, group):
        with ehd.Simulation(to_ehd(p), prec, row_kernel=False) as sim:
            sim.set_fields(f)
            sim.step(5)
            sim.step(3)
            a = sim.get_fields()
        o = O.Oracle(p)
        o.set_fields(f)
        o.step(8)
        r = o.get_fields()
        o.close()
        for k in O.FIELDS:
            n = np.linalg.norm(r[k])
            if np.abs(r[k]).max() <= 1e-9:
                continue
            eg, el = np.linalg.norm(g[k] - r[k]) / n, np.linalg.norm(a[k] - r[k]) / n
            assert eg < 2.0 * el + 1e-6, (k, eg, el)
