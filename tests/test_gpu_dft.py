"""The folded transforms and the two-sided z solve (csrc/dft.cu) against the
oracle's odd-extension DFT solve, at the sizes where their tiles change: one
point, the smallest odd and even widths, 64 and 65 folded values (126, 127,
130 points: one and two tiles of outputs), the last widths they may serve and
the first beyond them (run-time radix passes), widths on either side of the
choice between the two (360, 400, 500), even and odd numbers of interior
planes, and a depth whose columns need 16 modes a block.

Tolerances are those of the other Poisson tests (1e-10 FP64, 2e-6 FP32 of the
largest value): a folded sum of K <= 513 terms has a rounding error of about
0.2 sqrt(K) units (2.7e-7 at K = 513) relative to its rms, as the FFT's few
units are.
"""
import numpy as np
import pytest

from conftest import O, ehd, relerr

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 5), (2, 3, 6), (3, 2, 4), (126, 7, 6), (127, 5, 7), (130, 6, 5), (7, 126, 6),
          (5, 127, 7), (6, 130, 5), (1023, 3, 4), (3, 1024, 5), (1025, 2, 4), (2, 1025, 4),
          (64, 10, 12), (10, 64, 12), (4, 6, 700),
          (360, 4, 5), (4, 400, 6), (500, 3, 6)]


def case(shape, seed):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000)
    return p, M.random_fields(p, seed)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 2e-6)])
def test_poisson_matches_oracle(shape, prec, tol):
    p, f = case(shape, 8)
    o = O.Oracle(p)
    o.set_fields(f)
    o.poisson()
    o.efield()
    b = o.get_fields()
    o.close()
    with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), prec) as sim:
        sim.set_fields(f)
        sim.poisson()
        a = sim.get_fields()
    e = max(np.abs(b[k]).max() for k in ("ex", "ey", "ez"))
    assert relerr(a["phi"], b["phi"]) < tol, relerr(a["phi"], b["phi"])
    for k in ("ex", "ey", "ez"):
        assert np.abs(a[k] - b[k]).max() < tol * e, (k, np.abs(a[k] - b[k]).max() / e)


def test_group_launch_agrees_with_lone_contexts():
    """Grouped batch steps (one launch over the instances, blockIdx.z) on
    grids whose axes are both, or only one of them, folded."""
    cases = [case(s, 20 + i) for i, s in enumerate([(30, 25, 7), (30, 25, 7), (64, 22, 9),
                                                    (64, 22, 9), (22, 48, 9), (22, 48, 9)])]
    ps = [ehd.Params.from_dict(p.as_dict()) for p, _ in cases]
    with ehd.Batch(ps, "fp64") as b:
        b.set_mode(0)
        for sim, (_, f) in zip(b, cases):
            sim.set_fields(f)
        b.step(6)
        got = [sim.get_fields() for sim in b]
    for p, (_, f), g in zip(ps, cases, got):
        with ehd.Simulation(p, "fp64") as sim:
            sim.set_fields(f)
            sim.step(6)
            one = sim.get_fields()
        for k in O.FIELDS:
            assert relerr(g[k], one[k]) < 1e-11, (k, relerr(g[k], one[k]))
