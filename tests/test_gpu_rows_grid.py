"""The row kernel's two ways of placing the injector plane's CTAs (csrc/lbm.cu,
prepare_lbm_rows): with slots of their own beside the row walkers (256 x 16 x 17, 96
x 8 x 9: as many rows a CTA either way) and before walkers that fill every slot (200 x
30 x 17, 128 x 64 x 17: a row less a CTA), more injector rows than slots (256 x 150 x
5), and fewer rows than slots; the FP64 step against the per-node kernel.

The two differ in the order of the FP32 plane sums behind the references alone,
so the tolerance is that of the other comparisons of the two kernels (1e-11).
"""
import numpy as np
import pytest

from conftest import O, ehd, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(256, 16, 17), (96, 8, 9), (200, 30, 17), (128, 64, 17),
                                   (256, 150, 5), (32, 2, 4)])
def test_rows_and_injector_plane_match_the_node_kernel(shape):
    import make_golden as M
    nx, ny, nz = shape
    dz = 1.0 / (nz - 1)
    p = O.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=200, M=10, C=10, Fe=4000)
    f = M.random_fields(p, 29)
    out = []
    for kern in (0, 1):
        with ehd.Simulation(ehd.Params.from_dict(p.as_dict()), "fp64") as sim:
            sim.set_tuning(lbm_kernel=kern)
            sim.set_fields(f)
            sim.step(12)
            out.append(sim.get_fields())
    for k in ("rho", "q", "phi"):
        assert relerr(out[0][k], out[1][k]) < 1e-11, (k, relerr(out[0][k], out[1][k]))
    scale = max(np.abs(out[1][k]).max() for k in ("u", "v", "w"))
    for k in ("u", "v", "w"):
        assert np.abs(out[0][k] - out[1][k]).max() / scale < 1e-11, k
