"""FULLY_COUPLED systems of every size class of the cluster solve (one, two and
four rows a thread, and the one-CTA kernels past its limit) against the oracle,
with the tolerances of test_coupled_gpu.py; the one-launch and the region-split
step of the same scene give the same rows."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver
from tests._util import rel_l2

pytestmark = pytest.mark.gpu

TOL = {S.PRECISION_FP64: 1e-11, S.PRECISION_FP32_COMPENSATED: 1e-4}


def scene(r, n):
    h = 0.005
    sc = S.Scene(cell_size=h, divisions=(n, n + 1, n + 2), time_step=S.reference_time_step(h), pml_width=6)
    k = sc.time_step
    sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, (0.001, -0.0012, 0.0007), (r * h, 0, 0),
                                    accel_kind=S.ACCEL_GAUSSIAN_PULSATION, accel_amplitude=1e3, accel_t0=9 * k,
                                    accel_tau=3 * k))
    sc.objects.append(S.RigidObject(S.SHAPE_BOX, (0.0, 0.0, (r + 5.5) * h), (2.2 * h, 2.6 * h, 1.4 * h)))
    sc.sources.append(S.GaussianSource((0.0, (r + 3) * h, 0.0), 6 * k))
    sc.listeners = np.array([[(r + 4) * h, 0.0, 0.0], [0.0, -(r + 5) * h, 0.003]])
    sc.boundary_handling = S.BOUNDARY_FULLY_COUPLED
    return sc


@pytest.mark.parametrize("r,n,rows", [(3, 38, (1, 1000)), (13, 60, (2048, 4096)), (16, 66, (4097, 8192)),
                                      (22, 78, (8193, 16384)), (30, 94, (16385, 40000))])
def test_every_size_matches_the_oracle(oracle_lib, fdtd_lib, r, n, rows):
    sc = scene(r, n)
    yo = oracle_lib.OracleSolver(sc).step(24)
    assert np.abs(yo).max() > 0
    for precision, tol in TOL.items():
        with PML_WaveSolver(sc, precision=precision) as g:
            y = g.step(24)
            info = g.boundary_info()
        assert rows[0] <= info["rows"] <= rows[1] and info["iterations"] > 0
        assert rel_l2(y, yo) <= tol
        with PML_WaveSolver(sc, precision=precision, tile_y=8, graph_steps=8) as g:
            assert np.array_equal(g.step(24), y)
