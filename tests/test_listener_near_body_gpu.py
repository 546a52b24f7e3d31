"""Listeners whose stencil holds ghost cells: their rows read the pressure of the
step before beside the solid, so they must be done before the next step writes
that buffer.  Against the FP64 oracle over many steps, from a single solve (with
and without graphs) and as a batch member; tolerances of the listener parity tests."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.batch import SolveBatch
from acoustics_b200.solver import PML_WaveSolver
from tests._util import rel_l2

pytestmark = pytest.mark.gpu

TOL = {S.PRECISION_FP64: 1e-12, S.PRECISION_FP32_COMPENSATED: 1e-4}


def scene(dims):
    h = 0.005
    sc = S.Scene(cell_size=h, divisions=dims, time_step=S.reference_time_step(h), pml_width=6, steps=160)
    k = sc.time_step
    sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, (0.0, 0.0, 0.0), (0.03, 0, 0),
                                    accel_kind=S.ACCEL_GAUSSIAN_PULSATION, accel_amplitude=1e3, accel_t0=40 * k,
                                    accel_tau=12 * k))
    sc.sources.append(S.GaussianSource((0.0, 0.05, 0.01), 16 * k))
    r = 0.0355
    sc.listeners = np.array([[r, 0.001, 0.001], [-0.6 * r, 0.8 * r, 0.0], [0.001, -0.7 * r, 0.72 * r], [0.05, 0.05, 0.0]])
    return sc


@pytest.mark.parametrize("precision", sorted(TOL))
@pytest.mark.parametrize("dims", [(40, 42, 44), (72, 80, 76)])
def test_rows_beside_a_body_match_the_oracle(oracle_lib, fdtd_lib, precision, dims):
    sc = scene(dims)
    yo = oracle_lib.OracleSolver(sc).step(sc.steps)
    for graph_steps in (0, 16):
        with PML_WaveSolver(sc, precision=precision, graph_steps=graph_steps) as g:
            y = g.step(sc.steps)
        assert rel_l2(y, yo) <= TOL[precision], graph_steps
        for li in range(sc.n_listeners):
            assert rel_l2(y[:, li], yo[:, li]) <= 10 * TOL[precision], (graph_steps, li)
    with SolveBatch([sc, scene((48, 40, 44))], precision=precision, graph_steps=16, x_chunk=2, tile_y=8) as b:
        b.run()
        assert np.array_equal(b.output(0), y)
