"""Cells a body leaves by jumps of cells: where the whole stencil of a cell's fit was
solid too, it takes its neighbour's value, and that neighbour may be such a cell itself.
FP64 against the oracle, which goes over the cells one after the other, and FP32 too,
with the tolerances of the parity tests; FP32 twice, bit for bit."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver
from tests._util import rel_l2

pytestmark = pytest.mark.gpu

H = 0.004
BALL, PLATE = (S.SHAPE_SPHERE, (5.2 * H, 0, 0)), (S.SHAPE_BOX, (0.7 * H, 5.1 * H, 4.2 * H))
# (shape and size, start in cells, jump a step in cells) of each body
CASES = {
    "a cell and a half": [(BALL, (-3, 0, 0), (1.5, 0, 0))],
    "three cells": [(BALL, (-3.2, 0.3, 0), (3, 0, 0))],
    "three cells back": [(BALL, (3.2, 0.3, 0), (-3, 0, 0))],
    "five cells aslant": [(BALL, (0, -2, -2), (2.5, 2.5, 3))],
    "down": [(BALL, (0.1, 0.2, 3), (0, 0, -4))],
    "a plate": [(PLATE, (-2, 0, 0), (1.2, 0, 0))],
    "two": [(BALL, (-6, 0, 0), (2, 0, 0)), (BALL, (7, 1, 0), (0, -3, 0))],
    "a mesh": [("mesh", (-3, 0, 0), (3, 0, 1))],
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_values_of_left_cells(oracle_lib, fdtd_lib, name):
    sc = S.Scene(cell_size=H, divisions=(64, 60, 60), time_step=S.reference_time_step(H), pml_width=6)
    n, k = 8, sc.time_step
    for i, (shape, start, jump) in enumerate(CASES[name]):
        if shape == "mesh":
            sc.meshes.append(S.icosphere(5.2 * H, 2))
            shape = (S.SHAPE_MESH, (0, 0, 0))
        at = H * (np.asarray(start, dtype=float) + np.outer([0] * n + [1, 2, 1, 0, 1, 2], jump))
        sc.objects.append(S.RigidObject(shape[0], at[0], shape[1], mesh=0, motion=S.MOTION_KEYFRAMED,
                                        accel_kind=S.ACCEL_GAUSSIAN_TRANSLATION, accel_amplitude=800.0, accel_t0=0.0,
                                        accel_tau=20 * k, accel_dir=(0.6, 0.8, 0.0)))
        sc.tracks.append(S.KeyframeTrack(i, k, np.hstack([at, np.tile([1.0, 0.0, 0.0, 0.0], (len(at), 1))])))
    sc.sources.append(S.GaussianSource((0.0, 0.05, 0.01), 10 * k, width_space=0.1))
    sc.listeners = np.array([[0.07, 0.05, 0.05], [0.0, 0.06, -0.05]])
    for precision, tol in ((S.PRECISION_FP64, 1e-12), (S.PRECISION_FP32_COMPENSATED, 1e-4)):
        o, fields = oracle_lib.OracleSolver(sc), []
        yo = [o.step(m) for m in (n, 1, 1, 1, 3)]
        for _ in range(1 if precision == S.PRECISION_FP64 else 2):
            with PML_WaveSolver(sc, precision=precision) as g:
                for m, want in zip((n, 1, 1, 1, 3), yo):
                    assert rel_l2(g.step(m), want) <= tol
                fo, go = o.classification()
                fg, gg = g.GetGrid()
                assert np.array_equal(fo, fg)
                assert np.array_equal(go, gg)
                fields.append((g.field(S.FIELD_PRESSURE), g.field(S.FIELD_PRESSURE_PREV)))
        po = o.field(S.FIELD_PRESSURE)
        assert np.abs(po).max() > 0
        assert rel_l2(fields[0][0], po) <= tol
        for a, b in zip(*(fields * 2)[:2]):
            assert np.array_equal(a, b)
