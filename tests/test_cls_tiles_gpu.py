"""Moving analytic bodies against the oracle after every few steps: the one-launch
classification over tiles (flags and ghost faces: integers, no tolerance) and the
interior planes that start before it (listener rows and the pressure field, with
the tolerances of the parity tests): bodies at a corner of the grid, crossing
tiles, overlapping, leaving the PML's edge, below a cell, turned boxes and
ellipsoids, with a constraint, and so large or so many that no plane is apart."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver
from tests._util import rel_l2

pytestmark = pytest.mark.gpu

H = 0.004
TOL = {S.PRECISION_FP64: 1e-12, S.PRECISION_FP32_COMPENSATED: 1e-4}


def ball(c, r, v, shape=S.SHAPE_SPHERE, size=None, rotation=(1, 0, 0, 0, 1, 0, 0, 0, 1)):
    return S.RigidObject(shape, c, size or (r, 0, 0), rotation=rotation,
                         motion=S.MOTION_BALLISTIC if any(v) else S.MOTION_STATIC, velocity=v, gravity=(0, 0, -9.81))


A = np.deg2rad(31.0)
ROT = (np.cos(A), -np.sin(A), 0.0, np.sin(A), np.cos(A), 0.0, 0.0, 0.0, 1.0)
CASES = {
    "one": ((90, 40, 42), [ball((0.01, 0.0, 0.0), 0.02, (70, 20, 5))], False),
    "two apart": ((120, 38, 40), [ball((-0.12, 0.0, 0.0), 0.017, (60, 0, 0)), ball((0.12, 0.004, 0.0), 0.019, (-60, 0, 9))],
                  False),
    "overlapping": ((60, 44, 40), [ball((-0.012, 0.0, 0.0), 0.018, (40, 0, 0)), ball((0.012, 0.006, 0.0), 0.02, (-40, 0, 0)),
                                   ball((0.0, -0.01, 0.008), 0.012, (0, 0, 0))], False),
    "turned kinds": ((70, 44, 46), [ball((-0.06, 0.0, 0.0), 0, (80, 0, 0), S.SHAPE_BOX, (0.013, 0.02, 0.011), ROT),
                                    ball((0.06, 0.0, 0.004), 0, (0, 0, 0), S.SHAPE_ELLIPSOID, (0.02, 0.012, 0.01), ROT)],
                     False),
    "below a cell": ((64, 40, 40), [ball((0.0301, 0.0021, 0.0), 0.0011, (200, 80, 60))], False),
    "constraint": ((80, 40, 44), [ball((0.0, 0.0, 0.0), 0.02, (70, 0, 0))], True),
    "large": ((48, 48, 50), [ball((0.0, 0.0, 0.0), 0.055, (50, 30, 0))], False),
    "into the layer": ((60, 40, 40), [ball((0.07, 0.03, 0.03), 0.015, (180, 90, 90))], False),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_moving_bodies_match_the_oracle(oracle_lib, fdtd_lib, name):
    dims, bodies, constraint = CASES[name]
    sc = S.Scene(cell_size=H, divisions=dims, time_step=S.reference_time_step(H), pml_width=6)
    sc.objects.extend(bodies)
    if constraint:
        sc.constraints.append(S.PlaneConstraint(1, 1, -0.05))
    sc.sources.append(S.GaussianSource((0.0, 0.045, 0.0), 10 * sc.time_step))
    sc.listeners = np.array([[0.02, 0.05, 0.0], [-0.05, 0.045, 0.02], [0.0, -0.04, 0.05]])
    for precision, tol in TOL.items():
        o = oracle_lib.OracleSolver(sc)
        solid = 0
        with PML_WaveSolver(sc, precision=precision) as g:
            for n in (1, 1, 2, 9, 20, 20):
                yo, yg = o.step(n), g.step(n)
                fo, go = o.classification()
                fg, gg = g.GetGrid()
                assert np.array_equal(fo, fg)
                assert np.array_equal(go, gg)
                solid += int((fg & S.CELL_BULK == 0).sum())
            assert solid > 0
            assert np.abs(yo).max() > 0 and rel_l2(yg, yo) <= tol
            po = o.field(S.FIELD_PRESSURE)
            assert rel_l2(g.field(S.FIELD_PRESSURE), po) <= tol


@pytest.mark.parametrize("n_balls", [1, 2])
def test_planes_started_ahead_match_the_phased_order(fdtd_lib, n_balls):
    """A grid large enough that the interior planes out of the bodies' reach start
    before the classification (FP32), against the same solve with an x chunk that
    keeps the interior in one piece: the same bits."""
    sc = S.Scene(cell_size=H, divisions=(210, 120, 124), time_step=S.reference_time_step(H), pml_width=6)
    sc.objects.extend([ball((-0.2, 0.01, 0.0), 0.03, (90, 0, 0)), ball((0.25, 0.0, 0.02), 0.025, (-120, 30, 0))][:n_balls])
    sc.sources.append(S.GaussianSource((-0.1, 0.0, 0.02), 10 * sc.time_step))
    sc.listeners = np.array([[0.0, 0.05, 0.0], [-0.3, 0.1, 0.1]])
    out = []
    for x_chunk in (0, 4):
        with PML_WaveSolver(sc, precision=S.PRECISION_FP32_COMPENSATED, x_chunk=x_chunk) as g:
            out.append([g.step(60), g.field(S.FIELD_PRESSURE), g.field(S.FIELD_PRESSURE_PREV)])
    assert np.abs(out[0][1]).max() > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
