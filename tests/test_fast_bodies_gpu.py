"""Bodies that jump cells in one time step: the fit of a cell they leave lies as far
beyond it as they went, so the kernels that start before the classification (interior
planes in FP32, the PML shell) must leave those cells alone.  FP32 against the same
solve with its interior in one piece, bit for bit; FP64 against the oracle with the
tolerance of the parity tests.  Launches tell whether planes did start ahead."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver
from tests._util import rel_l2

pytestmark = pytest.mark.gpu

H = 0.004


def track(obj, start, jumps, step):
    """Keyframes a time step apart: obj goes by `jumps` cells (x, y, z) each step."""
    at = np.asarray(start) + H * np.vstack([np.zeros(3), np.cumsum(np.asarray(jumps, dtype=np.float64), axis=0)])
    return S.KeyframeTrack(obj, step, np.hstack([at, np.tile([1.0, 0.0, 0.0, 0.0], (len(at), 1))]))


# body radius in cells, its jump a step in cells, planes ahead of the classification
CASES = {
    "slow": (8.3, (0.3, 0, 0), True),
    "three cells": (8.3, (3, 0, 0), True),
    "eight cells": (8.3, (8, 1, 0), True),
    "eight cells back": (8.3, (-8, 0, 2), True),
    "out of its box": (4.2, (8, 0, 0), False),
    "a plate": (0.6, (1.4, 0, 0), False),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("kind", ["sphere", "mesh"])
def test_planes_ahead_keep_clear_of_the_fits(fdtd_lib, name, kind):
    r, jump, ahead = CASES[name]
    sc = S.Scene(cell_size=H, divisions=(230, 112, 116), time_step=S.reference_time_step(H), pml_width=6)
    steps = 8 if abs(jump[0]) > 2 else 12
    start = (-0.1 * np.sign(jump[0]), 0.01, 0.0)
    if kind == "mesh":
        sc.meshes.append(S.icosphere(r * H, 2) if r > 1 else S.box_mesh((r * H, 9 * H, 9 * H)))
    size = (r * H, 0, 0) if r > 1 else (r * H, 9 * H, 9 * H)
    sc.objects.append(S.RigidObject(S.SHAPE_MESH if kind == "mesh" else S.SHAPE_SPHERE if r > 1 else S.SHAPE_BOX,
                                    start, size, mesh=0, motion=S.MOTION_KEYFRAMED,
                                    accel_kind=S.ACCEL_GAUSSIAN_TRANSLATION, accel_amplitude=800.0, accel_t0=0.0,
                                    accel_tau=20 * sc.time_step, accel_dir=(1.0, 0.0, 0.0)))
    # sound where the fits lie, before the body starts
    sc.sources.append(S.GaussianSource((start[0], 0.0, 0.0), 10 * sc.time_step, width_space=0.1))
    sc.tracks.append(track(0, start, [(0, 0, 0)] * 6 + [jump] * steps, sc.time_step))
    sc.listeners = np.array([[0.3, 0.1, 0.1]])
    out = []
    for x_chunk in (0, 4):
        with PML_WaveSolver(sc, precision=S.PRECISION_FP32_COMPENSATED, x_chunk=x_chunk) as g:
            y = g.step(6)
            ys, launches = [y], []
            for _ in range(steps):
                ys.append(g.step(1))
                launches.append(g.last_launch_count())
            out.append((np.vstack(ys), g.field(S.FIELD_PRESSURE), g.field(S.FIELD_PRESSURE_PREV), launches,
                        g.overlapped_steps()))
    assert np.abs(out[0][1]).max() > 0
    for a, b in zip(out[0][:3], out[1][:3]):
        assert np.array_equal(a, b)
    # one interior launch more where planes started ahead; the sources, added by the
    # interior and ghost kernels, are a kernel of their own in the other solve.  (The
    # first of these steps finds the body where it was.)
    assert [a - b for a, b in zip(out[0][3], out[1][3])] == [0] + [0 if ahead else -1] * (steps - 1)


@pytest.mark.parametrize("jump", [0.4, 2.0, 5.0])
def test_shell_ahead_keeps_clear_of_the_fits(oracle_lib, fdtd_lib, jump):
    """A sphere that comes near the PML and leaves it again by jumps.  (FP64, whose shell
    writes over the p^{n-1} a fit reads; FP32 holds none in the PML, and takes p^n there.)"""
    sc = S.Scene(cell_size=H, divisions=(64, 44, 46), time_step=S.reference_time_step(H), pml_width=6)
    r = 7.2
    # interior faces lie 6 cells from the grid's; the body's far side two to three cells from one of them
    start = np.array([-(32 - 6 - 3.1 - r) * H, 0.0, 0.0])
    n = 6
    sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, start, (r * H, 0, 0), motion=S.MOTION_KEYFRAMED,
                                    accel_kind=S.ACCEL_GAUSSIAN_TRANSLATION, accel_amplitude=800.0, accel_t0=0.0,
                                    accel_tau=20 * sc.time_step, accel_dir=(1.0, 0.0, 0.0)))
    sc.tracks.append(track(0, start, [(0, 0, 0)] * n + [(jump, 0, 0)] * 3 + [(-jump, 0, 0)] * 3 + [(jump, 0, 0)] * 3,
                           sc.time_step))
    sc.sources.append(S.GaussianSource((0.02, 0.06, 0.0), 10 * sc.time_step, width_space=0.1))
    sc.listeners = np.array([[0.09, 0.05, 0.05], [0.0, 0.06, -0.05]])
    o = oracle_lib.OracleSolver(sc)
    with PML_WaveSolver(sc) as g:
        for k in (n, 3, 3, 3):
            yo, yg = o.step(k), g.step(k)
            fo, go = o.classification()
            fg, gg = g.GetGrid()
            assert np.array_equal(fo, fg)
            assert np.array_equal(go, gg)
            assert rel_l2(yg, yo) <= 1e-12
            assert rel_l2(g.field(S.FIELD_PRESSURE), o.field(S.FIELD_PRESSURE)) <= 1e-12
        assert g.overlapped_steps() > 0  # (the resting and the slow steps' shell did start ahead)
