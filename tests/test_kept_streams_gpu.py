"""Streams and pinned buffers of closed solvers serve the next ones: solves made and
closed one after another, side by side in threads, of both stream priorities (moving
bodies and static), of staging buffers that grow and shrink, with batches between and
the kept ones given back in the middle, each the same bit for bit as the first of its
scene (no tolerance)."""
import threading

import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200._lib import load
from acoustics_b200.batch import SolveBatch
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

H = 0.005


def scene(dims, listeners, moving):
    rng = np.random.default_rng(listeners)
    sc = S.Scene(cell_size=H, divisions=dims, time_step=S.reference_time_step(H), pml_width=6)
    k = sc.time_step
    sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, (0.001, 0.0, 0.002), (0.02, 0, 0), accel_kind=S.ACCEL_GAUSSIAN_PULSATION,
                                    accel_amplitude=500.0, accel_t0=10 * k, accel_tau=4 * k,
                                    motion=S.MOTION_BALLISTIC if moving else S.MOTION_STATIC,
                                    velocity=(30.0, 0.0, 0.0) if moving else (0.0, 0.0, 0.0)))
    sc.sources.append(S.GaussianSource((0.03, 0.02, 0.0), 6 * k))
    sc.listeners = rng.uniform(-0.04, 0.04, (listeners, 3))
    sc.steps = 30
    return sc


SCENES = [scene((40, 38, 41), 3, False), scene((38, 40, 39), 200, True), scene((41, 41, 40), 60, False),
          scene((40, 40, 37), 1, True)]


def solve(sc, precision):
    with PML_WaveSolver(sc, precision=precision) as g:
        one = g.step(7)
        g.stepSystem()
        row = g.FetchPressureData().copy()
        return [one, row, g.step(20), g.field(S.FIELD_PRESSURE)]


@pytest.mark.parametrize("precision", [S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED])
def test_solves_by_kept_streams(fdtd_lib, precision):
    load().fdtd_release_cached_memory(-1)
    want = [solve(sc, precision) for sc in SCENES]
    wrong = []

    def work(first):
        for i in range(6):
            m = (first + i) % len(SCENES)
            got = solve(SCENES[m], precision)
            if not all(np.array_equal(a, b) for a, b in zip(got, want[m])):
                wrong.append(m)
            if first == 0 and i == 2:
                load().fdtd_release_cached_memory(0)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for _ in range(2):
        with SolveBatch([SCENES[0], SCENES[2]], precision=precision, graph_steps=4) as b:
            b.run()
            rows = [b.output(0), b.output(1)]
        for m, y in zip((0, 2), rows):
            assert np.array_equal(y[:7], want[m][0])
        assert all(np.array_equal(a, b) for a, b in zip(solve(SCENES[1], precision), want[1]))
    load().fdtd_release_cached_memory(-1)
    assert all(np.array_equal(a, b) for a, b in zip(solve(SCENES[3], precision), want[3]))
