"""Read-backs through pinned buffers that solves share: fields, slices and single cells of
several solves read at the same time by as many threads, again after solves are closed
and the kept buffers given back, equal the values read one at a time (bit for bit)."""
import threading

import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200._lib import load
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

H = 0.005


def solve(n, precision):
    sc = S.Scene(cell_size=H, divisions=(n, n - 3, n + 2), time_step=S.reference_time_step(H), pml_width=6)
    sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, (0.001, 0.0, 0.002), (0.02, 0, 0)))
    sc.sources.append(S.GaussianSource((0.05, 0.02, 0.0), 5e-5, width_space=0.05))
    g = PML_WaveSolver(sc, precision=precision)
    g.step(5, record=False)
    return g


def view(g):
    n = g.n_cells
    return [g.FetchCell(n // 2).tobytes(), g.field(S.FIELD_PRESSURE).tobytes(), g.SampleAxisAlignedSlice(1, 0.0).tobytes(),
            g.FetchCell(n // 3).tobytes(), g.field(S.FIELD_PRESSURE_PREV).tobytes()]


def test_views_of_several_solves_at_once(fdtd_lib):
    solves = [solve(n, p) for n, p in ((40, 0), (44, 1), (61, 0), (97, 1), (33, 0), (72, 1))]
    want = [view(g) for g in solves]
    assert len(set(w[1] for w in want)) == len(want)
    wrong = []

    def reader(i):
        for _ in range(12):
            if view(solves[i]) != want[i]:
                wrong.append(i)

    for round_ in range(3):
        threads = [threading.Thread(target=reader, args=(i,)) for i in range(len(solves))]
        for t in threads:
            t.start()
        if round_ == 1:
            for _ in range(20):
                load().fdtd_release_cached_memory(-1)
        for t in threads:
            t.join()
        assert not wrong
    for g in solves[:3]:
        g.close()
    load().fdtd_release_cached_memory(-1)
    assert [view(g) for g in solves[3:]] == want[3:]
    for g in solves[3:]:
        g.close()
