"""A batched step's sources added by the interior and ghost kernels, and its advance
beside the field kernels: sources over a body, at the PML's edge, overlapping and
switched off, one to four a member, members of one step to many, every number of x
planes a thread, eager and by graphs, and more members than the interior's
parameter table holds, each member's rows the same bit for bit as its solve on its
own (no tolerance).  And the order of the reduced PML state's shell units (rows
with few z groups outside the z PML in one piece, others in two): the same fields
as the one-launch step."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.batch import SolveBatch
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

P64, P32 = S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED
H = 0.005


def scene(dims, pml=5, sources=1, off=0.0, body=True, seed=0, steps=30):
    rng = np.random.default_rng(seed)
    sc = S.Scene(cell_size=H, divisions=dims, time_step=S.reference_time_step(H), pml_width=pml)
    k = sc.time_step
    if body:
        sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, (0.002, 0.0, -0.001), (0.018, 0, 0),
                                        accel_kind=S.ACCEL_GAUSSIAN_TRANSLATION, accel_amplitude=1e3, accel_t0=12 * k,
                                        accel_tau=4 * k, accel_dir=(0.0, 0.6, 0.8)))
    edge = 0.5 * H * np.asarray(dims) - (pml + 1) * H
    places = [(0.021, 0.003, 0.0), tuple(edge), tuple(-edge), (0.0, -0.02, 0.004)]
    for i in range(sources):
        sc.sources.append(S.GaussianSource(places[i], (4 + i) * k, offset_time=off + 3 * i * k))
    sc.listeners = rng.uniform(-0.4 * H * min(dims), 0.4 * H * min(dims), (3, 3))
    sc.steps = steps
    return sc


def check(scenes, precision, **opt):
    with SolveBatch(scenes, precision=precision, **opt) as b:
        b.run()
        rows = [b.output(m) for m in range(len(scenes))]
    for m, sc in enumerate(scenes):
        with PML_WaveSolver(sc, precision=precision) as g:
            assert np.array_equal(rows[m], g.step(sc.steps)), f"member {m}"
    assert max(np.abs(y).max() for y in rows) > 0


@pytest.mark.parametrize("precision", [P64, P32])
@pytest.mark.parametrize("opt", [dict(x_chunk=2), dict(x_chunk=4, graph_steps=2), dict(x_chunk=8, graph_steps=16),
                                 dict(graph_steps=8, tile_y=16), dict(tile_y=1)], ids=str)
def test_batch_sources_and_advance(fdtd_lib, precision, opt):
    check([scene((30, 31, 33), sources=1, steps=57), scene((41, 28, 37), sources=4, seed=1, steps=1),
           scene((29, 35, 30), sources=2, seed=2, steps=2, body=False), scene((30, 30, 30), sources=0, seed=3, steps=34),
           scene((26, 27, 47), sources=3, off=0.0, seed=4, steps=41, body=False),
           scene((28, 28, 28), sources=1, off=1.0, seed=5, steps=23)], precision, **opt)


@pytest.mark.parametrize("precision", [P64, P32])
def test_more_members_than_the_parameter_table(fdtd_lib, precision):
    scenes = [scene((20 + i % 5, 21, 22 + i % 3), pml=4, sources=i % 3, seed=i, steps=6 + i % 7, body=False)
              for i in range(163)]
    check(scenes, precision, graph_steps=2)


@pytest.mark.parametrize("nz", [92, 103, 104, 105, 106, 107, 121])
@pytest.mark.parametrize("pml", [7, 8, 8.4])
def test_shell_units_in_one_piece_and_two(fdtd_lib, nz, pml):
    sc = scene((27, 29, nz), pml=pml, sources=2)
    out = []
    for opt in (dict(), dict(tile_y=3), dict(tile_y=8), dict(tile_y=64)):
        with PML_WaveSolver(sc, precision=P32, **opt) as g:
            rows = g.step(40)
            out.append([rows, g.field(S.FIELD_PRESSURE), g.field(S.FIELD_PRESSURE_PREV)])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
