"""The one-launch step of small static solves against the region-split kernels
(asked for by an explicit shell shape): the same expressions, so rows and every
field the same bit for bit (no tolerance).  Grids with every remainder of the
tiles, PML widths down to two cells and with a fraction, no interior at all,
zero to four sources (also switched off and beside a body), bodies of each
acceleration, a constraint, no listeners, air absorption, the full and the reduced
PML state, chunk lengths that cut graphs, and a snapshot in the middle."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200._lib import FDTDError
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

P64, P32 = S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED
H = 0.005


def scene(dims=(40, 41, 43), pml=6, bodies=1, sources=1, listeners=5, alpha=0.0, constraint=False, off=0.0, seed=0):
    rng = np.random.default_rng(seed)
    sc = S.Scene(cell_size=H, divisions=dims, time_step=S.reference_time_step(H), pml_width=pml, air_viscosity_alpha=alpha)
    k = sc.time_step
    kinds = [(S.SHAPE_SPHERE, (0.021, 0, 0), S.ACCEL_GAUSSIAN_PULSATION), (S.SHAPE_BOX, (0.012, 0.009, 0.02),
             S.ACCEL_GAUSSIAN_TRANSLATION), (S.SHAPE_ELLIPSOID, (0.02, 0.01, 0.012), S.ACCEL_NONE)]
    places = [(0.001, 0.002, -0.003), (0.03, -0.025, 0.01), (-0.035, 0.03, 0.004)]
    for (shape, size, accel), c in list(zip(kinds, places))[:bodies]:
        sc.objects.append(S.RigidObject(shape, c, size, accel_kind=accel, accel_amplitude=900.0, accel_t0=30 * k,
                                        accel_tau=9 * k, accel_dir=(0.6, 0.0, 0.8)))
    for i in range(sources):
        sc.sources.append(S.GaussianSource(tuple(rng.uniform(-0.03, 0.03, 3)), (8 + 3 * i) * k,
                                           offset_time=off + 5 * i * k))
    if constraint:
        sc.constraints.append(S.PlaneConstraint(2, 1, -0.045))
    half = 0.5 * H * np.asarray(dims) - H
    sc.listeners = rng.uniform(-half, half, (listeners, 3)) if listeners else None
    return sc


def fields(g):
    which = [S.FIELD_PRESSURE, S.FIELD_PRESSURE_PREV]
    if g.pml_state() == S.PML_STATE_FULL:
        which += [S.FIELD_PML_PX, S.FIELD_PML_PY, S.FIELD_PML_PZ, S.FIELD_VX, S.FIELD_VY, S.FIELD_VZ]
    return [g.field(w) for w in which]


CASES = {
    "odd": {}, "tiny": dict(dims=(17, 13, 15), pml=2, bodies=0), "row of one": dict(dims=(9, 40, 9), pml=4, bodies=0),
    "fraction": dict(dims=(31, 29, 37), pml=3.4, bodies=1), "no interior": dict(dims=(20, 22, 21), pml=11, bodies=0),
    "long z": dict(dims=(20, 19, 157), pml=6, bodies=0), "long x": dict(dims=(151, 18, 22), pml=5, bodies=0),
    "no source": dict(sources=0), "four sources": dict(sources=4), "source off": dict(off=1.0),
    "three bodies": dict(dims=(44, 45, 46), bodies=3), "air": dict(alpha=2e-6, bodies=2), "silent": dict(listeners=0),
    "many listeners": dict(listeners=67), "constraint": dict(constraint=True, bodies=2),
    "wide": dict(dims=(64, 66, 150), pml=8, bodies=3, sources=2),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("precision,state", [(P64, S.PML_STATE_AUTO), (P32, S.PML_STATE_AUTO), (P32, S.PML_STATE_FULL)])
def test_one_launch_equals_the_region_split_step(fdtd_lib, name, precision, state):
    sc = scene(**CASES[name])
    with PML_WaveSolver(sc, precision=precision, pml_state=state, tile_y=8) as g:
        want = [g.step(n) for n in (1, 2, 33, 40)]
        end = fields(g)
    for graph_steps in (0, 16):
        with PML_WaveSolver(sc, precision=precision, pml_state=state, graph_steps=graph_steps) as g:
            got = [g.step(n) for n in (1, 2, 33, 40)]
            for a, b in zip(got + fields(g), want + end):
                assert np.array_equal(a, b)
    # (the sources of the two grids without updated cells in reach are silent: see the next test)
    if sc.n_listeners and name not in ("source off", "no interior", "row of one"):
        assert max(np.abs(y).max() for y in want) > 0


@pytest.mark.parametrize("name", ["no interior", "row of one", "tiny", "long x"])
@pytest.mark.parametrize("precision,state", [(P64, S.PML_STATE_AUTO), (P32, S.PML_STATE_AUTO), (P32, S.PML_STATE_FULL)])
def test_one_launch_from_random_fields(fdtd_lib, name, precision, state):
    sc = scene(**CASES[name])
    rng = np.random.default_rng(7)
    p = rng.normal(size=sc.n_cells)
    out = []
    for tile_y in (8, 0):
        with PML_WaveSolver(sc, precision=precision, pml_state=state, tile_y=tile_y) as g:
            g.step(1)
            g.set_field(S.FIELD_PRESSURE, p)
            g.set_field(S.FIELD_PRESSURE_PREV, 0.9 * p)
            if g.pml_state() == S.PML_STATE_FULL:
                for w in (S.FIELD_PML_PX, S.FIELD_PML_PY, S.FIELD_PML_PZ):
                    g.set_field(w, p / 3.0)
            out.append([g.step(23)] + fields(g))
    assert np.abs(out[0][0]).max() > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_one_launch_continues_from_a_snapshot(fdtd_lib):
    sc = scene(bodies=2, sources=2)
    for precision in (P64, P32):
        with PML_WaveSolver(sc, precision=precision) as g:
            g.step(21)
            blob = g.snapshot()
            rows = g.step(30)
            end = fields(g)
        with PML_WaveSolver(sc, precision=precision) as g:
            g.restore(blob)
            assert np.array_equal(g.step(30), rows)
            for a, b in zip(fields(g), end):
                assert np.array_equal(a, b)
            g.Reinitialize_PML_WaveSolver(0.0)
            g.step(21)
            assert np.array_equal(g.step(30), rows)


@pytest.mark.parametrize("precision", [P64, P32])
def test_a_cell_that_is_not_finite_gives_the_same_rows_and_status(fdtd_lib, precision):
    """One NaN near a listener: the fit leaves the cell out, until it has spread."""
    sc = scene(bodies=0, listeners=3)
    out = []
    for tile_y in (0, 8):
        with PML_WaveSolver(sc, precision=precision, tile_y=tile_y) as g:
            g.step(12)
            p = g.field(S.FIELD_PRESSURE).reshape(sc.divisions)
            i = [int((sc.listeners[0][d] + 0.5 * H * sc.divisions[d]) / H - 0.5) for d in range(3)]
            p[tuple(i)] = np.nan
            g.set_field(S.FIELD_PRESSURE, p)
            log = []
            for _ in range(6):
                try:
                    log.append((0, g.step(1)))
                except FDTDError as e:
                    log.append((e.status, None))
            log.append((0, g.field(S.FIELD_PRESSURE)))
            out.append(log)
    for (sa, a), (sb, b) in zip(*out):
        assert sa == sb
        assert a is None or np.array_equal(a, b, equal_nan=True)
