"""Sources added by the interior and ghost kernels (the default) against the kernel
that adds them afterwards (asked for by x_chunk = 4, which keeps it): the same bits,
with one to four sources, beside a body, at the PML's edge, switched off, with air
absorption, and beside a moving body; and the shell's planes per thread that the
size chooses against eight."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

H = 0.005
CASES = {"one": dict(), "four": dict(sources=4), "air": dict(alpha=2e-6), "off": dict(off=2.0), "moving": dict(moving=True),
         "no body": dict(body=False), "two thirds of two waves": dict(dims=(150, 124, 122)),
         "three waves": dict(dims=(200, 190, 210))}


def scene(dims=(45, 46, 47), sources=1, alpha=0.0, off=0.0, moving=False, body=True):
    rng = np.random.default_rng(5)
    sc = S.Scene(cell_size=H, divisions=dims, time_step=S.reference_time_step(H), pml_width=8, air_viscosity_alpha=alpha)
    k = sc.time_step
    if body:
        sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, (0.002, 0.0, -0.001), (0.022, 0, 0),
                                        accel_kind=S.ACCEL_GAUSSIAN_TRANSLATION, accel_amplitude=1e3, accel_t0=20 * k,
                                        accel_tau=6 * k, motion=S.MOTION_BALLISTIC if moving else S.MOTION_STATIC,
                                        velocity=(60.0, 0.0, 20.0) if moving else (0.0, 0.0, 0.0)))
    edge = 0.5 * H * np.asarray(dims) - 9 * H
    places = [(0.03, 0.005, 0.0), tuple(edge), tuple(-edge), (0.0, -0.028, 0.01)]
    for i in range(sources):
        sc.sources.append(S.GaussianSource(places[i], (6 + i) * k, offset_time=off + 4 * i * k))
    sc.listeners = rng.uniform(-0.05, 0.05, (4, 3))
    return sc


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("precision", [S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED])
def test_fused_sources_equal_the_source_kernel(fdtd_lib, name, precision):
    sc = scene(**CASES[name])
    out = []
    # an explicit shell shape keeps small grids on the region-split step
    for opt in (dict(tile_y=8, x_chunk=4), dict(tile_y=8), dict(tile_y=8, graph_steps=8), dict()):
        with PML_WaveSolver(sc, precision=precision, **opt) as g:
            rows = g.step(45)
            out.append([rows, g.field(S.FIELD_PRESSURE), g.field(S.FIELD_PRESSURE_PREV)])
    assert np.abs(out[0][1]).max() > 0 or name == "off"
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
