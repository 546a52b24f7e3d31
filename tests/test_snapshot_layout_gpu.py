"""A binary snapshot names its layout: one of another layout (an older library's, or one
whose length is not this solver's) is refused as not matching, never read; one with room
behind it in its buffer is taken."""
import struct

import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200._lib import FDTDError
from acoustics_b200.solver import PML_WaveSolver
from tests._util import small_scene_with

pytestmark = pytest.mark.gpu

OLD_MAGIC = 0x314E53445446  # the layout before the step constants held the bodies' accelerations


def scene():
    return small_scene_with(S.RigidObject(S.SHAPE_SPHERE, (0.01, 0.0, 0.0), (0.02, 0, 0),
                                          accel_kind=S.ACCEL_GAUSSIAN_PULSATION, accel_amplitude=500.0, accel_t0=1e-4,
                                          accel_tau=4e-5))


@pytest.mark.parametrize("precision", [S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED])
def test_other_layouts_are_refused(fdtd_lib, precision):
    with PML_WaveSolver(scene(), precision=precision) as g:
        g.step(12)
        blob = bytes(g.snapshot())
        y = g.step(10)
        old = struct.pack("<Q", OLD_MAGIC) + blob[8:]
        for bad in (old, old + bytes(512), old[:-256]):
            with pytest.raises(FDTDError, match="does not match"):
                g.restore(bad)
        with pytest.raises(FDTDError, match="truncated"):
            g.restore(blob[:-1])
        g.restore(blob + bytes(64))
        assert np.array_equal(g.step(10), y)


def test_a_snapshot_of_another_scene_of_the_same_cell_count_is_refused(fdtd_lib):
    a, b = scene(), scene()
    b.pml_width = 4.0  # fewer cells in the compact PML arrays: another length
    b.sources.append(S.GaussianSource((0.0, -0.06, 0.0), 1e-4))
    with PML_WaveSolver(a) as g, PML_WaveSolver(b) as k:
        g.step(3)
        k.step(3)
        A, B = bytes(g.snapshot()), bytes(k.snapshot())
        assert len(A) != len(B)
        big, small, into = (A, B, k) if len(A) > len(B) else (B, A, g)
        with pytest.raises(FDTDError):
            into.restore(big)  # longer than this solver's
