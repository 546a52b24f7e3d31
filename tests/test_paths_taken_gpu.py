"""Which kernels a step takes, by its launches: the comparisons of one path with another
elsewhere mean something only while their two sides take different ones.  One launch a
step up to the limit on cells, several past it or with explicit shapes; one kernel less
where the interior and ghost kernels add the sources."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

H = 0.005
P64, P32 = S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED


def scene(dims, moving=False, constraint_in_pml=False):
    sc = S.Scene(cell_size=H, divisions=dims, time_step=S.reference_time_step(H), pml_width=6)
    sc.objects.append(S.RigidObject(S.SHAPE_SPHERE, (0.002, 0.0, -0.001), (0.022, 0, 0),
                                    motion=S.MOTION_BALLISTIC if moving else S.MOTION_STATIC,
                                    velocity=(20.0, 0.0, 0.0) if moving else (0.0, 0.0, 0.0)))
    if constraint_in_pml:
        sc.constraints.append(S.PlaneConstraint(1, 1, -0.06))
    sc.sources.append(S.GaussianSource((0.03, 0.005, 0.0), 6 * sc.time_step))
    return sc


def launches(sc, precision, **opt):
    """Launches of one step after the first ones (no listeners)."""
    with PML_WaveSolver(sc, precision=precision, **opt) as g:
        g.step(3)
        g.step(5)
        n = g.last_launch_count()
        assert n % 5 == 0
        return n // 5


# (cells on either side of the limits: 1.0 M in FP64, 1.6 M in FP32)
@pytest.mark.parametrize("precision,below,above", [(P64, (98, 100, 102), (101, 100, 102)),
                                                   (P32, (116, 117, 117), (117, 117, 118))])
def test_one_launch_up_to_the_limit(fdtd_lib, precision, below, above):
    assert launches(scene(below), precision) == 1
    assert launches(scene(above), precision) == 3  # ghost cells, interior, shell
    for opt in (dict(tile_y=8), dict(x_chunk=2), dict(tile_y=8, x_chunk=2)):
        assert launches(scene(below), precision, **opt) == 3
    assert launches(scene((44, 45, 46), constraint_in_pml=True), precision) > 1


@pytest.mark.parametrize("precision", [P64, P32])
@pytest.mark.parametrize("moving", [False, True])
def test_sources_take_a_launch_of_their_own_with_an_explicit_chunk(fdtd_lib, precision, moving):
    sc = scene((46, 45, 44), moving)
    fused, apart = (launches(sc, precision, tile_y=8, x_chunk=x) for x in (2, 4))
    assert apart == fused + 1
