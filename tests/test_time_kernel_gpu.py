"""The profiling hook times what a step runs: the ghost list of a moving scene (kept per
parity) is the one of the last classification in every launch, and a solve that steps in
one launch is timed by that launch (its region-split shell alone takes about three times
as long)."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

H = 0.004


@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("steps", [6, 7])
def test_ghost_list_launches_work_on_the_list(fdtd_lib, mesh, steps):
    sc = S.Scene(cell_size=H, divisions=(48, 44, 46), time_step=S.reference_time_step(H), pml_width=6)
    shape = dict(shape=S.SHAPE_MESH, size=(0, 0, 0), mesh=0) if mesh else dict(shape=S.SHAPE_SPHERE, size=(0.02, 0, 0))
    if mesh:
        sc.meshes.append(S.icosphere(0.02, 2))
    sc.objects.append(S.RigidObject(center=(0.001, 0.0, 0.0), motion=S.MOTION_BALLISTIC, velocity=(20.0, 0.0, 0.0),
                                    **shape))
    sc.sources.append(S.GaussianSource((0.02, 0.0, 0.0), 4e-5, width_space=0.2))
    with PML_WaveSolver(sc, precision=S.PRECISION_FP32_COMPENSATED) as g:
        g.step(steps)
        flags, faces = g.GetGrid()
        # the increment, which every launch adds to (FP64's two replays of one launch undo
        # one another); the source is wide, so the field is flat nowhere
        before = g.field(S.FIELD_PRESSURE_PREV)
        g.time_kernel(3, 1)
        changed = g.field(S.FIELD_PRESSURE_PREV) != before
        listed = np.unique(faces["neighbour_cell"])
        listed = listed[flags.ravel()[listed] & S.CELL_PML == 0]
        assert len(listed) > 100
        assert changed.ravel()[listed].mean() > 0.9
        assert not np.delete(changed.ravel(), listed).any()


@pytest.mark.parametrize("precision", [S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED])
def test_step_kernels_of_a_one_launch_solve(fdtd_lib, precision):
    sc = S.Scene(cell_size=H, divisions=(64, 64, 64), time_step=S.reference_time_step(H), pml_width=8)
    sc.sources.append(S.GaussianSource((0.0, 0.0, 0.0), 4e-5))
    with PML_WaveSolver(sc, precision=precision) as g:
        g.step(4)
        assert g.last_launch_count() <= 8  # (one a step, and the first step's tables)
        step, shell = (min(g.time_kernel(w, 64) for _ in range(5)) for w in (0, 2))
        assert step < shell
