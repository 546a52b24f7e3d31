"""The warp-per-brick solid test of scenes with mesh bodies against the oracle,
flag by flag and ghost face by ghost face: bodies smaller than a cell, boxes of
every remainder of the 2 x 4 x 4 bricks, bricks deep inside a body, several
bodies and a constraint in one brick, and a body whose every triangle is about
equally far from a cell (integers: no tolerance)."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

H = 0.004


def scene(bodies, constraint=False):
    sc = S.Scene(cell_size=H, divisions=(44, 46, 50), time_step=S.reference_time_step(H), pml_width=6)
    for mesh, center, velocity in bodies:
        moving = any(velocity)
        if isinstance(mesh, S.TriangleMesh):
            sc.meshes.append(mesh)
            sc.objects.append(S.RigidObject(S.SHAPE_MESH, center, (0, 0, 0), mesh=len(sc.meshes) - 1,
                                            motion=S.MOTION_BALLISTIC if moving else S.MOTION_STATIC, velocity=velocity))
        else:
            shape, size = mesh
            sc.objects.append(S.RigidObject(shape, center, size,
                                            motion=S.MOTION_BALLISTIC if moving else S.MOTION_STATIC, velocity=velocity))
    if constraint:
        sc.constraints.append(S.PlaneConstraint(1, 1, -0.06))
    sc.sources.append(S.GaussianSource((0.0, 0.05, 0.0), 4e-5))
    sc.listeners = np.array([[0.05, 0.05, 0.05]])
    return sc


REST = (0.0, 0.0, 0.0)
CASES = {
    "centred sphere": [(S.icosphere(0.0401, 3), (0.002, 0.002, 0.002), REST)],
    "below a cell": [(S.icosphere(0.0013, 1), (0.0021, 0.0019, 0.0001), REST),
                     (S.icosphere(0.0006, 0), (0.002, -0.018, 0.006), REST)],
    "thin plate": [(S.box_mesh((0.03, 0.0007, 0.022)), (0.001, 0.0005, -0.0005), REST)],
    "remainders": [(S.box_mesh((0.0101, 0.0143, 0.0062)), (-0.03, -0.002, 0.003), REST),
                   (S.icosphere(0.0177, 2), (0.024, 0.003, -0.004), REST)],
    "touching kinds": [(S.icosphere(0.016, 2), (-0.014, 0.0, 0.0), REST),
                       ((S.SHAPE_ELLIPSOID, (0.02, 0.011, 0.009)), (0.0195, 0.0, 0.001), REST),
                       ((S.SHAPE_BOX, (0.008, 0.012, 0.01)), (0.0, -0.028, 0.0), REST)],
    "moving": [(S.icosphere(0.015, 2), (-0.02, 0.001, 0.0), (90.0, 10.0, 0.0)),
               (S.box_mesh((0.009, 0.011, 0.008)), (0.022, 0.0, 0.002), (-80.0, 0.0, 20.0))],
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("constraint", [False, True])
def test_mesh_flags_and_faces_match_the_oracle(oracle_lib, fdtd_lib, name, constraint):
    sc = scene(CASES[name], constraint)
    o = oracle_lib.OracleSolver(sc)
    for precision in (S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED):
        with PML_WaveSolver(sc, precision=precision) as g:
            o = oracle_lib.OracleSolver(sc)
            for _ in range(3):
                o.step(7)
                g.step(7)
                fo, go = o.classification()
                fg, gg = g.GetGrid()
                assert np.array_equal(fo, fg)
                assert np.array_equal(go, gg)
            assert (fg & S.CELL_BULK == 0).any()
