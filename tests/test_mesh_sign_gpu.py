"""Mesh bodies whose signed distance changes sign away from the surface (closed and
consistently oriented, so they are accepted, but not the boundary of a solid): one
sphere inside another, two that overlap, a surface turned inside out; and hollow or
several-part bodies with a true inside.  Their flags are those of every cell's own
solid test, as the oracle makes it, flag by flag and face by face (integers: no
tolerance)."""
import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.solver import PML_WaveSolver

pytestmark = pytest.mark.gpu

H = 0.004


def joined(*parts):
    """One mesh of several: (mesh, offset, inside out)."""
    V, T, n = [], [], 0
    for mesh, offset, inward in parts:
        V.append(np.asarray(mesh.vertices) + np.asarray(offset))
        T.append((np.asarray(mesh.triangles)[:, ::-1] if inward else np.asarray(mesh.triangles)) + n)
        n += len(mesh.vertices)
    return S.TriangleMesh(np.vstack(V), np.vstack(T))


BIG, SMALL = S.icosphere(0.056, 3), S.icosphere(0.016, 2)
MESHES = {
    "nested": joined((BIG, (0, 0, 0), False), (SMALL, (0.001, 0, 0), False)),
    "overlapping": joined((S.icosphere(0.04, 2), (-0.012, 0, 0), False), (S.icosphere(0.036, 2), (0.014, 0.002, 0), False)),
    "inside out": joined((S.icosphere(0.03, 2), (0, 0, 0), True)),
    "hollow": joined((BIG, (0, 0, 0), False), (S.icosphere(0.03, 2), (0.001, 0, 0), True)),
    "two parts": joined((S.icosphere(0.02, 2), (-0.03, 0, 0), False), (S.box_mesh((0.012, 0.02, 0.01)), (0.03, 0, 0), False)),
}


@pytest.mark.parametrize("name", sorted(MESHES))
@pytest.mark.parametrize("moving", [False, True])
def test_flags_and_faces_match_the_oracle(oracle_lib, fdtd_lib, name, moving):
    if moving and name == "inside out":
        pytest.skip("the whole grid beside such a body would be fresh cells inside it")
    sc = S.Scene(cell_size=H, divisions=(52, 49, 50), time_step=S.reference_time_step(H), pml_width=6)
    sc.meshes.append(MESHES[name])
    sc.objects.append(S.RigidObject(S.SHAPE_MESH, (0.0012, -0.0007, 0.0004), (0, 0, 0), mesh=0,
                                    motion=S.MOTION_BALLISTIC if moving else S.MOTION_STATIC,
                                    velocity=(25.0, 10.0, 0.0) if moving else (0.0, 0.0, 0.0)))
    sc.sources.append(S.GaussianSource((0.0, 0.07, 0.0), 4e-5))
    sc.listeners = np.array([[0.07, 0.07, 0.06]])
    for precision in (S.PRECISION_FP64, S.PRECISION_FP32_COMPENSATED):
        o = oracle_lib.OracleSolver(sc)
        with PML_WaveSolver(sc, precision=precision) as g:
            for _ in range(2):
                o.step(5)
                g.step(5)
                fo, go = o.classification()
                fg, gg = g.GetGrid()
                assert np.array_equal(fo, fg)
                assert np.array_equal(go, gg)
            assert (fg & S.CELL_BULK == 0).any()
