"""Which meshes bound a solid, so that the sign of their distance changes at the surface
only: the classification's short cuts rest on it.  Known shapes, turned and moved; and
wherever the answer is yes, random points have the sign of their winding number."""
import ctypes as C

import numpy as np
import pytest

from acoustics_b200 import scene as S


def joined(*parts):
    """One mesh of several: (mesh, offset, inside out)."""
    V, T, n = [], [], 0
    for mesh, offset, inward in parts:
        V.append(np.asarray(mesh.vertices) + np.asarray(offset))
        T.append((np.asarray(mesh.triangles)[:, ::-1] if inward else np.asarray(mesh.triangles)) + n)
        n += len(mesh.vertices)
    return S.TriangleMesh(np.vstack(V), np.vstack(T))


def torus(R=0.03, r=0.01, n=24, m=12):
    u, v = np.meshgrid(np.arange(n), np.arange(m), indexing="ij")
    a, b = 2 * np.pi * u / n, 2 * np.pi * v / m
    V = np.stack([(R + r * np.cos(b)) * np.cos(a), (R + r * np.cos(b)) * np.sin(a), r * np.sin(b)], -1).reshape(-1, 3)
    at = lambda i, j: (i % n) * m + j % m  # noqa: E731
    T = []
    for i in range(n):
        for j in range(m):
            T += [(at(i, j), at(i + 1, j), at(i + 1, j + 1)), (at(i, j), at(i + 1, j + 1), at(i, j + 1))]
    return S.TriangleMesh(V, np.asarray(T, dtype=np.int32))


def split_box(half, n):
    """A box whose faces are n x n squares of two triangles: flat fans round its vertices."""
    V, T = [], []
    for axis in range(3):
        for s in (-1, 1):
            d1, d2 = (axis + 1) % 3, (axis + 2) % 3
            g = np.linspace(-1, 1, n + 1)
            base = len(V)
            for x in g:
                for y in g:
                    p = [0.0] * 3
                    p[axis], p[d1], p[d2] = s, x, y
                    V.append(p)
            for i in range(n):
                for j in range(n):
                    a, b, c, d = base + i * (n + 1) + j, base + (i + 1) * (n + 1) + j, base + (i + 1) * (n + 1) + j + 1, \
                        base + i * (n + 1) + j + 1
                    q = [(a, b, c), (a, c, d)]
                    T += q if s > 0 else [t[::-1] for t in q]
    V = np.asarray(V)
    uniq, inv = np.unique(np.round(V, 9), axis=0, return_inverse=True)
    return S.TriangleMesh(uniq * np.asarray(half), inv.reshape(-1)[np.asarray(T)].astype(np.int32))


def ell():
    """An L-shaped prism (a reflex edge, coplanar triangles, obtuse fans)."""
    P = np.array([(0, 0), (2, 0), (2, 1), (1, 1), (1, 2), (0, 2)], dtype=float)
    tri = [(0, 1, 2), (0, 2, 3), (0, 3, 4), (0, 4, 5)]
    V = np.vstack([np.c_[P, np.zeros(6)], np.c_[P, np.ones(6)]]) * 0.01
    T = [t[::-1] for t in tri] + [tuple(i + 6 for i in t) for t in tri]
    for i in range(6):
        j = (i + 1) % 6
        T += [(i, j, j + 6), (i, j + 6, i + 6)]
    return S.TriangleMesh(V, np.asarray(T, dtype=np.int32))


def cones_tip_to_tip(n=10):
    """Two cones that share their tip vertex (two fans round it)."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a)], -1) * 0.01
    V = [(0.0, 0.0, 0.0), (0, 0, 0.02), (0, 0, -0.02)]
    V += [(x, y, 0.02) for x, y in ring] + [(x, y, -0.02) for x, y in ring]
    T = []
    for i in range(n):
        j = (i + 1) % n
        T += [(0, 3 + j, 3 + i), (1, 3 + i, 3 + j), (0, 3 + n + i, 3 + n + j), (2, 3 + n + j, 3 + n + i)]
    return S.TriangleMesh(np.asarray(V), np.asarray(T, dtype=np.int32))


def dented(depth):
    """A box whose top middle is pushed down by `depth`: through the bottom past 2."""
    m = split_box((0.01, 0.01, 0.01), 2)
    V = m.vertices.copy()
    top = np.where((np.abs(V[:, 2] - 0.01) < 1e-9) & (np.abs(V[:, 0]) < 1e-9) & (np.abs(V[:, 1]) < 1e-9))[0]
    V[top, 2] -= depth * 0.01
    return S.TriangleMesh(V, m.triangles)


BALL = S.icosphere(0.02, 2)
CASES = {
    "icosphere": (BALL, 1), "fine icosphere": (S.icosphere(0.04, 3), 1), "coarse": (S.icosphere(0.01, 0), 1),
    "box": (S.box_mesh((0.01, 0.02, 0.03)), 1), "plate": (S.box_mesh((0.03, 0.0004, 0.02)), 1),
    "split box": (split_box((0.02, 0.01, 0.015), 4), 1), "torus": (torus(), 1), "L": (ell(), 1),
    "dent": (dented(1.5), 1), "side by side": (joined((BALL, (-0.03, 0, 0), False), (S.box_mesh((0.01,) * 3), (0.03, 0, 0), False)), 1),
    "through the bottom": (dented(2.5), 0), "spindle torus": (torus(R=0.008), 0), "pinched": (cones_tip_to_tip(), 0),
    "inside out": (joined((BALL, (0, 0, 0), True)), 0),
    "nested": (joined((BALL, (0, 0, 0), False), (S.icosphere(0.008, 1), (0, 0, 0), False)), 0),
    "overlapping": (joined((BALL, (-0.012, 0, 0), False), (BALL, (0.012, 0.001, 0), False)), 0),
    "touching boxes": (joined((S.box_mesh((0.01,) * 3), (-0.01, 0, 0), False), (S.box_mesh((0.01,) * 3), (0.01, 0, 0), False)), 0),
    "one inward": (joined((BALL, (-0.03, 0, 0), False), (BALL, (0.03, 0, 0), True)), 0),
}


def bounds_solid(lib, mesh):
    V, T = np.ascontiguousarray(mesh.vertices, dtype=np.float64), np.ascontiguousarray(mesh.triangles, dtype=np.int32)
    d = S.MeshDesc()
    d.n_vertices, d.n_triangles = len(V), len(T)
    d.vertices = V.ctypes.data_as(C.POINTER(C.c_double))
    d.triangles = T.ctypes.data_as(C.POINTER(C.c_int32))
    f = lib.fdtd_debug_mesh_bounds_solid
    f.restype = C.c_int
    return f(C.byref(d)), d, (V, T)


def winding(V, T, q):
    """Generalised winding number (solid angles of all triangles over 4 pi)."""
    a, b, c = (V[T[:, k]][None] - q[:, None] for k in range(3))
    la, lb, lc = (np.linalg.norm(x, axis=-1) for x in (a, b, c))
    num = np.einsum("pti,pti->pt", a, np.cross(b, c))
    den = la * lb * lc + np.einsum("pti,pti->pt", a, b) * lc + np.einsum("pti,pti->pt", b, c) * la + \
        np.einsum("pti,pti->pt", c, a) * lb
    return (2 * np.arctan2(num, den)).sum(axis=1) / (4 * np.pi)


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("turned", [False, True])
def test_known_shapes(fdtd_lib, name, turned):
    mesh, want = CASES[name]
    V = np.asarray(mesh.vertices, dtype=np.float64)
    if turned:
        q = np.linalg.qr(np.random.default_rng(2).normal(size=(3, 3)))[0]
        V = V @ (q * np.sign(np.linalg.det(q))).T + np.array([0.3, -0.2, 0.1])
    mesh = S.TriangleMesh(V, mesh.triangles)
    got, desc, (V, T) = bounds_solid(fdtd_lib, mesh)
    assert got == want
    if want:
        rng = np.random.default_rng(3)
        lo, hi = V.min(0), V.max(0)
        q = lo + (hi - lo) * rng.uniform(-0.3, 1.3, (400, 3))
        out = np.zeros(len(q))
        assert fdtd_lib.fdtd_mesh_signed_distance(C.byref(desc), C.c_int64(len(q)), q.ctypes.data_as(C.c_void_p),
                                                  out.ctypes.data_as(C.c_void_p)) == 0
        w = winding(V, T, q)
        off = np.abs(out) > 1e-9
        assert np.array_equal(out[off] < 0, w[off] > 0.5)
        assert (out < 0).any() and (out > 0).any()


def test_random_bumpy_spheres(fdtd_lib):
    """Spheres with displaced vertices: a yes is only ever given where the sign is right."""
    rng = np.random.default_rng(11)
    yes = 0
    for amp in (0.0, 0.02, 0.1, 0.3, 0.6, 0.9, 1.5):
        base = S.icosphere(1.0, 2)
        V = base.vertices * (1 + amp * rng.uniform(-1, 1, (len(base.vertices), 1))) + 0.05 * amp * rng.normal(size=base.vertices.shape)
        got, desc, (V, T) = bounds_solid(fdtd_lib, S.TriangleMesh(V, base.triangles))
        yes += got
        if got == 1:
            q = rng.uniform(-1.6, 1.6, (500, 3))
            out = np.zeros(len(q))
            assert fdtd_lib.fdtd_mesh_signed_distance(C.byref(desc), C.c_int64(len(q)), q.ctypes.data_as(C.c_void_p),
                                                      out.ctypes.data_as(C.c_void_p)) == 0
            assert np.array_equal(out < 0, winding(V, T, q) > 0.5)
    assert 2 <= yes <= 6
